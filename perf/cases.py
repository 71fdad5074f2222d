"""The search work that is timed when a kernel or a host path changes.

Each case is a dict of plain values; `prepare` makes what a program has in
hand before the call (the chunk and its index on the device, host query
arrays, device buffers of the operator calls), `run` is one pass through the
public entry points of `gzb`, `work` what the path cannot do without.

Calls (`case["call"]`):

  search     raw protein queries -> SEG, cutoffs and hash lists on the
             device -> presearch -> build results, against a resident chunk
             (what `aln` does per query batch once its database is loaded)
  reads      the same for DNA reads (six-frame translation first)
  presearch  the presearch alone of a resident query set (a chunk loop's
             inner step), its merged lists read back
  slots      the chunk loop over a database stored in the engine's slots
  load       `gzb.search.search` on a chunk that is not resident: upload,
             index build, presearch, build results, sort
  gapped     GappedExtenderGpu on device buffers of chained seeds
  ungapped   UngappedExtenderGpu with trigger on device buffers
  distance   DistanceCalculatorGpu on device buffers
  prepare    query preparation of device-resident reads (translation, SEG,
             per-query cutoffs)

Sequences follow the laws of `gzb.workload` (log-normal lengths, residues
from the Robinson background, 30 % of the queries planted homologs at 30 to
90 % identity with indels), drawn on the GPU.
"""
from __future__ import annotations

import math
import os
import sys
from types import SimpleNamespace

import numpy as np
import torch

_PACKAGE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                        "ghostz-gpu_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

from gzb import native as N  # noqa: E402
from gzb import params as P  # noqa: E402
from gzb import search as S  # noqa: E402
from gzb import workload as W  # noqa: E402

MEAN_PROTEIN = 360      # residues: exp(0.6^2 / 2) * 300
SEED_SPACING = 64       # database residues per seed of the operator cases
SEED_MATCH = 12         # residues around a seed that match in the reduced alphabet


def listed():
    return [
        # one query against a small database, nothing to hide latency behind
        # (an interactive look-up)
        {"name": "search-1-x-20k", "call": "search", "proteins": 20_000, "queries": 1,
         "median": 300, "sigma": 0.0, "filter": True, "clustering": True, "mode": "eager"},
        # the small benchmark configuration, end to end
        {"name": "search-1k-x-20k", "call": "search", "proteins": 20_000, "queries": 1_000,
         "median": 300, "sigma": 0.6, "filter": True, "clustering": True, "mode": "eager"},
        # a batch of an odd size without SEG and without clustering
        {"name": "search-3k-x-301k-plain-index", "call": "search", "proteins": 301_003,
         "queries": 3_001, "median": 300, "sigma": 0.6, "filter": False, "clustering": False,
         "mode": "eager"},
        # the benchmark's presearch: its 10,000 queries, a chunk of 1.5 M
        # proteins, one graph
        {"name": "presearch-10k-x-1.5M", "call": "presearch", "proteins": 1_500_000,
         "queries": 10_000, "median": 300, "sigma": 0.6, "filter": True, "clustering": True,
         "mode": "graph"},
        # query lengths from 20 to 8,000 (the uneven configuration's law)
        {"name": "presearch-uneven-4k-x-700k", "call": "presearch", "proteins": 700_000,
         "queries": 4_000, "median": 250, "sigma": 1.0, "filter": True, "clustering": True,
         "mode": "graph"},
        # the plain schedule (one launch per stage, hit order), read back whole
        {"name": "presearch-plain-2k-x-400k", "call": "presearch", "proteins": 400_000,
         "queries": 2_000, "median": 300, "sigma": 0.6, "filter": True, "clustering": True,
         "mode": "plain"},
        # sequencing reads, end to end
        {"name": "reads-30k-x-400k", "call": "reads", "proteins": 400_000, "reads": 30_000,
         "length": 150, "filter": True, "clustering": True, "mode": "graph"},
        # a database of several chunks kept in HBM, uneven queries
        {"name": "slots-2k-x-4x100k", "call": "slots", "proteins": 100_000, "chunks": 4,
         "queries": 2_000, "median": 250, "sigma": 1.0, "filter": True, "clustering": True,
         "mode": "graph"},
        # a chunk that has to be uploaded and indexed before it is searched
        {"name": "load-300-x-200k", "call": "load", "proteins": 200_000, "queries": 300,
         "median": 300, "sigma": 0.6, "filter": True, "clustering": True},
        # the operators a host program calls itself
        {"name": "gapped-operator-300k", "call": "gapped", "seeds": 300_000, "reverse": False,
         "bits": 15.0},
        {"name": "ungapped-operator-3M", "call": "ungapped", "seeds": 3_000_000},
        {"name": "prepare-150k-reads", "call": "prepare", "reads": 150_000, "length": 150,
         "filter": True},
    ]


def _log_size(rng, lo, hi):
    """A size spread over [lo, hi] on a log scale, round ones no more likely
    than odd ones."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["search", "search", "presearch", "presearch", "presearch", "reads",
                       "slots", "load", "gapped", "ungapped", "distance", "prepare"])
    if call in ("gapped", "ungapped", "distance"):
        c = {"call": call, "seeds": _log_size(rng, 500, {"gapped": 600_000,
                                                         "ungapped": 4_000_000,
                                                         "distance": 4_000_000}[call])}
        if call == "gapped":
            c["reverse"] = rng.random() < 0.5
            # the presearch's X-drop, or the build results step's
            c["bits"] = rng.choice([15.0, 25.0])
        return c
    if call == "prepare":
        return {"call": call, "reads": _log_size(rng, 100, 200_000),
                "length": rng.choice([75, 100, 101, 150, 151, 250, 301]),
                "filter": rng.random() < 0.8}
    c = {"call": call, "proteins": _log_size(rng, 2_000, 700_000), "clustering":
         rng.random() < 0.8, "filter": rng.random() < 0.8}
    if call == "reads":
        c["reads"] = _log_size(rng, 20, 30_000)
        c["length"] = rng.choice([75, 100, 101, 150, 151, 250, 301])
    else:
        c["queries"] = _log_size(rng, 1, 5_000)
        c["median"], c["sigma"] = rng.choice([(300, 0.6), (300, 0.6), (250, 1.0), (60, 0.4)])
    if call == "slots":
        c["chunks"] = rng.randint(2, 4)
        c["proteins"] = max(1_000, c["proteins"] // c["chunks"])
    if call == "load":
        c["proteins"] = min(c["proteins"], 300_000)
        c["queries"] = min(c["queries"], 1_000)
    else:
        c["mode"] = rng.choice(["graph", "graph", "eager", "plain"])
    return c


# ---------------------------------------------------------------------------
# sequences, drawn on the GPU


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _background():
    f = np.array([P.ROBINSON[ch] for ch in P.REGULAR])
    return f / f.sum()


def _residues(g, n):
    cdf = torch.tensor(np.cumsum(_background())[:-1], dtype=torch.float32, device="cuda")
    out = torch.empty(n, dtype=torch.uint8, device="cuda")
    step = 1 << 26
    for a in range(0, n, step):
        b = min(n, a + step)
        u = torch.rand(b - a, generator=g, device="cuda")
        out[a:b] = torch.bucketize(u, cdf, out_int32=True, right=True).to(torch.uint8)
    return out


def _lengths(g, n, median, sigma, lo, hi):
    x = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    return (median * torch.exp(sigma * x)).round().clamp(lo, hi).to(torch.int64)


def _join(residues, lengths):
    """Sequences back to back as [delim s0 delim s1 ... delim]: (codes,
    first-residue offsets)."""
    n = len(lengths)
    ends = torch.cumsum(lengths + 1, 0)
    starts = ends - lengths
    codes = torch.full((int(ends[-1]) + 1,), P.DELIMITER, dtype=torch.uint8, device="cuda")
    owner = torch.repeat_interleave(torch.arange(n, device="cuda", dtype=torch.int32), lengths)
    at = torch.arange(int(lengths.sum()), device="cuda") + 1 + owner
    codes[at] = residues
    return codes, starts


def _database(g, n, median=300, sigma=0.6, lo=30, hi=3000):
    lengths = _lengths(g, n, median, sigma, lo, hi)
    total = int(lengths.sum()) + n + 1
    codes = _residues(g, total)
    ends = torch.cumsum(lengths + 1, 0)
    codes[0] = P.DELIMITER
    codes[ends] = P.DELIMITER
    starts = ends - lengths
    offsets = torch.cat([starts, torch.tensor([total], device="cuda")])
    db = W.Database(codes=codes.cpu().numpy(), offsets=offsets.cpu().numpy().astype(np.uint32),
                    number_sequences=n)
    return db, codes, starts, lengths


def _substitutions(lam=0.3176):
    """Row r: cumulative chances of what residue r is replaced by."""
    t = _background()[None, :] * np.exp(lam * P.blosum62()[:20, :20])
    np.fill_diagonal(t, 0.0)
    return torch.tensor(np.cumsum(t / t.sum(1, keepdims=True), 1), dtype=torch.float32,
                        device="cuda")


def _geometric(g, n, mean=3.0):
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64).clamp_min(1e-12)
    return (torch.log(u) / math.log(1.0 - 1.0 / mean)).floor().to(torch.int64) + 1


def _queries(g, n, sources, median, sigma, homologs=0.3):
    """Raw protein queries in the engine layout (host codes, offsets,
    lengths): unrelated ones, and homologs of the database sequences
    (sources: list of (codes, starts, lengths))."""
    hi = 3000 if sigma < 1.0 else 8000
    lo = 30 if sigma < 1.0 else 20
    lengths = _lengths(g, n, median, sigma, lo, hi)
    planted = torch.rand(n, generator=g, device="cuda") < homologs
    codes, starts, slen = sources[0]
    which = torch.randint(0, len(starts), (n,), generator=g, device="cuda")
    chunk = torch.randint(0, len(sources), (n,), generator=g, device="cuda")
    base_len = lengths.clone()
    base_at = torch.zeros(n, dtype=torch.int64, device="cuda")
    for k, (_, st, ln) in enumerate(sources):
        w = which % len(st)
        mine = planted & (chunk == k)
        # a homolog is as long as its source
        base_len = torch.where(mine, ln[w].clamp(max=hi), base_len)
        base_at = torch.where(mine, st[w], base_at)
    total = int(base_len.sum())
    owner = torch.repeat_interleave(torch.arange(n, device="cuda"), base_len)
    first = torch.cumsum(base_len, 0) - base_len
    within = torch.arange(total, device="cuda") - first[owner]
    res = _residues(g, total)
    for k, (cs, _, _) in enumerate(sources):
        mine = (planted & (chunk == k))[owner]
        res[mine] = cs[(base_at[owner] + within)[mine]]
    identity = (0.3 + 0.6 * torch.rand(n, generator=g, device="cuda"))[owner]
    change = planted[owner] & (torch.rand(total, generator=g, device="cuda") > identity)
    at = change.nonzero()[:, 0]
    u = torch.rand(len(at), generator=g, device="cuda")
    rows = _substitutions()[res[at].long()]
    res[at] = (rows < u[:, None]).sum(1).clamp(max=19).to(torch.uint8)
    # insertions behind a residue, deletions of a run of residues
    event = planted[owner] & (torch.rand(total, generator=g, device="cuda") < 0.02)
    run = _geometric(g, total)
    insert = event & (torch.rand(total, generator=g, device="cuda") < 0.5)
    delete = event & ~insert
    edge = torch.zeros(total + 1, dtype=torch.int64, device="cuda")
    seq_end = (first + base_len)[owner]
    d_at = delete.nonzero()[:, 0]
    edge.index_add_(0, d_at, torch.ones_like(d_at))
    edge.index_add_(0, torch.minimum(d_at + run[d_at], seq_end[d_at]), -torch.ones_like(d_at))
    copies = torch.where(torch.cumsum(edge, 0)[:total] > 0, 0, 1)
    copies = copies + torch.where(insert, run, 0)
    copies[first] = copies[first].clamp_min(1)  # no query is empty
    out_owner = torch.repeat_interleave(owner, copies)
    source = torch.repeat_interleave(torch.arange(total, device="cuda"), copies)
    out = res[source]
    inserted = torch.ones(len(out), dtype=torch.bool, device="cuda")
    inserted[1:] = source[1:] == source[:-1]
    inserted[0] = False
    out = torch.where(inserted, _residues(g, len(out)), out)
    qlen = torch.bincount(out_owner, minlength=n)
    codes, starts = _join(out, qlen)
    return SimpleNamespace(codes=codes.cpu().numpy(),
                           offsets=(starts - 1).cpu().numpy().astype(np.uint32),
                           lengths=(qlen + 2).cpu().numpy().astype(np.uint32))


def _seed_pairs(g, n):
    """n seed positions whose surroundings match in the reduced alphabet, as
    the seed search finds them: query codes and database codes on the device
    (with the padding the operators ask for), per seed the query id, query
    position and database position, and the number of queries."""
    nq = max(1, min(2_000, n // 50))
    lengths = _lengths(g, nq, 300, 0.6, 60, 3000)
    q, starts = _join(_residues(g, int(lengths.sum())), lengths)
    db_len = n * SEED_SPACING + 2 * SEED_SPACING
    db = _residues(g, db_len)
    ends = torch.cumsum(_lengths(g, db_len // MEAN_PROTEIN + 1, 300, 0.6, 30, 3000), 0)
    db[ends[ends < db_len]] = P.DELIMITER
    db[0] = P.DELIMITER
    db[-1] = P.DELIMITER
    qid = torch.randint(0, nq, (n,), generator=g, device="cuda")
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    margin = SEED_MATCH
    span = (lengths - 2 * margin)[qid]
    qpos = starts[qid] + margin + (u * span).to(torch.int64)
    dpos = torch.arange(n, device="cuda") * SEED_SPACING + SEED_SPACING
    dpos = dpos + torch.randint(-8, 9, (n,), generator=g, device="cuda")
    # the reduced alphabet's groups: a residue is kept or replaced inside
    groups, _ = P.reduced_code_map()
    group = groups[:20]
    peers = torch.tensor(np.array([[np.flatnonzero(group == group[r])[k % (group == group[r]).sum()]
                                    for k in range(12)] for r in range(20)]),
                         dtype=torch.uint8, device="cuda")
    for t in range(-SEED_MATCH // 2, SEED_MATCH // 2):
        src = q[qpos + t].long()
        like = peers[src, torch.randint(0, 12, (n,), generator=g, device="cuda")]
        keep = torch.rand(n, generator=g, device="cuda") < 0.6
        new = torch.where(keep, src.to(torch.uint8), like)
        old = db[dpos + t]
        db[dpos + t] = torch.where(old == P.DELIMITER, old, new)
    def padded(codes):
        t = torch.full((len(codes) + 2 * N.PAD,), P.DELIMITER, dtype=torch.uint8, device="cuda")
        t[N.PAD:N.PAD + len(codes)] = codes
        return t
    return SimpleNamespace(q=padded(q), db=padded(db), nq=nq, lengths=lengths,
                           qid=qid.to(torch.int32), qpos=qpos.to(torch.int32),
                           dpos=dpos.to(torch.int32))


# ---------------------------------------------------------------------------


def _schedule(case):
    return N.SCHEDULE_PLAIN if case.get("mode") == "plain" else N.SCHEDULE_BATCHED


def _engine(case, params, dbs):
    e = N.PresearchEngine(0)
    e.set_params(params)
    e.set_graph(case.get("mode") == "graph")
    for k, db in enumerate(dbs):
        e.set_database(db, chunk_id=k)
        if len(dbs) > 1:
            e.swap_database(k)
    return e


def prepare(case, seed):
    g = _generator(seed * 7919 + 11)
    call = case["call"]
    if call in ("ungapped", "distance"):
        return _prepare_seeds(case, g)
    if call == "gapped":
        return _prepare_gapped(case, g)
    if call == "prepare":
        db, _, _, _ = _database(g, 2_000)
        reads = W.make_reads(db, case["reads"], seed, read_length=case["length"])
        return _prepare_reads(case, reads)
    params = P.make_params(clustering=case["clustering"])
    made = [_database(g, case["proteins"]) for _ in range(case.get("chunks", 1))]
    dbs = [m[0] for m in made]
    st = {"case": case, "params": params, "dbs": dbs}
    if call == "reads":
        reads = W.make_reads(dbs[0], case["reads"], seed, read_length=case["length"])
        st.update(engine=_engine(case, params, dbs), dna=reads.dna, offsets=reads.offsets)
        return st
    raw = _queries(g, case["queries"], [m[1:] for m in made], case["median"], case["sigma"])
    if call == "load":
        codes, cut, trig = N.prepare_protein_queries(raw.codes, raw.offsets, raw.lengths,
                                                     filter=case["filter"])
        q = W.Queries(codes=codes, offsets=raw.offsets, lengths=raw.lengths, cutoffs=cut,
                      triggers=trig)
        real = raw.lengths.astype(np.int64) - 2
        st.update(engine=N.PresearchEngine(0),
                  prepared=S.PreparedQueries(queries=q, real_lengths=real.astype(np.uint32)))
        return st
    e = _engine(case, params, dbs)
    st.update(engine=e, raw=raw)
    if call in ("presearch", "slots"):
        e.set_protein_queries(raw.codes, raw.offsets, raw.lengths, filter=case["filter"])
    return st


def _prepare_gapped(case, g):
    """Seeds for the gapped operator: the ungapped hits of a presearch, one
    of each query's diagonals (the chain filter leaves about that), and the
    sequences they lie in."""
    n = case["seeds"]
    # about 0.64 chained hits per query and 1,000 proteins
    queries = max(40, min(2_000, n // 100))
    proteins = max(1_000, min(600_000, int(1.8e3 * n / queries)))
    params = P.make_params()
    db, codes, starts, lengths = _database(g, proteins)
    raw = _queries(g, queries, [(codes, starts, lengths)], 300, 0.6)
    e = N.PresearchEngine(0)
    e.set_params(params)
    e.set_database(db)
    e.set_protein_queries(raw.codes, raw.offsets, raw.lengths)
    e.presearch(N.SCHEDULE_BATCHED)
    qid, qpos, dpos = (a.astype(np.int64) for a in e.hits())
    e.close()
    diagonal = (qid << 40) + dpos - qpos
    keep = np.sort(np.unique(diagonal, return_index=True)[1])[:n]
    qpos = raw.offsets[qid].astype(np.int64) + qpos
    assert qpos.min() > 0 and qpos.max() < len(raw.codes) and dpos.max() < db.length
    back = 1 if case["reverse"] else 0
    q, q_address = N.device_sequence(raw.codes, P.DELIMITER)
    d, d_address = N.device_sequence(db.codes, P.DELIMITER)
    op = N.GappedExtenderGpu()
    op.SetQueries(P.DELIMITER, q_address)
    op.SetDatabase(d_address)
    matrix = N.device_matrix(P.blosum62())
    cutoff = P.normalized_to_nominal(case["bits"], P.GAPPED_LAMBDA, P.GAPPED_K)
    op.SetScoreParameters(matrix, P.NUMBER_LETTERS, 11, 1, cutoff)
    seeds = [torch.from_numpy((a[keep] - back).astype(np.int32)).cuda()
             for a in (qpos, dpos)]
    return {"case": case, "op": op, "keep": (q, d, matrix), "seeds": seeds,
            "at": [torch.empty_like(s) for s in seeds], "scores": torch.empty_like(seeds[0])}


def _prepare_seeds(case, g):
    s = _seed_pairs(g, case["seeds"])
    if case["call"] == "distance":
        op = N.DistanceCalculatorGpu()
        similar, _ = P.reduced_code_map()
        table = np.zeros(32, np.uint8)
        table[:len(similar)] = similar
        keep = torch.from_numpy(table).cuda()
        op.SetQueries(s.q.data_ptr() + N.PAD)
        op.SetDatabase(s.db.data_ptr() + N.PAD)
        op.SetReducedCodeMap(keep)
        op.SetSubsequenceLength(10)
        out = torch.empty(len(s.qpos), dtype=torch.int8, device="cuda")
    else:
        op = N.UngappedExtenderGpu()
        matrix = N.device_matrix(P.blosum62())
        # per-query cutoffs as query preparation finds them (7 and 22 bits)
        cut = torch.randint(15, 19, (s.nq,), device="cuda", dtype=torch.int32)
        trig = torch.randint(44, 52, (s.nq,), device="cuda", dtype=torch.int32)
        cut.copy_(15 + s.lengths % 4)
        trig.copy_(44 + s.lengths % 8)
        keep = (matrix, cut, trig)
        op.SetQueries(P.DELIMITER, s.q.data_ptr() + N.PAD, cut, trig)
        op.SetDatabase(s.db.data_ptr() + N.PAD)
        op.SetScoreMatrix(matrix, P.NUMBER_LETTERS)
        out = torch.empty(len(s.qpos), dtype=torch.int8, device="cuda")
    return {"case": case, "op": op, "keep": keep, "s": s, "out": out}


def _prepare_reads(case, reads):
    lengths = np.diff(reads.offsets).astype(np.uint32)
    out_offsets, qlen, total = N.translated_layout(lengths)
    n = len(lengths)
    return {"case": case, "n": n,
            "dna": torch.from_numpy(reads.dna).cuda(),
            "offsets": torch.from_numpy(reads.offsets[:-1].astype(np.int64)).cuda(),
            "lengths": torch.from_numpy(lengths.view(np.int32).copy()).cuda(),
            "out_offsets": torch.from_numpy(out_offsets.astype(np.int64)).cuda(),
            "qlen": torch.from_numpy(qlen.view(np.int32).copy()).cuda(),
            "out": torch.empty(total, dtype=torch.uint8, device="cuda"),
            "cut": torch.empty(n, dtype=torch.int32, device="cuda"),
            "trig": torch.empty(n, dtype=torch.int32, device="cuda"),
            "status": torch.zeros(1, dtype=torch.int32, device="cuda"),
            "matrix": P.blosum62()}


def _padded(rows, width):
    """Alignment records of all queries as one array of whole numbers (slots
    past a query's count hold nothing: zeros), and how many each has."""
    counts = np.array([len(r) for r in rows], np.int32)
    out = np.zeros((len(rows), width, 14), np.int32)
    for i, r in enumerate(rows):
        out[i, :len(r)] = r.view(np.int32).reshape(-1, 14)
    return {"counts": counts, "rows": out}


def _alignments(state):
    """The build results step into the caller's pinned arrays, as a program
    over the C ABI keeps them."""
    e = state["engine"]
    n, width = e.number_queries, int(state["params"]["max_number_results"])
    if "counts" not in state:
        state["counts"] = torch.zeros(n, dtype=torch.int32).pin_memory()
        state["rows"] = torch.zeros(n, width, 14, dtype=torch.int32).pin_memory()
    counts, rows = state["counts"].numpy(), state["rows"].numpy()
    N.check(N.lib().gzb_engine_build_alignments(e.h, N.hptr(counts), N.hptr(rows), None))
    rows[np.arange(width)[None, :] >= counts[:, None]] = 0
    return {"counts": counts, "rows": rows}


def _merged(counts, records):
    """The merged lists; a query's slots past its count hold nothing."""
    rows = records.view(np.int32).reshape(len(counts), -1, 9)
    rows[np.arange(rows.shape[1])[None, :] >= counts[:, None]] = 0
    return {"counts": counts.astype(np.int32), "records": rows}


def run(state):
    case = state["case"]
    call = case["call"]
    if call == "gapped":
        at, seeds, scores = state["at"], state["seeds"], state["scores"]
        at[0].copy_(seeds[0])
        at[1].copy_(seeds[1])
        state["op"].ExtendOneSideScoreOnlyAsync(len(scores), case["reverse"], None, None, None,
                                                at[0], at[1], scores)
        return {"scores": scores, "query": at[0], "database": at[1]}
    if call == "ungapped":
        s = state["s"]
        state["op"].ExtendWithTriggerAsync(len(s.qid), None, None, None, None, s.qid, s.qpos,
                                           s.dpos, state["out"])
        return state["out"]
    if call == "distance":
        s = state["s"]
        state["op"].CalculateDistancesAsync(len(s.qpos), None, None, None, s.qpos, s.dpos,
                                            state["out"])
        return state["out"]
    if call == "prepare":
        n, out = state["n"], state["out"]
        N.translate_dna_queries_async(state["dna"], state["offsets"], state["lengths"], n,
                                      state["out_offsets"], out, P.DELIMITER)
        if case["filter"]:
            N.seg_translated_queries_async(out, state["out_offsets"], state["lengths"], n,
                                           state["status"])
        N.query_karlin_cutoffs_async(out, state["out_offsets"], state["qlen"], n,
                                     state["matrix"], state["cut"], state["trig"])
        return {"codes": out, "cutoffs": state["cut"], "triggers": state["trig"],
                "status": state["status"]}
    e = state["engine"]
    if call == "load":
        return _padded(S.search(e, state["params"], state["prepared"], state["dbs"]),
                       int(state["params"]["max_number_results"]))
    schedule = _schedule(case)
    if call == "reads":
        cut, trig = e.set_translated_queries(state["dna"], state["offsets"],
                                             filter=case["filter"])
    elif call == "search":
        raw = state["raw"]
        cut, trig = e.set_protein_queries(raw.codes, raw.offsets, raw.lengths,
                                          filter=case["filter"])
    if call in ("reads", "search"):
        e.reset_results()
        e.presearch(schedule)
        return dict(_alignments(state), cutoffs=cut, triggers=trig)
    e.reset_results()
    for k in range(len(state["dbs"])):
        if call == "slots":
            e.swap_database(k)
        e.presearch(schedule)
        if call == "slots":
            e.swap_database(k)
    return _merged(*e.result_rows())


def work(case):
    """Bytes: every input read once, every output written once.  Operations:
    the integer operations of the DP cells and residue pairs that chance hits
    of this many residue pairs lead to, at 10 a cell and 4 a pair (the
    benchmark's counters: 1.0e-5 cells and 1.2e-5 pairs per query residue and
    database residue)."""
    call = case["call"]
    if call == "gapped":
        return {"bytes": 12 * case["seeds"], "flops": 10 * 1000 * case["seeds"]}
    if call == "ungapped":
        return {"bytes": 13 * case["seeds"] + 60 * case["seeds"], "flops": 200 * case["seeds"]}
    if call == "distance":
        return {"bytes": 29 * case["seeds"], "flops": 20 * case["seeds"]}
    if call == "prepare":
        return {"bytes": 3 * case["length"] * case["reads"],
                "flops": 12 * 2 * case["length"] * case["reads"]}
    residues = case["proteins"] * case.get("chunks", 1) * MEAN_PROTEIN
    if call == "reads":
        letters = 2 * case["length"] * case["reads"]
        n = case["reads"]
    else:
        letters = case["queries"] * case["median"] * math.exp(case["sigma"] ** 2 / 2)
        n = case["queries"]
    ops = (10 * 1.0e-5 + 4 * 1.2e-5) * letters * residues
    return {"bytes": int(residues + letters + 360 * n), "flops": int(ops)}


def exact(case, seed):
    """Every output is a whole number or a byte (scores, positions, counts,
    residue codes), which have to stay what they are; none is a computed
    floating value."""
    return None
