"""The seed search over X-drops and score matrices on both sides of what its
windows take: all queries narrow or wide, some of each, matrix entries at and
beyond the window tables' range.  Hits, results and counters equal the
oracle's, the residue pairs examined those of the dealt walker (a walk a seed,
pair by pair), and windows are evaluated only where most queries are narrow."""
import numpy as np
import pytest

from gzb import params as P
from gzb import workload as W
from kernel_trace import kernels
from test_gpu_engine import _compare, _small, engine  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu

# X-drops of the first and of the other queries, matrix scale, windows
CASES = [((30, 30), 1, True), ((31, 31), 1, False), ((127, 127), 1, False),
         ((128, 128), 1, False), ((900, 900), 1, False), ((15, 127), 1, True),
         ((15, 128), 1, True), ((1, 32767), 1, True), ((30, 30), 11, True),
         ((30, 30), 12, False), ((180, 180), 12, False)]


@pytest.fixture(scope="module")
def chunk():
    return _small(n_db=800, n_q=60)


def _params(scale):
    p = P.make_params(matrix=P.blosum62() * scale, gap_open=11 * scale, gap_extension=scale)
    one = P.make_params()
    for name in ("code_scores", "seed_threshold"):
        p[name] = one[name]
    p["gapped_cutoff"] = one["gapped_cutoff"] * scale
    return p


@pytest.mark.parametrize("cutoffs,scale,windows", CASES)
@pytest.mark.parametrize("graph", [False, True])
def test_hits_match_oracle(engine, oracle, chunk, cutoffs, scale, windows, graph):  # noqa: F811
    from gzb import native as N
    db, q = chunk
    params = _params(scale)
    cut = np.full(q.number, cutoffs[0], np.int32)
    cut[int(0.6 * q.number):] = cutoffs[1]
    trig = (np.full(q.number, 60) * scale).astype(np.int32)
    q = W.Queries(codes=q.codes, offsets=q.offsets, lengths=q.lengths, cutoffs=cut, triggers=trig)
    engine.set_graph(graph)
    try:
        _compare(engine, oracle, params, db, q, schedule=N.SCHEDULE_BATCHED)
        steps = engine.counters()["ungapped_steps"]
        engine.reset_results()
        names = kernels(lambda: engine.presearch(N.SCHEDULE_BATCHED))
        for stage in ("seed", "member"):
            assert any(f"{stage}_kernel(" in n for n in names) == windows
            assert any(f"{stage}_lane_kernel(" in n for n in names) != windows
        engine.set_tile(N.SCHEDULE_BATCHED, N.TILE_SEED_WALKER, N.SEED_WALKER_DEALT)
        engine.reset_results()
        engine.presearch(N.SCHEDULE_BATCHED)
        assert engine.counters()["ungapped_steps"] == steps
    finally:
        engine.set_tile(N.SCHEDULE_BATCHED, N.TILE_SEED_WALKER, N.SEED_WALKER_UNIT)
        engine.set_graph(False)


@pytest.mark.parametrize("call", ["protein", "translated"])
def test_prepared_queries(engine, chunk, call):  # noqa: F811
    """Cutoffs found on the device decide as well: the default 7 bits and 40."""
    from gzb import native as N
    db, _ = chunk
    engine.set_params(P.make_params())
    engine.set_database(db)
    for bits, windows in ((7.0, True), (40.0, False), (7.0, True)):
        if call == "protein":
            seqs = [db.codes[db.offsets[s]:db.offsets[s + 1] - 1] for s in range(20)]
            raw = W.pack_queries(seqs, cutoffs=(np.zeros(20, np.int32), np.zeros(20, np.int32)))
            cut, _ = engine.set_protein_queries(raw.codes, raw.offsets, raw.lengths,
                                                ungapped_bits=bits)
        else:
            reads = W.make_reads(db, 30, 5, read_length=150)
            cut, _ = engine.set_translated_queries(reads.dna, reads.offsets, ungapped_bits=bits)
        assert (np.median(cut) <= 30) == windows
        engine.reset_results()
        names = kernels(lambda: engine.presearch(N.SCHEDULE_BATCHED))
        assert any("seed_kernel(" in n for n in names) == windows
        assert any("seed_lane_kernel(" in n for n in names) != windows
