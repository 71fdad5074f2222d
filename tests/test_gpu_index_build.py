"""Database index and query lists at the edges of the kernels that build
them: hash lengths around the eight residues that are hashed in registers,
chunk lengths off the four positions a thread takes, every window length
class, and buckets around the sizes at which the clustering changes its path
(32 entries a warp's registers, 64, 128, 256, a block above, 65,536 entries
in a block's flags).  All arrays equal the oracle's."""
import numpy as np
import pytest

from gzb import params as P
from gzb import workload as W

pytestmark = pytest.mark.gpu

INDEX = ("nc_keys", "nc_offsets", "nc_values", "rep_keys", "rep_offsets", "rep_positions",
         "member_offsets", "member_positions")
LISTS = ("hashes", "offsets", "check_counts", "query_ids", "positions")


@pytest.fixture(scope="module")
def engine():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gzb import native as N
    e = N.PresearchEngine(0)
    yield e
    e.close()


def _database(sequences):
    """[d] seq [d] seq ... [d] of the given code arrays."""
    parts, offsets, at = [np.array([P.DELIMITER], np.uint8)], [1], 1
    for s in sequences:
        parts += [s, parts[0]]
        at += len(s) + 1
        offsets.append(at)
    return W.Database(codes=np.concatenate(parts).astype(np.uint8),
                      offsets=np.array(offsets, np.uint32), number_sequences=len(sequences))


@pytest.mark.parametrize("sets,length,window,extra", [
    (P.DEFAULT_REDUCED_SETS, 8, 10, 0), (P.DEFAULT_REDUCED_SETS, 8, 16, 1),
    (P.DEFAULT_REDUCED_SETS, 7, 1, 2), (P.DEFAULT_REDUCED_SETS, 6, 9, 3),
    ("ARNDCQEGH ILMFVWYPSTK", 8, 15, 0), ("ARNDCQEGH ILMFVWYPSTK", 9, 10, 1),
    ("ARNDCQEGH ILMFVWYPSTK", 16, 16, 2)])
def test_hash_and_window_lengths(engine, oracle, sets, length, window, extra):
    p = P.make_params(subsequence_length=window, reduced_sets=sets,
                      seed_threshold=39 if length <= 8 else 80)
    p["max_hash_length"] = length
    p["min_hash_length"] = min(length, 6)
    rng = np.random.default_rng(100 * length + window)
    seqs = [rng.integers(0, 20, n).astype(np.uint8)
            for n in list(range(1, 40)) + list(rng.integers(100, 400, 60)) + [200 + extra]]
    db = _database(seqs + [W.mutate(rng, s, 0.95) for s in seqs[::2]])
    q = W.make_queries(db, 40, 2701, median=60)
    engine.set_params(p)
    engine.set_database(db)
    engine.set_queries(q)
    got, exp = engine.index_arrays(), oracle.db_index(p, db.codes)
    for name in INDEX:
        assert np.array_equal(got[name], exp[name]), name
    got, exp = engine.list_arrays(), oracle.query_lists(p, q)
    for name in LISTS:
        assert np.array_equal(got[name], exp[name]), name
    assert len(exp["positions"]) > 0


SIZES = (1, 2, 3, 30, 31, 32, 33, 34, 63, 64, 65, 95, 127, 128, 129, 160, 255, 256, 257, 258,
         288, 289, 513, 1000, 3000)


@pytest.mark.parametrize("sizes", [SIZES, (65535, 300), (65536,), (65700, 40)],
                         ids=["edges", "65535", "65536", "65700"])
@pytest.mark.parametrize("changed", [0, 2, 10])
def test_bucket_sizes(engine, oracle, sizes, changed):
    """Each bucket's entries share a core and, with `changed` residues of the
    window drawn anew, one of a few surroundings: `changed` 0 gives large
    clusters, 10 hardly any."""
    if changed == 10 and max(sizes) > 3000:
        sizes = [min(s, 3000) for s in sizes]  # (the oracle compares every pair)
    p = P.make_params()
    rng = np.random.default_rng(sum(sizes) + changed)
    sequences = []
    for n in sizes:
        core = rng.integers(0, 20, 8).astype(np.uint8)
        families = rng.integers(0, 20, (7, 24)).astype(np.uint8)
        families[:, 8:16] = core
        s = families[rng.integers(0, 7, n)]
        for _ in range(changed):
            at = rng.choice(np.r_[0:8, 16:24], n)
            s[np.arange(n), at] = rng.integers(0, 20, n)
        sequences += list(s)
    order = rng.permutation(len(sequences))
    db = _database([sequences[i] for i in order])
    engine.set_params(p)
    engine.set_database(db)
    got, exp = engine.index_arrays(), oracle.db_index(p, db.codes)
    for name in INDEX:
        assert np.array_equal(got[name], exp[name]), name
    assert len(exp["member_positions"]) > 0 or changed == 10
