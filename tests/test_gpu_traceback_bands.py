"""Build results where the traced extension changes its path: rows a lane
short of, at and beyond one and two steps of 32 columns, bands around the 224
columns a warp keeps and beyond them (the thread kernels redo those), gap
costs that open and extend in every order, and extensions that end within a
few residues of a sequence's end.  Every alignment equals the oracle's."""
import numpy as np
import pytest

from gzb import params as P
from gzb import workload as W
from test_gpu_build_results import _check, engine  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gap_open,gap_extension", [(11, 1), (1, 1), (5, 2), (3, 7)])
@pytest.mark.parametrize("cutoff", [1, 14, 15, 16, 31, 64, 95, 104, 112, 113, 130, 260])
def test_bands(engine, oracle, gap_open, gap_extension, cutoff):  # noqa: F811
    rng = np.random.default_rng(2800 + cutoff)
    db = W.make_database(200, 2801, median=700)
    seqs = []
    for s in range(0, 36, 2):
        src = db.codes[db.offsets[s]:db.offsets[s + 1] - 1]
        seqs.append(W.mutate(rng, src, rng.uniform(0.5, 0.95), indel_p=0.03))
    q = W.pack_queries(seqs)
    p = P.make_params(gap_open=gap_open, gap_extension=gap_extension)
    p["gapped_cutoff"] = min(cutoff, 26)
    p["result_gapped_cutoff"] = cutoff
    engine.set_params(p)
    engine.set_database(db)
    engine.set_queries(q)
    engine.presearch(0)
    assert _check(engine, oracle, p, db, q) > 10


def test_short_ends(engine, oracle, params):  # noqa: F811
    """Queries that are a homolog's piece, cut so that one side or both reach
    the query's or the subject's end within 0 to 70 residues."""
    db = W.make_database(120, 2901, median=160, lo=60, hi=400)
    rng = np.random.default_rng(2902)
    seqs = []
    for s in range(72):
        src = db.codes[db.offsets[s]:db.offsets[s + 1] - 1]
        cut = s % 72
        piece = src[: max(40, len(src) - cut)] if s % 2 else src[min(cut, len(src) - 40):]
        seqs.append(W.mutate(rng, piece, 0.92, indel_p=0.01))
    q = W.pack_queries(seqs)
    engine.set_params(params)
    engine.set_database(db)
    engine.set_queries(q)
    engine.presearch(0)
    assert _check(engine, oracle, params, db, q) > 40
