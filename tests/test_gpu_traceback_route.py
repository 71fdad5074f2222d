"""Bands of up to 256 columns stay with the build results step's warp kernel
(no thread kernel runs), wider ones do not; both equal the oracle."""
import numpy as np
import pytest

from gzb import params as P
from gzb import workload as W
from kernel_trace import kernels
from test_gpu_build_results import _check, engine  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu


# the widest band of these sides has some 2 (X-drop - 11) + 30 columns
@pytest.mark.parametrize("cutoff,redone", [(90, False), (106, False), (108, False), (116, False),
                                           (122, False), (130, True)])
def test_wide_bands(engine, oracle, cutoff, redone):  # noqa: F811
    rng = np.random.default_rng(7)
    db = W.make_database(12, 31, median=700, lo=600, hi=900)
    q = W.pack_queries([W.mutate(rng, db.codes[db.offsets[s]:db.offsets[s + 1] - 1], 0.9,
                                 indel_p=0.0) for s in range(12)])
    p = P.make_params()
    p["result_gapped_cutoff"] = cutoff
    engine.set_params(p)
    engine.set_database(db)
    engine.set_queries(q)
    engine.presearch(0)
    assert _check(engine, oracle, p, db, q) >= 12
    names = kernels(lambda: engine.build_alignments())
    assert any("tb_side_warp_kernel" in n for n in names)
    assert any("tb_walk_kernel" in n for n in names) == redone
