"""Code scores on both sides of what the hashes in registers pack (24 bits
with the sign): the index and the query lists equal the oracle's."""
import numpy as np
import pytest

from gzb import params as P
from gzb import workload as W
from test_gpu_index_build import INDEX, LISTS, engine  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1, 762600, 762601, 1 << 20, 1 << 24])
def test_scaled_scores(engine, oracle, scale):  # noqa: F811
    p = P.make_params()
    p["code_scores"] *= scale           # 11 * 762,600 is the last that fits
    p["seed_threshold"] = 39 * scale
    db = W.make_database(300, 71, median=120)
    q = W.make_queries(db, 40, 72, median=60)
    engine.set_params(p)
    engine.set_database(db)
    engine.set_queries(q)
    got, exp = engine.index_arrays(), oracle.db_index(p, db.codes)
    assert all(np.array_equal(got[name], exp[name]) for name in INDEX)
    got, exp = engine.list_arrays(), oracle.query_lists(p, q)
    assert all(np.array_equal(got[name], exp[name]) for name in LISTS)
