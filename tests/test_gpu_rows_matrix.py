"""Score matrices whose entries the grouped rows do not admit: the
thread-per-extension kernels run the general rows themselves.  Every extension
equals the oracle's, and an engine hands none of them on."""
import numpy as np
import pytest

from gzb import params as P
from gzb import workload as W
from kernel_trace import kernels
from test_gpu_operators import _concat, _gapped_gpu, torch_cuda  # noqa: F401

pytestmark = pytest.mark.gpu

KERNELS = ["ROWS", "LANE", "DEAL", "STATIC"]


def _matrix():
    m = P.blosum62()
    stop = P.LETTERS.index("*")
    m[stop, :] = m[:, stop] = -2000
    return m


@pytest.mark.parametrize("kernel", KERNELS)
def test_operator_matches_oracle(torch_cuda, oracle, kernel):  # noqa: F811
    from gzb import native as N
    m = _matrix()
    params = P.make_params(matrix=m)
    rng = np.random.default_rng(5)
    A = [W.random_residues(rng, n) for n in (1, 2, 31, 32, 33, 64, 65, 300) for _ in range(9)]
    B = [W.mutate(rng, a, 0.85) for a in A]
    for s in B[::3]:
        s[len(s) // 2] = P.LETTERS.index("*")
    qc, qs = _concat(A, 25)
    dc, ds = _concat(B, 25)
    was = N.get_tile_parameter(N.TILE_GAPPED_KERNEL)
    N.set_tile_parameter(N.TILE_GAPPED_KERNEL, getattr(N, "GAPPED_KERNEL_" + kernel))
    try:
        for rev in (False, True):
            at = [(len(a) if len(a) < len(b) else len(b)) - 1 if rev else 0 for a, b in zip(A, B)]
            qpos = [int(s) + k for s, k in zip(qs, at)]
            dpos = [int(s) + k for s, k in zip(ds, at)]
            s, q, d, cells = _gapped_gpu(torch_cuda, params, qc, dc, qpos, dpos, rev, 38, matrix=m)
            total = 0
            for i in range(len(A)):
                es, eq, ed, ec = oracle.gapped_one_side(params, qc, qpos[i], dc, dpos[i], rev, 38)
                assert (int(s[i]), int(q[i]), int(d[i])) == (es, qpos[i] + eq, dpos[i] + ed), i
                total += ec
            assert cells == total
    finally:
        N.set_tile_parameter(N.TILE_GAPPED_KERNEL, was)


@pytest.mark.parametrize("kernel", KERNELS)
def test_engine_hands_nothing_on(torch_cuda, kernel):  # noqa: F811
    from gzb import native as N
    db = W.make_database(300, 61, median=200)
    rng = np.random.default_rng(62)
    q = W.pack_queries([W.mutate(rng, db.codes[db.offsets[s]:db.offsets[s + 1] - 1], 0.8)
                        for s in range(0, 60, 2)])
    e = N.PresearchEngine(0)
    try:
        e.set_params(P.make_params(matrix=_matrix()))
        e.set_database(db)
        e.set_queries(q)
        e.set_tile(N.SCHEDULE_BATCHED, N.TILE_GAPPED_KERNEL, getattr(N, "GAPPED_KERNEL_" + kernel))
        e.presearch(N.SCHEDULE_BATCHED)
        c = e.counters()
        assert c["gapped_extensions"] > 50
        assert c["gapped_fallbacks"] == 0
        e.reset_results()
        names = kernels(lambda: e.presearch(N.SCHEDULE_BATCHED))
        assert not any("gapped" in n and "true>" in n for n in names)
    finally:
        e.close()
