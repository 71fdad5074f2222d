"""Every thread-per-extension kernel that runs the grouped rows
(csrc/gzb_row.cuh), and the ones it hands extensions on to, against the
oracle at the sizes where rows can go wrong: queries of every remainder by
the group of four columns, bands at the edge of the ring, scores at the edge
of a band's range, gap penalties and X-drops on both sides of the rule."""
import numpy as np
import pytest

from gzb import params as P
from gzb import workload as W
from test_gpu_operators import _concat, _gapped_gpu, torch_cuda  # noqa: F401

pytestmark = pytest.mark.gpu

KERNELS = [("rows", 64), ("rows", 32), ("rows", 128), ("lane", 64), ("deal", 64), ("static", 64)]


@pytest.mark.parametrize("kernel,width", KERNELS)
@pytest.mark.parametrize("go,ge,cutoff", [(11, 1, 26), (11, 1, 52), (4, 0, 10), (3, 2, 959),
                                          (3, 2, 960), (0, 0, 20)])
def test_rows_kernels_match_oracle(torch_cuda, oracle, kernel, width, go, ge, cutoff):  # noqa: F811
    from gzb import native as N
    params = P.make_params(gap_open=go, gap_extension=ge)
    rng = np.random.default_rng(cutoff + go + width)
    A, B = [], []
    for n in list(range(1, 34)) * 3 + [60, 61, 62, 63, 64, 65, 66, 127, 300, 700, 1500]:
        a = W.random_residues(rng, n)
        A.append(a)
        B.append(W.mutate(rng, a, rng.uniform(0.5, 1.0)))
    qc, qs = _concat(A, 25)
    dc, ds = _concat(B, 25)
    n = len(A)
    at = [int(rng.integers(0, min(len(A[i]), len(B[i])))) for i in range(n)]
    qpos = [qs[i] + at[i] for i in range(n)]
    dpos = [ds[i] + at[i] for i in range(n)]
    ids = {"rows": N.GAPPED_KERNEL_ROWS, "lane": N.GAPPED_KERNEL_LANE,
           "deal": N.GAPPED_KERNEL_DEAL, "static": N.GAPPED_KERNEL_STATIC}
    was = [N.get_tile_parameter(t) for t in (N.TILE_GAPPED_KERNEL, N.TILE_BAND_WIDTH)]
    N.set_tile_parameter(N.TILE_GAPPED_KERNEL, ids[kernel])
    N.set_tile_parameter(N.TILE_BAND_WIDTH, width)
    try:
        for rev in (False, True):
            s, q, d, cells = _gapped_gpu(torch_cuda, params, qc, dc, qpos, dpos, rev, cutoff)
            total = 0
            for i in range(n):
                es, eq, ed, ec = oracle.gapped_one_side(params, qc, qpos[i], dc, dpos[i], rev,
                                                        cutoff)
                total += ec
                assert (int(s[i]), int(q[i]), int(d[i])) == \
                    (es, int(qpos[i]) + eq, int(dpos[i]) + ed), (i, rev)
            assert cells == total
    finally:
        N.set_tile_parameter(N.TILE_GAPPED_KERNEL, was[0])
        N.set_tile_parameter(N.TILE_BAND_WIDTH, was[1])


@pytest.mark.parametrize("top", [900, 4000])
def test_large_matrix_entries(torch_cuda, oracle, top):  # noqa: F811
    """Scores that outgrow a band, and entries the rows do not admit."""
    m = np.full((20, 20), -2, np.int32)
    np.fill_diagonal(m, top)
    params = P.make_params(matrix=m)
    rng = np.random.default_rng(top)
    A = [rng.integers(0, 20, n).astype(np.uint8) for n in (1, 5, 20, 31, 32, 33, 200)]
    B = [W.mutate(rng, a, 0.9) for a in A]
    qc, qs = _concat(A, 25)
    dc, ds = _concat(B, 25)
    s, q, d, _ = _gapped_gpu(torch_cuda, params, qc, dc, list(qs), list(ds), False, 26, matrix=m)
    for i in range(len(A)):
        es, eq, ed, _ = oracle.gapped_one_side(params, qc, int(qs[i]), dc, int(ds[i]), False, 26)
        assert (int(s[i]), int(q[i]), int(d[i])) == (es, int(qs[i]) + eq, int(ds[i]) + ed), i
