"""The ungapped operator at the edges of its window evaluation against the
oracle: cutoffs and scores in and beyond the window tables' range, a
delimiter that is no residue code, seeds at sequence ends, sequences longer
and shorter than a window, and counts off a warp's 32."""
import numpy as np
import pytest

from gzb import params as P
from gzb import workload as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 20000])
@pytest.mark.parametrize("delimiter,scale,cutoffs", [
    (25, 1, (1, 40)), (25, 1, (100, 180)), (31, 1, (5, 25)), (200, 1, (5, 25)),
    (25, 11, (50, 127)), (25, 12, (50, 127)), (25, 20, (300, 900))])
def test_flags_match_oracle(oracle, n, delimiter, scale, cutoffs):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gzb import native as N
    rng = np.random.default_rng(n + delimiter + scale)
    matrix = P.blosum62() * scale
    p = P.make_params(matrix=matrix)
    p["delimiter"] = delimiter

    def concat(seqs):
        starts, parts, at = [], [[delimiter]], 1
        for s in seqs:
            starts.append(at)
            parts += [s, [delimiter]]
            at += len(s) + 1
        return np.concatenate(parts).astype(np.uint8), np.array(starts)
    A = [W.random_residues(rng, int(rng.choice([1, 3, 30, 33, 65, 200]))) for _ in range(200)]
    B = [W.mutate(rng, a, rng.uniform(0.3, 1.0)) if len(a) > 3 else a for a in A]
    B = [b if len(b) else a for a, b in zip(A, B)]
    (qc, qs), (dc, ds) = concat(A), concat(B)
    ids = rng.integers(0, len(A), n)
    qp = np.array([qs[i] + rng.integers(0, len(A[i])) for i in ids])
    dp = np.array([ds[i] + min(max(a - qs[i] + rng.integers(-1, 2), 0), len(B[i]) - 1)
                   for i, a in zip(ids, qp)])
    cut = rng.integers(*cutoffs, len(A)).astype(np.int32)
    trig = (scale * rng.integers(0, 60, len(A))).astype(np.int32)
    _, qa = keep_q = N.device_sequence(qc, delimiter)
    _, da = keep_d = N.device_sequence(dc, delimiter)
    tm = N.device_matrix(matrix)
    tcut, ttrig = torch.from_numpy(cut).cuda(), torch.from_numpy(trig).cuda()
    u = N.UngappedExtenderGpu()
    u.SetQueries(delimiter, qa, tcut, ttrig)
    u.SetDatabase(da)
    u.SetScoreMatrix(tm, matrix.shape[0])
    dev = [torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(3)]
    out = torch.full((n,), -1, dtype=torch.int8, device="cuda")
    flags = np.zeros(n, np.int8)
    u.ExtendWithTriggerAsync(n, ids.astype(np.uint32), qp.astype(np.uint32),
                             dp.astype(np.uint32), flags, *dev, out)
    torch.cuda.synchronize()
    exp = np.array([oracle.ungapped_with_trigger(p, qc, int(a), dc, int(b), int(cut[i]),
                                                 int(trig[i])) > trig[i]
                    for i, a, b in zip(ids, qp, dp)], np.int8)
    assert np.array_equal(flags, exp)
    assert n < 1000 or 0 < exp.sum() < n
    del keep_q, keep_d
