"""Which rows the gapped operator runs: the grouped ones where a gap fits into
the X-drop and a row's share of the gap extension is small, else one column at
a time (both are compared with the oracle in test_gpu_rows.py and
test_gpu_operators.py)."""
import numpy as np
import pytest

from gzb import params as P
from kernel_trace import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("go,ge,cutoff,grouped", [
    (11, 1, 38, True), (11, 1, 12, True), (11, 1, 11, False), (11, 24, 35, True),
    (11, 24, 34, False), (11, 25, 400, False), (11, 100, 38, False), (0, 1, 1, True),
    (11, 1, 960, False)])
def test_rows_by_penalties(go, ge, cutoff, grouped):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gzb import native as N
    codes = np.random.default_rng(1).integers(0, 20, 200).astype(np.uint8)
    keep, at = N.device_sequence(codes, P.DELIMITER)
    matrix = N.device_matrix(P.blosum62())
    q, d, scores = (torch.full((64,), 100, dtype=torch.int32, device="cuda") for _ in range(3))
    op = N.GappedExtenderGpu()
    op.SetQueries(P.DELIMITER, at)
    op.SetDatabase(at)
    op.SetScoreParameters(matrix, P.NUMBER_LETTERS, go, ge, cutoff)
    names = kernels(lambda: op.ExtendOneSideScoreOnlyAsync(64, False, None, None, None, q, d,
                                                           scores))
    rows = [n for n in names if "gapped_rows_kernel" in n]
    assert len(rows) == 1
    assert ("true" in rows[0]) == grouped and ("false" in rows[0]) != grouped
    del keep
