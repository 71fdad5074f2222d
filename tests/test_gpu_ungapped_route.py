"""Which kernel the ungapped operator runs: the window kernel for a delimiter
that is a residue code, the pair by pair one for any other (its flags are
compared in test_gpu_ungapped.py)."""
import numpy as np
import pytest

from gzb import params as P
from kernel_trace import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("delimiter,kernel", [(25, "ungapped_trigger"), (31, "ungapped_trigger"),
                                              (32, "ungapped_pairs"), (255, "ungapped_pairs")])
def test_kernel_by_delimiter(delimiter, kernel):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gzb import native as N
    codes = np.random.default_rng(1).integers(0, 20, 200).astype(np.uint8)
    keep, at = N.device_sequence(codes, delimiter)
    one = [torch.full((64,), v, dtype=torch.int32, device="cuda") for v in (0, 100, 100, 15, 40)]
    out = torch.empty(64, dtype=torch.int8, device="cuda")
    matrix = N.device_matrix(P.blosum62())
    op = N.UngappedExtenderGpu()
    op.SetQueries(delimiter, at, one[3], one[4])
    op.SetDatabase(at)
    op.SetScoreMatrix(matrix, P.NUMBER_LETTERS)
    names = kernels(lambda: op.ExtendWithTriggerAsync(64, None, None, None, None, *one[:3], out))
    assert [n for n in names if "ungapped" in n] and all(kernel in n for n in names
                                                         if "ungapped" in n)
    del keep
