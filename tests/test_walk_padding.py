"""The ungapped operator's window evaluation with anything but delimiters
around the sequences: the bytes behind a delimiter decide nothing and index
nothing outside the score tables.  On the CPU (the same source compiled for
the host, the memory behind the table set to scores that would show), then the
operator itself."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from gzb import params as P

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
PAD = 64


def _sequences(rng, n, pad):
    """One sequence between delimiters, each pad byte anything but a code."""
    q = rng.integers(32, 256, (2, n + 2 * pad + 2)).astype(np.uint8)
    q[:, pad:pad + n + 2] = rng.integers(0, 20, n + 2)
    same = rng.random(n + 2) < 0.5
    q[1, pad:pad + n + 2][same] = q[0, pad:pad + n + 2][same]
    q[:, pad] = q[:, pad + n + 1] = P.DELIMITER
    return q


@pytest.mark.parametrize("behind", [0x7ffe7ffe, 0x00ff00ff, 0x80018001])
def test_windows_ignore_what_lies_behind_a_delimiter(tmp_path_factory, behind):
    if shutil.which("nvcc") is None:
        pytest.skip("no nvcc")
    lib = str(tmp_path_factory.mktemp("walk") / "walk_padding_host.so")
    subprocess.check_call(["nvcc", "-std=c++17", "-O2", "-shared", "-Xcompiler", "-fPIC",
                           "-gencode", "arch=compute_100a,code=sm_100a",
                           "-I", os.path.join(ROOT, "ghostz-gpu_b200", "csrc"),
                           "-I", os.path.join(ROOT, "include"),
                           os.path.join(HERE, "walk_padding_host.cu"), "-o", lib])
    lib = C.CDLL(lib)
    m = np.zeros((32, 32), np.int32)
    m[:25, :25] = P.blosum62()
    rng = np.random.default_rng(1)
    p = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731
    for n in (1, 5, 31, 33, 70):
        q, d = _sequences(rng, n, PAD)
        pos = np.arange(PAD + 1, PAD + 1 + n).astype(np.uint32)
        hits = []
        for pad in (False, True):
            s = [x.copy() for x in (q, d)]
            if pad:
                for x in s:
                    x[:PAD] = x[PAD + n + 2:] = P.DELIMITER
            out = np.zeros(n, np.int32)
            lib.walk_window_hits(p(s[0]), p(s[1]), C.c_uint64(n), p(pos), p(pos), p(m),
                                 P.DELIMITER, 15, 20, C.c_uint32(behind), p(out))
            hits.append(out)
        assert np.array_equal(*hits)


@pytest.mark.gpu
@pytest.mark.parametrize("cutoff", [15, 127, 128, 400])
def test_operator_ignores_what_lies_behind_a_delimiter(oracle, cutoff):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gzb import native as N
    rng = np.random.default_rng(cutoff)
    params = P.make_params()
    matrix = N.device_matrix(P.blosum62())
    for n in (1, 5, 31, 33, 70, 300):
        q, d = _sequences(rng, n, PAD)
        pos = np.arange(PAD + 1, PAD + 1 + n).astype(np.uint32)
        trigger = 30
        op = N.UngappedExtenderGpu()
        dev = [torch.from_numpy(x.copy()).cuda() for x in (q, d)]
        cut = torch.full((1,), cutoff, dtype=torch.int32, device="cuda")
        trig = torch.full((1,), trigger, dtype=torch.int32, device="cuda")
        op.SetQueries(P.DELIMITER, dev[0].data_ptr(), cut, trig)
        op.SetDatabase(dev[1].data_ptr())
        op.SetScoreMatrix(matrix, P.NUMBER_LETTERS)
        ids = torch.zeros(n, dtype=torch.int32, device="cuda")
        at = torch.from_numpy(pos.astype(np.int32)).cuda()
        out = torch.full((n,), -1, dtype=torch.int8, device="cuda")
        op.ExtendWithTriggerAsync(n, None, None, None, None, ids, at, at, out)
        torch.cuda.synchronize()
        # (the oracle's sequences stop at their delimiters, too)
        exp = [oracle.ungapped_with_trigger(params, q, int(a), d, int(a), cutoff, trigger) > trigger
               for a in pos]
        assert out.cpu().numpy().astype(bool).tolist() == exp
