"""The grouped rows of the gapped extension (csrc/gzb_row.cuh) against the
oracle, on the CPU: the same source compiled for the host.  Scores, positions
and DP cell counts are whole numbers and have to be equal."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from gzb import params as P
from gzb import workload as W

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
PAD = 64


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("no nvcc")
    lib = str(tmp_path_factory.mktemp("row_dp") / "row_dp_host.so")
    subprocess.check_call(["nvcc", "-std=c++17", "-O2", "-shared", "-Xcompiler", "-fPIC",
                           "-gencode", "arch=compute_100a,code=sm_100a",
                           "-I", os.path.join(ROOT, "ghostz-gpu_b200", "csrc"),
                           "-I", os.path.join(ROOT, "include"),
                           os.path.join(HERE, "row_dp_host.cu"), "-o", lib])
    return C.CDLL(lib)


def _run(rows, width, q, q0, d, d0, delim, go, ge, cutoff, rev, matrix):
    out = (C.c_int32 * 3)()
    cells = C.c_uint64()
    m = np.ascontiguousarray(matrix, np.int32)
    st = rows.row_extend(width, C.c_void_p(q.ctypes.data), C.c_uint64(q0),
                         C.c_void_p(d.ctypes.data), C.c_uint64(d0), delim, go, ge, cutoff,
                         int(rev), C.c_void_p(m.ctypes.data), m.shape[0], out, C.byref(cells))
    return st, (out[0], out[1], out[2], cells.value)


def _buffer(rng, parts, delim, letters):
    """[pad, delim, part 0, delim, part 1, delim, pad] and the first part's start;
    the neighbour behind the delimiter is a sequence of its own."""
    pad = np.full(PAD, delim, np.uint8)
    other = rng.integers(0, letters, 20).astype(np.uint8)
    return np.concatenate([pad, other, [delim], parts, [delim], other, pad]).astype(np.uint8), \
        PAD + 21


def _pair(rng, n, letters):
    a = rng.integers(0, letters, n).astype(np.uint8)
    b = a.copy()
    m = rng.random(n) < rng.uniform(0, 0.5)
    b[m] = rng.integers(0, letters, int(m.sum()))
    if n > 8 and rng.random() < 0.6:
        at, k = int(rng.integers(1, n - 4)), int(rng.integers(1, 6))
        b = np.delete(b, slice(at, at + k)) if rng.random() < 0.5 else \
            np.insert(b, at, rng.integers(0, letters, k)).astype(np.uint8)
    return a, b


# gap penalties and X-drops: no gap column at all (X-drop below a gap), one,
# many; free extension; X-drop 0; a wide X-drop that only short queries hold
@pytest.mark.parametrize("go,ge,cutoff", [(11, 1, 26), (11, 1, 52), (11, 1, 11), (11, 1, 12),
                                          (0, 1, 5), (5, 3, 40), (4, 0, 10), (11, 1, 0),
                                          (7, 2, 200), (40, 10, 959)])
@pytest.mark.parametrize("width", [32, 64])
def test_rows_match_oracle(rows, oracle, go, ge, cutoff, width):
    rng = np.random.default_rng(go * 1000 + ge * 100 + cutoff + width)
    done = handed = 0
    for it in range(400):
        protein = it % 2 == 0
        letters = 20 if protein else int(rng.integers(2, 8))
        if protein:
            matrix, delim = P.blosum62(), 25
        else:
            matrix = rng.integers(-4, 1, (letters, letters)).astype(np.int32)
            np.fill_diagonal(matrix, rng.integers(1, 8, letters))
            delim = letters
        # every remainder of a query's length by the group of four columns
        a, b = _pair(rng, int(rng.integers(1, 24)) if it % 3 else int(rng.integers(24, 220)),
                     letters)
        q, q0 = _buffer(rng, a, delim, letters)
        d, d0 = _buffer(rng, b, delim, letters)
        i = int(rng.integers(0, len(a)))
        j = int(np.clip(i + rng.integers(-2, 3), 0, len(b) - 1))
        params = P.make_params(matrix=matrix, gap_open=go, gap_extension=ge)
        params["delimiter"] = delim
        rev = bool(rng.random() < 0.5)
        st, got = _run(rows, width, q, q0 + i, d, d0 + j, delim, go, ge, cutoff, rev, matrix)
        if st == 2:
            handed += 1
            continue
        assert st == 1
        assert got == oracle.gapped_one_side(params, q, q0 + i, d, d0 + j, rev, cutoff), \
            (it, i, j, rev)
        done += 1
    assert done > 100


def test_long_homologs_and_score_limit(rows, oracle):
    """Thousands of rows (the per-row share of every score grows), and scores
    past what a band holds, which are handed on rather than wrapped."""
    rng = np.random.default_rng(3)
    states = set()
    for top, n in ((6, 3000), (6, 9000), (11, 4000)):
        matrix = np.full((20, 20), -4, np.int32)
        np.fill_diagonal(matrix, top)
        a = rng.integers(0, 20, n).astype(np.uint8)
        b = a.copy()
        b[::97] = rng.integers(0, 20, len(b[::97]))
        q, q0 = _buffer(rng, a, 25, 20)
        d, d0 = _buffer(rng, b, 25, 20)
        params = P.make_params(matrix=matrix)
        st, got = _run(rows, 64, q, q0, d, d0, 25, 11, 1, 26, False, matrix)
        states.add(st)
        if st == 1:
            assert got == oracle.gapped_one_side(params, q, q0, d, d0, False, 26)
    assert states == {1, 2}


@pytest.mark.parametrize("go,ge,cutoff,admitted", [
    (11, 1, 26, True), (11, 1, 959, True), (11, 1, 960, False), (11, 1, -1, False),
    (0, 0, 26, False), (1023, 0, 26, True), (1023, 1, 26, False), (0, 1023, 26, True)])
def test_admitted_parameters(rows, go, ge, cutoff, admitted):
    matrix = np.full((20, 20), -1, np.int32)
    rng = np.random.default_rng(1)
    q, q0 = _buffer(rng, np.zeros(5, np.uint8), 25, 20)
    st, _ = _run(rows, 64, q, q0, q, q0, 25, go, ge, cutoff, False, matrix)
    fits = -1 + ge < 1024 - cutoff
    assert (st != -1) == (admitted and fits)


# The first row's columns reach the query's end where a gap is cheap: the
# delimiter's column is no cell, whatever the score table holds for its byte
# (codes from 32 on read a neighbouring row's entries, a delimiter below the
# matrix's side its own).
@pytest.mark.parametrize("delim", [19, 25, 31, 34, 50, 63, 64, 100, 200, 255])
@pytest.mark.parametrize("go,ge,cutoff", [(0, 1, 30), (1, 1, 30), (2, 3, 60), (4, 0, 10)])
def test_delimiter_column_is_no_cell(rows, oracle, delim, go, ge, cutoff):
    rng = np.random.default_rng(delim * 100 + go + ge)
    matrix = P.blosum62()[:20, :20]
    matrix[:, 19] = matrix[19, :] = 9
    done = 0
    for n in list(range(1, 14)) * 12:
        letters = 19
        a, b = (rng.integers(0, letters, k).astype(np.uint8) for k in (n, int(rng.integers(1, 30))))
        q, q0 = _buffer(rng, a, delim, letters)
        d, d0 = _buffer(rng, b, delim, letters)
        params = P.make_params(matrix=matrix, gap_open=go, gap_extension=ge)
        params["delimiter"] = delim
        for rev in (False, True):
            i, j = (len(a) - 1, len(b) - 1) if rev else (0, 0)
            st, got = _run(rows, 32, q, q0 + i, d, d0 + j, delim, go, ge, cutoff, rev, matrix)
            if st == 1:
                assert got == oracle.gapped_one_side(params, q, q0 + i, d, d0 + j, rev, cutoff), \
                    (n, rev)
                done += 1
    assert done > 100
