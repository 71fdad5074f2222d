"""The query statistics of many queries at once (four lanes a query) against
the oracle and against the same queries a few at a time (a warp per query),
bit for bit: counts off the eight queries of a block, queries whose series needs
more rounds than the buffers hold, and matrices whose score ranges lie on
both sides of what those buffers are sized for."""
import numpy as np
import pytest

from gzb import params as P
from test_gpu_karlin import _cases, _layout, native  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu


def _many(oracle, n):
    cases = []
    while len(cases) < n:
        cases += _cases(oracle, 60 + len(cases))
    return cases[:n]


@pytest.mark.parametrize("n", [2047, 2048, 2049, 2056, 2311])
def test_many_match_oracle(native, oracle, params, n):  # noqa: F811
    cases = _many(oracle, n)
    codes, offsets, lengths = _layout(cases)
    cut, trig, kar = native.query_karlin_cutoffs(codes, offsets, lengths)
    for i, q in enumerate(cases):
        lam, k, h, c, t = oracle.query_karlin(params, q)
        assert (np.float32(lam), np.float32(k), np.float32(h)) == tuple(kar[i]), i
        assert (int(cut[i]), int(trig[i])) == (c, t), i


@pytest.mark.parametrize("low,high", [(-1, 11), (-4, 1), (-4, 3), (-4, 12), (-4, 15), (-12, 6),
                                      (-13, 6), (-16, 15)])
def test_many_match_few(native, oracle, low, high):  # noqa: F811
    m = P.blosum62().astype(np.int32)
    m = np.clip(m, low, high)
    m[17, 17], m[0, 24] = high, low
    if low < -4:
        m[m < 0] -= 2
        m = np.clip(m, low, high)
    cases = _many(oracle, 2100)
    codes, offsets, lengths = _layout(cases)
    many = native.query_karlin_cutoffs(codes, offsets, lengths, matrix=m)
    for a in range(0, len(cases), 1050):
        part = cases[a:a + 1050]
        few = native.query_karlin_cutoffs(*_layout(part), matrix=m)
        for x, y in zip(many, few):
            assert np.array_equal(x[a:a + 1050], y, equal_nan=x.dtype.kind == "f")
