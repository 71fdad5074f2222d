"""The query statistics of many queries whatever their lengths: compositions
counted over every start and end within 16 bytes, empty queries, and long ones,
which must not make the other queries wait."""
import numpy as np
import pytest

from gzb import params as P

pytestmark = pytest.mark.gpu


def _torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _call(torch, codes, offsets, lengths):
    from gzb import native as N
    n = len(lengths)
    dev = [torch.from_numpy(a).cuda() for a in (codes, offsets.astype(np.int64),
                                                lengths.astype(np.int32))]
    out = [torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2)]
    matrix = P.blosum62()
    return lambda: N.query_karlin_cutoffs_async(*dev, n, matrix, *out), out


def test_any_alignment_and_length():
    torch = _torch()
    rng = np.random.default_rng(1)
    n = 2100
    lengths = np.concatenate([rng.integers(0, 40, n - 3), [1000, 70000, 17]])
    # queries that overlap and lie anywhere: no byte outside a query counts
    codes = rng.integers(0, 20, 80000).astype(np.uint8)
    offsets = rng.integers(0, len(codes) - lengths + 1)
    offsets[:16] = len(codes) - lengths[:16]
    run, out = _call(torch, codes, offsets, lengths)
    run()
    many = [o.cpu().numpy() for o in out]
    for a in range(0, n, 700):  # a warp a query
        part, got = _call(torch, codes, offsets[a:a + 700], lengths[a:a + 700])
        part()
        for x, y in zip(many, got):
            assert np.array_equal(x[a:a + 700], y.cpu().numpy())


@pytest.mark.parametrize("lengths", ["one of 35,000", "10,000 each"])
def test_long_queries_take_little_longer(lengths):
    torch = _torch()
    rng = np.random.default_rng(2)

    def time(ln):
        codes = rng.integers(0, 20, int(ln.sum())).astype(np.uint8)
        run, _ = _call(torch, codes, np.cumsum(ln) - ln, ln)
        times = []
        for _ in range(30):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            run()
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)
    long = np.full(2048, 300)
    if lengths == "10,000 each":
        long[:] = 10000
    else:
        long[1000] = 35000
    # (a warp a query: 1.0 of the time of 300 each; a byte a lane, one query
    # after another by one warp: 1.6 and 2.4)
    assert time(long) < 1.4 * time(np.full(2048, 300))
