"""An engine's page-locked staging: not made for its first large uploads, whose
copies would not pay for it, but once they add up to 128 MB; chunks uploaded
through it, at lengths around the least staged one and off its pieces and on
another stream, give the index of a page-locked upload."""
import numpy as np
import pytest

from gzb import params as P
from gzb import workload as W
from kernel_trace import kernels

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _chunk(length, seed):
    rng = np.random.default_rng(seed)
    codes = rng.integers(0, 20, length).astype(np.uint8)
    offsets = np.arange(1, length - 300, 300, dtype=np.uint32)
    codes[offsets - 1] = P.DELIMITER
    codes[-1] = P.DELIMITER
    offsets = np.append(offsets, length).astype(np.uint32)
    return W.Database(codes=codes, offsets=offsets, number_sequences=len(offsets) - 1)


def _pinned_copies(call):
    return sum("Memcpy HtoD (Pinned" in n for n in kernels(call))


def test_staging_is_made_when_it_pays():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gzb import native as N
    small, large = _chunk(8 * MB, 1), _chunk(60 * MB, 2)
    e = N.PresearchEngine(0)
    try:
        e.set_params(P.make_params())
        assert _pinned_copies(lambda: e.set_database(small)) < 8       # 8 MB
        assert _pinned_copies(lambda: e.set_database(large)) < 8       # 68
        assert _pinned_copies(lambda: e.set_database(large)) >= 60     # 128
        assert _pinned_copies(lambda: e.set_database(small)) >= 8
        for length in (8 * MB - 1, 8 * MB, 8 * MB + 1, 16 * MB + 12345):
            db = _chunk(length, length)
            pinned = W.Database(codes=torch.from_numpy(db.codes).pin_memory().numpy(),
                                offsets=db.offsets, number_sequences=db.number_sequences)
            e.set_database(pinned)
            want = e.export_index()
            for stream in (None, torch.cuda.Stream().cuda_stream, 2):
                e.set_database(db, stream=stream)
                assert np.array_equal(e.export_index(stream=stream), want)
            db.codes[-2] = 32
            with pytest.raises(N.GzbError, match="below 32"):
                e.set_database(db)
    finally:
        e.close()
