"""Large uploads: from pageable memory (staged by several threads) and from
page-locked memory (copied directly) a chunk gives the same index, at lengths
around the least staged one and off the staging's pieces, repeatedly and on
another stream; a bad code in the last piece is refused."""
import numpy as np
import pytest

from gzb import params as P
from gzb import workload as W

pytestmark = pytest.mark.gpu
LEAST = 8 << 20


@pytest.mark.parametrize("length", [LEAST - 1, LEAST, LEAST + 1, 2 * LEAST + 12345])
def test_pageable_and_pinned_uploads(length):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gzb import native as N
    rng = np.random.default_rng(length)
    codes = rng.integers(0, 20, length).astype(np.uint8)
    offsets = np.arange(1, length - 300, 300, dtype=np.uint32)
    codes[offsets - 1] = P.DELIMITER
    codes[-1] = P.DELIMITER
    offsets = np.append(offsets, length).astype(np.uint32)
    pinned = torch.from_numpy(codes).pin_memory().numpy()
    e = N.PresearchEngine(0)
    try:
        e.set_params(P.make_params())
        blobs = []
        stream = torch.cuda.Stream()
        for source, s in ((pinned, None), (codes, None), (codes, stream.cuda_stream),
                          (codes, None)):
            db = W.Database(codes=source, offsets=offsets, number_sequences=len(offsets) - 1)
            e.set_database(db, stream=s) if s else e.set_database(db)
            blobs.append(e.export_index())
        assert all(np.array_equal(blobs[0], b) for b in blobs[1:])
        bad = codes.copy()
        bad[-2] = 32
        with pytest.raises(N.GzbError, match="below 32"):
            e.set_database(W.Database(codes=bad, offsets=offsets,
                                      number_sequences=len(offsets) - 1))
    finally:
        e.close()


def test_per_thread_default_stream():
    """The per-thread default stream's handle means another stream in every
    thread: the staged pieces have to arrive between the work queued before
    and after the upload on the calling thread's."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gzb import native as N
    per_thread = 2  # cudaStreamPerThread
    length = 48 << 20
    rng = np.random.default_rng(5)
    offsets = np.arange(1, length - 300, 300, dtype=np.uint32)
    chunks = []
    for _ in range(2):
        codes = rng.integers(0, 20, length).astype(np.uint8)
        codes[offsets - 1] = P.DELIMITER
        codes[-1] = P.DELIMITER
        chunks.append(codes)
    offs = np.append(offsets, length).astype(np.uint32)
    e = N.PresearchEngine(0)
    try:
        e.set_params(P.make_params())

        def index(codes, **stream):
            db = W.Database(codes=codes, offsets=offs, number_sequences=len(offs) - 1)
            e.set_database(db, **stream)
            return e.export_index(**stream)
        want = [index(torch.from_numpy(c).pin_memory().numpy()) for c in chunks]
        for k in (0, 1, 0, 1, 1, 0):
            assert np.array_equal(index(chunks[k], stream=per_thread), want[k])
    finally:
        e.close()
