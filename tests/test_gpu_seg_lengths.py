"""SEG masking at the edges of its kernels against the oracle, bit for bit:
stretches around the 127 letters that are trimmed in registers, sequences
around 32 windows and around the windows kept in shared memory, and enough
short reads that a warp looks for marked frames several at a time."""
import numpy as np
import pytest

from gzb import params as P
from gzb import workload as W
from test_gpu_seg import _low_complexity_protein, _reads, native  # noqa: F401

pytestmark = pytest.mark.gpu

LETTERS = np.frombuffer(b"ARNDCQEGHILKMFPSTWYV", np.uint8)


def _stretch(rng, length, kinds, around):
    s = LETTERS[rng.integers(0, 20, length + 2 * around)].copy()
    pool = LETTERS[rng.choice(20, size=kinds, replace=False)]
    s[around:around + length] = pool[rng.integers(0, kinds, length)]
    return bytes(s)


def test_stretches_and_lengths(native, oracle):  # noqa: F811
    rng = np.random.default_rng(170)
    prots = [_stretch(rng, n, kinds, around)
             for n in (1, 12, 31, 33, 64, 100, 115, *range(120, 136), 160, 227, 228, 300, 700)
             for kinds in (1, 2, 4) for around in (0, 40)]
    prots += [bytes([c]) * n for c in b"AX*" for n in (12, 43, 44, 127, 128, 138, 139, 140, 500)]
    prots += [_low_complexity_protein(rng, n) for n in (43, 44, 45, 75, 76, 4106, 4107, 4108, 5000)
              for _ in range(4)]
    seqs = [native.encode_protein_for_seg(p) for p in prots]
    zero = np.zeros(len(seqs), np.int32)
    q = W.pack_queries(seqs, cutoffs=(zero, zero))
    codes, _, _ = native.prepare_protein_queries(q.codes, q.offsets, q.lengths)
    masked = 0
    for i, p in enumerate(prots):
        exp = oracle.protein_query_seg(p, P.DELIMITER)
        o, n = int(q.offsets[i]), int(q.lengths[i])
        assert np.array_equal(codes[o:o + n - 1], exp[:-1]), (i, len(p), p)
        masked += bool((codes[o + 1:o + n - 1] == 24).any())
    assert masked > 100


@pytest.mark.parametrize("repeat", [1, 9, 40])
def test_many_reads(native, oracle, repeat):  # noqa: F811
    """(The repeated copies of the reads are masked as the first ones.)"""
    rng = np.random.default_rng(171 + repeat)
    reads, _, _ = _reads(rng, 701)
    exp = [oracle.translate_query_seg(r, P.DELIMITER) for r in reads]
    order = rng.permutation(np.repeat(np.arange(len(reads)), repeat))
    dna = np.frombuffer(b"".join(reads[i] for i in order), np.uint8).copy()
    offsets = np.zeros(len(order) + 1, np.uint64)
    offsets[1:] = np.cumsum([len(reads[i]) for i in order])
    codes, offs, lens, _, _ = native.prepare_translated_queries(dna, offsets)
    for r, i in enumerate(order):
        assert np.array_equal(codes[int(offs[r]):int(offs[r]) + int(lens[r])], exp[i]), (r, i)
