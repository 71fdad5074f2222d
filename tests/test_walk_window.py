"""The seed search's window evaluation (csrc/gzb_walk.cuh) on the CPU: the
same source compiled for the host, against the pair by pair walk.  Every seed
it settles is no hit, with the walk's own number of residue pairs; a seed that
could be a hit, or whose walk leaves the window, is never settled.  Its exact
form decides hits, too, and leaves open only walks that leave the window."""
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


@pytest.fixture(scope="module")
def windows(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("no nvcc")
    lib = str(tmp_path_factory.mktemp("walk") / "walk_window_host.so")
    subprocess.check_call(["nvcc", "-std=c++17", "-O2", "-shared", "-Xcompiler", "-fPIC",
                           "-gencode", "arch=compute_100a,code=sm_100a",
                           "-I", os.path.join(ROOT, "ghostz-gpu_b200", "csrc"),
                           "-I", os.path.join(ROOT, "include"),
                           os.path.join(HERE, "walk_window_host.cu"), "-o", lib])
    return C.CDLL(lib)


def _side(q, d, i, j, step, m, delim, cutoff):
    """(best, pairs examined) of one side, pair by pair."""
    best = score = pairs = 0
    while q[i] != delim and d[j] != delim:
        score += int(m[d[j], q[i]])
        pairs += 1
        best = max(best, score)
        if best - score >= cutoff:
            break
        i += step
        j += step
    return best, pairs


# X-drops from one pair to more than a window holds, scores at the admitted
# edge, and delimiters at every distance from the seed
@pytest.mark.parametrize("cutoff,top,worst", [(15, 9, -4), (1, 5, -1), (127, 127, -127),
                                              (30, 2, -1), (16, 11, -127)])
def test_settled_seeds(windows, cutoff, top, worst):
    rng = np.random.default_rng(cutoff)
    delim, n = 25, 4000
    m = np.zeros((32, 32), np.int32)
    m[:25, :25] = rng.integers(worst, 1, (25, 25))
    np.fill_diagonal(m[:25, :25], rng.integers(1, top + 1, 25))
    q = np.full(n + 2 * PAD, delim, np.uint8)
    q[PAD:-PAD] = rng.integers(0, 25, n)
    d = q.copy()
    change = rng.random(len(d)) < 0.6
    d[change] = rng.integers(0, 25, int(change.sum()))
    for s in (q, d):
        s[rng.random(len(s)) < 0.02] = delim
        s[:PAD] = s[-PAD:] = delim
    qpos = rng.integers(PAD, PAD + n, 3000).astype(np.uint32)
    # unrelated pairs, and every relative alignment
    dpos = np.where(rng.random(3000) < 0.5, qpos, rng.integers(PAD, PAD + n, 3000)).astype(np.uint32)
    trigger = 3 * cutoff
    settled = np.zeros(3000, np.int32)
    steps = np.zeros(3000, np.int32)
    hits = np.zeros(3000, np.int32)
    p = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731
    windows.walk_windows(p(q), p(d), C.c_uint64(3000), p(qpos), p(dpos), p(m), delim, cutoff,
                         trigger, p(settled), p(steps), p(hits))
    for i in range(3000):
        a, b = int(qpos[i]), int(dpos[i])
        rb, rn = _side(q, d, a - 1, b - 1, -1, m, delim, cutoff)
        fb, fn = _side(q, d, a, b, 1, m, delim, cutoff)
        if settled[i]:
            assert rb + fb <= trigger, i
            assert steps[i] == rn + fn, i
            assert hits[i] == 0, i
        # open only where a walk leaves the window
        assert hits[i] == (rb + fb > trigger) or (hits[i] < 0 and max(rn, fn) >= 32), i
    assert settled.sum() > 0 or cutoff == 127  # (no walk of the wide X-drop ends in a window)


def test_blosum_seeds_are_settled(windows):
    """With the search's own parameters nine unrelated seeds in ten settle."""
    rng = np.random.default_rng(4)
    m = np.zeros((32, 32), np.int32)
    m[:25, :25] = P.blosum62()
    q = np.full(20000 + 2 * PAD, 25, np.uint8)
    d = q.copy()
    q[PAD:-PAD] = rng.integers(0, 20, 20000)
    d[PAD:-PAD] = rng.integers(0, 20, 20000)
    qpos = rng.integers(PAD, PAD + 20000, 5000).astype(np.uint32)
    dpos = rng.integers(PAD, PAD + 20000, 5000).astype(np.uint32)
    settled = np.zeros(5000, np.int32)
    steps = np.zeros(5000, np.int32)
    p = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731
    windows.walk_windows(p(q), p(d), C.c_uint64(5000), p(qpos), p(dpos), p(m), 25, 15, 41,
                         p(settled), p(steps), None)
    assert settled.mean() > 0.9
