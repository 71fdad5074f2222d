// gzb_walk.cuh -- the ungapped X-drop extension of a seed over a window of
// 32 residues either side, without branches (the seed search's first pass).
//
// SeedSearcher::UngappedExtend (src/seed_searcher.h:133-158) walks from the
// seed both ways until the score falls `cutoff` below its best or a
// delimiter is met, and asks whether the two bests sum to more than
// `trigger`.  Nine walks in ten end within 32 pairs on either side, and
// 987 seeds in 1,000 stay far below the trigger.  walk_window evaluates
// 32 pairs of both sides for every seed: where both walks end and even the
// windows' largest scores (an upper bound of the bests) do not exceed the
// trigger, the seed is settled, with the exact number of pairs the walks
// examined; the other seeds' walks go on from their windows' ends (walk_on),
// 32 of them together, and those near the trigger are left to walk_hit.
//
// Both sides are computed in one word, reverse in the low half and forward in
// the high half, scores doubled.  Per pair of pairs: two table words (the
// forward table's entries are << 16), score, running best, drop below it,
// and a sticky flag whose sum counts the steps from the walk's end on.  A
// delimiter's entry is odd, so that bit 0 of the drop tells a walk that a
// delimiter ended.  Exact for matrix entries up to kWalkMaxEntry in size and
// cutoffs 1 .. kWalkMaxCutoff.
//
// The 64 bytes around a position are read as three aligned 32-byte words: a
// scattered request costs the L1 cache one cycle per lane's 32-byte sector
// that misses, and at least ten a request whatever its width.  Measured on a
// B200, 32 random windows of an L2-resident chunk an SM: 97 cycles (three
// 32-byte loads a lane), 114 (five 16-byte loads), 161 (not allocated in
// L1); twenty 4-byte loads cost ten cycles each even where all hit.
#pragma once

#include <cstdint>

#include "gzb_kernels.cuh"
#include "gzb_row.cuh"

namespace gzb {

constexpr int kWindow = 32;           // residue pairs either side
constexpr int kWalkMaxEntry = 127;
constexpr int kWalkMaxCutoff = 127;
constexpr int kWalkStop = -513;       // a delimiter's (doubled) entry
constexpr uint32_t kWalkBias = 0x5000;       // keeps a half from borrowing
constexpr uint32_t kWalkBiasExact = 0x6200;  // (over 31 steps of 256 more)
constexpr int kWalkFlag = 0x400;      // set in a drop of at least cutoff

// Score table: the doubled score of (query code a, database code b) at byte
// 256 a + 4 (a ^ b) (reverse) and, << 16, 128 bytes behind (forward).  The
// XOR puts pairs that share a code into different banks.
constexpr int kWindowTableBytes = 32 * 256;

__host__ __device__ __forceinline__ int window_entry(int a, int b, int score, int delim) {
  return a == delim || b == delim ? kWalkStop : 2 * score;
}

// Fills the table; returns (on every thread) whether the matrix is admitted.
__device__ __forceinline__ bool load_window_table(uint32_t tbl, const int32_t *m, int delim,
                                                  int stride = 32) {
  bool fits = true;
  for (int i = threadIdx.x; i < 32 * 32; i += blockDim.x) {
    const int a = i >> 5, x = i & 31, b = a ^ x;
    const int score = m[b * stride + a];
    fits = fits && score >= -kWalkMaxEntry && score <= kWalkMaxEntry;
    const int v = window_entry(a, b, score, delim);
    row_store(tbl + 256 * a + 4 * x, (uint32_t)v);
    row_store(tbl + 256 * a + 4 * x + 128, (uint32_t)v << 16);
  }
  return __syncthreads_and(fits) != 0;
}

// The 32-byte words that hold s[-32 .. 31] (between s - 63 and s + 63).
struct WindowWords {
  uint32_t w[24];
};

__host__ __device__ __forceinline__ void fetch_window(const uint8_t *s, WindowWords &ww) {
  const uintptr_t p = (uintptr_t)s;
  const uintptr_t start = (p - kWindow) & ~(uintptr_t)31;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
#ifdef __CUDA_ARCH__
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(ww.w[8 * i]), "=r"(ww.w[8 * i + 1]), "=r"(ww.w[8 * i + 2]),
          "=r"(ww.w[8 * i + 3]), "=r"(ww.w[8 * i + 4]), "=r"(ww.w[8 * i + 5]),
          "=r"(ww.w[8 * i + 6]), "=r"(ww.w[8 * i + 7])
        : "l"(start + 32 * i));
#else
    for (int j = 0; j < 8; ++j) ww.w[8 * i + j] = reinterpret_cast<const uint32_t *>(start)[8 * i + j];
#endif
  }
}

// The residues s[-32 .. 31] of the fetched words, four a word.
__host__ __device__ __forceinline__ void align_window(const uint8_t *s, const WindowWords &ww,
                                                      uint32_t a[16]) {
  const uint32_t p = (uint32_t)(uintptr_t)s;
  const int shift = 8 * (int)(p & 3);
  const uint32_t start = p - kWindow;
  const bool by4 = (start & 16) != 0, by2 = (start & 8) != 0, by1 = (start & 4) != 0;
  uint32_t w[20];
#pragma unroll
  for (int i = 0; i < 20; ++i) w[i] = by4 ? ww.w[i + 4] : ww.w[i];
#pragma unroll
  for (int i = 0; i < 18; ++i) w[i] = by2 ? w[i + 2] : w[i];
#pragma unroll
  for (int i = 0; i < 17; ++i) w[i] = by1 ? w[i + 1] : w[i];
#pragma unroll
  for (int i = 0; i < 16; ++i) a[i] = row_funnel_r(w[i], w[i + 1], shift);
}

// byte J of x | byte J of a << 8 (x below 128: its sign bit fills the rest)
template <int J>
__host__ __device__ __forceinline__ uint32_t window_offset(uint32_t x, uint32_t a) {
#ifdef __CUDA_ARCH__
  return walk_offset<J>(x, a);
#else
  return ((x >> (8 * J)) & 0xffu) | (((a >> (8 * J)) & 0xffu) << 8);
#endif
}

__host__ __device__ __forceinline__ uint32_t window_addmax(uint32_t a, uint32_t b, uint32_t c) {
#ifdef __CUDA_ARCH__
  return __viaddmax_u16x2(a, b, c);  // per half max(a + b, c)
#else
  const uint32_t lo = ((a & 0xffffu) + (b & 0xffffu)) & 0xffffu, hi = ((a >> 16) + (b >> 16)) & 0xffffu;
  const uint32_t cl = c & 0xffffu, ch = c >> 16;
  return (lo > cl ? lo : cl) | ((hi > ch ? hi : ch) << 16);
#endif
}

// Both walks over the window; a byte of q or d of 32 or more is no table
// address.  bests: the sum of the two sides' largest
// (doubled) scores, from after a walk's end too unless kExact, where a score
// falls by 256 a step from there on and so stays below its best.  steps and
// delimiters (per half): the steps from the end on, and of those the ones
// where a delimiter had been met.
struct WindowWalk {
  int bests;
  int best[2], score[2];  // per side, doubled (score: at the window's end)
  int steps[2], delimiters[2];

  // the residue pairs side i's walk examines, if it ends in the window
  __host__ __device__ __forceinline__ int pairs(int i) const {
    return kWindow + 1 - steps[i] - (delimiters[i] == steps[i] ? 1 : 0);
  }
  __host__ __device__ __forceinline__ bool ended(int i) const { return steps[i] > 0; }
  // side i in a word: an ended walk's pairs and (an upper bound of) its
  // best, an open one's best and its drop below it
  __host__ __device__ __forceinline__ uint32_t side(int i) const {
    return ended(i) ? 0x80000000u | (uint32_t)((best[i] + 1) >> 1) << 16 | (uint32_t)pairs(i)
                    : (uint32_t)(best[i] >> 1) << 16 | (uint32_t)((best[i] - score[i]) >> 1);
  }
};

template <bool kExact>
__host__ __device__ __forceinline__ WindowWalk walk_both(uint32_t tbl, const uint32_t q[16],
                                                         const uint32_t d[16], int cutoff) {
  constexpr uint32_t bias = kExact ? kWalkBiasExact : kWalkBias;
  const uint32_t add = 0x10001u * (uint32_t)(kWalkFlag - 2 * cutoff);
  uint32_t score = 0x10001u * bias;
  uint32_t best = score + add;  // best + add
  uint32_t flags = 0, sum = 0;
#define GZB_WINDOW_PAIR(J)                                                       \
  {                                                                              \
    const uint32_t r = row_load_const(tbl + window_offset<3 - (J)>(xr, q[7 - k])); \
    const uint32_t f = row_load_const(tbl + window_offset<(J)>(xf, q[8 + k]) + 128); \
    score = score + r + f;                                                       \
    if (kExact) score -= (flags >> 2) & (0x10001u * (kWalkFlag >> 2));           \
    best = window_addmax(score, add, best);                                      \
    flags = (flags | (best - score)) & (0x10001u * (kWalkFlag | 1));             \
    sum += flags;                                                                \
  }
#pragma unroll
  for (int k = 0; k < kWindow / 4; ++k) {
    const uint32_t xr = (q[7 - k] ^ d[7 - k]) << 2, xf = (q[8 + k] ^ d[8 + k]) << 2;
    GZB_WINDOW_PAIR(0)
    GZB_WINDOW_PAIR(1)
    GZB_WINDOW_PAIR(2)
    GZB_WINDOW_PAIR(3)
  }
#undef GZB_WINDOW_PAIR
  WindowWalk w;
  w.steps[0] = (int)(sum & 0xffffu) / kWalkFlag;
  w.steps[1] = (int)(sum >> 16) / kWalkFlag;
  w.delimiters[0] = (int)(sum & (kWalkFlag - 1));
  w.delimiters[1] = (int)((sum >> 16) & (kWalkFlag - 1));
  const int zero = (int)((add & 0xffffu) + bias);
  w.best[0] = (int)(best & 0xffffu) - zero;
  w.best[1] = (int)(best >> 16) - zero;
  w.score[0] = (int)(score & 0xffffu) - (int)bias;
  w.score[1] = (int)(score >> 16) - (int)bias;
  w.bests = w.best[0] + w.best[1];
  return w;
}

// Whether the seed is settled as no hit; *steps then holds the residue pairs
// its two walks examine.  If not, side[0] and side[1] (reverse and forward)
// say where its walks are.
__host__ __device__ __forceinline__ bool walk_window(uint32_t tbl, const uint32_t q[16],
                                                     const uint32_t d[16], int cutoff,
                                                     int trigger, int *steps, uint32_t side[2]) {
  const WindowWalk w = walk_both<false>(tbl, q, d, cutoff);
  *steps = w.pairs(0) + w.pairs(1);
  side[0] = w.side(0);
  side[1] = w.side(1);
  return w.ended(0) && w.ended(1) && w.bests <= 2 * trigger;
}

#ifdef __CUDACC__
constexpr uint32_t kSideUnknown = 0xffffffffu;  // no window: the whole walk is to do

// The walks of a seed that its window leaves open, from the window's ends:
// true if it is no hit, with the pairs that both walks examine.  False where
// a walk could have stopped at the trigger, which walk_hit settles.
__device__ __forceinline__ bool walk_on(const uint8_t *q, const uint8_t *d, const char *tbl,
                                        int cutoff, int trigger, const uint32_t side[2],
                                        int *steps) {
  int n = 0, best[2];
  for (int i = 0; i < 2; ++i) {
    best[i] = (int)((side[i] >> 16) & 0x7fffu);
    n += side[i] >> 31 ? (int)(side[i] & 0xffffu) : kWindow;
  }
  if (side[0] == kSideUnknown || best[0] + best[1] > trigger) return false;
  if (!(side[0] >> 31))
    best[0] = walk_side<-1>(q - 1 - kWindow, d - 1 - kWindow, tbl, cutoff, trigger - best[1], &n,
                            best[0] - (int)(side[0] & 0xffffu), best[0]);
  if (best[0] + best[1] > trigger) return false;
  if (!(side[1] >> 31))
    best[1] = walk_side<1>(q + kWindow, d + kWindow, tbl, cutoff, trigger - best[0], &n,
                           best[1] - (int)(side[1] & 0xffffu), best[1]);
  *steps = n;
  return best[0] + best[1] <= trigger;
}
#endif

// 1: a hit (scores the walks reach sum to more than the trigger), 0: none
// (both walks end), -1: open.  The bytes behind a delimiter may be anything:
// their low five bits stand in, which no score or flag depends on.
__host__ __device__ __forceinline__ int walk_window_hit(uint32_t tbl, const uint32_t q[16],
                                                        const uint32_t d[16], int cutoff,
                                                        int trigger) {
  uint32_t qc[16], dc[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    qc[i] = q[i] & kCodeBits;
    dc[i] = d[i] & kCodeBits;
  }
  const WindowWalk w = walk_both<true>(tbl, qc, dc, cutoff);
  return w.bests > 2 * trigger ? 1 : w.steps[0] > 0 && w.steps[1] > 0 ? 0 : -1;
}

// Items waiting in shared memory until 32 of them are there, one stack per
// warp: a warp finds seeds, member work and hits with whatever lanes have
// one, and walks or writes them 32 at a time.
#ifdef __CUDACC__
template <typename T>
struct WarpStack {
  static constexpr uint32_t kCapacity = 64;  // 31 waiting and 32 more
  T *item;
  uint32_t n = 0;  // the same on every lane
  // the lanes with `have` add theirs (all lanes call it)
  __device__ __forceinline__ void push(bool have, T v) {
    const unsigned m = __ballot_sync(0xffffffffu, have);
    if (have) item[n + __popc(m & ((1u << (threadIdx.x & 31)) - 1u))] = v;
    n += __popc(m);
    __syncwarp();
  }
  // the newest 32 (fewer: all), one per lane; false on lanes without one
  __device__ __forceinline__ bool pop(T *v) {
    const uint32_t take = n < 32 ? n : 32, lane = threadIdx.x & 31;
    n -= take;
    if (lane < take) *v = item[n + lane];
    __syncwarp();
    return lane < take;
  }
  // pops into a global list: one atomic for the warp
  __device__ __forceinline__ void flush(T *list, unsigned long long *count,
                                        unsigned long long cap) {
    const uint32_t take = n < 32 ? n : 32, lane = threadIdx.x & 31;
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(count, (unsigned long long)take);
    base = __shfl_sync(0xffffffffu, base, 0);
    T v;
    if (pop(&v) && base + lane < cap) list[base + lane] = v;
  }
};
#endif

}  // namespace gzb
