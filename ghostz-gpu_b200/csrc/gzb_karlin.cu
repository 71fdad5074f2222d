// gzb_karlin.cu -- per-query ungapped Karlin-Altschul statistics and the
// integer cutoffs derived from them, on the device (query preparation).
//
// For every query the reference builds (ProteinQuery / TranslatedDnaQuery,
// SetStaticalParameters) it takes the query's letter composition against
// the Robinson background (Statistics::CalculateUngappedKarlinParameters,
// src/statistics.cpp:205-229), solves lambda, H and K
// (ext/karlin/src/karlin.c, BlastKarlinBlkCalc), and turns them into the
// ungapped X-drop and the gapped-extension trigger
// (src/aligner_gpu.cpp:228-238, src/statistics.cpp:28-43).
//
// Few queries take a warp each (karlin_kernel: the score distribution's
// j-fold convolutions for K are spread over the lanes, the serial sums stay
// on lane 0), many four lanes each (karlin_group_kernel).  Both first run
// with buffers for the rounds of the K series that nearly every query needs;
// one that needs more is marked and redone by a warp with buffers for all
// 100.  Every sum keeps the reference's order.  All arithmetic uses
// explicitly rounded operations (no fused multiply-add), so the float
// results agree with the reference's x86-64 build bit for bit; exp, pow and
// log are CUDA's double-precision functions.
#include <cuda_runtime.h>

#include <cstdint>
#include <cmath>

#include "ghostz_b200.h"
#include "gzb_common.h"

namespace gzb {

namespace {

constexpr int kKarlinIterMax = 100;           // BLAST_KARLIN_K_ITER_MAX
// A first pass gives each warp convolution buffers for kFastIter rounds of
// the K series (the series usually ends after 10-15), so more warps fit on
// an SM; a query that needs more rounds is marked and redone by a second
// pass with buffers for all kKarlinIterMax rounds.
constexpr int kFastIter = 24, kFastWarps = 4;
constexpr int kFullWarps = 2;
constexpr int32_t kPending = INT32_MIN;       // cutoff of a query left to the second pass
constexpr int kMaxLetters = 32;
constexpr int kMaxRange = 31;                 // highest - lowest score
constexpr int kMaxRegular = 19;               // ARNDCQEGHILKMFPSTWYV

// Robinson & Robinson background, ARNDCQEGHILKMFPSTWYV order
// (src/statistics.cpp:154-176)
constexpr double kRobinson[20] = {78.05, 51.29, 44.87, 53.64, 19.25, 42.64, 62.95,
                                  73.77, 21.99, 51.42, 90.19, 57.44, 22.43, 38.56,
                                  52.03, 71.20, 58.41, 13.30, 32.16, 64.41};

struct KarlinArgs {
  double background[kMaxLetters];        // normalised letter probabilities
  // letter pairs grouped by score (score low + s owns pairs
  // [pair_begin[s], pair_begin[s + 1])), in (c1, c2) order within a group
  uint8_t pair_c1[kMaxLetters * kMaxLetters];
  uint8_t pair_c2[kMaxLetters * kMaxLetters];
  uint16_t pair_begin[kMaxRange + 2];
  int number_letters;                    // codes 0 .. number_letters-1
  int low, high;                         // score range of the matrix
  float ungapped_bits, trigger_bits, ln2;
};

__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double ddiv(double a, double b) { return __ddiv_rn(a, b); }

__device__ bool range_bad(int lo, int hi) {
  return lo >= 0 || hi <= 0 || lo < -10000 || hi > 1000 || hi - lo > 11000;
}

__device__ long gcd_long(long a, long b) {
  long c;
  b = b < 0 ? -b : b;
  if (b > a) c = a, a = b, b = c;
  while (b != 0) {
    c = a % b;
    a = b;
    b = c;
  }
  return a;
}

// (sp[i * kStride]: the probability of score i)

// sum_i sp[i] exp(x i) the way the reference forms it: a running power
// from pow(exp(x), lo - 1), or exp(x i) per term once that underflows
template <int kStride>
__device__ double power_sum(const double *sp, int lo, int hi, double x) {
  const double x0 = exp(x);
  double x1 = pow(x0, (double)(lo - 1));
  double sum = 0.0;
  if (x1 > 0.0) {
    for (int i = lo; i <= hi; ++i) {
      x1 = dmul(x1, x0);
      sum = dadd(sum, dmul(sp[i * kStride], x1));
    }
  } else {
    for (int i = lo; i <= hi; ++i) sum = dadd(sum, dmul(sp[i * kStride], exp(dmul(x, (double)i))));
  }
  return sum;
}

// lambda by bisection (BlastKarlinLambdaBis)
template <int kStride>
__device__ double lambda_bisect(const double *sp, int lo, int hi) {
  if (range_bad(lo, hi)) return -1.0;
  double lambda = 0.0, up = 0.5;
  for (int guard = 0; guard < 2048; ++guard) {
    up = dmul(up, 2.0);
    if (power_sum<kStride>(sp, lo, hi, up) >= 1.0) break;
    lambda = up;
  }
  for (int j = 0; j < 17; ++j) {
    const double mid = ddiv(dadd(lambda, up), 2.0);
    if (power_sum<kStride>(sp, lo, hi, mid) > 1.0)
      up = mid;
    else
      lambda = mid;
  }
  return ddiv(dadd(lambda, up), 2.0);
}

// lambda by Newton-Raphson from 0.5 (BlastKarlinLambdaNR)
template <int kStride>
__device__ double lambda_newton(const double *sp, int lo, int hi) {
  if (range_bad(lo, hi)) return -1.0;
  double lambda = 0.5;
  for (int j = 0; j < 20; ++j) {
    double sum = -1.0, slope = 0.0;
    if (lambda < 0.01) break;
    const double x0 = exp(lambda);
    double x1 = pow(x0, (double)(lo - 1));
    if (x1 == 0.0) break;
    for (int i = lo; i <= hi; ++i) {
      x1 = dmul(x1, x0);
      const double t = dmul(sp[i * kStride], x1);
      sum = dadd(sum, t);
      slope = dadd(slope, dmul(t, (double)i));
    }
    const double step = ddiv(sum, slope);
    lambda = dsub(lambda, step);
    if (fabs(ddiv(step, lambda)) < 1.0e-5) {
      if (lambda > 1.0e-5) return lambda;
      break;
    }
  }
  return lambda_bisect<kStride>(sp, lo, hi);
}

// relative entropy (BlastKarlinLtoH)
template <int kStride>
__device__ double entropy(const double *sp, int lo, int hi, double lambda) {
  if (lambda < 0.0 || range_bad(lo, hi)) return -1.0;
  const double etolam = exp(lambda);
  double etolami = pow(etolam, (double)(lo - 1)), av = 0.0;
  if (etolami > 0.0) {
    for (int s = lo; s <= hi; ++s) {
      etolami = dmul(etolami, etolam);
      av = dadd(av, dmul(dmul(sp[s * kStride], (double)s), etolami));
    }
  } else {
    for (int s = lo; s <= hi; ++s)
      av = dadd(av, dmul(dmul(sp[s * kStride], (double)s), exp(dmul(lambda, (double)s))));
  }
  return dmul(lambda, av);
}

// K from the series' state after its rounds (sum: the last term; p[i *
// stride]: probability of score low + i); -1 where it has no value
__device__ double karlin_k(double sum, double oldsum, double oldsum2, double Sum, int j,
                           double av, double etolam, double lambda, int low, int range,
                           const double *p, int stride) {
  double sumlimit = 0.01;
  const double ratio = ddiv(oldsum, oldsum2);
  if (ratio >= dsub(1.0, dmul(sumlimit, 0.001))) return -1.0;
  sumlimit = dmul(sumlimit, 0.01);
  while (sum > sumlimit) {
    oldsum = dmul(oldsum, ratio);
    ++j;
    sum = ddiv(oldsum, (double)j);
    Sum = dadd(Sum, sum);
  }
  long delta = -low;
  for (int i = 1; i <= range && delta > 1; ++i)
    if (p[i * stride] != 0.0) delta = gcd_long(delta, i);
  const double e2 = exp(dmul(-2.0, Sum));
  if (dmul((double)delta, etolam) > 0.05) {
    const double etolami = pow(etolam, (double)(-delta));
    return ddiv(dmul((double)delta, e2), dmul(av, dsub(1.0, etolami)));
  }
  return ddiv(dmul((double)(-delta), e2),
              dmul(av, dsub(exp(dmul((double)(-delta), lambda)), 1.0)));
}

// NormalizedCutoff2NominalCutoff and Normalized2Nominal in float; ln K is
// the float nearest the exact logarithm
__device__ void store_cutoffs(const KarlinArgs &a, uint32_t r, float l, float h, double K,
                              int32_t *cutoffs, int32_t *triggers, float *karlin) {
  const float k = (float)K;
  const float c = __fdiv_rn(__fmul_rn(a.ungapped_bits, a.ln2), l);
  const float t =
      __fdiv_rn(__fadd_rn(__fmul_rn(a.trigger_bits, a.ln2), (float)log((double)k)), l);
  cutoffs[r] = (int32_t)floorf(c);
  triggers[r] = (int32_t)floorf(t);
  if (karlin) {
    karlin[3 * (size_t)r] = l;
    karlin[3 * (size_t)r + 1] = k;
    karlin[3 * (size_t)r + 2] = h;
  }
}

// kGroup lanes a query, 32 / kGroup queries a block (of one warp).  A query's
// convolutions are some 25,000 multiplications and additions, and each of
// its serial sums would keep only one lane of a warp busy, so with many
// queries those go side by side.  One buffer a query, in shared memory, its
// entries a row apart: a round replaces it from its end, kOut entries a lane
// at a time, each of which reads only entries up to its own.  The entries
// slide through registers: a step is a load of an entry and one of a
// probability for kOut products, and rows of zeros below and above the
// entries take the place of bounds (a zero's term leaves a sum as it is).
// What bounds it is the latency of double precision chains: the shared memory
// holds the buffers of some 88 queries an SM, which four lanes a query make
// eleven warps.  150,000 reads' frames: 4.61 ms with a warp a query, 2.43 with
// a lane, 1.58 with two, 1.41 with four.  `rounds`: those the buffer holds
// (karlin_rounds).
constexpr int kOut = 8;
constexpr int kGroup = 4;
constexpr int kRow = 32 / kGroup;  // queries a block: entries of a row

__host__ __device__ constexpr int karlin_steps(int range) {  // scores, a multiple of kOut
  return (range + kOut) / kOut * kOut;
}

// The compositions are counted by all warps of the block, 16 bytes a lane,
// over its queries' residues back to back; one of them goes on alone, on
// another of the SM's four schedulers in each of the blocks that share it (the
// first warp of every block: 3,072 queries 160 us, this way 117).  With the
// block's only warp taking the queries one after the other, a byte a lane,
// long ones waited: 3,072 queries of 308, 2,000 and 10,000 residues, and of 308
// with one of 35,000 among them, 117, 147, 279 and 191 us; this way 118, 121,
// 142 and 119 (a warp a query 156, 155, 160 and 154).
constexpr int kCountMost = 8;  // warps

// Warps a block, by the blocks an SM gets: as many as fit its registers, and
// one where the blocks are warps enough (6,144 queries of 308 and of 10,000
// residues with four warps 138 and 176 us, with one 118 and 225, a warp a query
// 218 and 228).
inline int karlin_warps(uint32_t blocks_per_sm) {
  return blocks_per_sm <= 2 ? kCountMost : blocks_per_sm <= 5 ? 4 : 1;
}

__global__ void __launch_bounds__(32 * kCountMost, 3)
    karlin_group_kernel(KarlinArgs a, const uint8_t *__restrict__ codes,
                        const uint64_t *__restrict__ offsets,
                        const uint32_t *__restrict__ lengths, uint32_t n, int rounds, int sms,
                        int32_t *__restrict__ cutoffs, int32_t *__restrict__ triggers,
                        float *__restrict__ karlin) {
  extern __shared__ double columns[];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x / 32;
  const int column = lane % kRow, part = lane / kRow;
  const int low = a.low, high = a.high, range = high - low;
  const int steps = karlin_steps(range);
  double *p = columns + column;          // [steps]: zero past the range
  double *buf = p + kRow * 2 * steps;    // [-steps ..]: zero rows below the entries
  const int rows = rounds * range + 1 + kOut * kGroup;
  const uint32_t r0 = blockIdx.x * kRow, r = r0 + column;
  const int nl = a.number_letters;
  // compositions, then frequencies with a pseudo-count for absent letters,
  // normalised
  int *count = reinterpret_cast<int *>(columns + kRow * (2 * steps + kMaxLetters));
  for (int i = threadIdx.x; i < 33 * kRow; i += blockDim.x) count[i] = 0;
  const uint64_t begin = r < n ? (uint64_t)(codes + offsets[r]) : 0;
  const uint64_t end = r < n ? begin + lengths[r] : 0;
  const uint32_t pieces = end > begin ? (uint32_t)((end - (begin & ~15ull) + 15) / 16) : 0;
  uint32_t last = pieces;  // the pieces of the queries up to the column's
  for (int d = 1; d < kRow; d <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, last, d, kRow);
    if (column >= d) last += t;
  }
  const uint32_t all = __shfl_sync(0xffffffffu, last, kRow - 1);
  __shared__ uint32_t one;
  if (threadIdx.x == 0) one = 0;
  __syncthreads();
  uint32_t slot;  // (its low two bits: the scheduler)
  asm volatile("mov.u32 %0, %%warpid;" : "=r"(slot));
  if (lane == 0 && (slot & 3) == blockIdx.x / sms % 4) one = warp;
  for (uint32_t i0 = 32 * warp; i0 < all; i0 += blockDim.x) {
    const uint32_t i = i0 + lane;
    int k = 0;  // the query piece i is of
#pragma unroll
    for (int j = 0; j < kRow - 1; ++j) k += i >= __shfl_sync(0xffffffffu, last, j);
    const uint32_t first = __shfl_sync(0xffffffffu, last - pieces, k);
    const uint64_t from = __shfl_sync(0xffffffffu, begin, k), to = __shfl_sync(0xffffffffu, end, k);
    if (i < all) {
      // (an aligned piece with a residue of the query in it)
      const uint64_t at = (from & ~15ull) + 16ull * (i - first);
      const uint4 v = __ldg(reinterpret_cast<const uint4 *>(at));
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const uint32_t c = (w[j / 4] >> (8 * (j & 3))) & 0xffu;
        if (c <= kMaxRegular && at + j >= from && at + j < to) atomicAdd(&count[33 * k + c], 1);
      }
    }
  }
  __syncthreads();
  if (warp != one) return;
  double total = 0.0;
  for (int c = 0; c < nl; ++c) {
    const int k = count[33 * column + c];
    const double f = (double)k + (k < 1 ? 1.0 : 0.0);
    buf[kRow * c] = f;
    total = dadd(total, f);
  }
  __syncwarp();
  for (int c = part; c < nl; c += kGroup) buf[kRow * c] = ddiv(buf[kRow * c], total);
  __syncwarp();
  double s = 0.0;
  for (int i = 0; i <= range; ++i) {
    double acc = 0.0;
    for (int k = a.pair_begin[i]; k < a.pair_begin[i + 1]; ++k)
      acc = dadd(acc, dmul(buf[kRow * a.pair_c1[k]], a.background[a.pair_c2[k]]));
    p[kRow * i] = acc;
    if (acc > 0.0) s = dadd(s, acc);
  }
  __syncwarp();
  for (int i = part; i < steps; i += kGroup)
    p[kRow * i] = i <= range ? (p[kRow * i] > 0.0 ? ddiv(p[kRow * i], s) : p[kRow * i]) : 0.0;
  for (int i = part - steps; i < rows; i += kGroup) buf[kRow * i] = i == 0 ? 1.0 : 0.0;
  __syncwarp();
  const double *sp = p - kRow * low;
  const float l = (float)lambda_newton<kRow>(sp, low, high);
  const float h = (float)entropy<kRow>(sp, low, high, (double)l);
  const double lambda = (double)l, H = (double)h;
  const double av = ddiv(H, lambda), etolam = exp(lambda);
  const bool valid = r < n && lambda > 0.0 && H > 0.0, closed = low == -1 || high == 1;
  double sum = 1.0, oldsum = 1.0, oldsum2 = 1.0, Sum = 0.0;
  int j = 0;
  // (every lane takes part in the rounds, for the queries still in need)
  bool open = valid && !closed;
  for (int round = 0; round < rounds && __any_sync(0xffffffffu, open); ++round) {
    const int top = (round + 1) * range;  // the last entry after this round
    for (int k0 = top / (kOut * kGroup) * (kOut * kGroup); k0 >= 0; k0 -= kOut * kGroup) {
      double *at = buf + kRow * (k0 + kOut * part);
      double acc[kOut], w[kOut], next[kOut];
#pragma unroll
      for (int e = 0; e < kOut; ++e) {
        acc[e] = 0.0;
        w[e] = at[kRow * e];
      }
      for (int u0 = 0; u0 < steps; u0 += kOut) {
#pragma unroll
        for (int e = 0; e < kOut; ++e) next[e] = at[-kRow * (u0 + 1 + e)];
#pragma unroll
        for (int t = 0; t < kOut; ++t) {
          const double pu = p[kRow * (u0 + t)];
#pragma unroll
          for (int e = 0; e < kOut; ++e)
            acc[e] = dadd(acc[e], dmul(e >= t ? w[e - t] : next[t - e - 1], pu));
        }
#pragma unroll
        for (int e = 0; e < kOut; ++e) w[e] = next[kOut - 1 - e];
      }
      __syncwarp();
#pragma unroll
      for (int e = 0; e < kOut; ++e) at[kRow * e] = acc[e];
      __syncwarp();
    }
    if (open) {
      const int lo = (round + 1) * low;
      double etolami = pow(etolam, (double)(lo - 1));
      s = 0.0;
      int i = 0;
#pragma unroll 4
      for (; i < -lo; ++i) {
        etolami = dmul(etolami, etolam);
        s = dadd(s, dmul(buf[kRow * i], etolami));
      }
#pragma unroll 4
      for (; i <= top; ++i) s = dadd(s, buf[kRow * i]);
      oldsum2 = oldsum;
      oldsum = s;
      ++j;
      sum = ddiv(s, (double)j);
      Sum = dadd(Sum, sum);
      open = sum > 0.01;
    }
    __syncwarp();
  }
  if (r >= n || part != 0) return;
  if (open) {
    cutoffs[r] = kPending;
    return;
  }
  double K = -1.0;
  if (valid)
    K = closed ? dmul(av, dsub(1.0, ddiv(1.0, etolam)))
               : karlin_k(sum, oldsum, oldsum2, Sum, j, av, etolam, lambda, low, range, p, kRow);
  store_cutoffs(a, r, l, h, K, cutoffs, triggers, karlin);
}

// Rounds karlin_group_kernel's buffers hold, so that eleven blocks share an
// SM's 228 KB (and 24 at most: the series ends after 12 to 15 rounds for
// nearly every composition); their bytes.
int karlin_rounds(int range, size_t *bytes) {
  const size_t most = 20172, row = kRow * sizeof(double);
  const int steps = karlin_steps(range), extra = 2 * steps + kOut * kGroup + 1;
  int rounds = ((int)(most / row) - extra) / range;
  if (rounds > kFastIter) rounds = kFastIter;
  if (rounds < 1) rounds = 1;
  int rows = extra + rounds * range;
  // (the compositions' counts lie above the frequencies)
  const int start = 2 * steps + kMaxLetters + (int)((33 * kRow * sizeof(int) + row - 1) / row);
  if (rows < start) rows = start;
  *bytes = rows * row;
  return rounds;
}

// From this many queries on, karlin_group_kernel is the faster whatever their
// lengths: 2,048 queries of 50, 308, 2,000 and 10,000 residues 102, 102, 104
// and 113 us, a warp a query 124, 124, 125 and 129 (1,536 of 308: 107).
constexpr uint32_t kGroupQueries = 2048;
// And where its buffers hold the rounds that most queries need (a range of up
// to 15 scores; a wider one takes a warp a query).
constexpr int kGroupRounds = 15;

// kIter: rounds of the K series the buffers hold.  kRetry: the second pass
// (only queries whose cutoff holds kPending).  The first pass runs eight
// blocks per SM (its grid), so it is bounded to the 64 registers that let
// all eight stay resident at once.
template <int kWarps, int kIter, bool kRetry>
__global__ void __launch_bounds__(kWarps * 32, kRetry ? 1 : 8)
    karlin_kernel(KarlinArgs a, const uint8_t *__restrict__ codes,
                  const uint64_t *__restrict__ offsets, const uint32_t *__restrict__ lengths,
                  uint32_t n, int32_t *__restrict__ cutoffs, int32_t *__restrict__ triggers,
                  float *__restrict__ karlin) {
  extern __shared__ double dist[];  // per warp: two convolution buffers
  __shared__ int count[kWarps][kMaxLetters];
  __shared__ double freq[kWarps][kMaxLetters];
  __shared__ double prob[kWarps][kMaxRange + 1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int low = a.low, high = a.high, range = high - low;
  const int cap = kIter * range + 1;
  double *buf0 = dist + (size_t)w * 2 * cap, *buf1 = buf0 + cap;
  const int nl = a.number_letters;
  const uint32_t warps = gridDim.x * kWarps;
  uint32_t first = 0, marked = 0;  // marked ones of the 32 queries from `first` on (kRetry)
  for (uint64_t at = (uint64_t)(blockIdx.x * kWarps + w) * (kRetry ? 32 : 1); at < n || marked;) {
    uint32_t r = (uint32_t)at;
    if (kRetry) {
      if (!marked) {
        first = (uint32_t)at;
        marked = __ballot_sync(0xffffffffu, at + lane < n && cutoffs[at + lane] == kPending);
        at += 32ull * warps;
        if (!marked) continue;
      }
      r = first + __ffs(marked) - 1;
      marked &= marked - 1;
    } else {
      at += warps;
    }
    // composition of regular letters over the whole query
    count[w][lane] = 0;
    __syncwarp();
    const uint8_t *q = codes + offsets[r];
    const uint32_t len = lengths[r];
    for (uint32_t i = lane; i < len; i += 32) {
      const uint8_t c = q[i];
      if (c <= kMaxRegular) atomicAdd(&count[w][c], 1);
    }
    __syncwarp();
    // frequencies with a pseudo-count for absent letters, normalised
    if (lane < nl) freq[w][lane] = (double)count[w][lane] + (count[w][lane] < 1 ? 1.0 : 0.0);
    __syncwarp();
    double total = 0.0;
    if (lane == 0)
      for (int c = 0; c < nl; ++c) total = dadd(total, freq[w][c]);
    total = __shfl_sync(0xffffffffu, total, 0);
    if (lane < nl) freq[w][lane] = ddiv(freq[w][lane], total);
    __syncwarp();
    // score probabilities: lane s accumulates score low + s over its letter
    // pairs in the reference's (c1, c2) order
    if (lane <= range) {
      double acc = 0.0;
      for (int i = a.pair_begin[lane]; i < a.pair_begin[lane + 1]; ++i)
        acc = dadd(acc, dmul(freq[w][a.pair_c1[i]], a.background[a.pair_c2[i]]));
      prob[w][lane] = acc;
    }
    __syncwarp();
    if (lane == 0) {
      double s = 0.0;
      for (int i = 0; i <= range; ++i)
        if (prob[w][i] > 0.0) s = dadd(s, prob[w][i]);
      for (int i = 0; i <= range; ++i)
        if (prob[w][i] > 0.0) prob[w][i] = ddiv(prob[w][i], s);
    }
    __syncwarp();
    const double *sp = prob[w] - low;  // sp[score]
    const double *p = prob[w];         // p[u] = probability of score low + u
    // lambda and H on lane 0, rounded to float as BlastKarlinBlkCalc keeps them
    float l = 0.f, h = 0.f;
    if (lane == 0) {
      l = (float)lambda_newton<1>(sp, low, high);
      h = (float)entropy<1>(sp, low, high, (double)l);
    }
    l = __shfl_sync(0xffffffffu, l, 0);
    h = __shfl_sync(0xffffffffu, h, 0);
    // K (BlastKarlinLHtoK)
    const double lambda = (double)l, H = (double)h;
    double K = -1.0;
    bool pending = false;  // the series needs more rounds than the buffers hold
    if (lambda > 0.0 && H > 0.0) {
      const double av = ddiv(H, lambda);
      const double etolam = exp(lambda);
      if (low == -1 || high == 1) {
        K = dmul(av, dsub(1.0, ddiv(1.0, etolam)));
      } else {
        double sumlimit = 0.01;
        double sum = 1.0, oldsum = 1.0, oldsum2 = 1.0, Sum = 0.0;
        int lo = 0, hi = 0, j = 0;
        double *cur = buf0, *nxt = buf1;
        if (lane == 0) cur[0] = 1.0;
        __syncwarp();
        while (j < kIter && sum > sumlimit) {
          lo += low;
          hi += high;
          const int top = hi - lo;
          for (int k = lane; k <= top; k += 32) {
            const int first = range - (top - k) > 0 ? range - (top - k) : 0;
            const int last = k < range ? k : range;
            double s = 0.0;
            for (int u = first; u <= last; ++u) s = dadd(s, dmul(cur[k - u], p[u]));
            nxt[k] = s;
          }
          __syncwarp();
          double s = 0.0;
          if (lane == 0) {
            double etolami = pow(etolam, (double)(lo - 1));
            int i = lo, idx = 0;
            for (; i != 0; ++i, ++idx) {
              etolami = dmul(etolami, etolam);
              s = dadd(s, dmul(nxt[idx], etolami));
            }
            for (; i <= hi; ++i, ++idx) s = dadd(s, nxt[idx]);
          }
          s = __shfl_sync(0xffffffffu, s, 0);
          __syncwarp();
          oldsum2 = oldsum;
          oldsum = s;
          double *t = cur;
          cur = nxt;
          nxt = t;
          ++j;
          sum = ddiv(s, (double)j);
          Sum = dadd(Sum, sum);
        }
        if (kIter < kKarlinIterMax && j == kIter && sum > sumlimit)
          pending = true;
        else
          K = karlin_k(sum, oldsum, oldsum2, Sum, j, av, etolam, lambda, low, range, p, 1);
      }
    }
    if (lane == 0 && pending) cutoffs[r] = kPending;
    if (lane == 0 && !pending) store_cutoffs(a, r, l, h, K, cutoffs, triggers, karlin);
    __syncwarp();
  }
}

}  // namespace

}  // namespace gzb

extern "C" int gzb_query_karlin_cutoffs(const uint8_t *d_codes, const uint64_t *d_offsets,
                                        const uint32_t *d_lengths, uint32_t number_queries,
                                        const int32_t *score_matrix, uint32_t number_letters,
                                        float ungapped_bits, float trigger_bits,
                                        int32_t *d_cutoffs, int32_t *d_triggers,
                                        float *d_karlin, void *stream) {
  using namespace gzb;
  GZB_CHECK(score_matrix, GZB_ERR_INVALID, "gzb_query_karlin_cutoffs: null score matrix");
  GZB_CHECK(number_letters > kMaxRegular && number_letters <= kMaxLetters, GZB_ERR_INVALID,
            "gzb_query_karlin_cutoffs: %u letters (protein alphabets of 20..32 codes)",
            number_letters);
  KarlinArgs a;
  int lo = score_matrix[0], hi = score_matrix[0];
  for (uint32_t i = 0; i < number_letters * number_letters; ++i) {
    lo = score_matrix[i] < lo ? score_matrix[i] : lo;
    hi = score_matrix[i] > hi ? score_matrix[i] : hi;
  }
  GZB_CHECK(lo < 0 && hi > 0, GZB_ERR_INVALID,
            "gzb_query_karlin_cutoffs: scores must span negative and positive values");
  GZB_CHECK(hi - lo <= kMaxRange, GZB_ERR_OVERFLOW,
            "gzb_query_karlin_cutoffs: score range %d exceeds %d", hi - lo, kMaxRange);
  int at = 0;
  for (int s = 0; s <= hi - lo; ++s) {
    a.pair_begin[s] = (uint16_t)at;
    for (uint32_t c1 = 0; c1 < number_letters; ++c1)
      for (uint32_t c2 = 0; c2 < number_letters; ++c2)
        if (score_matrix[c1 * number_letters + c2] == lo + s) {
          a.pair_c1[at] = (uint8_t)c1;
          a.pair_c2[at] = (uint8_t)c2;
          ++at;
        }
  }
  a.pair_begin[hi - lo + 1] = (uint16_t)at;
  // background, normalised in the reference's order (Statistics::Statistics)
  double sum = 0.0;
  for (int c = 0; c < kMaxLetters; ++c) a.background[c] = c < 20 ? kRobinson[c] : 0.0;
  for (uint32_t c = 0; c < number_letters; ++c) sum += a.background[c];
  for (uint32_t c = 0; c < number_letters; ++c) a.background[c] /= sum;
  a.number_letters = (int)number_letters;
  a.low = lo;
  a.high = hi;
  a.ungapped_bits = ungapped_bits;
  a.trigger_bits = trigger_bits;
  a.ln2 = (float)std::log(2.0);
  if (number_queries == 0) return GZB_OK;
  GZB_CHECK(d_codes && d_offsets && d_lengths && d_cutoffs && d_triggers, GZB_ERR_INVALID,
            "gzb_query_karlin_cutoffs: null buffer");
  int device = 0, sms = 148;
  GZB_CUDA(cudaGetDevice(&device));
  GZB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  const int range = hi - lo;
  // pass 1: buffers for kFastIter rounds; pass 2: the queries it left
  const size_t smem_fast = (size_t)kFastWarps * 2 * (kFastIter * range + 1) * sizeof(double);
  const size_t smem_full = (size_t)kFullWarps * 2 * (kKarlinIterMax * range + 1) * sizeof(double);
  auto fast = karlin_kernel<kFastWarps, kFastIter, false>;
  auto full = karlin_kernel<kFullWarps, kKarlinIterMax, true>;
  GZB_CUDA(cudaFuncSetAttribute(fast, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_fast));
  GZB_CUDA(cudaFuncSetAttribute(full, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_full));
  size_t smem_group = 0;
  const int rounds = karlin_rounds(range, &smem_group);
  if (number_queries >= kGroupQueries && rounds >= kGroupRounds) {
    GZB_CUDA(cudaFuncSetAttribute(karlin_group_kernel,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_group));
    const uint32_t blocks = (number_queries + kRow - 1) / kRow;
    karlin_group_kernel<<<blocks, 32 * karlin_warps((blocks + sms - 1) / sms), smem_group,
                          (cudaStream_t)stream>>>(
        a, d_codes, d_offsets, d_lengths, number_queries, rounds, sms, d_cutoffs,
        d_triggers, d_karlin);
  } else {
    const uint64_t want_fast = (number_queries + kFastWarps - 1) / kFastWarps;
    const uint64_t most_fast = (uint64_t)sms * 8;
    fast<<<(unsigned)(want_fast < most_fast ? want_fast : most_fast), kFastWarps * 32, smem_fast,
           (cudaStream_t)stream>>>(a, d_codes, d_offsets, d_lengths, number_queries, d_cutoffs,
                                   d_triggers, d_karlin);
  }
  GZB_CUDA(cudaGetLastError());
  const uint64_t want_full = (number_queries + 32 * kFullWarps - 1) / (32 * kFullWarps);
  const uint64_t most_full = (uint64_t)sms * 4;
  full<<<(unsigned)(want_full < most_full ? want_full : most_full), kFullWarps * 32, smem_full,
         (cudaStream_t)stream>>>(a, d_codes, d_offsets, d_lengths, number_queries, d_cutoffs,
                                 d_triggers, d_karlin);
  GZB_CUDA(cudaGetLastError());
  return GZB_OK;
}
