// gzb_row.cuh -- one database row of the gapped X-drop extension, four
// columns at a time (the thread-per-extension kernels' inner step).
//
// The recurrence of GappedExtender::ExtendOneSideScoreOnly
// (src/gapped_extender.cpp:306-471), exact for the parameters row_dp_exact
// admits; other parameters run lane_init / lane_row.  What differs from
// those is how a row is laid out and evaluated:
//
//  * Row r's scores carry an extra gap_ext * (r + 1), so that a vertical gap
//    passes from row to row unchanged; the diagonal's share is in the score
//    table, the threshold takes gap_ext per row.
//  * A band cell is one word, best score in the low half, vertical gap in
//    the high half, and scores are computed as value << 16.  The word itself
//    then serves as the vertical gap: its low half is a fraction below one
//    score unit, which no comparison against a whole score can see
//    (floor(x) >= t exactly when x >= t), and the diagonal is word << 16.  A
//    cell needs no unpacking, one three-way maximum and three add-maximum
//    instructions.  All scores carry kRowBias, which keeps the low halves
//    positive.
//  * The threshold t = max - X-drop is kept as (t << 16) - tag: a cell that
//    raises the maximum leaves its place in the row in the tag (1, 2, ...;
//    0: the maximum is an earlier row's).  A tag is smaller than the gap
//    between a score's largest fraction and the next whole score, so
//    comparisons come out as with t << 16, and a later cell with the same
//    score has a larger tag and changes nothing.
//  * The horizontal gap and a pruned cell's vertical gap are not reset: a
//    pruned cell's score s is below the threshold t = max - X-drop, so the
//    gaps it passes on (s - gap, or a gap that was not above s) are below t
//    as well, and t only rises.  They can neither keep a cell nor grow the
//    band, as long as kInitScore is below every threshold (X-drop < 1024).
//    A pruned cell's word is reset, its best score is the next row's
//    diagonal.
//  * A row is evaluated in whole groups of four columns, from the group of
//    the band's left boundary column to the group of its right end or
//    further while the horizontal gap stays above the threshold (which is
//    how the reference grows the band).  The columns a group adds on either
//    side hold kEmptyCell and stay pruned: left of the boundary every cell
//    was pruned when the boundary passed it, and right of the band every
//    cell was pruned or not reached yet.  Two cases need a word rewritten at
//    the row's end: the boundary column 0 when the band leaves it while its
//    vertical gap is still alive, and the last kept column when the
//    reference adds no sentinel behind it.
//  * The band's new edges are the first and last kept column, from one
//    pruned flag per column.
//
// The query residues of a group are one word (a byte per column, four times
// the residue code); groups are set up once, a few ahead of the band.
//
// What bounds it (gapped_rows_kernel on 300,000 extensions of the 2,000-query
// search, ncu): instruction issue, 75 % of the slots, ALU instructions half
// of them; 108 warp instructions per group of a row, of which some 30 are the
// row's own work.  A row costs the widest of its 32 bands (8.7 groups, the
// mean band has 6).  Against one column at a time with a 32-bit cell pair
// unpacked and packed: 10,000 queries x 1,500,000 proteins, gapped stage
// 62.1 -> 45.7 ms (20 G cells); a lone long extension's row takes half the
// time, so 1,000 x 20,000 went from 2.6 to 1.7 ms.  Tried on the same case:
// one cell at a time in this arithmetic 67 ms (the lanes part at every
// branch); cells addressed through pointers 51.2 ms (64-bit address
// arithmetic); two groups per loop turn 45.7 against 47.1 ms; the pruned
// cells selected by a sign mask 48.7 ms, additions moved to the multiply-add
// pipe 47.1 ms.
#pragma once

#include <cstdint>

#include "gzb_kernels.cuh"

namespace gzb {

// ---- instructions the step is made of (host forms for tests on the CPU)
__host__ __device__ __forceinline__ int row_max3(int a, int b, int c) {
#ifdef __CUDA_ARCH__
  return __vimax3_s32(a, b, c);
#else
  const int m = a > b ? a : b;
  return m > c ? m : c;
#endif
}
__host__ __device__ __forceinline__ int row_addmax(int a, int b, int c) {  // max(a + b, c)
#ifdef __CUDA_ARCH__
  return __viaddmax_s32(a, b, c);
#else
  const int s = (int)((unsigned)a + (unsigned)b);
  return s > c ? s : c;
#endif
}
// (high half of s) | (high half of g) << 16
__host__ __device__ __forceinline__ uint32_t row_pack(int s, int g) {
#ifdef __CUDA_ARCH__
  return __byte_perm((uint32_t)s, (uint32_t)g, 0x7632);
#else
  return ((uint32_t)s >> 16) | ((uint32_t)g & 0xffff0000u);
#endif
}
__host__ __device__ __forceinline__ uint32_t row_funnel_r(uint32_t lo, uint32_t hi, int n) {
#ifdef __CUDA_ARCH__
  return __funnelshift_r(lo, hi, n);
#else
  return n ? (lo >> n) | (hi << (32 - n)) : lo;
#endif
}
__host__ __device__ __forceinline__ uint32_t row_reverse_bytes(uint32_t w) {
#ifdef __CUDA_ARCH__
  return __byte_perm(w, 0, 0x0123);
#else
  return __builtin_bswap32(w);
#endif
}
// The band and the score table are addressed by their 32-bit shared-memory
// addresses (on the host, offsets into row_host_memory): with pointers the
// compiler computes every address of the cell loop in 64 bits.
struct RowGroup {
  uint32_t w[4];
};
inline char *row_host_memory = nullptr;  // host only
__host__ __device__ __forceinline__ uint32_t row_load(uint32_t a) {
#ifdef __CUDA_ARCH__
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
#else
  return *reinterpret_cast<uint32_t *>(row_host_memory + a);
#endif
}
__host__ __device__ __forceinline__ void row_store(uint32_t a, uint32_t v) {
#ifdef __CUDA_ARCH__
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
#else
  *reinterpret_cast<uint32_t *>(row_host_memory + a) = v;
#endif
}
__host__ __device__ __forceinline__ RowGroup row_load4(uint32_t a) {
#ifdef __CUDA_ARCH__
  RowGroup g;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(g.w[0]), "=r"(g.w[1]), "=r"(g.w[2]), "=r"(g.w[3])
               : "r"(a)
               : "memory");
  return g;
#else
  return *reinterpret_cast<RowGroup *>(row_host_memory + a);
#endif
}
__host__ __device__ __forceinline__ void row_store4(uint32_t a, const RowGroup &g) {
#ifdef __CUDA_ARCH__
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(g.w[0]), "r"(g.w[1]),
               "r"(g.w[2]), "r"(g.w[3])
               : "memory");
#else
  *reinterpret_cast<RowGroup *>(row_host_memory + a) = g;
#endif
}
// a score-table entry (the table does not change)
__host__ __device__ __forceinline__ uint32_t row_load_const(uint32_t a) {
#ifdef __CUDA_ARCH__
  uint32_t v;
  asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
#else
  return *reinterpret_cast<uint32_t *>(row_host_memory + a);
#endif
}
// byte j of w, plus a
template <int J>
__host__ __device__ __forceinline__ uint32_t row_byte_plus(uint32_t w, uint32_t a) {
#ifdef __CUDA_ARCH__
  return __dp4a(w, 1u << (8 * J), a);
#else
  return ((w >> (8 * J)) & 0xffu) + a;
#endif
}
// the warp's lanes meet
__host__ __device__ __forceinline__ void row_meet() {
#ifdef __CUDA_ARCH__
  __syncwarp();
#endif
}
// whether any lane of the warp has `p` (all call it)
__host__ __device__ __forceinline__ bool row_any(bool p) {
#ifdef __CUDA_ARCH__
  return __any_sync(0xffffffffu, p) != 0;
#else
  return p;
#endif
}
// lowest / highest set bit of a non-zero word
__host__ __device__ __forceinline__ int row_low_bit(uint32_t v) {
#ifdef __CUDA_ARCH__
  return __ffs((int)v) - 1;
#else
  return __builtin_ctz(v);
#endif
}
__host__ __device__ __forceinline__ int row_high_bit(uint32_t v) {
#ifdef __CUDA_ARCH__
  return 31 - __clz((int)v);
#else
  return 31 - __builtin_clz(v);
#endif
}

// a band cell: best score and vertical gap (biased so that the fraction a
// low half makes, 1024 .. 30719, and a tag of up to 34816 stay below one
// score unit)
constexpr int kRowBias = 2048;
__host__ __device__ constexpr uint32_t row_cell(int best, int gap) {
  return (uint32_t)(uint16_t)(int16_t)(best + kRowBias) |
         ((uint32_t)(uint16_t)(int16_t)(gap + kRowBias) << 16);
}
__host__ __device__ constexpr int row_score(int v) {  // a score as rows compute it
  return (int)((unsigned)(v + kRowBias) << 16);
}
constexpr uint32_t kEmptyCell = row_cell(kInitScore, kInitScore);
constexpr int kNoDelimiter = 0x3fffffff;
constexpr int kRowMaxBest = 28671;   // the largest maximum (and row share) a band holds
constexpr int kRowMaxScore = 1023;   // the largest matrix entry, gap or X-drop

// Whether row_init / row_step are exact for these parameters: the initial
// score below every threshold (see above), values that fit the halves, and
// a gap that costs something (a gap never ties with the maximum).
__host__ __device__ inline bool row_dp_exact(int gap_open, int gap_ext, int cutoff) {
  return cutoff >= 0 && cutoff <= kRowMaxScore - 64 && gap_open >= 0 && gap_ext >= 0 &&
         gap_open <= kRowMaxScore && gap_ext <= kRowMaxScore && gap_open + gap_ext >= 1 &&
         gap_open + gap_ext <= kRowMaxScore;
}

// Whether they are also the faster form.  A row costs one group of four
// columns at least, so where no gap fits into the X-drop and the band is one
// column wide, one column at a time is; and a row's share of gap_ext uses up
// the halves' range, past which an extension starts anew on a warp (after some
// 1,000 rows of a homolog at kRowMaxGapExt).  One column at a time and grouped,
// in us: 600,000 extensions with penalties 11/1, X-drop 11 479 and 541, X-drop
// 12 659 and 577; 300,000 with 11/24, X-drop 38 665 and 615, 120 1,547 and
// 1,369, 240 3,442 and 3,137; with 11/28, X-drop 60 707 and 683, 120 1,427 and
// 1,817, 240 2,723 and 2,828; 100,000 with 11/100, X-drop 38 309 and 544.
constexpr int kRowMaxGapExt = 24;

__host__ __device__ inline bool row_dp_pays(int gap_open, int gap_ext, int cutoff) {
  return gap_open + gap_ext <= cutoff && gap_ext <= kRowMaxGapExt;
}

// Whether a matrix entry keeps a pruned cell's diagonal below every
// threshold and the values of a row inside int16.
__host__ __device__ __forceinline__ bool row_entry_fits(int v, int gap_ext, int cutoff) {
  return v >= -kRowMaxScore && v + gap_ext < -kInitScore - cutoff;
}

// The score table of a block: row x (database residue) at word
// kMatrixStride * x, (score + gap_ext) << 16; a query residue's byte
// indexes its row directly.  Words past the table are readable for any
// residue byte.
constexpr int kRowTableWords = kMatrixStride * kMatrixStride + 64;

__host__ __device__ __forceinline__ int row_table_entry(int v, int gap_ext) {
  return (int)((unsigned)(v + gap_ext) << 16);
}

// Loads the table; returns (on every thread) whether its entries fit.
__device__ __forceinline__ bool load_row_table(int *tbl, const GappedJob &job, const int32_t *m,
                                               int number_letters, int stride) {
  bool fits = true;
  for (int i = threadIdx.x; i < kRowTableWords; i += blockDim.x) {
    const int r = i / kMatrixStride, c = i % kMatrixStride;
    int v = 0;
    if (r < number_letters && c < number_letters) v = m[r * stride + c];
    fits = fits && row_entry_fits(v, job.gap_ext, job.cutoff);
    tbl[i] = row_table_entry(v, job.gap_ext);
  }
  return __syncthreads_and(fits) != 0;
}

// The band of one extension: W columns, a circular buffer of W / 4 groups;
// [group][thread][column] cells (a group is one 16-byte access, and a warp's
// lanes never share a bank whatever groups they are at) and [group][thread]
// residue words.
template <int W, int STRIDE>
struct RowBand {
  static_assert(W >= 16 && (W & (W - 1)) == 0 && W <= 128, "a power of two up to 128 columns");
  static constexpr int kGroups = W / 4;
  uint32_t cell;  // this thread's group 0 (16-byte aligned)
  uint32_t res;   // this thread's word of group 0
  __host__ __device__ __forceinline__ uint32_t slot(int g) const {
    return (uint32_t)(g & (kGroups - 1));
  }
  __host__ __device__ __forceinline__ uint32_t group(int g) const {
    return cell + slot(g) * (16 * STRIDE);
  }
  __host__ __device__ __forceinline__ uint32_t column(int c) const {
    return group(c >> 2) + 4 * (uint32_t)(c & 3);
  }
  __host__ __device__ __forceinline__ uint32_t residues(int g) const {
    return res + slot(g) * (4 * STRIDE);
  }
};

struct RowExt {
  const uint8_t *q0;
  const uint8_t *dn;  // the residue after xr
  int inc;
  int bs, be;         // band [bs, be) as the reference counts it
  int delim_at;       // column of the query's delimiter (kNoDelimiter: not seen)
  int groups;         // groups set up so far
  int thr;            // row_score(running maximum - X-drop + gap_ext * rows)
  int best;           // running maximum
  int col, at;        // its column and row (0 and -1: none yet)
  int row;            // the next row
  int xr;             // its residue, loaded one row ahead
  uint32_t cells;
  // the maximum's query and database offsets
  __host__ __device__ __forceinline__ int pos0() const { return (col - 1) * inc; }
  __host__ __device__ __forceinline__ int pos1() const { return at * inc; }
};

// The residues of group g's columns (column c holds query residue c - 1)
// and the delimiter's column if it lies there.
template <class Band>
__host__ __device__ __forceinline__ void row_residues(const Band &band, RowExt &x, int g,
                                                      int delim) {
  const uint8_t *s = x.q0 + (4 * g - 1) * x.inc;
  const uintptr_t a = (uintptr_t)s - (x.inc > 0 ? 0 : 3);
  const uint32_t *p = (const uint32_t *)(a & ~(uintptr_t)3);
  uint32_t w = row_funnel_r(p[0], p[1], 8 * (int)(a & 3));
  if (x.inc < 0) w = row_reverse_bytes(w);
  uint32_t z = w ^ (0x01010101u * (uint32_t)delim);
  if (g == 0) z |= 0xffu;  // column 0 is not a residue
  const uint32_t hit = (z - 0x01010101u) & ~z & 0x80808080u;  // its lowest set bit is exact
  if (hit && x.delim_at == kNoDelimiter) x.delim_at = 4 * g + (row_low_bit(hit) >> 3);
  row_store(band.residues(g), (w & 0x3f3f3f3fu) << 2);
}

// A group the band has not reached: residues, empty cells.
template <class Band>
__host__ __device__ __forceinline__ void row_new_group(const Band &band, RowExt &x, int delim) {
  const int g = x.groups++;
  row_residues(band, x, g, delim);
  row_store4(band.group(g), RowGroup{{kEmptyCell, kEmptyCell, kEmptyCell, kEmptyCell}});
}

// The band ends at the query's end: its last column's best score is no
// diagonal for the delimiter's column, which its group evaluates with it.
template <class Band>
__host__ __device__ __forceinline__ void row_end_diagonal(const Band &band, int last) {
  const uint32_t a = band.column(last);
  row_store(a, (row_load(a) & 0xffff0000u) | (kEmptyCell & 0xffffu));
}

// Row -1 (src/gapped_extender.cpp:345-364): the gap row along the query.
template <int W, int STRIDE>
__host__ __device__ __forceinline__ int row_init(const GappedJob &job,
                                                 const RowBand<W, STRIDE> &band, RowExt &x,
                                                 const uint8_t *q0, const uint8_t *d0,
                                                 bool reverse) {
  using Band = RowBand<W, STRIDE>;
  const int inc = reverse ? -1 : 1;
  const int delim = job.delim;
  const int ge = job.gap_ext, gi = job.gap_open + job.gap_ext;
  x.q0 = q0;
  x.dn = d0 + inc;
  x.inc = inc;
  x.thr = row_score(-job.cutoff);
  x.best = 0;
  x.col = 0;
  x.at = -1;
  x.row = 0;
  x.cells = 0;
  x.groups = 0;
  x.delim_at = kNoDelimiter;
  x.xr = d0[0];
  if (q0[0] == delim || x.xr == delim) return kLaneDone;
  // columns 1 .. k hold the gap row's scores at or above -X-drop
  int k = 0;
  if (job.cutoff >= gi) k = ge == 0 ? W : (job.cutoff - gi) / ge + 1;
  if (k >= W) k = W;  // (overflows below unless the query ends first)
  int score = -gi;
  for (;;) {
    const int g = x.groups++;
    row_residues(band, x, g, delim);
    RowGroup cell;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = 4 * g + j;
      cell.w[j] = kEmptyCell;
      // a gap cell's vertical gap is as row 0 uses it
      if (c == 0) {
        cell.w[j] = row_cell(0, -gi + ge);
      } else {
        if (c <= k && c < x.delim_at) cell.w[j] = row_cell(score, score - gi + ge);
        score -= ge;
      }
    }
    row_store4(band.group(g), cell);
    const int end = (k < x.delim_at - 1 ? k : x.delim_at - 1) + 1;  // first column not set
    if (4 * x.groups > end) {
      x.bs = 0;
      x.be = end < x.delim_at ? end + 1 : end;  // the sentinel column
      if (end >= x.delim_at) row_end_diagonal(band, end - 1);
      break;
    }
    if (x.groups == Band::kGroups) return kLaneOverflow;
  }
  if (x.be > 4 * x.groups) {
    if (x.groups == Band::kGroups) return kLaneOverflow;
    row_new_group(band, x, delim);
  }
  return kLaneRunning;
}

// One database row (src/gapped_extender.cpp:366-470) of every lane whose
// `st` is kLaneRunning; the whole warp calls it.
template <int W, int STRIDE>
__host__ __device__ __forceinline__ int row_step(const GappedJob &job, uint32_t tbl,
                                                 const RowBand<W, STRIDE> &band, RowExt &x,
                                                 int st) {
  using Band = RowBand<W, STRIDE>;
  constexpr int kAhead = 2;  // groups set up beyond the band's when some lane needs one
  if (st == kLaneRunning && x.xr == job.delim) st = kLaneDone;
  const int gi = (int)((unsigned)-(job.gap_open + job.gap_ext) << 16);
  const int ge = (int)((unsigned)-job.gap_ext << 16);
  bool go = false;  // the extension goes on after this row
  int last = 0, edge = 0;
  if (st == kLaneRunning) {
    const uint32_t row = tbl + 4u * kMatrixStride * (uint32_t)x.xr;
    x.xr = *x.dn;  // the next row's residue (the chunk is padded)
    x.dn += x.inc;
    // a vertical gap opened in this row, as the next row uses it
    const int gv = gi - ge;
    int cut = (int)((unsigned)-job.cutoff << 16);  // less the cell's tag
    const int g0 = x.bs >> 2, gn = (x.be + 3) >> 2;
    // groups that may be evaluated: set up, in the ring, not past the query
    int limit = (x.delim_at + 3) >> 2;
    limit = limit < x.groups ? limit : x.groups;
    limit = limit < g0 + Band::kGroups ? limit : g0 + Band::kGroups;
    const int thr0 = (int)((unsigned)x.thr - (unsigned)ge);
    int thr = thr0;
    int gap = row_score(kInitScore);  // the horizontal gap
    uint32_t prev = kEmptyCell;       // the column before
    // first and last group with a kept column: 16 * group + pruned flags
    // (column 0 of the group in bit 3); `flags` are the newest group's
    int kf = kNoDelimiter, kl = 0;
    uint32_t flags = 15, skip = g0 == 0 ? 8 : 0;  // column 0 is no cell
    int g = g0;
    RowGroup cur = row_load4(band.group(g));
    uint32_t res = row_load(band.residues(g));
#pragma unroll 2
    do {
      const RowGroup w = cur;
      const int sc[4] = {
          (int)row_load_const(row_byte_plus<0>(res, row)), (int)row_load_const(row_byte_plus<1>(res, row)),
          (int)row_load_const(row_byte_plus<2>(res, row)), (int)row_load_const(row_byte_plus<3>(res, row))};
      cur = row_load4(band.group(g + 1));
      res = row_load(band.residues(g + 1));
      if (flags != 15) {
        kl = 16 * g + (int)flags;  // (of group g - 1: settled at the end)
        kf = kf < kl ? kf : kl;
      }
      RowGroup o;
      flags = skip;
      skip = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const unsigned diag = (j ? w.w[j - 1] : prev) << 16;
        const int s = row_max3((int)(diag + (unsigned)sc[j]), (int)w.w[j], gap);
        const bool drop = s < thr;
        thr = row_addmax(s, --cut, thr);
        gap = row_addmax(s, gi, (int)((unsigned)gap + (unsigned)ge));
        const uint32_t cell = row_pack(s, row_addmax(s, gv, (int)w.w[j]));
        o.w[j] = drop ? kEmptyCell : cell;
        if (drop) flags |= 8u >> j;
      }
      prev = w.w[3];
      row_store4(band.group(g), o);
      ++g;
      // past the band while the horizontal gap lives
    } while ((g < gn || gap >= thr) && g < limit);
    // the maximum, its column if this row raised it, the threshold
    const int clean = (int)(((unsigned)thr + 0xffffu) & 0xffff0000u);
    x.best += (int)((unsigned)clean - (unsigned)thr0) >> 16;
    if (clean != thr0) {
      x.col = 4 * g0 + (int)((unsigned)clean - (unsigned)thr) - 1;
      x.at = x.row;
    }
    ++x.row;
    x.thr = clean;
    x.cells += (uint32_t)(x.be - x.bs - 1);
    // ---- the band's new edges
    const int top = 4 * g - 1;  // the last column evaluated
    if (top >= x.delim_at) {
      // horizontal gaps that ran past the query's end are no cells
      flags |= (2u << (top - x.delim_at)) - 1;
      for (int c = x.delim_at; c <= top; ++c) row_store(band.column(c), kEmptyCell);
    }
    if (flags != 15) {
      kl = 16 * g + (int)flags;
      kf = kf < kl ? kf : kl;
    }
    if (kf == kNoDelimiter) {
      st = kLaneDone;
    } else if ((clean >> 16) + job.cutoff > kRowMaxBest + kRowBias - 2 * kRowMaxScore) {
      // a later row's values might not fit int16: the maximum has to leave
      // room for one more score
      st = kLaneOverflow;
    } else {
      go = true;
      const int first = 4 * (kf >> 4) - 1 - row_high_bit(~(unsigned)kf & 15u);
      last = 4 * (kl >> 4) - 1 - row_low_bit(~(unsigned)kl & 15u);
      if (gap >= clean && last == top) {
        // the horizontal gap goes on past the groups set up
        while (gap >= clean && last + 1 < x.delim_at) {
          if (((last + 1) >> 2) >= x.groups) {
            if (((last + 1) >> 2) - g0 >= Band::kGroups) {
              st = kLaneOverflow;
              go = false;
              break;
            }
            row_new_group(band, x, job.delim);
            if (last + 1 >= x.delim_at) break;
          }
          ++last;
          row_store(band.column(last), row_pack(gap, (int)((unsigned)gap + (unsigned)gv)));
          gap = (int)((unsigned)gap + (unsigned)ge);
        }
      }
      if (first > 1 && g0 == 0) row_store(band.column(0), kEmptyCell);
      x.bs = first - 1;
      // the column whose residue the reference tests (:461): the old right
      // end where the band shrank, else the column after the last
      const int grown = last + 1 - x.be;
      edge = grown < 0 ? x.be : last + 1;
      x.cells += (uint32_t)(grown < 0 ? 0 : grown);
    }
  }
  if (row_any(go && (edge >> 2) >= x.groups)) {
    // every lane that is short of groups ahead sets its up now, so that the
    // warp comes here every few rows only
    if (go) {
      int want = (edge >> 2) + kAhead + 1;
      const int room = (x.bs >> 2) + Band::kGroups;
      want = want < room ? want : room;
      while (x.groups < want) row_new_group(band, x, job.delim);
    }
    row_meet();
  }
  if (go) {
    x.be = last + 2;  // with the sentinel column (an empty cell)
    if ((edge >> 2) >= x.groups || ((x.be - 1) >> 2) - (x.bs >> 2) >= Band::kGroups) {
      st = kLaneOverflow;
    } else if (edge >= x.delim_at) {
      // no sentinel
      x.be = last + 1;
      row_end_diagonal(band, last);
    }
  }
  row_meet();
  return st;
}

}  // namespace gzb
