// The grouped rows of gzb_row.cuh on the host, one extension a call
// (tests/test_row_dp.py).
#include <cstring>
#include <vector>

#include "gzb_row.cuh"

using namespace gzb;

template <int W>
static int extend(const GappedJob &job, const uint8_t *q0, const uint8_t *d0, int reverse,
                  const int32_t *matrix, int letters, int32_t *out, uint64_t *cells) {
  constexpr int kTable = 16, kCells = 8192, kRes = 16384;  // 16-byte aligned offsets
  static std::vector<uint32_t> memory(8192);
  for (auto &w : memory) w = 0xFCFCFCFCu;  // a band starts with whatever was there
  row_host_memory = reinterpret_cast<char *>(memory.data());
  bool fits = true;
  for (int i = 0; i < kRowTableWords; ++i) {
    const int r = i / kMatrixStride, c = i % kMatrixStride;
    const int v = r < letters && c < letters ? matrix[r * letters + c] : 0;
    fits = fits && row_entry_fits(v, job.gap_ext, job.cutoff);
    row_store(kTable + 4 * i, (uint32_t)row_table_entry(v, job.gap_ext));
  }
  if (!fits) return -1;
  RowBand<W, 2> band{kCells, kRes};
  RowExt x;
  int st = row_init(job, band, x, q0, d0, reverse != 0);
  while (st == kLaneRunning) st = row_step(job, kTable, band, x, st);
  out[0] = x.best;
  out[1] = x.pos0();
  out[2] = x.pos1();
  *cells = x.cells;
  return st;
}

// 1: done, 2: handed on (band or score too large), -1: the parameters are
// not admitted
extern "C" int row_extend(int width, const uint8_t *q, uint64_t q0, const uint8_t *d, uint64_t d0,
                          int delim, int gap_open, int gap_ext, int cutoff, int reverse,
                          const int32_t *matrix, int letters, int32_t *out, uint64_t *cells) {
  if (!row_dp_exact(gap_open, gap_ext, cutoff)) return -1;
  GappedJob job{q, d, delim, gap_open, gap_ext, cutoff};
  return width == 32 ? extend<32>(job, q + q0, d + d0, reverse, matrix, letters, out, cells)
                     : extend<64>(job, q + q0, d + d0, reverse, matrix, letters, out, cells);
}
