// walk_window_hit of gzb_walk.cuh on the host, with everything a byte's
// address could reach behind the window table set (tests/test_walk_padding.py).
#include <vector>

#include "gzb_walk.cuh"

using namespace gzb;

extern "C" void walk_window_hits(const uint8_t *q, const uint8_t *d, uint64_t n,
                                 const uint32_t *qpos, const uint32_t *dpos, const int32_t *m32,
                                 int delim, int cutoff, int trigger, uint32_t behind,
                                 int32_t *hits) {
  std::vector<uint32_t> memory(1 << 16, behind);
  row_host_memory = reinterpret_cast<char *>(memory.data());
  for (int a = 0; a < 32; ++a)
    for (int x = 0; x < 32; ++x) {
      const int v = window_entry(a, a ^ x, m32[(a ^ x) * 32 + a], delim);
      row_store(256 * a + 4 * x, (uint32_t)v);
      row_store(256 * a + 4 * x + 128, (uint32_t)v << 16);
    }
  for (uint64_t i = 0; i < n; ++i) {
    WindowWords w;
    uint32_t qa[16], da[16];
    fetch_window(q + qpos[i], w);
    align_window(q + qpos[i], w, qa);
    fetch_window(d + dpos[i], w);
    align_window(d + dpos[i], w, da);
    hits[i] = walk_window_hit(0, qa, da, cutoff, trigger);
  }
}
