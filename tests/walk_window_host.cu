// The window evaluation of gzb_walk.cuh on the host (tests/test_walk_window.py).
#include <vector>

#include "gzb_walk.cuh"

using namespace gzb;

// settled[i], steps[i] and (unless null) hits[i] of seeds (qpos[i], dpos[i])
extern "C" void walk_windows(const uint8_t *q, const uint8_t *d, uint64_t n, const uint32_t *qpos,
                             const uint32_t *dpos, const int32_t *m32, int delim, int cutoff,
                             int trigger, int32_t *settled, int32_t *steps, int32_t *hits) {
  std::vector<uint32_t> memory(kWindowTableBytes / 4);
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
    uint32_t side[2];
    settled[i] = walk_window(0, qa, da, cutoff, trigger, &steps[i], side) ? 1 : 0;
    if (hits) hits[i] = walk_window_hit(0, qa, da, cutoff, trigger);
  }
}
