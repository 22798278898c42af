// Host build of the device cell rasterizer (raster.cuh) against the oracle's rasterizer (the
// reference's banded DDA): every 4 x 32 window of a canvas, for random lines of all slopes and
// directions, of whole-pixel coordinates and of the largest extents. The device's reciprocal is an
// approximation; here it is off by up to 3 ulp either way.
// Usage: raster_rows_check <seed> <lines>; exit status 0 when all match.
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "b2d_oracle.h"

#define __device__
#define __forceinline__ inline
using std::max;
using std::min;
static inline uint32_t atomicAdd(uint32_t* p, uint32_t v) { uint32_t o = *p; *p += v; return o; }
static int g_ulp = 0;
static inline float fast_rcp(float x) {
  if (x == 0.0f) return 0.0f;                  // not used: a vertical segment crosses no cell boundary
  float r = 1.0f / x;
  uint32_t b; memcpy(&b, &r, 4);
  b += uint32_t(g_ulp);
  memcpy(&r, &b, 4);
  return r;
}
#include "raster.cuh"

using namespace blgpu;

static long check(int w, int rows, DevSeg g, uint32_t sign) {
  std::vector<uint32_t> grid(size_t(rows) * size_t(w + 2));
  std::fill(grid.begin(), grid.end(), 0u);
  b2d_oracle_rasterize_line(g.x0, g.y0, g.x1, g.y1, sign, 64, w, rows, grid.data());
  long bad = 0;
  // every window near the line, and the first and last ones
  const int t_min = (min(g.x0, g.x1) >> 8) / 32, t_max = (max(g.x0, g.x1) >> 8) / 32, t_end = (w + 31) / 32;
  for (int row0 = (g.y0 >> 8) & ~3; row0 <= (g.y1 - 1) >> 8 && row0 < rows; row0 += 4) {
    for (int t = 0; t < t_end; t++) {
      if (t != 0 && t + 1 != t_end && (t < t_min - 1 || t > t_max + 1)) continue;
      uint32_t cells[4 * 32] = {}, bd[4] = {};
      ras::WindowSink cs{cells, bd, t * 32};
      ras::segment_to_window(g, sign, row0, 4, cs);
      for (int r = 0; r < 4 && row0 + r < rows; r++) {
        uint32_t left = 0;
        const uint32_t* line = &grid[size_t(row0 + r) * size_t(w + 2)];
        for (int x = 0; x < t * 32; x++) left += line[x];
        if (left != bd[r]) bad++;
        for (int x = 0; x < 32 && t * 32 + x < w; x++) if (line[t * 32 + x] != cells[r * 32 + x]) bad++;
      }
    }
  }
  if (bad) printf("mismatch %d x %d: (%d, %d) - (%d, %d) sign %u, %ld values\n", w, rows, g.x0, g.y0, g.x1, g.y1, sign, bad);
  return bad;
}

int main(int argc, char** argv) {
  const uint64_t seed = argc > 1 ? strtoull(argv[1], nullptr, 10) : 1;
  const long n = argc > 2 ? atol(argv[2]) : 1000;
  std::mt19937_64 rng(seed);
  auto u = [&](int lo, int hi) { return int(lo + int64_t(rng() % uint64_t(hi - lo + 1))); };
  long bad = 0;
  for (long i = 0; i < n && bad < 20; i++) {
    g_ulp = u(-3, 3);
    int w = u(1, 200), h = u(1, 40);
    DevSeg g;
    const int kind = u(0, 7);
    if (kind == 0 && i % 16 == 0) { w = u(1000, 65535); h = u(1, 12); }
    if (kind == 1 && i % 16 == 0) { w = u(1, 40); h = u(1000, 65535); }
    const int W = w * 256, H = h * 256;
    g.x0 = u(0, W); g.x1 = u(0, W); g.y0 = u(0, H); g.y1 = u(0, H);
    if (kind == 2) { g.x1 = min(W, max(0, g.x0 + u(-300, 300))); g.y1 = min(H, max(0, g.y0 + u(-300, 300))); }
    if (kind == 3) { g.x0 &= ~255; g.x1 &= ~255; }
    if (kind == 4) { g.y0 &= ~255; g.y1 &= ~255; }
    if (kind == 5) { g.x0 &= ~127; g.x1 &= ~127; g.y0 &= ~63; g.y1 &= ~63; }
    if (kind == 6) { const int d = min(min(W - g.x0, H - g.y0), u(0, 4000)); g.x1 = g.x0 + d; g.y1 = g.y0 + d; }
    if (kind == 7) { g.x1 = g.x0 + u(-2, 2); g.x1 = min(W, max(0, g.x1)); }
    if (g.y0 > g.y1) { std::swap(g.y0, g.y1); std::swap(g.x0, g.x1); }
    if (g.y0 == g.y1) continue;
    bad += check(w, h, g, uint32_t(rng() & 1u));
  }
  printf("mismatches %ld\n", bad);
  return bad ? 1 : 0;
}
