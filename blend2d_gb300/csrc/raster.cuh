// raster.cuh - the reference's analytic cells, evaluated per (segment, pixel row).
//
// The reference walks a segment with an integer DDA (AnalyticRasterizer, blend2d/raster/
// analyticrasterizer_p.h:289-1166): cell[x] += (cover << 9) - area, cell[x + 1] += area. Its
// accumulators are rounded divisions in disguise. After k steps the x at a row boundary and the y
// at a cell boundary are
//   X(y) = x0 +- floor(((y - y0) * |dx| + ceil(dy / 2)) / dy)
//   Y(x) = y0 +  floor((|x - x0| * dy + ceil(|dx| / 2)) / |dx|)
// because the error term starts at (d >> 1) - 1 and every step keeps 0 <= error < d. So a row's
// cells need only the row's entry and exit x and one Y per cell boundary crossed, whatever the
// segment did above it: there is no state to advance to the row, no case per slope or direction,
// and no 64-bit division. A segment that runs to the left is the mirror image of one that runs to
// the right: with u = -x its cells are walked in the same order, the cover of a cell splits
// between its near side ((cover << 9) - area) and its far side (area) the same way, and only the
// column of a side differs. One detail of the DDA is kept: a steep segment (dy >= |dx|) takes the
// crossing's y modulo the row, a shallow one relative to it (the two differ when rounding puts
// the crossing on the next row's top).
//
// A window is 4 rows x 32 columns. Contributions left of it are summed into a per-row backdrop (the
// coverage carried in from the left), contributions right of it are dropped. All sums are modular
// u32, so the windows' partial sums equal the reference's band sums.
#pragma once

#include "blgpu_internal.h"

namespace blgpu {
namespace ras {

#ifdef __CUDACC__
__device__ __forceinline__ float fast_rcp(float x) {   // within 1 ulp; inf for 0 (a vertical segment's, not used)
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
#endif

// floor((a * b + (d + 1) / 2) / d) for 0 <= a, b, d < 2^24, a * b / d < 2^24 (+ rounding), d > 0;
// `rcp` ~ 1 / d to a few ulp. The quotient is estimated in FP32 (off by 8 at most: the product's
// and the reciprocal's relative errors on a quotient below 2^24) and corrected by its remainder,
// which fits 32 bits because |remainder| <= 8 d.
__device__ __forceinline__ int div_round(int a, int b, int d, float rcp) {
  int q = int(float(a) * float(b) * rcp);
  int r = int(uint32_t(a) * uint32_t(b) + uint32_t((d + 1) >> 1) - uint32_t(q) * uint32_t(d));
  while (r < 0) { q--; r += d; }
  while (r >= d) { q++; r -= d; }
  return q;
}

// Cells of one window: 4 x 32 sums and a per-row backdrop, both in shared memory.
struct WindowSink {
  uint32_t* cells;
  uint32_t* backdrop;
  int tx0;
  __device__ __forceinline__ void add(int row, int x, uint32_t v) {
    const int cx = x - tx0;
    if (cx < 0) atomicAdd(&backdrop[row], v);
    else if (cx < kTileW) atomicAdd(&cells[row * kTileW + cx], v);
  }
};

// All cells of one segment in the window's rows [row0, row0 + rows). Rows outside, cells inside: one
// flat loop over all cells, its row step in a branch, measured slower (coverage of the 512-canvas
// batch 9.7 against 5.2 ms: the lanes do not meet again after the branch).
template<typename Sink>
__device__ __forceinline__ void segment_to_window(const DevSeg& g, uint32_t sign, int row0, int rows, Sink& cs) {
  const int r0 = max(g.y0 >> 8, row0), r1 = min((g.y1 - 1) >> 8, row0 + rows - 1);
  if (r0 > r1) return;
  const uint32_t sm = 0u - sign;
  const bool rtl = g.x1 < g.x0;
  const int flip = rtl ? -1 : 0;                     // u = (x ^ flip) - flip
  const int u0 = (g.x0 ^ flip) - flip, u1 = (g.x1 ^ flip) - flip;
  const int dx = u1 - u0, dy = g.y1 - g.y0;
  const bool steep = dy >= dx;
  const float rdx = fast_rcp(float(dx)), rdy = fast_rcp(float(dy));
  // the cells whose sides lie in the window, in u
  const int c_lo = (rtl ? -(cs.tx0 + kTileW) : cs.tx0 - 1), c_hi = (rtl ? -cs.tx0 : cs.tx0 + kTileW - 1);

  int ub = r0 > (g.y0 >> 8) ? u0 + div_round((r0 << 8) - g.y0, dx, dy, rdy) : u0;
  for (int r = r0; r <= r1; r++) {
    const int top = r << 8;
    const int ua = ub;
    const bool last = g.y1 <= top + 256;
    ub = last ? u1 : u0 + div_round(top + 256 - g.y0, dx, dy, rdy);
    const int yt = max(g.y0 - top, 0), yb = last ? g.y1 - top : 256;
    const int ca = ua >> 8, ce = ub > ua ? (ub - 1) >> 8 : ca;
    // y of the boundary between cells c - 1 and c
    auto cross = [&](int c) {
      const int y = g.y0 + div_round((c << 8) - u0, dy, dx, rdx);
      return steep ? (y & 255) : y - top;
    };
    const int row = r - row0;
    int y_prev = yt;
    int c = ca;
    if (ca < c_lo) {
      y_prev = ce < c_lo ? yb : cross(c_lo);
      c = c_lo;
      if (!rtl) atomicAdd(&cs.backdrop[row], ((uint32_t(y_prev - yt) ^ sm) - sm) << 9);
    }
    int f_in = c == ca ? ua & 255 : 0;
    uint32_t carry = 0;
    const int c_end = min(ce, c_hi);
    if (c <= c_end) {
      for (; c <= c_end; c++) {
        const bool end = c == ce;
        const int y = end ? yb : cross(c + 1);
        const int f_out = end ? ub - (ce << 8) : 256;
        const uint32_t cover = (uint32_t(y - y_prev) ^ sm) - sm;
        const uint32_t area = cover * uint32_t(f_in + f_out);
        cs.add(row, (c ^ flip) - flip, carry + (cover << 9) - area);
        carry = area;
        y_prev = y;
        f_in = 0;
      }
      cs.add(row, (c ^ flip) - flip, carry);
    }
    if (rtl && ce > c_hi) atomicAdd(&cs.backdrop[row], ((uint32_t(yb - y_prev) ^ sm) - sm) << 9);
  }
}

}  // namespace ras
}  // namespace blgpu
