// kernels.cu - the sm_103a render pipeline (K0 LUT build, K1 edge build, K2 binning, K3 fine).
//
// Built with -fmad=false: the FP64 edge builder and the FP32 radial/conic fetchers must not be
// contracted into FMAs, because the reference computes every a*b+c unfused.
#include <cuda_runtime.h>
#include <stdint.h>

#include "blgpu_internal.h"
#include "edge_build.cuh"
#include "pipeline.cuh"
#include "raster.cuh"

namespace blgpu {

// ---------------------------------------------------------------------------------------------
// K0 - gradient LUTs (interpolation.cpp:19-156, interpolation_sse2.cpp:18-171,
// interpolation_avx2.cpp:18-177), one warp per table: the spans are written in the order of the
// reference's sequential span writer (later spans overwrite earlier ones).
// ---------------------------------------------------------------------------------------------

__device__ __forceinline__ uint32_t rgba32_of(uint64_t v) {
  uint32_t b = uint32_t(v >> 8) & 0xFFu, g = uint32_t(v >> 24) & 0xFFu;
  uint32_t r = uint32_t(v >> 40) & 0xFFu, a = uint32_t(v >> 56) & 0xFFu;
  return (a << 24) | (r << 16) | (g << 8) | b;
}
__device__ __forceinline__ uint32_t simd_div255(uint32_t x) { return (((x + 0x80u) & 0xFFFFu) * 0x101u) >> 16; }
__device__ __forceinline__ uint32_t sat8(uint32_t v) { return v > 255u ? 255u : v; }
__device__ __forceinline__ uint32_t premul_avx2_short_span(uint32_t c) {
  uint32_t a = c >> 24;
  return (sat8(simd_div255(a | (255u * a))) << 24) | (sat8(simd_div255((c >> 16) & 255u)) << 16) |
         (sat8(simd_div255((c >> 8) & 255u)) << 8) | sat8(simd_div255(c & 255u));
}
// Channels times alpha over 255, two to a word. The SIMD builders' product (x + 128) * 257 >> 16 is the
// same number, (y + (y >> 8)) >> 8 with y = x + 128, so both kinds of builder use this one.
__device__ __forceinline__ uint32_t premul(uint32_t c) {
  uint32_t a = c >> 24;
  uint32_t v = c | 0xFF000000u;
  uint32_t rb = (v & 0x00FF00FFu) * a + 0x00800080u;
  uint32_t ag = ((v >> 8) & 0x00FF00FFu) * a + 0x00800080u;
  rb = (rb + ((rb >> 8) & 0x00FF00FFu)) & 0xFF00FF00u;
  ag = (ag + ((ag >> 8) & 0x00FF00FFu)) & 0xFF00FF00u;
  return ag | (rb >> 8);
}
__device__ __forceinline__ int round_to_int(double x) {
  int y = (x >= -2147483648.5 && x < 2147483647.5) ? __double2int_rn(x) : INT32_MIN;
  return y + (double(y) - x == -0.5);
}

// One interpolation span of a LUT builder: the FP64 part of the builder (stop positions and the
// per-channel increments) is evaluated once per span, one lane per stop; entries only do integer work.
struct LutSpan {
  uint32_t start, count;   // simd: first entry and i (entries start .. start + i); scalar: start, cnt
  uint32_t c0, c1;         // colours at both ends (scalar: after its equal-position rule)
  int32_t inc[4];          // simd: dx per channel (b, g, r, a); scalar: r, g, b, a increments
  uint32_t pos[4];         // simd: the first entry's channels, 8.23 with the rounding half
};

// The entries of one span, by a warp. Lane l has the entries that are l modulo 32, of every span: where a
// span begins on the entry the one before it ends on, it overwrites it, as in the reference's builders.
__device__ __forceinline__ void lut_span_simd(const LutSpan& q, uint32_t* lut, uint32_t size, int lane, bool avx2) {
  const uint32_t start = q.start, end = min(start + q.count, size - 1u);
  uint32_t e = (start & ~31u) + uint32_t(lane);
  if (q.count <= 1) {
    const uint32_t c0 = avx2 ? premul_avx2_short_span(q.c0) : premul(q.c0), c1 = avx2 ? premul_avx2_short_span(q.c1) : premul(q.c1);
    if (e < start) e += 32;                    // at most two entries
    if (e <= end) lut[e] = e == start ? c0 : c1;
    return;
  }
  // every channel stays within 0 .. 255: the increments are truncated towards zero
  uint32_t v[4], step[4];
#pragma unroll
  for (int ch = 0; ch < 4; ch++) {
    v[ch] = q.pos[ch] + uint32_t(q.inc[ch]) * (e - start);
    step[ch] = uint32_t(q.inc[ch]) * 32u;
  }
  for (; e <= end; e += 32) {
    if (e >= start)
      lut[e] = premul((v[0] >> 23) | ((v[1] >> 15) & 0xFF00u) | ((v[2] >> 7) & 0xFF0000u) | ((v[3] << 1) & 0xFF000000u));
#pragma unroll
    for (int ch = 0; ch < 4; ch++) v[ch] += step[ch];
  }
}

__device__ __forceinline__ void lut_span_scalar(const LutSpan& q, uint32_t* lut, uint32_t size, int lane) {
  constexpr uint32_t kMask = 0xFFu << 23, kHalf = 1u << 22;
  const uint32_t start = q.start, end = min(start + q.count, size), c0 = q.c0, first = premul(c0);
  const bool flat = c0 == q.c1, opaque = ((c0 & q.c1) >> 24) == 0xFFu;
  for (uint32_t e = (start & ~31u) + uint32_t(lane); e < end; e += 32) {
    if (e < start) continue;
    uint32_t v = first;
    if (!flat && e != start) {
      const uint32_t j = e - start;
      const uint32_t r = ((c0 << 7) & kMask) + kHalf + j * uint32_t(q.inc[0]);
      const uint32_t g = ((c0 << 15) & kMask) + kHalf + j * uint32_t(q.inc[1]);
      const uint32_t b = ((c0 << 23) & kMask) + kHalf + j * uint32_t(q.inc[2]);
      const uint32_t a = opaque ? kMask : ((c0 >> 1) & kMask) + kHalf + j * uint32_t(q.inc[3]);
      v = premul(((a & kMask) << 1) | ((r & kMask) >> 7) | ((g & kMask) >> 15) | ((b & kMask) >> 23));
    }
    lut[e] = v;
  }
}

// 64-bit LUT of dithered gradients: interpolate_prgb64 (interpolation.cpp:161-288). Same span walk
// as the scalar 32-bit builder (a span covers (p1 >> 8) - (p0 >> 8) + 1 entries, its first entry is
// premultiplied c0, later ones step 16.15 fixed-point positions), with 16-bit channels and
// premultiplication by udiv65535 (scalar_p.h:37, :179-222).
struct LutSpan64 {
  uint32_t start, count;
  uint64_t c0, c1;
  uint32_t inc[4];         // r, g, b, a
};

__device__ __forceinline__ uint32_t udiv65535(uint32_t x) { return ((x + 0x8000u) + ((x + 0x8000u) >> 16)) >> 16; }

__device__ __forceinline__ uint64_t premul64(uint64_t c) {
  const uint32_t a = uint32_t(c >> 48);
  const uint32_t r = udiv65535((uint32_t(c >> 32) & 0xFFFFu) * a);
  const uint32_t g = udiv65535((uint32_t(c >> 16) & 0xFFFFu) * a);
  const uint32_t b = udiv65535((uint32_t(c) & 0xFFFFu) * a);
  return (uint64_t(a) << 48) | (uint64_t(r) << 32) | (uint64_t(g) << 16) | uint64_t(b);
}

constexpr uint32_t kLut64Shift = 15, kLut64Mask = 0xFFFFu << 15;

__device__ __forceinline__ void lut_span64(const LutSpan64& q, uint64_t* lut, uint32_t size, int lane) {
  constexpr uint32_t kHalf = 1u << (kLut64Shift - 1);
  const uint32_t start = q.start, end = min(start + q.count, size);
  const uint64_t c0 = q.c0, first = premul64(c0);
  const bool flat = c0 == q.c1, opaque = ((c0 & q.c1) >> 48) == 0xFFFFu;
  const uint32_t r0 = uint32_t((c0 >> (32 - kLut64Shift)) & kLut64Mask) + kHalf;
  const uint32_t g0 = uint32_t((c0 >> (16 - kLut64Shift)) & kLut64Mask) + kHalf;
  const uint32_t b0 = uint32_t((c0 << kLut64Shift) & kLut64Mask) + kHalf;
  const uint32_t a0 = uint32_t((c0 >> (48 - kLut64Shift)) & kLut64Mask) + kHalf;
  for (uint32_t e = (start & ~31u) + uint32_t(lane); e < end; e += 32) {
    if (e < start) continue;
    uint64_t v = first;
    if (!flat && e != start) {
      const uint32_t j = e - start;
      const uint32_t r = r0 + j * q.inc[0], g = g0 + j * q.inc[1], b = b0 + j * q.inc[2];
      if (opaque) {
        v = (uint64_t(r & kLut64Mask) << (32 - kLut64Shift)) | (uint64_t(g & kLut64Mask) << (16 - kLut64Shift)) |
            (uint64_t(b & kLut64Mask) >> kLut64Shift) | 0xFFFF000000000000ull;
      }
      else {
        const uint32_t a = (a0 + j * q.inc[3]) >> kLut64Shift;
        v = (uint64_t(a) << 48) | (uint64_t(udiv65535((r >> kLut64Shift) * a)) << 32) |
            (uint64_t(udiv65535((g >> kLut64Shift) * a)) << 16) | uint64_t(udiv65535((b >> kLut64Shift) * a));
      }
    }
    lut[e] = v;
  }
}

// Warp-wide build of one 64-bit LUT, 32 stops per chunk like the 32-bit scalar path below.
__device__ void lut_build64(const DevLutJob& job, const DevStop* s, uint64_t* lut, LutSpan64* spans, int lane) {
  const uint32_t n = job.stop_count;
  const uint64_t first_c = s[0].rgba64;
  const double fWidth = double(int32_t(job.lut_size - 1u) << 8);
  uint32_t car_u0 = 0, span_end = 0;
  uint64_t car_c = first_c;
  for (uint32_t si = 0; si < n; si += 32) {
    const uint32_t k = si + uint32_t(lane);
    const int ns = int(min(32u, n - si));
    uint64_t c1 = 0;
    uint32_t u1 = 0;
    if (k < n) {
      c1 = s[k].rgba64;
      u1 = uint32_t(round_to_int(s[k].offset * fWidth));
    }
    uint32_t u0 = __shfl_up_sync(0xFFFFFFFFu, u1, 1);
    uint64_t c0 = __shfl_up_sync(0xFFFFFFFFu, c1, 1);
    if (lane == 0) { u0 = car_u0; c0 = car_c; }
    if (lane < ns) {
      LutSpan64 sp;
      const uint32_t i = (u1 >> 8) - (u0 >> 8);
      if (i == 0) c0 = c1;
      sp.start = u0 >> 8;
      sp.count = i + 1u;
      sp.c0 = c0;
      sp.c1 = c1;
      if (c0 != c1 && sp.count > 1) {
        const int32_t div = int32_t(sp.count - 1u);
        sp.inc[0] = uint32_t(int32_t(uint32_t((c1 >> (32 - kLut64Shift)) & kLut64Mask) -
                                     uint32_t((c0 >> (32 - kLut64Shift)) & kLut64Mask)) / div);
        sp.inc[1] = uint32_t(int32_t(uint32_t((c1 >> (16 - kLut64Shift)) & kLut64Mask) -
                                     uint32_t((c0 >> (16 - kLut64Shift)) & kLut64Mask)) / div);
        sp.inc[2] = uint32_t(int32_t(uint32_t((c1 << kLut64Shift) & kLut64Mask) -
                                     uint32_t((c0 << kLut64Shift) & kLut64Mask)) / div);
        sp.inc[3] = uint32_t(int32_t(uint32_t((c1 >> (48 - kLut64Shift)) & kLut64Mask) -
                                     uint32_t((c0 >> (48 - kLut64Shift)) & kLut64Mask)) / div);
      }
      spans[lane] = sp;
    }
    car_u0 = __shfl_sync(0xFFFFFFFFu, u1, ns - 1);
    car_c = __shfl_sync(0xFFFFFFFFu, c1, ns - 1);
    __syncwarp();
    span_end = spans[ns - 1].start + spans[ns - 1].count;
    for (int j = 0; j < ns; j++) lut_span64(spans[j], lut, job.lut_size, lane);
    __syncwarp();
  }
  // the trailing fill is the last stop's colour; entry 0 is the first stop's
  const uint64_t tail = premul64(car_c);
  for (uint32_t e = (span_end & ~31u) + uint32_t(lane); e < job.lut_size; e += 32)
    if (e >= span_end) lut[e] = tail;
  if (lane == 0) lut[0] = premul64(first_c);
}

// One warp per LUT. The span table is built 32 stops at a time, one stop per lane: a span depends
// only on its stop and the one before it (position and colour, passed up one lane; the previous
// chunk's last stop is carried), so the FP64 stop positions and increments of a chunk are computed
// in parallel. The spans follow one another from entry 0 on without a gap (the stops are sorted), and the
// warp writes them in order, 32 entries at a time, then the entries after the last one and entry 0.
// Bound: instruction issue. An entry that looked through all spans for its own, with a second pass over
// the table for its end and its first entry: 198,000 tables of 512 canvases of the batch 0.93 -> 0.46
// ms (on the side stream, beside the curves: frame 14.86 -> 14.40), 20,000 tables of curve paths 0.118
// -> 0.054, 4,000 dithered ones 0.035 -> 0.017, one table 0.020 -> 0.010.
constexpr int kLutWarps = 8;

__global__ void __launch_bounds__(32 * kLutWarps) lut_kernel(const DevLutJob* jobs, const DevStop* stops, uint32_t* luts,
                                                             const uint32_t* counts) {
  const uint32_t num_jobs = counts[kCntLutJobs];
  __shared__ LutSpan spans_all[kLutWarps][32];
  __shared__ LutSpan64 spans64_all[kLutWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t jid = blockIdx.x * kLutWarps + uint32_t(warp);
  if (jid >= num_jobs) return;                         // whole warps leave together
  LutSpan* spans = spans_all[warp];
  const DevLutJob job = jobs[jid];
  const DevStop* s = stops + job.stop_first;
  if (job.variant == kLut64) {                         // offset is even: 8-byte aligned entries
    lut_build64(job, s, reinterpret_cast<uint64_t*>(luts + job.lut_offset), spans64_all[warp], lane);
    return;
  }
  const uint32_t n = job.stop_count;
  const bool scalar = job.variant == kLutScalar;
  const bool avx2 = job.variant == kLutAVX2;
  uint32_t* lut = luts + job.lut_offset;
  const uint32_t first_c = rgba32_of(s[0].rgba64);
  const double fWidth = double(int32_t(job.lut_size - 1u) << 8);
  uint32_t car_u0 = 0, car_c = first_c, span_end = 0;
  for (uint32_t si = (!scalar && s[0].offset == 0.0 && n > 1) ? 1u : 0u; si < n; si += 32) {
    const uint32_t k = si + uint32_t(lane);
    const int ns = int(min(32u, n - si));
    uint32_t c1 = 0, u1 = 0;
    if (k < n) {
      c1 = rgba32_of(s[k].rgba64);
      u1 = uint32_t(round_to_int(s[k].offset * fWidth));
    }
    uint32_t u0 = __shfl_up_sync(0xFFFFFFFFu, u1, 1), c0 = __shfl_up_sync(0xFFFFFFFFu, c1, 1);
    if (lane == 0) { u0 = car_u0; c0 = car_c; }
    if (lane < ns) {
      LutSpan sp;
      sp.start = u0 >> 8;
      if (scalar) {                                     // interpolation.cpp, one stop
        const uint32_t i = (u1 >> 8) - (u0 >> 8);
        if (i == 0) c0 = c1;
        sp.count = i + 1u;
        sp.c0 = c0;
        sp.c1 = c1;
        if (c0 != c1 && sp.count > 1) {
          const uint32_t kMask = 0xFFu << 23;
          const int32_t div = int32_t(sp.count - 1u);
          sp.inc[0] = int32_t(((c1 << 7) & kMask) - ((c0 << 7) & kMask)) / div;
          sp.inc[1] = int32_t(((c1 << 15) & kMask) - ((c0 << 15) & kMask)) / div;
          sp.inc[2] = int32_t(((c1 << 23) & kMask) - ((c0 << 23) & kMask)) / div;
          sp.inc[3] = int32_t(((c1 >> 1) & kMask) - ((c0 >> 1) & kMask)) / div;
        }
      }
      else {                                            // interpolation_sse2.cpp and _avx2.cpp, one stop
        sp.count = (u1 >> 8) - (u0 >> 8);
        sp.c0 = c0;
        sp.c1 = c1;
        if (sp.count > 1) {
          const double scale = double(1 << 23) / double(int(sp.count));
          for (int ch = 0; ch < 4; ch++) {
            const int32_t cc = int32_t((c0 >> (8 * ch)) & 255u);
            const int32_t dd = int32_t((c1 >> (8 * ch)) & 255u) - cc;
            const double pv = double(dd) * scale;
            sp.inc[ch] = (pv > -2147483649.0 && pv < 2147483648.0) ? __double2int_rz(pv) : INT32_MIN;
            sp.pos[ch] = (uint32_t(cc) << 23) + (1u << 22);
          }
        }
      }
      spans[lane] = sp;
    }
    // carry the chunk's last stop
    car_u0 = __shfl_sync(0xFFFFFFFFu, u1, ns - 1);
    car_c = __shfl_sync(0xFFFFFFFFu, c1, ns - 1);
    __syncwarp();
    span_end = spans[ns - 1].start + spans[ns - 1].count + (scalar ? 0u : 1u);
    for (int j = 0; j < ns; j++) {
      if (scalar) lut_span_scalar(spans[j], lut, job.lut_size, lane);
      else lut_span_simd(spans[j], lut, job.lut_size, lane, avx2);
    }
    __syncwarp();
  }
  // the trailing fill is the last stop's colour; entry 0 is the first stop's
  const uint32_t tail = premul(car_c);
  for (uint32_t e = (span_end & ~31u) + uint32_t(lane); e < job.lut_size; e += 32)
    if (e >= span_end) lut[e] = tail;
  if (lane == 0) lut[0] = premul(first_c);
}

// ---------------------------------------------------------------------------------------------
// K1 - FP64 edge building. The reference's builder walks a command's figures sequentially, but
// the cells it produces depend only on the multiset of segments, and the segments of one line or
// curve depend only on that line's or curve's own points: clipping decisions come from the
// points' clip flags, the previous curve ends exactly on this one's first point, and the
// left/right border runs it accumulates are vertical lines at the clip box's x0/x1, whose cells
// add up the same whether consecutive runs are merged or not. So `classify` splits every
// analytic command into items (lines, curves, closing lines) and `edge_items` builds each item
// on its own thread with the reference's clipping builder, appending segments with batched
// atomics. An invalid point (NaN) makes the reference reject the whole command; here it marks the
// command invalid and binning drops it.
// ---------------------------------------------------------------------------------------------

enum : uint32_t { kCmdHasSegments = 1u, kCmdInvalid = 2u };

__device__ __forceinline__ void init_builder(eb::Builder& b, const DevCanvas& cv) {
  b.cx0 = 0.0; b.cy0 = 0.0; b.cx1 = double(cv.w) * 256.0; b.cy1 = double(cv.h) * 256.0;
  b.icx0 = eb::trunc_i(b.cx0); b.icx1 = eb::trunc_i(b.cx1);
  const double tol = 0.20 * 256.0;
  b.tol_sq = tol * tol;
  b.acc_x0_y0 = b.acc_x0_y1 = b.acc_x1_y0 = b.acc_x1_y1 = b.cy0;
  b.px = b.py = 0; b.psign = 0; b.pasc = false;
}

// work_counter words of the cubic and of the quadratic / conic curves
template<int DEG>
struct CurveWords {
  static constexpr uint32_t kCurves = DEG == 3 ? 2 : 21;     // curves of the curve list
  static constexpr uint32_t kPieces = DEG == 3 ? 23 : 25;    // their monotonic pieces
  static constexpr uint32_t kSafe = DEG == 3 ? 28 : 34;      // pieces the safe loop flattens
  static constexpr uint32_t kClip = kSafe + 1;               // the other ones
  static constexpr uint32_t kTreeQueue = kSafe + 2, kClipQueue = kSafe + 3;
  static constexpr uint32_t kHanded = DEG == 3 ? 38 : 39;    // subtrees of clipped pieces handed to the tree flattener
};
// Walks the figures of a command the way add_from_source does (edgebuilder_p.h:1032-1070), by a warp,
// 32 vertices at a time, and calls fn(kind, a, b, has) for every vertex's line, curve or closing line
// (at most one; all lanes call it, `has` says whether the lane's vertex has an item).
// What a vertex is depends on what came before it only through a state of four values - seeking a
// figure's move, expecting a command, one or two vertices of a curve still to pass - so each vertex is
// a function on the states (2 bits per state), and a scan of the functions' compositions gives every
// lane the state it starts from.
template<typename Fn>
__device__ __forceinline__ void for_each_item(const uint8_t* cmd, int n, int lane, Fn&& fn) {
  if (!cmd) {                                       // a polygon: one figure of lines
    for (int base = 0; base < n; base += 32) {
      const int i = base + lane;
      // vertex i's line ends at i; vertex 0 stands for the closing line
      fn(uint32_t(kItemLine), i ? i - 1 : n - 1, i, i < n);
    }
    return;
  }
  enum : uint32_t { kSeek = 0, kNext = 1, kPass1 = 2, kPass2 = 3 };
  uint32_t state = kSeek, conics_before = 0;        // conic commands among the 32 vertices before
  int start = 0;
  for (int base = 0; base < n; base += 32) {
    const int i = base + lane;
    const uint32_t c = i < n ? cmd[i] : 255u;
    const bool quad = c == 2u && i <= n - 2, cubic = c == 4u && i < n - 2, conic = c == 3u && i < n - 2;
    const uint32_t figure = c == 0u ? kNext : kSeek;     // a vertex that ends a figure may begin another
    const uint32_t next = c == 1u ? kNext : cubic ? kPass2 : (quad || conic) ? kPass1 : figure;
    uint32_t acc = i < n ? figure | (next << 2) | (kNext << 4) | (kPass1 << 6) : 0xE4u;   // past the end: unchanged
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t f = __shfl_up_sync(0xFFFFFFFFu, acc, o);      // first f, then acc
      const uint32_t both = ((acc >> (2u * (f & 3u))) & 3u) | (((acc >> (2u * ((f >> 2) & 3u))) & 3u) << 2) |
                            (((acc >> (2u * ((f >> 4) & 3u))) & 3u) << 4) | (((acc >> (2u * (f >> 6))) & 3u) << 6);
      if (lane >= o) acc = both;
    }
    const uint32_t before = __shfl_up_sync(0xFFFFFFFFu, acc, 1);
    const uint32_t st = lane ? (before >> (2u * state)) & 3u : state;
    const bool expects = st == kNext && i < n;
    const bool other = c != 1u && !quad && !cubic && !conic;       // ends the figure: its closing line
    const uint32_t starts = __ballot_sync(0xFFFFFFFFu, c == 0u && st <= kNext);
    const uint32_t conics = __ballot_sync(0xFFFFFFFFu, conic && st == kNext);
    const uint32_t starts_before = starts & ((1u << lane) - 1u);
    const int figure_start = starts_before ? base + 31 - __clz(starts_before) : start;
    // the point before a vertex is the vertex before it, but a conic ends on the vertex after its own
    const bool after_conic = lane >= 2 ? (conics >> (lane - 2)) & 1u : (conics_before >> (30 + lane)) & 1u;
    const int prev = after_conic ? i : i - 1;
    fn(cubic ? uint32_t(kItemCubic) : quad ? uint32_t(kItemQuad) : conic ? uint32_t(kItemConic) : uint32_t(kItemLine),
       prev, other ? figure_start : i, expects);
    if (starts) start = base + 31 - __clz(starts);
    conics_before = conics;
    state = (__shfl_sync(0xFFFFFFFFu, acc, 31) >> (2u * state)) & 3u;
  }
  // the last figure's closing line
  fn(uint32_t(kItemLine), n - 1, start, state == kNext && lane == 0);
}

// One warp per command (four in turn in frames of many commands): the finite check, then one item per
// line and curve. Lines go to the item list (edge_items_kernel); cubic curves to the front of the
// curve list and quadratic / conic curves to its back. A block counts its commands' items, takes
// room for all of them with one atomic per list and walks them again to write them. One thread per
// command, walking its vertices in turn, and three atomics a command: 20,000 curve paths 43 -> 28 us,
// 10,000 stroke outlines of 230 vertices 515 -> 99 us, the 395,000 commands of 512
// batch canvases 311 -> 260 us.
constexpr int kClassifyWarps = 8;
constexpr uint32_t kClassifyMax = 4;           // commands per warp

__global__ void __launch_bounds__(32 * kClassifyWarps) classify_kernel(FrameView f, uint32_t per_warp) {
  __shared__ uint3 room[kClassifyWarps * kClassifyMax];       // counts, then first places
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u, num_cmds = f.counts[kCntCmds];
  const uint32_t block_first = blockIdx.x * kClassifyWarps * per_warp;
  if (block_first >= num_cmds) return;                        // whole blocks leave together
  uint32_t whole = 0;                                         // bit k: the warp's command k is built whole
  for (uint32_t k = 0; k < per_warp; k++) {
    const uint32_t c = block_first + uint32_t(w) * per_warp + k;
    uint32_t lines = 0, cubics = 0, quads = 0;
    if (c < num_cmds && f.cmds[c].kind == kFillAnalytic) {
      const DevCmd& cmd = f.cmds[c];
      const int n = int(cmd.geom_count);
      const uint32_t geom = cmd.geom_first;
      if (lane == 0) {
        f.cmd_bbox[c] = make_int4(INT32_MAX, INT32_MAX, INT32_MIN, INT32_MIN);
        f.cmds_rw[c].status = 0u;
      }
      // A command with a non-finite transformed point is built whole, by one thread, exactly as the
      // reference builds it (its clip flags then depend on the order points are visited in). With
      // coordinates and matrix below 2^500 no transformed point overflows: only larger ones (or
      // infinities and NaNs) are transformed to see.
      const DevXform& xf = f.xforms[cmd.xform];
      const double2* xy = reinterpret_cast<const double2*>(f.verts) + geom;
      auto large = [](double v) { return ((uint32_t(__double2hiint(v)) >> 20) & 0x7FFu) >= 1023u + 500u; };
      bool finite = true;
      const bool large_m = large(xf.m[0]) | large(xf.m[1]) | large(xf.m[2]) | large(xf.m[3]) | large(xf.m[4]) | large(xf.m[5]);
      for (int i = lane; i < n; i += 32) {
        const double2 p = xy[i];
        if (large_m | large(p.x) | large(p.y)) {
          double tx, ty;
          if (xf.affine) { tx = p.x * xf.m[0] + p.y * xf.m[2] + xf.m[4]; ty = p.x * xf.m[1] + p.y * xf.m[3] + xf.m[5]; }
          else { tx = p.x * xf.m[0] + xf.m[4]; ty = p.y * xf.m[3] + xf.m[5]; }
          finite &= isfinite(tx) & isfinite(ty);
        }
      }
      if (!__all_sync(0xFFFFFFFFu, finite)) {
        whole |= 1u << k;
        lines = 1;
      }
      else {
        for_each_item(cmd.geom == kGeomPath ? f.path_cmds + geom : nullptr, n, lane, [&](uint32_t kind, int, int, bool has) {
          lines += uint32_t(__popc(__ballot_sync(0xFFFFFFFFu, has && kind == kItemLine)));
          cubics += uint32_t(__popc(__ballot_sync(0xFFFFFFFFu, has && kind == kItemCubic)));
          quads += uint32_t(__popc(__ballot_sync(0xFFFFFFFFu, has && (kind == kItemQuad || kind == kItemConic))));
        });
      }
    }
    if (lane == 0) room[uint32_t(w) * per_warp + k] = make_uint3(lines, cubics, quads);
  }
  __syncthreads();
  if (w == 0) {
    const bool on = uint32_t(lane) < kClassifyWarps * per_warp;
    const uint3 mine = on ? room[lane] : make_uint3(0u, 0u, 0u);
    uint3 sum = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, sum.x, o), y = __shfl_up_sync(0xFFFFFFFFu, sum.y, o),
                     z = __shfl_up_sync(0xFFFFFFFFu, sum.z, o);
      if (lane >= o) { sum.x += x; sum.y += y; sum.z += z; }
    }
    uint32_t bx = 0, by = 0, bz = 0;
    if (lane == 31) {
      if (sum.x) bx = atomicAdd(f.work_counter + 1, sum.x);
      if (sum.y) by = atomicAdd(f.work_counter + CurveWords<3>::kCurves, sum.y);
      if (sum.z) bz = atomicAdd(f.work_counter + CurveWords<2>::kCurves, sum.z);
      // cubics fill the curve list from the front and quadratics from the back: together, and each
      // list on its own, they must fit (the bound is one item per vertex)
      if (bx + sum.x > f.item_capacity || by + sum.y > f.item_capacity || bz + sum.z > f.item_capacity)
        atomicOr(f.error_flags, kErrItems);
    }
    bx = __shfl_sync(0xFFFFFFFFu, bx, 31);
    by = __shfl_sync(0xFFFFFFFFu, by, 31);
    bz = __shfl_sync(0xFFFFFFFFu, bz, 31);
    if (on) room[lane] = make_uint3(bx + sum.x - mine.x, by + sum.y - mine.y, bz + sum.z - mine.z);
  }
  __syncthreads();
  for (uint32_t k = 0; k < per_warp; k++) {
    const uint32_t c = block_first + uint32_t(w) * per_warp + k;
    if (c >= num_cmds || f.cmds[c].kind != kFillAnalytic) continue;
    uint3 at = room[uint32_t(w) * per_warp + k];
    if ((whole >> k) & 1u) {
      if (lane == 0 && at.x < f.item_capacity) f.items[at.x] = DevItem{c, kItemWhole, 0u, 0u};
      continue;
    }
    const DevCmd& cmd = f.cmds[c];
    for_each_item(cmd.geom == kGeomPath ? f.path_cmds + cmd.geom_first : nullptr, int(cmd.geom_count), lane,
                  [&](uint32_t kind, int a, int b, bool has) {
      const uint32_t l = __ballot_sync(0xFFFFFFFFu, has && kind == kItemLine);
      const uint32_t cu = __ballot_sync(0xFFFFFFFFu, has && kind == kItemCubic);
      const uint32_t q = __ballot_sync(0xFFFFFFFFu, has && (kind == kItemQuad || kind == kItemConic));
      if (has) {
        const DevItem it{c, kind, uint32_t(a), uint32_t(b)};
        if (kind == kItemLine) {
          const uint32_t at_l = at.x + uint32_t(__popc(l & lt));
          if (at_l < f.item_capacity) f.items[at_l] = it;
        }
        else if (kind == kItemCubic) {
          const uint32_t at_c = at.y + uint32_t(__popc(cu & lt));
          if (at_c < f.item_capacity) f.curve_items[at_c] = it;
        }
        else {
          const uint32_t at_q = at.z + uint32_t(__popc(q & lt));
          if (at_q < f.item_capacity) f.curve_items[f.item_capacity - 1u - at_q] = it;
        }
      }
      at.x += uint32_t(__popc(l));
      at.y += uint32_t(__popc(cu));
      at.z += uint32_t(__popc(q));
    });
  }
}

// The end of a curve's or piece's builder: border runs emitted, segments flushed, the command's
// bbox, status and binning bound updated.
__device__ __forceinline__ void finish_curve(FrameView& f, eb::Builder& b, uint32_t cmd, uint32_t& rows) {
  b.done();
  b.sink.flush();
  if (b.sink.n) {
    int4* bb = f.cmd_bbox + cmd;
    atomicMin(&bb->x, b.sink.xmin);
    atomicMin(&bb->y, b.sink.ymin);
    atomicMax(&bb->z, b.sink.xmax);
    atomicMax(&bb->w, b.sink.ymax);
    atomicOr(&f.cmds_rw[cmd].status, kCmdHasSegments);
    rows += b.sink.rows;
  }
}

// The lanes' subdivision stacks live in local memory with the top entry in registers
// (eb::CachedStack). Holding the next eight entries in shared memory instead measured slower on
// the batched workload (piece kernel 10.8 -> 14.2 ms): the shared-memory carve-out shrinks the L1
// that the stacks' and the segment sinks' local memory hits in.
constexpr int kCurveThreads = 128;
constexpr uint32_t kSplitBlocksPerSM = 8;      // of each kind of curve
// Idle lanes a warp waits for before it takes new pieces: each refill's set-up costs the warp its
// FP64 instructions whatever the number of lanes refilled. On the batched workload 24 and 28
// measured 246-248 ms per step, 16 and 20 250 ms, 32 251 ms, 8 257 ms and 4 259 ms.
constexpr uint32_t kPieceRefillLanes = 24;
// ... and lanes at a leaf it waits for before it clips and emits them (8, 12, 16 and 20 measured 18.78,
// 18.70, 18.65 and 18.58 ms on the same canvases, 1.827, 1.823, 1.822 and 1.829 ms on 20,000 curve paths).
constexpr uint32_t kPieceLeafLanes = 16;

// Curves in three kernels, each with the cubic curves in the first half of its blocks and the
// quadratic and conic ones in the second, so that neither kind's tail waits for the other's and a
// frame without one kind loses blocks that leave at once, not launches. (Not alternating blocks: the
// even ones go to one half of the SMs, and a frame of cubics alone took twice as long.)
// curve_split_kernel does curve_to's set-up - transform, clip flags, a curve entirely on one side of the
// clip box, the split into monotonic pieces - and writes the pieces. edge_pieces_kernel flattens the clipped
// pieces lane-scheduled; edge_tree_kernel then flattens what no clip touches. A piece is built by its own
// builder: the border runs a curve accumulates are vertical lines at the clip box's x0/x1 whose cells add
// up the same whether the runs of consecutive pieces are merged or not.
//
// In curve_split_kernel a warp takes up to 32 curves and its lanes share their work: a lane per curve for
// the transform, the polynomial and the sorting of its cuts, a lane per (curve, candidate set) for
// the roots, a lane per piece for the pieces, whatever curve they belong to. A thread per curve ran the
// piece loop as often as the warp's most divided curve asks (8 times for 3.4 pieces on average), and in a
// small frame went through all of it alone. Frames with few curves give each warp fewer. Bound: the FP64
// pipe. 512 canvases of the batch 2.13 -> 1.77 ms, 20,000 curve paths 0.22 -> 0.19, a 64x64 icon 0.048 ->
// 0.016 (4, 5, 6 and 8 blocks an SM measured alike).
constexpr int kSplitWarps = 4;

// A kind's part of the piece list: the pieces the safe loop flattens from its front, the clipped ones from
// its back. The cubic curves' part takes the most pieces they can have, 8 a curve of three vertices; of
// three entries per vertex that leaves two per vertex and more for the quadratic and conic ones, which
// have at most 3 pieces in two vertices.
struct PieceList {
  uint32_t* at;
  uint32_t n;
};
template<int DEG>
__device__ __forceinline__ PieceList piece_list(const FrameView& f) {
  const unsigned long long most = (eb::kCubicCands + 1ull) * min(f.work_counter[CurveWords<3>::kCurves], f.item_capacity);
  const uint32_t cubic = most < f.piece_capacity ? uint32_t(most) : f.piece_capacity;
  return DEG == 3 ? PieceList{f.piece_list, cubic} : PieceList{f.piece_list + cubic, f.piece_capacity - cubic};
}

template<int DEG>
struct SplitShared {
  static constexpr int kCands = DEG == 3 ? eb::kCubicCands : 2;
  double pt[2 * (DEG + 1)][32];      // the curves' points
  double poly[2 * DEG][32];          // their polynomials without the constant term (the first point)
  double t[kCands][32];              // their candidates, then their cuts in order
  uint32_t end[32];                  // pieces of the curves up to and with this one
  uint32_t cuts[32];
  uint32_t cmd[32];
  uint32_t any[32];
};

// One vertical run at a side of the clip box per lane that has one (Builder::emit_left / emit_right of a
// builder that accumulated y0 to y1): segment, bounds, binning bound.
__device__ __forceinline__ void emit_runs(FrameView& f, bool has, int x, double y0, double y1, uint32_t cmd, int lane, uint32_t& rows) {
  const int a = has ? eb::trunc_i(y0) : 0, b = has ? eb::trunc_i(y1) : 0;
  has = a != b;
  const uint32_t set = __ballot_sync(0xFFFFFFFFu, has);
  if (!set) return;
  uint32_t base = 0;
  if (lane == __ffs(set) - 1) base = atomicAdd(f.totals + 0, uint32_t(__popc(set)));
  base = __shfl_sync(0xFFFFFFFFu, base, __ffs(set) - 1) + uint32_t(__popc(set & ((1u << lane) - 1u)));
  if (!has) return;
  const int ya = min(a, b), yb = max(a, b);
  if (base < f.seg_capacity) {
    f.segs[base] = DevSeg{x, ya, x, yb};
    f.seg_meta[base] = (cmd << 1) | uint32_t(a > b);
  }
  const uint32_t strips = (uint32_t((yb - 1) >> 8) >> kStripShift) - (uint32_t(ya >> 8) >> kStripShift) + 1u;
  rows += uint32_t(((((x + 256) >> 8) + 1) >> kTileShift) - (((x - 256) >> 8) >> kTileShift) + 1) + 3u * strips;
  int4* bb = f.cmd_bbox + cmd;
  atomicMin(&bb->x, x);
  atomicMin(&bb->y, ya);
  atomicMax(&bb->z, x);
  atomicMax(&bb->w, yb);
  atomicOr(&f.cmds_rw[cmd].status, kCmdHasSegments);
}

template<int DEG>
__device__ __forceinline__ eb::Poly<DEG> shared_poly(const SplitShared<DEG>& sh, int j) {
  auto term = [&](int i) { return eb::Pt{sh.poly[2 * i][j], sh.poly[2 * i + 1][j]}; };
  const eb::Pt c0{sh.pt[0][j], sh.pt[1][j]};
  if constexpr (DEG == 3) return eb::Poly<3>{term(0), term(1), term(2), c0};
  else return eb::Poly<2>{term(0), term(1), c0};
}

template<int DEG>
__device__ void split_curves(FrameView& f, SplitShared<DEG>& sh, uint32_t block, uint32_t blocks) {
  using W = CurveWords<DEG>;
  constexpr int kCands = SplitShared<DEG>::kCands;
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t n_cubic = min(f.work_counter[CurveWords<3>::kCurves], f.item_capacity);
  const uint32_t n_items = DEG == 3 ? n_cubic : min(f.work_counter[CurveWords<2>::kCurves], f.item_capacity - n_cubic);
  const uint32_t warps = blocks * kSplitWarps;
  const uint32_t share = min(32u, (n_items + warps - 1u) / warps);      // curves a warp takes at a time
  const PieceList list = piece_list<DEG>(f);
  uint32_t rows = 0;
  for (uint32_t first = (block * kSplitWarps + (threadIdx.x >> 5)) * share; first < n_items; first += warps * share) {
    const int count = int(min(share, n_items - first));
    // a lane per curve: transform and clip flags (LaneCurve::prepare's set-up)
    uint32_t pieces = 0, cmd_i = 0;
    double run0 = 0.0, run1 = 0.0;
    int run_x = 0;
    bool run = false;
    if (lane < count) {
      const DevItem it = f.curve_items[DEG == 3 ? first + uint32_t(lane) : f.item_capacity - 1u - (first + uint32_t(lane))];
      const DevCmd& cmd = f.cmds[it.cmd];
      const DevXform& xf = f.xforms[cmd.xform];
      eb::Builder b;
      init_builder(b, f.canvases[cmd.canvas]);
      eb::Src src;
      src.xy = f.verts + 2ull * cmd.geom_first;
      src.affine = xf.affine != 0;
      src.m00 = xf.m[0]; src.m01 = xf.m[1]; src.m10 = xf.m[2]; src.m11 = xf.m[3]; src.m20 = xf.m[4]; src.m21 = xf.m[5];
      eb::Pt pts[DEG + 1];
      pts[0] = src.tf(int(it.a));
      pts[1] = src.tf(int(it.b));
      if (DEG == 3) pts[2] = src.tf(int(it.b) + 1);
      pts[DEG] = src.tf(int(it.b) + (DEG == 3 || it.kind == kItemConic ? 2 : 1));
      cmd_i = it.cmd;
      uint32_t common = 15u, any = 0;
#pragma unroll
      for (int i = 0; i <= DEG; i++) {
        const uint32_t fl = b.fxy(pts[i]);
        common &= fl;
        any |= fl;
        sh.pt[2 * i][lane] = pts[i].x;
        sh.pt[2 * i + 1][lane] = pts[i].y;
      }
      sh.cmd[lane] = cmd_i;
      sh.any[lane] = any;
      if (common) {
        if (!(common & (eb::CF_Y0 | eb::CF_Y1))) {
          run = true;
          run_x = (common & eb::CF_X0) ? b.icx0 : b.icx1;
          run0 = eb::dclamp(pts[0].y, b.cy0, b.cy1);
          run1 = eb::dclamp(pts[DEG].y, b.cy0, b.cy1);
        }
      }
      else {
        pieces = 1;
        eb::Pt terms[DEG];
        if constexpr (DEG == 3) {
          const eb::Poly<3> p = eb::curve_poly(pts[0], pts[1], pts[2], pts[3]);
          terms[0] = p.a; terms[1] = p.b; terms[2] = p.c;
        }
        else {
          const eb::Poly<2> p = eb::curve_poly(pts[0], pts[1], pts[2]);
          terms[0] = p.a; terms[1] = p.b;
        }
#pragma unroll
        for (int i = 0; i < DEG; i++) { sh.poly[2 * i][lane] = terms[i].x; sh.poly[2 * i + 1][lane] = terms[i].y; }
      }
    }
    emit_runs(f, run, run_x, run0, run1, cmd_i, lane, rows);
    const uint32_t live = __ballot_sync(0xFFFFFFFFu, pieces != 0u);
    if (!live) continue;
    __syncwarp();
    // a lane per (curve, candidate set)
    constexpr int kSets = DEG == 3 ? eb::kCubicSets : 2;
    for (int task = lane; task < kSets * count; task += 32) {
      const int set = task / count, j = task - set * count;
      if (!((live >> j) & 1u)) continue;
      if constexpr (DEG == 3) {
        double c[2];
        eb::cubic_candidates(shared_poly<3>(sh, j), set, c);
        if (set == 0) sh.t[0][j] = c[0];
        else { sh.t[2 * set - 1][j] = c[0]; sh.t[2 * set][j] = c[1]; }
      }
      else {
        const double a = sh.pt[set][j], b = sh.pt[2 + set][j], c = sh.pt[4 + set][j];
        sh.t[set][j] = (a - b) / (a - b * 2.0 + c);
      }
    }
    __syncwarp();
    // a lane per curve: its cuts in order, each once
    if (pieces) {
      uint32_t n = 0;
      if constexpr (DEG == 3) {
        // positive doubles order like their bits
        unsigned long long v[kCands];
#pragma unroll
        for (int k = 0; k < kCands; k++) v[k] = (unsigned long long)__double_as_longlong(sh.t[k][lane]);
#pragma unroll
        for (int i = 1; i < kCands; i++) {
#pragma unroll
          for (int k = i; k > 0; k--) {
            const unsigned long long lo = min(v[k - 1], v[k]), hi = max(v[k - 1], v[k]);
            v[k - 1] = lo;
            v[k] = hi;
          }
        }
        const unsigned long long none = (unsigned long long)__double_as_longlong(eb::kNoCut);
        unsigned long long last = 0;
#pragma unroll
        for (int k = 0; k < kCands; k++) {
          if (v[k] != none && v[k] != last) { sh.t[n][lane] = __longlong_as_double((long long)v[k]); n++; }
          last = v[k];
        }
      }
      else {
        const double ex = sh.t[0][lane], ey = sh.t[1][lane];
        const double t0 = eb::dmin(ex, ey), t1 = eb::dmax(ex, ey);
        if ((t0 > 0.0) & (t0 < 1.0)) sh.t[n++][lane] = t0;
        if ((t1 > eb::dmax(t0, 0.0)) & (t1 < 1.0)) sh.t[n++][lane] = t1;
      }
      sh.cuts[lane] = n;
      pieces = n + 1u;
    }
    uint32_t end = pieces;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, end, o);
      if (lane >= o) end += v;
    }
    sh.end[lane] = end;
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, end, 31);
    __syncwarp();
    // a lane per piece; its first point is the last one of the piece before it, on the lane below or
    // of the last lane's piece of the step before
    eb::Pt carry{0.0, 0.0};
    for (uint32_t at0 = 0; at0 < total; at0 += 32) {
      const uint32_t at = at0 + uint32_t(lane);
      const bool on = at < total;
      int j = 0;
      if (on) {
#pragma unroll
        for (int step = 16; step; step >>= 1)
          if (sh.end[j + step - 1] <= at) j += step;
      }
      eb::Pt out[DEG + 1];
      bool keep = false, safe = false;
      run = false;
      cmd_i = sh.cmd[j];
      const uint32_t any = sh.any[j];
      const uint32_t n = on ? sh.cuts[j] : 0u, k = on ? at - (j ? sh.end[j - 1] : 0u) : 0u;
      const eb::Poly<DEG> p = shared_poly<DEG>(sh, j);
      const double t1 = k < n ? sh.t[k][j] : 1.0;
      eb::Pt to{sh.pt[2 * DEG][j], sh.pt[2 * DEG + 1][j]};
      if (k < n) to = eb::poly_point(p, t1);
      eb::Pt from{__shfl_up_sync(0xFFFFFFFFu, to.x, 1), __shfl_up_sync(0xFFFFFFFFu, to.y, 1)};
      if (lane == 0) from = carry;
      carry = eb::Pt{__shfl_sync(0xFFFFFFFFu, to.x, 31), __shfl_sync(0xFFFFFFFFu, to.y, 31)};
      if (k == 0) from = eb::Pt{sh.pt[0][j], sh.pt[1][j]};
      if (on) {
        if (n == 0) {
#pragma unroll
          for (int i = 0; i <= DEG; i++) out[i] = eb::Pt{sh.pt[2 * i][j], sh.pt[2 * i + 1][j]};
        }
        else {
          eb::poly_piece(p, k ? sh.t[k - 1][j] : 0.0, t1, from, to, out);
        }
        eb::Builder b;
        init_builder(b, f.canvases[f.cmds[cmd_i].canvas]);
        keep = true;
        if (any) {
          // pieces outside the clip box end here, with at most a run at its side
          uint32_t sign;
          const eb::PieceOutside where = eb::piece_outside(out, DEG, b, run0, run1, sign);
          keep = where == eb::kCrosses;
          run = where >= eb::kLeftRun;
          run_x = where == eb::kLeftRun ? b.icx0 : b.icx1;
          if (sign) { const double t = run0; run0 = run1; run1 = t; }
        }
        safe = keep && eb::piece_flattens_safe(out, DEG, any, b);
      }
      emit_runs(f, run, run_x, run0, run1, cmd_i, lane, rows);
      // one atomic per step for the pieces, the safe ones (listed from the front of the kind's list) and
      // the others (from its back)
      const uint32_t kept = __ballot_sync(0xFFFFFFFFu, keep), safes = __ballot_sync(0xFFFFFFFFu, safe);
      const uint32_t clips = kept & ~safes;
      if (!kept) continue;
      uint32_t place = 0;
      if (lane == 0) place = atomicAdd(f.work_counter + W::kPieces, uint32_t(__popc(kept)));
      if (lane == 1 && safes) place = atomicAdd(f.work_counter + W::kSafe, uint32_t(__popc(safes)));
      if (lane == 2 && clips) place = atomicAdd(f.work_counter + W::kClip, uint32_t(__popc(clips)));
      const uint32_t base = __shfl_sync(0xFFFFFFFFu, place, 0), bs = __shfl_sync(0xFFFFFFFFu, place, 1),
                     bc = __shfl_sync(0xFFFFFFFFu, place, 2);
      if (keep) {
        const uint32_t idx = base + uint32_t(__popc(kept & lt));
        const uint32_t li = safe ? bs + uint32_t(__popc(safes & lt)) : bc + uint32_t(__popc(clips & lt));
        if (idx >= f.piece_capacity || li >= list.n) {
          atomicOr(f.error_flags, kErrPieces);
        }
        else {
          DevPiece pc;
#pragma unroll
          for (int i = 0; i <= DEG; i++) pc.p[i] = make_double2(out[i].x, out[i].y);
          pc.cmd = cmd_i;
          pc.any = any;
          pc.node = 0u;
          const uint32_t to = DEG == 3 ? idx : f.piece_capacity - 1u - idx;
          f.pieces[to] = pc;
          list.at[safe ? li : list.n - 1u - li] = to;
        }
      }
    }
    __syncwarp();
  }
  rows = __reduce_add_sync(0xFFFFFFFFu, rows);
  if (lane == 0 && rows) atomicAdd(f.totals + 1, rows);
}

__global__ void __launch_bounds__(32 * kSplitWarps, kSplitBlocksPerSM) curve_split_kernel(FrameView f) {
  __shared__ SplitShared<3> shared[kSplitWarps];
  const uint32_t half = gridDim.x / 2u;
  const int w = threadIdx.x >> 5;
  if (blockIdx.x >= half) split_curves<2>(f, reinterpret_cast<SplitShared<2>&>(shared[w]), blockIdx.x - half, half);
  else split_curves<3>(f, shared[w], blockIdx.x, half);
}

// The clipped pieces: the clipping state machine, one step of a lane's piece per iteration of a
// warp-wide loop. Only the nodes on the way to a clip are walked here: a subtree inside the clip box
// is handed to the tree flattener, as a piece in the gap between the cubic pieces (from the front of
// the piece array) and the others (from its back), while there is room (half of the gap each). A
// clipped piece then costs its lane some seven steps on average, not one per leaf. Bound: latency - of instruction
// fetches, every warp being somewhere else in the state machine, then FP64 - with 7 to 9 of 32 lanes active. Against flattening every leaf here, one kernel per kind of curve, all
// quadratic pieces included: large shapes on 1023x767 0.65 -> 0.06 ms (the tree flattener 0.07 ->
// 0.04), 10,000 stroked paths (quadratic outlines) 0.94 -> 0.06 (tree 0.03 -> 0.30), a 64x64 icon
// 0.10 -> 0.04, 20,000 curve paths on 1920x1080 0.17 -> 0.13, 512 canvases of the batch 3.04 -> 2.12
// (there mostly because pieces outside the box end in curve_split_kernel, 1.92 -> 2.16).

// The gap's entries for handed-over subtrees of one kind.
__device__ __forceinline__ uint32_t handed_room(const FrameView& f, uint32_t n_cubic, uint32_t n_quad) {
  return n_cubic + n_quad < f.piece_capacity ? (f.piece_capacity - n_cubic - n_quad) / 2u : 0u;
}

// Pieces a warp takes at a time: all its idle lanes can hold, or, in frames whose pieces are fewer
// than the launch's lanes, an even share of them once all its lanes are idle, so that every warp has
// some.
__device__ __forceinline__ uint32_t piece_share(uint32_t n_items, uint32_t blocks) {
  const uint32_t warps = blocks * (kCurveThreads / 32);
  return min(32u, (n_items + warps - 1u) / warps);
}

template<int DEG>
__device__ void flatten_clipped(FrameView& f, uint32_t blocks) {
  using W = CurveWords<DEG>;
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t n_cubic = min(f.work_counter[CurveWords<3>::kPieces], f.piece_capacity);
  const uint32_t n_quad = min(f.work_counter[CurveWords<2>::kPieces], f.piece_capacity - n_cubic);
  const uint32_t n_mine = DEG == 3 ? n_cubic : n_quad;
  const PieceList list = piece_list<DEG>(f);
  const uint32_t n_items = min(f.work_counter[W::kClip], min(n_mine, list.n));
  const uint32_t room = handed_room(f, n_cubic, n_quad), share = piece_share(n_items, blocks);
  uint32_t* queue = f.work_counter + W::kClipQueue;
  using Lane = eb::LaneCurve<DEG, eb::CachedStack<DEG>>;
  eb::Builder b;
  Lane lc;
  enum Phase : int { kIdle = 0, kStepping, kAtLeaf, kDone };
  int phase = kIdle;
  bool exhausted = false;
  uint32_t cur = 0, rows = 0;
  // few pieces: no lane waits for others
  const uint32_t refill_lanes = share == 32u ? kPieceRefillLanes : 33u, leaf_lanes = share == 32u ? kPieceLeafLanes : 1u;

  for (;;) {
    // hand the next pieces of the list to the idle lanes (one atomic per warp), once enough lanes
    // are idle that the set-up's and the ending's instructions serve several pieces at once
    const uint32_t want = __ballot_sync(0xFFFFFFFFu, phase == kDone || (phase == kIdle && !exhausted));
    const bool none = !__any_sync(0xFFFFFFFFu, phase == kStepping || phase == kAtLeaf);
    if (want && (uint32_t(__popc(want)) >= refill_lanes || none)) {
      if (phase == kDone) {
        finish_curve(f, b, cur, rows);
        phase = kIdle;
      }
      const int leader = __ffs(want) - 1;
      const uint32_t take = none ? min(uint32_t(__popc(want)), share) : uint32_t(__popc(want));
      uint32_t base = 0;
      if (lane == leader) base = atomicAdd(queue, take);
      base = __shfl_sync(0xFFFFFFFFu, base, leader);
      if (base >= n_items) exhausted = true;
      const uint32_t rank = uint32_t(__popc(want & lt));
      if (((want >> lane) & 1u) && !exhausted && rank < take) {
        const uint32_t t = base + rank;
        if (t >= n_items) {
          exhausted = true;
        }
        else {
          const uint32_t pi = list.at[list.n - 1u - t];
          // a list entry is written only for a piece that fit in the piece array; with a frame
          // that overflowed it (reported by curve_split), an entry may be stale: the lane then
          // stays idle and takes another piece
          if (DEG == 3 ? pi < n_cubic : (pi < f.piece_capacity && pi >= f.piece_capacity - n_quad)) {
            const DevPiece pc = f.pieces[pi];
            cur = pc.cmd;
            init_builder(b, f.canvases[f.cmds[cur].canvas]);
            b.sink.init(f.segs, f.seg_meta, f.totals + 0, f.seg_capacity, cur);
            eb::Pt pts[DEG + 1];
#pragma unroll
            for (int i = 0; i <= DEG; i++) pts[i] = eb::Pt{pc.p[i].x, pc.p[i].y};
            phase = lc.begin_piece(b, pts, pc.any) ? kStepping : kDone;
          }
        }
      }
    }
    if (__all_sync(0xFFFFFFFFu, phase == kIdle && exhausted)) break;   // the list is exhausted
    bool hand = false;
    if (phase == kStepping) {
      const int r = lc.template step<true>(b);
      if (r == Lane::kStepLeaf) phase = kAtLeaf;
      hand = r == Lane::kStepHand;
    }
    // leaves, where the clips are: together, when enough lanes stand at one or no lane can step on
    const uint32_t leaves = __ballot_sync(0xFFFFFFFFu, phase == kAtLeaf);
    if (leaves && (uint32_t(__popc(leaves)) >= leaf_lanes || !__any_sync(0xFFFFFFFFu, phase == kStepping))) {
      if (phase == kAtLeaf) {
        lc.leaf(b);
        phase = kStepping;
      }
    }
    const uint32_t hands = __ballot_sync(0xFFFFFFFFu, hand);
    if (hands) {
      const int leader = __ffs(hands) - 1;
      uint32_t at = 0;
      if (lane == leader) at = atomicAdd(f.work_counter + W::kHanded, uint32_t(__popc(hands)));
      at = __shfl_sync(0xFFFFFFFFu, at, leader) + uint32_t(__popc(hands & lt));
      if (hand) {
        if (at < room) {
          DevPiece pc;
#pragma unroll
          for (int i = 0; i <= DEG; i++) pc.p[i] = make_double2(lc.mc.p[i].x, lc.mc.p[i].y);
          pc.cmd = cur;
          pc.any = 0;
          pc.node = kPieceNode | (lc.sign << 8) | uint32_t(lc.mc.sp);
          f.pieces[DEG == 3 ? n_cubic + at : f.piece_capacity - 1u - n_quad - at] = pc;
          // the subtree's segments count towards this command's bounds where they are emitted
          lc.skip_node(b);
        }
        else {
          lc.split_node(b);
        }
      }
    }
    if (phase == kStepping && lc.state == eb::kLsDone && !lc.next_piece(b, true)) phase = kDone;
  }
  rows = __reduce_add_sync(0xFFFFFFFFu, rows);
  if (lane == 0 && rows) atomicAdd(f.totals + 1, rows);
}

// `few`: the blocks of each kind that work while the pieces are no more than four per lane of them;
// more pieces bring in the launch's other blocks. Eight blocks an SM measured 18.20 ms against three's
// 18.70 on 512 canvases of the batch (a million clipped pieces), but 1.862 against 1.823 on 20,000
// curve paths (20,000 pieces).
__global__ void __launch_bounds__(kCurveThreads) edge_pieces_kernel(FrameView f, uint32_t few) {
  const uint32_t half = gridDim.x / 2u, block = blockIdx.x % half;
  const bool quads = blockIdx.x >= half;
  const uint32_t n = f.work_counter[quads ? CurveWords<2>::kClip : CurveWords<3>::kClip];
  const uint32_t blocks = min(half, max(few, n / (4u * kCurveThreads)));
  if (block >= blocks) return;
  if (quads) flatten_clipped<2>(f, blocks);
  else flatten_clipped<3>(f, blocks);
}

// The pieces the safe loop flattens (those of curves inside the clip box, and the inside pieces of
// clipped curves: eb::piece_flattens_safe) and the subtrees edge_pieces_kernel handed over, flattened as subdivision trees (eb::TreeNode)
// whose nodes the lanes of a warp share. A lane splits its node, goes on with the left half and keeps the
// right half on its own stack, unless a lane of the warp is out of work: then the right half goes
// to that lane through shared memory. So lanes do not sit idle while other lanes' trees still have
// nodes, and the FP64 instructions (whose cost to the pipe does not depend on the active lanes)
// serve more of them. The segments are those of the loop flattener, in another order; they are
// appended for the warp with one atomic per step, and each lane accumulates the command bounds
// finish_curve would for the run of segments it emits for one command. Bound: the FP64 pipe (a split's
// 12 additions) and the latency of the exchange. The flatness test is decided in 32 bits
// (eb::flat_guess) for all but one node in a thousand: 2.35 -> 1.68 ms on 512 canvases of the batch,
// 0.32 -> 0.23 on 20,000 curve paths.

// Idle lanes a warp of the tree flattener waits for before it takes new pieces, and its blocks per
// SM. With the 32-bit flatness test 3 blocks and refills of 16 lanes measured 19.42 ms on 512 canvases
// of the batch and 1.863 ms on 20,000 curve paths, 4 and 8 19.36 and 1.851, 4 and 16 19.24 and 1.835,
// 5 and 16 19.18 and 1.836, 5 and 24 19.18 and 1.833.
constexpr int kTreeRefillLanes = 16;
constexpr int kTreeBlocksPerSM = 5;     // of each kind of curve

template<int DEG>
struct alignas(16) TreeXchg {
  double x[DEG + 1], y[DEG + 1];
  uint32_t cmd, level, sign, pad;
};

template<int DEG>
__device__ void flatten_trees(FrameView& f, TreeXchg<DEG>* xchg, uint32_t blocks) {
  using W = CurveWords<DEG>;
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t n_cubic = min(f.work_counter[CurveWords<3>::kPieces], f.piece_capacity);
  const uint32_t n_quad = min(f.work_counter[CurveWords<2>::kPieces], f.piece_capacity - n_cubic);
  const PieceList list = piece_list<DEG>(f);
  const uint32_t n_safe = min(f.work_counter[W::kSafe], min(DEG == 3 ? n_cubic : n_quad, list.n));
  const uint32_t n_items = n_safe + min(f.work_counter[W::kHanded], handed_room(f, n_cubic, n_quad));
  const uint32_t share = piece_share(n_items, blocks);
  uint32_t* queue = f.work_counter + W::kTreeQueue;
  const double tol = 0.20 * 256.0;
  const double tol_sq = tol * tol;                    // init_builder's
  eb::TreeNode<DEG> cur;
  eb::TreeNode<DEG> stack[eb::kStackLevels];
  int nst = 0;
  uint32_t cmd = 0, sign = 0;
  bool busy = false, exhausted = false;
  // bounds of the segments emitted for command acc_cmd since the last flush
  uint32_t acc_cmd = 0xFFFFFFFFu, acc_rows = 0, rows = 0;
  int xmin = INT32_MAX, ymin = INT32_MAX, xmax = INT32_MIN, ymax = INT32_MIN;
  auto flush_bounds = [&]() {
    if (acc_cmd == 0xFFFFFFFFu) return;
    int4* bb = f.cmd_bbox + acc_cmd;
    atomicMin(&bb->x, xmin);
    atomicMin(&bb->y, ymin);
    atomicMax(&bb->z, xmax);
    atomicMax(&bb->w, ymax);
    atomicOr(&f.cmds_rw[acc_cmd].status, kCmdHasSegments);
    rows += acc_rows;
    acc_cmd = 0xFFFFFFFFu;
    acc_rows = 0;
    xmin = ymin = INT32_MAX;
    xmax = ymax = INT32_MIN;
  };

  for (;;) {
    // new pieces for the idle lanes, as edge_pieces_kernel takes them
    const uint32_t want = __ballot_sync(0xFFFFFFFFu, !busy && !exhausted);
    const bool none = !__any_sync(0xFFFFFFFFu, busy);
    if (want && ((share == 32u && __popc(want) >= kTreeRefillLanes) || none)) {
      const int leader = __ffs(want) - 1;
      const uint32_t take = none ? min(uint32_t(__popc(want)), share) : uint32_t(__popc(want));
      uint32_t base = 0;
      if (lane == leader) base = atomicAdd(queue, take);
      base = __shfl_sync(0xFFFFFFFFu, base, leader);
      if (base >= n_items) exhausted = true;
      const uint32_t rank = uint32_t(__popc(want & lt));
      if (!busy && !exhausted && rank < take) {
        const uint32_t t = base + rank;
        if (t >= n_items) {
          exhausted = true;
        }
        else {
          const uint32_t e = t - n_safe;         // a handed-over subtree when t >= n_safe
          const uint32_t pi = t < n_safe ? list.at[t] : DEG == 3 ? n_cubic + e : f.piece_capacity - 1u - n_quad - e;
          // an entry of a piece that did not fit in the piece array (the frame fails) is skipped
          if (t >= n_safe || (DEG == 3 ? pi < n_cubic : pi < f.piece_capacity && pi >= f.piece_capacity - n_quad)) {
            const DevPiece pc = f.pieces[pi];
            eb::Pt pts[DEG + 1];
#pragma unroll
            for (int i = 0; i <= DEG; i++) pts[i] = eb::Pt{pc.p[i].x, pc.p[i].y};
            if (pc.node & kPieceNode) {          // oriented and bounded already
#pragma unroll
              for (int i = 0; i <= DEG; i++) cur.p[i] = pts[i];
              cur.level = int(pc.node & 0xFFu);
              sign = (pc.node >> 8) & 1u;
            }
            else {
              cur = eb::tree_root<DEG>(pts, sign);
            }
            cmd = pc.cmd;
            nst = 0;
            busy = true;
          }
        }
      }
    }
    if (__all_sync(0xFFFFFFFFu, !busy && exhausted)) break;

    eb::TreeNode<DEG> left, right;
    const bool leaf = busy && eb::tree_step<DEG>(cur, tol_sq, left, right);
    const bool split = busy && !leaf;

    // a leaf's segment (Builder::add after desc_open, Sink::emit), one atomic for the warp
    int x0 = 0, y0 = 0, x1 = 0, y1 = 0;
    if (leaf) {
      x0 = eb::trunc_i(cur.p[0].x); y0 = eb::trunc_i(cur.p[0].y);
      x1 = eb::trunc_i(cur.p[DEG].x); y1 = eb::trunc_i(cur.p[DEG].y);
    }
    const bool emit = leaf && y0 != y1;
    const uint32_t em = __ballot_sync(0xFFFFFFFFu, emit);
    if (em) {
      const int leader = __ffs(em) - 1;
      uint32_t base = 0;
      if (lane == leader) base = atomicAdd(f.totals + 0, uint32_t(__popc(em)));
      base = __shfl_sync(0xFFFFFFFFu, base, leader);
      if (emit) {
        const uint32_t idx = base + uint32_t(__popc(em & lt));
        if (idx < f.seg_capacity) {
          f.segs[idx] = DevSeg{x0, y0, x1, y1};
          f.seg_meta[idx] = (cmd << 1) | sign;
        }
        if (cmd != acc_cmd) { flush_bounds(); acc_cmd = cmd; }
        // Sink::emit's bounds and seglist-entry bound
        const uint32_t strips = (uint32_t((y1 - 1) >> 8) >> kStripShift) - (uint32_t(y0 >> 8) >> kStripShift) + 1u;
        const int lo = min(x0, x1) - 256, hi = max(x0, x1) + 256;
        const uint32_t tiles = uint32_t((((hi >> 8) + 1) >> kTileShift) - ((lo >> 8) >> kTileShift) + 1);
        acc_rows += tiles + 3u * strips;
        ymin = min(ymin, y0);
        ymax = max(ymax, y1);
        xmin = min(xmin, min(x0, x1));
        xmax = max(xmax, max(x0, x1));
      }
    }
    if (leaf) {
      if (nst) cur = stack[--nst];
      else busy = false;
    }

    // the right halves of this step's splits go first to the lanes out of work
    const uint32_t idle = __ballot_sync(0xFFFFFFFFu, !busy);
    const uint32_t donors = __ballot_sync(0xFFFFFFFFu, split);
    const int k = min(__popc(idle), __popc(donors));
    if (split) {
      const int r = __popc(donors & lt);
      if (r < k) {
        TreeXchg<DEG>& x = xchg[r];
#pragma unroll
        for (int i = 0; i <= DEG; i++) { x.x[i] = right.p[i].x; x.y[i] = right.p[i].y; }
        x.cmd = cmd;
        x.level = uint32_t(right.level);
        x.sign = sign;
      }
      else {
        stack[nst++] = right;
      }
      cur = left;
    }
    __syncwarp();
    if (!busy) {
      const int q = __popc(idle & lt);
      if (q < k) {
        const TreeXchg<DEG>& x = xchg[q];
#pragma unroll
        for (int i = 0; i <= DEG; i++) cur.p[i] = eb::Pt{x.x[i], x.y[i]};
        cur.level = int(x.level);
        cmd = x.cmd;
        sign = x.sign;
        nst = 0;
        busy = true;
      }
    }
    __syncwarp();
  }
  flush_bounds();
  rows = __reduce_add_sync(0xFFFFFFFFu, rows);
  if (lane == 0 && rows) atomicAdd(f.totals + 1, rows);
}

__global__ void __launch_bounds__(kCurveThreads) edge_tree_kernel(FrameView f) {
  __shared__ TreeXchg<3> xchg[kCurveThreads / 32][32];
  const int w = threadIdx.x >> 5;
  const uint32_t half = gridDim.x / 2u;
  if (blockIdx.x >= half) flatten_trees<2>(f, reinterpret_cast<TreeXchg<2>*>(xchg[w]), half);
  else flatten_trees<3>(f, xchg[w], half);
}

// Lines, and commands built whole: classify_kernel's item list.
__global__ void __launch_bounds__(256) edge_items_kernel(FrameView f) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t rows = 0;
  bool emitted = false;                        // the lane built an item whose segments count
  eb::Builder b;
  const uint32_t n_items = min(f.work_counter[1], f.item_capacity);
  if (t < n_items) {
    const DevItem it = f.items[t];
    const DevCmd cmd = f.cmds[it.cmd];
    const DevCanvas cv = f.canvases[cmd.canvas];
    const DevXform xf = f.xforms[cmd.xform];
    init_builder(b, cv);
    b.sink.init(f.segs, f.seg_meta, f.totals + 0, f.seg_capacity, it.cmd);
    eb::Src src;
    src.xy = f.verts + 2ull * cmd.geom_first;
    src.cmd = cmd.geom == kGeomPath ? f.path_cmds + cmd.geom_first : nullptr;
    src.affine = xf.affine != 0;
    src.m00 = xf.m[0]; src.m01 = xf.m[1]; src.m10 = xf.m[2]; src.m11 = xf.m[3]; src.m20 = xf.m[4]; src.m21 = xf.m[5];
    eb::Pt a = src.tf(int(it.a));
    uint32_t a_flags = b.fxy(a);
    int rc = 0;
    if (it.kind == kItemWhole) {
      src.i = 0;
      src.n = int(cmd.geom_count);
      rc = eb::build(b, src);                  // includes done()
    }
    else {
      src.i = src.n = 0;                       // no further lines: line_to builds exactly this one
      rc = eb::line_to(b, src, a, a_flags, src.tf(int(it.b)));
    }
    if (rc) {
      atomicOr(&f.cmds_rw[it.cmd].status, kCmdInvalid);
    }
    else {
      if (it.kind != kItemWhole) b.done();
      emitted = true;
    }
  }
  // What is left in the lanes' sinks (a line item's one segment, mostly) goes out with one atomic
  // for the warp, and the command bounds with one set of atomics per command of the warp (the
  // items of a polygon or path sit in consecutive lanes): Sink::flush and finish_curve's work.
  const int lane = threadIdx.x & 31;
  const uint32_t nb = emitted ? uint32_t(b.sink.nb) : 0u;
  uint32_t incl = nb;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= o) incl += v;
  }
  const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
  if (total) {
    uint32_t base = 0;
    if (lane == 31) base = atomicAdd(f.totals + 0, total);
    base = __shfl_sync(0xFFFFFFFFu, base, 31) + incl - nb;
    for (uint32_t k = 0; k < nb; k++) {
      if (base + k < f.seg_capacity) {
        f.segs[base + k] = b.sink.buf[k];
        f.seg_meta[base + k] = (b.sink.cmd << 1) | b.sink.sbuf[k];
      }
    }
  }
  const bool has = emitted && b.sink.n;
  const uint32_t key = has ? b.sink.cmd : 0xFFFFFFFFu;
  const uint32_t peers = __match_any_sync(0xFFFFFFFFu, key);
  if (has) {
    const int x0 = __reduce_min_sync(peers, b.sink.xmin), y0 = __reduce_min_sync(peers, b.sink.ymin);
    const int x1 = __reduce_max_sync(peers, b.sink.xmax), y1 = __reduce_max_sync(peers, b.sink.ymax);
    if (lane == __ffs(peers) - 1) {
      int4* bb = f.cmd_bbox + key;
      atomicMin(&bb->x, x0);
      atomicMin(&bb->y, y0);
      atomicMax(&bb->z, x1);
      atomicMax(&bb->w, y1);
      atomicOr(&f.cmds_rw[key].status, kCmdHasSegments);
    }
    rows = b.sink.rows;
  }
  rows = __reduce_add_sync(0xFFFFFFFFu, rows);
  if (lane == 0 && rows) atomicAdd(f.totals + 1, rows);
}

// ---------------------------------------------------------------------------------------------
// Exclusive scan of u32 (three-phase, recursive on block sums).
// ---------------------------------------------------------------------------------------------

constexpr int kScanThreads = 512;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* smem, uint32_t& total) {
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) smem[warp] = x;
  __syncthreads();
  int nw = blockDim.x >> 5;
  if (warp == 0) {
    uint32_t w = lane < nw ? smem[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xFFFFFFFFu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < nw) smem[lane] = w;
  }
  __syncthreads();
  uint32_t warp_off = warp ? smem[warp - 1] : 0u;
  total = smem[nw - 1];
  __syncthreads();
  return warp_off + x - v;
}

__global__ void scan_tiles_kernel(const uint32_t* in, uint32_t* out, uint32_t* block_sums, uint32_t n) {
  __shared__ uint32_t smem[32];
  uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  uint32_t v[kScanItems];
  uint32_t sum = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) { v[k] = (base + k < n) ? in[base + k] : 0u; sum += v[k]; }
  uint32_t total;
  uint32_t off = block_exclusive_scan(sum, smem, total);
#pragma unroll
  for (int k = 0; k < kScanItems; k++) { if (base + k < n) out[base + k] = off; off += v[k]; }
  if (threadIdx.x == 0 && block_sums) block_sums[blockIdx.x] = total;
}

__global__ void scan_add_kernel(uint32_t* out, const uint32_t* block_offsets, uint32_t n) {
  uint32_t i = blockIdx.x * kScanTile + threadIdx.x;
  uint32_t add = block_offsets[blockIdx.x];
  for (int k = 0; k < kScanItems; k++, i += kScanThreads)
    if (i < n) out[i] += add;
}

// The frame's four scans - slots, gradient row states and conic row runs per command, list entries per
// list row - with their totals, together: one launch of a block per array while the longest has at
// most kScanSmall elements, else three launches over all four. Each array on its own, with a launch
// for its total, took 8 launches on small frames and 16 on larger ones, at 2 to 3 us each.
struct ScanJobs {
  const uint32_t* in[4];
  uint32_t* out[4];
  uint32_t* total[4];
  uint32_t* sums[4];                   // a word per tile of kScanTile elements
  uint32_t n[4];
};
constexpr uint32_t kScanSmall = 16384;
constexpr int kScanWide = 1024;        // threads of the blocks that walk a whole array

// One array (in may equal out), by one block; the total goes to `total`.
__device__ __forceinline__ void scan_by_block(const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* total, uint32_t* smem) {
  uint32_t carry = 0;
  for (uint32_t first = 0; first < n; first += uint32_t(kScanWide * kScanItems)) {
    const uint32_t base = first + threadIdx.x * kScanItems;
    uint32_t v[kScanItems], sum = 0, all;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) { v[k] = base + k < n ? in[base + k] : 0u; sum += v[k]; }
    uint32_t off = carry + block_exclusive_scan(sum, smem, all);
#pragma unroll
    for (int k = 0; k < kScanItems; k++) { if (base + k < n) out[base + k] = off; off += v[k]; }
    carry += all;
  }
  if (threadIdx.x == 0 && total) *total = carry;
}

__global__ void __launch_bounds__(kScanWide) scan_arrays_kernel(ScanJobs j, int of_sums) {
  __shared__ uint32_t smem[32];
  const int a = blockIdx.x;
  if (of_sums) scan_by_block(j.sums[a], j.sums[a], (j.n[a] + kScanTile - 1) / kScanTile, j.total[a], smem);
  else scan_by_block(j.in[a], j.out[a], j.n[a], j.total[a], smem);
}

__global__ void __launch_bounds__(kScanThreads) scan_arrays_tiles_kernel(ScanJobs j) {
  __shared__ uint32_t smem[32];
  const int a = blockIdx.y;
  const uint32_t n = j.n[a], base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  if (blockIdx.x * kScanTile >= n) return;
  uint32_t v[kScanItems], sum = 0, total;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) { v[k] = base + k < n ? j.in[a][base + k] : 0u; sum += v[k]; }
  uint32_t off = block_exclusive_scan(sum, smem, total);
#pragma unroll
  for (int k = 0; k < kScanItems; k++) { if (base + k < n) j.out[a][base + k] = off; off += v[k]; }
  if (threadIdx.x == 0) j.sums[a][blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) scan_arrays_add_kernel(ScanJobs j) {
  const int a = blockIdx.y;
  const uint32_t n = j.n[a];
  if (blockIdx.x * kScanTile >= n) return;
  const uint32_t add = j.sums[a][blockIdx.x];
  uint32_t i = blockIdx.x * kScanTile + threadIdx.x;
#pragma unroll
  for (int k = 0; k < kScanItems; k++, i += kScanThreads)
    if (i < n) j.out[a][i] += add;
}

// ---------------------------------------------------------------------------------------------
// K2 - binning
// ---------------------------------------------------------------------------------------------

// Between the halves: the sizes the counting half produced must fit the arrays the rendering half
// writes (they always do in an eager run, whose arrays are sized from them; a graph frame's are
// sized by capacities). Otherwise the rendering half is skipped and the host re-runs the frame.
__global__ void frame_gate_kernel(FrameView f) {
  const uint32_t* t = f.totals;
  const bool over = t[0] > min(f.seg_capacity, f.num_segs) || t[1] > f.num_seglist || t[2] > f.num_cmdrows ||
                    t[3] > f.num_row_entries || t[4] > f.num_row_states || t[6] > f.num_row_runs;
  if (over) {
    f.work_counter[kSkipWord] = 1u;
    atomicOr(f.error_flags, kErrCapacity);
  }
}

__device__ __forceinline__ bool frame_skipped(const FrameView& f) { return f.work_counter[kSkipWord] != 0u; }

// Tile/row bookkeeping: canvas of every global tile and list row.
__device__ __forceinline__ void tile_setup(const FrameView& f, uint32_t i, uint32_t* row_canvas) {
  const uint32_t num_canvases = f.counts[kCntCanvases];
  // binary search the canvas owning tile i / row i
  if (i < f.counts[kCntTiles]) {
    uint32_t lo = 0, hi = num_canvases - 1;
    while (lo < hi) { uint32_t mid = (lo + hi + 1) >> 1; if (f.canvases[mid].tile_base <= i) lo = mid; else hi = mid - 1; }
    f.tile_canvas[i] = lo;
  }
  const uint32_t log2 = kTileShift - f.list_shift;
  if (i < (f.counts[kCntRows] << log2)) {
    uint32_t lo = 0, hi = num_canvases - 1;
    while (lo < hi) { uint32_t mid = (lo + hi + 1) >> 1; if ((f.canvases[mid].row_base << log2) <= i) lo = mid; else hi = mid - 1; }
    row_canvas[i] = lo;
  }
}

// Tile ranges of every command (empty commands get 0xFFFFFFFF) and its number of tile rows; the same
// launch does the tiles' and list rows' bookkeeping.
__global__ void cmd_tiles_kernel(FrameView f, uint32_t* cmdrow_counts_per_cmd, uint32_t* row_counts, uint32_t* row_canvas) {
  uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  tile_setup(f, c, row_canvas);
  if (c >= f.counts[kCntCmds]) {
    // entries beyond the frame's commands (up to the capacity the scans run over) count nothing
    if (c < f.num_cmds) { cmdrow_counts_per_cmd[c] = 0; f.rs_count[c] = 0; f.rb_count[c] = 0; }
    return;
  }
  const DevCmd cmd = f.cmds[c];
  const DevCanvas cv = f.canvases[cmd.canvas];
  int x0, y0, x1, y1;   // inclusive pixel range
  bool empty = false;
  if (cmd.kind == kFillAnalytic) {
    // pixel bbox of the coverage: rows [ymin >> 8, (ymax - 1) >> 8], columns [xmin >> 8, xmax >> 8]
    const uint32_t st = cmd.status;
    empty = (st & kCmdInvalid) || !(st & kCmdHasSegments);
    f.cmds_rw[c].status = (st & kCmdInvalid) ? 1u : (empty ? 2u : 0u);
    const int4 bb = f.cmd_bbox[c];
    x0 = max(bb.x >> 8, 0); y0 = max(bb.y >> 8, 0);
    x1 = min(bb.z >> 8, cv.w - 1); y1 = min((bb.w - 1) >> 8, cv.h - 1);
    if (!empty) {
      f.cmds_rw[c].box[0] = x0; f.cmds_rw[c].box[1] = y0;
      f.cmds_rw[c].box[2] = x1; f.cmds_rw[c].box[3] = y1;
    }
  }
  else if (cmd.kind == kFillBoxA || cmd.kind == kFillMaskA) {
    x0 = cmd.box[0]; y0 = cmd.box[1]; x1 = cmd.box[2] - 1; y1 = cmd.box[3] - 1;
  }
  else {
    x0 = cmd.box[0] >> 8; y0 = cmd.box[1] >> 8; x1 = ((cmd.box[2] + 255) >> 8) - 1; y1 = ((cmd.box[3] + 255) >> 8) - 1;
  }
  x0 = max(x0, 0); y0 = max(y0, 0); x1 = min(x1, cv.w - 1); y1 = min(y1, cv.h - 1);
  if (x0 > x1 || y0 > y1) empty = true;
  if (empty) {
    f.cmd_tile_x[c] = 0xFFFFFFFFu;
    f.cmd_tile_y[c] = 0xFFFFFFFFu;
    f.cmd_xr[c] = 0x0000FFFFu;   // x0 = 65535 > x1 = 0: overlaps nothing
    f.cmd_yr[c] = 0x0000FFFFu;
    cmdrow_counts_per_cmd[c] = 0;
    f.rs_count[c] = 0;
    f.rb_count[c] = 0;
    return;
  }
  const uint32_t fetch = f.styles[cmd.style].fetch;
  f.rs_count[c] = px::has_row_table(fetch) ? uint32_t(y1 - y0 + 1) : 0u;
  // conic row runs: the reference restarts the fetcher at each band of an analytic fill, once for
  // a box fill
  f.rb_count[c] = fetch != kFetchConic ? 0u
                : cmd.kind == kFillAnalytic ? uint32_t(y1 / cv.band_height - y0 / cv.band_height + 1) : 1u;
  f.cmd_xr[c] = uint32_t(x0) | (uint32_t(x1) << 16);
  f.cmd_yr[c] = uint32_t(y0) | (uint32_t(y1) << 16);
  uint32_t tx0 = uint32_t(x0) >> kTileShift, tx1 = uint32_t(x1) >> kTileShift;
  // the command's list rows (1 << list_shift pixel rows each)
  uint32_t ty0 = uint32_t(y0) >> f.list_shift, ty1 = uint32_t(y1) >> f.list_shift;
  f.cmd_tile_x[c] = tx0 | (tx1 << 16);
  f.cmd_tile_y[c] = ty0 | (ty1 << 16);
  // segment lists are kept per (command, strip row, tile column)
  cmdrow_counts_per_cmd[c] = cmd.kind == kFillAnalytic
      ? ((uint32_t(y1) >> kStripShift) - (uint32_t(y0) >> kStripShift) + 1u) * (tx1 - tx0 + 1u) : 0u;

  const uint32_t row_base = cv.row_base << (kTileShift - f.list_shift);
  for (uint32_t r = ty0; r <= ty1; r++) atomicAdd(&row_counts[row_base + r], 1u);
}

// Segments per (command, strip row, tile column) slot: a segment belongs to every slot its cells
// can touch within each strip row. The first pass counts the slots' segments; tiles entirely right of
// a segment get its per-row cover in their backdrop (added once, at the first tile right of it; a
// prefix over tile columns carries it on). The second pass writes the (segment, mask index) work
// items, grouped by slot in mask order, so the items of consecutive masks are contiguous.
//
// A lane's unit of work is one strip row of one segment: a warp lays the strip rows of its 32
// segments end to end and walks them 32 at a time, so a segment that crosses the whole canvas costs
// the warp what as many short ones do. `per_warp`: 32 segments, or 8 in frames whose segments would
// fill less than one wave of warps, so that the few long ones spread over the SMs. Bound: the
// latency of the units' atomics. Count and scatter pass, against one thread per segment walking all
// its strip rows: 83,000 edges of 20,000 pattern quads on 4096x4096 0.48 + 0.48 -> 0.23 + 0.11 ms
// (32 a warp: 0.23 + 0.19); 27,000 segments of large shapes on 1023x767 0.18 + 0.18 -> 0.02 + 0.05
// ms (32 a warp: 0.05 + 0.11).
constexpr int kBinWarps = 8;
constexpr int kStripsPerTile = kTileH / kStripRows;

template<bool kScatter>
__global__ void __launch_bounds__(32 * kBinWarps) seg_bin_kernel(FrameView f, uint32_t per_warp) {
  if (frame_skipped(f)) return;
  __shared__ DevSeg seg_all[kBinWarps][32];
  __shared__ uint4 par_all[kBinWarps][32];     // first strip row, slot of (strip row 0, tile column 0), tile columns | sign << 15, segment
  __shared__ uint32_t end_all[kBinWarps][32];  // strip rows of the segments up to and with this one
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t first = (blockIdx.x * kBinWarps + uint32_t(w)) * per_warp, s = first + uint32_t(lane);
  // the segments the edge builders emitted must all have found a place in the segment array
  if (s == 0 && !kScatter && f.totals[0] > f.seg_capacity) atomicOr(f.error_flags, kErrSegments);
  const uint32_t n = min(f.totals[0], min(f.seg_capacity, f.num_segs));
  if (first >= n) return;                      // whole warps leave together
  uint32_t rows = 0;
  if (uint32_t(lane) < per_warp && s < n) {
    const uint32_t sm = f.seg_meta[s];
    const uint32_t c = sm >> 1;
    const uint32_t ctx = f.cmd_tile_x[c];
    if (ctx != 0xFFFFFFFFu) {
      const uint32_t yr = f.cmd_yr[c];
      const int sr0 = int((yr & 0xFFFFu) >> kStripShift), sr1 = int((yr >> 16) >> kStripShift);
      const DevSeg g = f.segs[s];
      const int r0 = max((g.y0 >> 8) >> kStripShift, sr0), r1 = min(((g.y1 - 1) >> 8) >> kStripShift, sr1);
      const uint32_t tx0 = ctx & 0xFFFFu, ntx = (ctx >> 16) - tx0 + 1u;
      rows = uint32_t(max(r1 - r0 + 1, 0));
      seg_all[w][lane] = g;
      // modulo 2^32: the slots the units compute from it are the command's
      par_all[w][lane] = make_uint4(uint32_t(r0), f.cmdrow_base[c] - uint32_t(sr0) * ntx - tx0, ctx | ((sm & 1u) << 15), s);   // tile columns are below 2^11
    }
  }
  uint32_t end = rows;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, end, o);
    if (lane >= o) end += v;
  }
  end_all[w][lane] = end;
  const uint32_t total = __shfl_sync(0xFFFFFFFFu, end, 31);
  __syncwarp();
  for (uint32_t u = uint32_t(lane); u < total; u += 32) {
    int k = 0;                                 // the unit's segment: the first whose end lies beyond u
#pragma unroll
    for (int step = 16; step; step >>= 1)
      if (end_all[w][k + step - 1] <= u) k += step;
    const DevSeg g = seg_all[w][k];
    const uint4 par = par_all[w][k];
    const int r = int(par.x + (u - (k ? end_all[w][k - 1] : 0u)));
    const int tx0 = int(par.z & 0x7FFFu), tx1 = int(par.z >> 16);
    int t_first, t_last;
    strip_tile_range(g, r, t_first, t_last);
    const int t0 = max(t_first, tx0), t1 = min(t_last, tx1);
    const uint32_t row_slot = par.y + uint32_t(r) * uint32_t(tx1 - tx0 + 1);
    for (int t = t0; t <= t1; t++) {
      const uint32_t slot = row_slot + uint32_t(t);
      if (!kScatter) {
        atomicAdd(&f.slot_mask[slot], 1u);
      }
      else {
        const uint32_t m = f.slot_mask[slot] - 1u;
        if (m >= f.mask_capacity) continue;    // no masks: nothing below a covering command (or too many, reported)
        const uint32_t pos = atomicAdd(&f.mask_cursor[m], 1u);
        if (pos >= f.num_seglist) { atomicOr(f.error_flags, kErrSeglist); continue; }
        f.entries[pos] = make_uint2(par.w, m);
      }
    }
    if (!kScatter && t_last + 1 <= tx1) {
      const uint32_t sm = 0u - ((par.z >> 15) & 1u);
      uint32_t* bd = f.backdrop + size_t(row_slot + uint32_t(max(t_last + 1, tx0))) * kStripRows;
      const int ya = max(g.y0 >> 8, r << kStripShift), yb = min((g.y1 - 1) >> 8, (r << kStripShift) + kStripRows - 1);
      for (int y = ya; y <= yb; y++) {
        const int top = max(g.y0, y << 8), bot = min(g.y1, (y + 1) << 8);
        const uint32_t cov = (uint32_t(bot - top) ^ sm) - sm;
        atomicAdd(&bd[y & (kStripRows - 1)], cov << 9);
      }
    }
  }
}

// Slots of the frame: the binning count from the device totals, within the arrays' capacity.
__device__ __forceinline__ uint32_t frame_slots(const FrameView& f) { return min(f.totals[2], f.num_cmdrows); }

// The last command whose first slot is <= x (so x is one of its slots), by the whole warp.
__device__ __forceinline__ uint32_t slot_command(const FrameView& f, uint32_t x, uint32_t num_cmds, int lane) {
  uint32_t lo = 0, hi = num_cmds;              // cmdrow_base[lo] <= x; the answer is below hi
  while (hi - lo > 1) {
    const uint32_t step = (hi - lo + 31u) / 32u, k = lo + uint32_t(lane) * step;
    const uint32_t below = __ballot_sync(0xFFFFFFFFu, k < hi && f.cmdrow_base[k] <= x);
    lo += (31u - uint32_t(__clz(below))) * step;
    hi = min(hi, lo + step);
  }
  return lo;
}

// The commands of 32 consecutive slots from `it` on (each lane's is returned), found from command `c` at
// or before them: those after it whose first slot is not beyond the lane's. Leaves c at the last
// lane's command.
__device__ __forceinline__ uint32_t slot_commands(const FrameView& f, uint32_t& c, uint32_t it, uint32_t end,
                                                  uint32_t num_cmds, int lane) {
  const uint32_t s = it + uint32_t(lane), last = min(it + 31u, end - 1u);
  uint32_t mine = c;
  for (;;) {
    const uint32_t k = c + 1u + uint32_t(lane);
    const uint32_t b = k < num_cmds ? f.cmdrow_base[k] : 0xFFFFFFFFu;
    if (__shfl_sync(0xFFFFFFFFu, b, 0) > last) break;
    uint32_t pos = 0;
#pragma unroll
    for (int step = 16; step; step >>= 1)
      if (__shfl_sync(0xFFFFFFFFu, b, int(pos) + step - 1) <= s) pos += uint32_t(step);
    const uint32_t b31 = __shfl_sync(0xFFFFFFFFu, b, 31);
    if (pos == 31u && b31 <= s) pos = 32u;
    if (mine == c) mine = c + pos;             // later rounds only move the lanes beyond this one's commands
    if (b31 > last) break;
    c += 32u;
  }
  c = __shfl_sync(0xFFFFFFFFu, mine, 31);
  return mine;
}

// After the count pass, in two passes over the slots with the occlusion pass between them (it needs
// the prefixes, and tells which slots need no masks). First the backdrop deltas become prefixes over the
// tile columns of every (command, strip row). A warp takes the (command, strip row)s that begin in its
// kPrefixSlots slots, whole, 32 slots at a time (a segmented scan: several narrow rows or a part of a
// wide one). Bound: the backdrops' bytes (16 B read per slot, written where they change).
constexpr int kLayoutWarps = 8;
constexpr uint32_t kLayoutSlots = 128, kPrefixSlots = 256;

__global__ void __launch_bounds__(32 * kLayoutWarps) backdrop_prefix_kernel(FrameView f) {
  if (frame_skipped(f)) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t n = frame_slots(f), num_cmds = f.counts[kCntCmds];
  const uint64_t x0 = (uint64_t(blockIdx.x) * kLayoutWarps + uint32_t(w)) * kPrefixSlots;
  if (x0 >= n) return;
  // the first (command, strip row) beginning at or after x; `c` its command if it is inside one
  uint32_t c = 0;
  auto row_start = [&](uint64_t x) -> uint32_t {
    if (x >= n) return n;
    c = slot_command(f, uint32_t(x), num_cmds, lane);
    const uint32_t ctx = f.cmd_tile_x[c];
    const uint32_t ntx = (ctx >> 16) - (ctx & 0xFFFFu) + 1u;
    const uint32_t past = (uint32_t(x) - f.cmdrow_base[c]) % ntx;
    return past ? min(n, uint32_t(x) + ntx - past) : uint32_t(x);
  };
  const uint32_t end = row_start(x0 + kPrefixSlots);
  const uint32_t begin = row_start(x0);        // leaves c at x0's command: at or before begin's
  uint4 carry = make_uint4(0u, 0u, 0u, 0u);    // the last slot's prefix of the slots before
  for (uint32_t it = begin; it < end; it += 32) {
    const uint32_t s = it + uint32_t(lane);
    const bool on = s < end;
    const uint4 v = on ? *reinterpret_cast<const uint4*>(f.backdrop + size_t(s) * kStripRows) : make_uint4(0u, 0u, 0u, 0u);
    if (!__any_sync(0xFFFFFFFFu, (v.x | v.y | v.z | v.w | carry.x | carry.y | carry.z | carry.w) != 0u)) continue;
    const uint32_t mine = slot_commands(f, c, it, end, num_cmds, lane);
    uint32_t col = 0;
    if (on) {
      const uint32_t ctx = f.cmd_tile_x[mine];
      col = (s - f.cmdrow_base[mine]) % ((ctx >> 16) - (ctx & 0xFFFFu) + 1u);
    }
    uint4 p = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t px = __shfl_up_sync(0xFFFFFFFFu, p.x, o), py = __shfl_up_sync(0xFFFFFFFFu, p.y, o);
      const uint32_t pz = __shfl_up_sync(0xFFFFFFFFu, p.z, o), pw = __shfl_up_sync(0xFFFFFFFFu, p.w, o);
      if (lane >= o && col >= uint32_t(o)) { p.x += px; p.y += py; p.z += pz; p.w += pw; }
    }
    if (col > uint32_t(lane)) { p.x += carry.x; p.y += carry.y; p.z += carry.z; p.w += carry.w; }
    if (on && (p.x != v.x || p.y != v.y || p.z != v.z || p.w != v.w))
      *reinterpret_cast<uint4*>(f.backdrop + size_t(s) * kStripRows) = p;
    carry = make_uint4(__shfl_sync(0xFFFFFFFFu, p.x, 31), __shfl_sync(0xFFFFFFFFu, p.y, 31),
                       __shfl_sync(0xFFFFFFFFu, p.z, 31), __shfl_sync(0xFFFFFFFFu, p.w, 31));
  }
}

// Then the slots with segments that no later command covers (cull_kernel) get their mask index, the
// mask's record and its first work item, in place of the segment count; the others get none. A warp
// takes 128 slots, packs those with segments together (in large shapes one in 50 has any) and looks up
// the places of 32 of them at a time; a block takes its masks and work items from one 64-bit counter with
// one atomic, so masks and items come in the same order and need no scan over the frame. Bound: the
// latency of the look-ups. Both passes in place of one warp per command for the prefix, two frame-wide
// scans and a flag and a compaction pass over the slots: 2.4 -> 0.46 ms for the 46 M slots of 20,000
// pattern quads on 4096x4096, 0.36 -> 0.03 ms for large shapes on 1023x767, and 8 to 12 launches fewer.
// Unpacked, with the look-ups of every 32 slots that have one with segments: 0.225 ms of the former, now
// 0.175; 256 and 512 slots a warp slowed small frames (unpacked: 32 canvases 26 -> 39 and 64 us for both passes).
__global__ void __launch_bounds__(32 * kLayoutWarps) slot_compact_kernel(FrameView f) {
  if (frame_skipped(f)) return;
  constexpr int kSteps = int(kLayoutSlots) / 32;
  __shared__ uint32_t masks_of[kLayoutWarps], items_of[kLayoutWarps];
  __shared__ uint2 live_all[kLayoutWarps][kLayoutSlots];      // the warp's slots with segments and their counts
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t n = frame_slots(f), num_cmds = f.counts[kCntCmds];
  const uint64_t x0 = (uint64_t(blockIdx.x) * kLayoutWarps + uint32_t(w)) * kLayoutSlots;
  if (x0 - uint64_t(w) * kLayoutSlots >= n) return;   // whole blocks leave together
  uint2* live = live_all[w];
  uint32_t num_live = 0;
  {
    uint32_t v[kSteps];
#pragma unroll
    for (int k = 0; k < kSteps; k++) {
      const uint64_t s = x0 + uint64_t(32 * k + lane);
      v[k] = s < n ? f.slot_mask[s] : 0u;
    }
#pragma unroll
    for (int k = 0; k < kSteps; k++) {
      const uint32_t some = __ballot_sync(0xFFFFFFFFu, v[k] != 0u);
      if (v[k]) live[num_live + uint32_t(__popc(some & lt))] = make_uint2(uint32_t(x0) + 32u * uint32_t(k) + uint32_t(lane), v[k]);
      num_live += uint32_t(__popc(some));
    }
  }
  if (!__syncthreads_or(int(num_live != 0u))) return;         // no slot of the block has segments
  // the slots' commands are mostly all among the 32 after the first slot's: one load for all of them
  const uint32_t c = num_live ? slot_command(f, uint32_t(x0), num_cmds, lane) : 0u;
  const uint32_t next = num_live && c + 1u + uint32_t(lane) < num_cmds ? f.cmdrow_base[c + 1u + uint32_t(lane)] : 0xFFFFFFFFu;
  const bool near = uint64_t(__shfl_sync(0xFFFFFFFFu, next, 31)) >= x0 + kLayoutSlots;
  uint32_t slot[kSteps], count[kSteps], mine[kSteps], place[kSteps], my_masks = 0, my_items = 0;
#pragma unroll
  for (int k = 0; k < kSteps; k++) {
    slot[k] = count[k] = mine[k] = place[k] = 0u;
    if (uint32_t(32 * k) >= num_live) continue;
    const bool on = uint32_t(32 * k + lane) < num_live;
    if (on) { slot[k] = live[32 * k + lane].x; count[k] = live[32 * k + lane].y; }
    uint32_t m = c;
    if (near) {
      uint32_t pos = 0;
#pragma unroll
      for (int step = 16; step; step >>= 1)
        if (__shfl_sync(0xFFFFFFFFu, next, int(pos) + step - 1) <= slot[k]) pos += uint32_t(step);
      m += pos;
    }
    else {
      for (uint32_t hi = num_cmds; hi - m > 1u;) {            // first slots: m's at or before the slot, hi's after it
        const uint32_t mid = m + (hi - m) / 2u;
        if (f.cmdrow_base[mid] <= slot[k]) m = mid;
        else hi = mid;
      }
    }
    if (on) {
      const uint32_t ctx = f.cmd_tile_x[m], tx0 = ctx & 0xFFFFu, ntx = (ctx >> 16) - tx0 + 1u;
      const uint32_t local = slot[k] - f.cmdrow_base[m], row = local / ntx;
      const uint32_t tx = tx0 + local - row * ntx, sr = ((f.cmd_yr[m] & 0xFFFFu) >> kStripShift) + row;
      const DevCanvas& cv = f.canvases[f.cmds[m].canvas];
      const uint32_t tile = cv.tile_base + (sr >> (kTileShift - kStripShift)) * uint32_t(cv.tiles_x) + tx;
      mine[k] = m;
      place[k] = tx | (sr << 16);
      if (m < f.strip_cmd[tile * kStripsPerTile + (sr & (kStripsPerTile - 1u))]) {
        f.slot_mask[slot[k]] = 0u;
        count[k] = 0u;
      }
    }
    my_masks += uint32_t(__popc(__ballot_sync(0xFFFFFFFFu, count[k] != 0u)));
    my_items += __reduce_add_sync(0xFFFFFFFFu, count[k]);
  }
  if (lane == 0) { masks_of[w] = my_masks; items_of[w] = my_items; }
  __syncthreads();
  if (w == 0) {
    uint32_t m = lane < kLayoutWarps ? masks_of[lane] : 0u, t = lane < kLayoutWarps ? items_of[lane] : 0u;
    const uint32_t m1 = m, t1 = t;
#pragma unroll
    for (int o = 1; o < kLayoutWarps; o <<= 1) {
      const uint32_t vm = __shfl_up_sync(0xFFFFFFFFu, m, o), vt = __shfl_up_sync(0xFFFFFFFFu, t, o);
      if (lane >= o) { m += vm; t += vt; }
    }
    unsigned long long base = 0;
    if (lane == kLayoutWarps - 1 && m)
      base = atomicAdd(reinterpret_cast<unsigned long long*>(f.work_counter + kMaskAlloc),
                       ((unsigned long long)m << 32) | t);
    base = __shfl_sync(0xFFFFFFFFu, base, kLayoutWarps - 1);
    if (lane < kLayoutWarps) { masks_of[lane] = uint32_t(base >> 32) + m - m1; items_of[lane] = uint32_t(base) + t - t1; }
  }
  __syncthreads();
  uint32_t mask_at = masks_of[w], item_at = items_of[w];
#pragma unroll
  for (int k = 0; k < kSteps; k++) {
    const uint32_t some = __ballot_sync(0xFFFFFFFFu, count[k] != 0u);
    if (!some) continue;
    uint32_t incl = count[k];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += t;
    }
    if (count[k]) {
      const uint32_t idx = mask_at + uint32_t(__popc(some & lt));
      f.slot_mask[slot[k]] = idx + 1u;
      if (idx < f.mask_capacity) {
        const uint32_t x = (place[k] & 0xFFFFu) << kTileShift, y = (place[k] >> 16) << kStripShift;
        const DevCmd& cmd = f.cmds[mine[k]];
        const DevCanvas& cv = f.canvases[cmd.canvas];
        f.mask_cursor[idx] = item_at + incl - count[k];
        // what the coverage pass needs of the slot
        f.mask_info[idx] = make_uint4((x + min(uint32_t(cv.w) - x, uint32_t(kTileW)) - 1u) |
                                          ((y + min(uint32_t(cv.h) - y, uint32_t(kStripRows)) - 1u) << 16),
                                      mine[k], (cmd.flags << 16) | cmd.alpha, slot[k]);
      }
    }
    mask_at += uint32_t(__popc(some));
    item_at += __shfl_sync(0xFFFFFFFFu, incl, 31);
  }
}

// Device properties the launch shapes depend on, queried once (thread-safe static
// initialization: the runtime's two pipeline lanes launch from two threads).
static int device_sms() {
  static const int v = [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
  }();
  return v;
}
// Canvas transfers with page-locked host images: one block column per canvas, one warp per row,
// 4-byte words across the lanes. One launch moves every canvas of a frame, with any strides on
// either side (a DMA copy per canvas pays a per-row cost on the many short rows of small canvases).
__global__ void __launch_bounds__(256) canvas_copy_kernel(const DevXfer* xfers, uint32_t n, int to_host) {
  const uint32_t i = blockIdx.x;
  if (i >= n) return;
  const DevXfer t = xfers[i];
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  for (int y = int(blockIdx.y) * warps + (threadIdx.x >> 5); y < t.h; y += int(gridDim.y) * warps) {
    if (t.a8) {      // strides in bytes
      const uint8_t* src = reinterpret_cast<const uint8_t*>(to_host ? t.dev : t.host) +
                           int64_t(y) * (to_host ? t.dev_stride : t.host_stride);
      uint8_t* dst = reinterpret_cast<uint8_t*>(to_host ? t.host : t.dev) + int64_t(y) * (to_host ? t.host_stride : t.dev_stride);
      for (int x = lane; x < t.w; x += 32) dst[x] = src[x];
      continue;
    }
    const uint32_t* src = to_host ? t.dev + int64_t(y) * t.dev_stride : t.host + int64_t(y) * t.host_stride;
    uint32_t* dst = to_host ? t.host + int64_t(y) * t.host_stride : t.dev + int64_t(y) * t.dev_stride;
    // 16-byte accesses when both rows start at 16-byte boundaries: a quarter of the instructions
    // and of the link transactions, so the copy takes less from the kernels it runs beside
    if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0) {
      const int w4 = t.w >> 2;
      for (int x = lane; x < w4; x += 32)
        reinterpret_cast<uint4*>(dst)[x] = reinterpret_cast<const uint4*>(src)[x];
      for (int x = (w4 << 2) + lane; x < t.w; x += 32) dst[x] = src[x];
    }
    else {
      for (int x = lane; x < t.w; x += 32) dst[x] = src[x];
    }
  }
}

int launch_canvas_copy(const DevXfer* xfers, uint32_t n, int to_host, cudaStream_t st) {
  if (!n) return 0;
  // blocks per canvas: enough in all to keep the link busy, also for a single canvas (a 1023x767 one,
  // 3.1 MB, took 92 us with 16 blocks)
  const uint32_t rows = min(max(uint32_t(device_sms()) * 8u / n, 16u), 256u);
  canvas_copy_kernel<<<dim3(n, rows), 256, 0, st>>>(xfers, n, to_host);
  return 1;
}

int launch_frame_gate(const FrameView& f, cudaStream_t st) {
  frame_gate_kernel<<<1, 1, 0, st>>>(f);
  return 1;
}

// Command-list records: word 0.w is the command's kind (bits 0-1), flags (2-3), alpha (4-11), its style's
// fetch kind and dither flag; word 1.z the style with bit 31 set when it is solid, its colour in 1.w.
constexpr uint32_t kRecSolid = 0x80000000u;
constexpr uint32_t kRecFetchShift = 16, kRecDither = 1u << 20;

// Per tile row: commands overlapping the row in painter's order (one block per row).
__global__ void row_fill_kernel(FrameView f, const uint32_t* row_canvas) {
  __shared__ uint32_t smem[32];
  uint32_t row = blockIdx.x;
  const uint32_t log2 = kTileShift - f.list_shift;
  if (row >= (f.counts[kCntRows] << log2) || frame_skipped(f)) return;        // whole blocks leave together
  const DevCanvas cv = f.canvases[row_canvas[row]];
  uint32_t r = row - (cv.row_base << log2);
  uint32_t out = f.row_offsets[row];
  uint32_t copies = 0;
  for (uint32_t base = 0; base < cv.cmd_count; base += blockDim.x) {
    uint32_t c = cv.cmd_first + base + threadIdx.x;
    uint32_t flag = 0;
    if (base + threadIdx.x < cv.cmd_count) {
      uint32_t ty = f.cmd_tile_y[c];
      flag = (ty != 0xFFFFFFFFu && (ty & 0xFFFFu) <= r && (ty >> 16) >= r) ? 1u : 0u;
      copies += flag & f.cmds[c].flags;               // bit 0: SrcCopy
    }
    uint32_t total;
    uint32_t pos = block_exclusive_scan(flag, smem, total);
    if (flag) {
      // everything the composite needs of the command to test it against a strip and find its
      // slot, gathered once here for every strip of the list row
      // A solid fill's colour (DevCmd::color) takes the place of the row-state base it does not
      // use, with bit 31 of the style word saying so: the composite then loads neither the command
      // nor the style.
      const DevCmd& cmd = f.cmds[c];
      const uint32_t ctx = f.cmd_tile_x[c];
      const DevStyle& style = f.styles[cmd.style];
      const bool solid = style.fetch == kFetchSolid;
      const uint32_t meta = cmd.kind | (cmd.flags << 2) | (cmd.alpha << 4) | (style.fetch << kRecFetchShift) |
                            (style.dither ? kRecDither : 0u);
      uint4* rec = f.row_recs + 2u * (out + pos);
      f.row_box[out + pos] = make_uint2(f.cmd_xr[c], f.cmd_yr[c]);
      rec[0] = make_uint4(c, f.cmd_xr[c], f.cmd_yr[c], meta);
      rec[1] = make_uint4(f.cmdrow_base[c], (ctx & 0xFFFFu) | (((ctx >> 16) - (ctx & 0xFFFFu) + 1u) << 16),
                          cmd.style | (solid ? kRecSolid : 0u), solid ? cmd.color : f.rs_base[c]);
    }
    out += total;
  }
  uint32_t total_copies;
  block_exclusive_scan(copies, smem, total_copies);
  if (threadIdx.x == 0) f.row_copies[row] = total_copies;
}

// ---------------------------------------------------------------------------------------------
// K3a - coverage. A slot is (analytic command, strip row, tile column): 4 rows x 32 pixels. One
// warp takes kSlots consecutive slots with segments (by mask index), whose work items are
// contiguous: its lanes evaluate the items' cells (raster.cuh: straight arithmetic per pixel row, so
// neither slope nor direction parts the lanes) into the slots' cells in shared memory (atomicAdd:
// u32 sums commute) and their left-of-tile cover into the slots' backdrops; then it sweeps slot by
// slot (8-lane shuffle prefix per row from the backdrop) into 128 8-bit masks and leaves the cells
// zero for its next slots. No barrier wider than the warp. Bound: issue slots (79 % of cycles on 512
// canvases of the batch), about half of them the sweeps. Measured against one block per 64 slots running the reference's DDA on
// items sorted by its code paths, the whole pass with its slot layout: 0.82 -> 0.35 ms on 1920x1080 with
// 20,000 curve paths, 9.7 -> 4.0 ms on 512 canvases of the batch.
// ---------------------------------------------------------------------------------------------

constexpr int kFineWarps = kFineThreads / 32;
constexpr int kFineBlocksPerSM = 4;
constexpr uint32_t kCullBlocksPerSM = 8;
constexpr int kSlotPixels = kStripRows * kTileW;
constexpr int kCoverWarps = 4;

template<int kSlots>
__global__ void __launch_bounds__(32 * kCoverWarps) coverage_kernel(FrameView f, bool occlusion) {
  __shared__ __align__(16) uint32_t cells_all[kCoverWarps][kSlots][kSlotPixels];
  __shared__ __align__(16) uint32_t bd_all[kCoverWarps][kSlots][kStripRows];
  __shared__ uint32_t org_all[kCoverWarps][kSlots];   // the slot's last column and row on the canvas
  __shared__ uint2 meta_all[kCoverWarps][kSlots];     // command flags << 16 | alpha, command
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (frame_skipped(f)) return;
  const uint32_t all_masks = f.work_counter[kMaskAlloc + 1], num_masks = min(all_masks, f.mask_capacity);
  if (blockIdx.x == 0 && threadIdx.x == 0 && all_masks > f.mask_capacity) atomicOr(f.error_flags, kErrMasks);
  const uint32_t groups = (num_masks + kSlots - 1) / kSlots;
  const uint32_t first = blockIdx.x * kCoverWarps + uint32_t(warp);
  if (first >= groups) return;
  uint32_t(*cells)[kSlotPixels] = cells_all[warp];
  uint32_t(*bd)[kStripRows] = bd_all[warp];
  uint32_t* org = org_all[warp];
  uint2* meta = meta_all[warp];
#pragma unroll
  for (int j = 0; j < kSlots; j++) *reinterpret_cast<uint4*>(&cells[j][lane * 4]) = make_uint4(0u, 0u, 0u, 0u);

  for (uint32_t grp = first; grp < groups; grp += gridDim.x * kCoverWarps) {
    const uint32_t m0 = grp * kSlots;
    const int nk = int(min(uint32_t(kSlots), num_masks - m0));
    if (lane < nk) {
      const uint4 info = f.mask_info[m0 + uint32_t(lane)];
      org[lane] = info.x;
      meta[lane] = make_uint2(info.z, info.y);
      *reinterpret_cast<uint4*>(bd[lane]) = *reinterpret_cast<const uint4*>(f.backdrop + size_t(info.w) * kStripRows);
    }
    // a mask's cursor now stands at the end of its items, where the next mask's begin
    const uint32_t e0 = m0 ? f.mask_cursor[m0 - 1u] : 0u, e1 = min(f.mask_cursor[m0 + uint32_t(nk) - 1u], f.num_seglist);
    __syncwarp();
    for (uint32_t e = e0 + uint32_t(lane); e < e1; e += 32) {
      const uint2 it = f.entries[e];
      const int j = int(it.y - m0);
      const uint32_t o = org[j];
      ras::WindowSink sink{cells[j], bd[j], int(o & 0xFFFFu & ~uint32_t(kTileW - 1))};
      ras::segment_to_window(f.segs[it.x], f.seg_meta[it.x] & 1u, int((o >> 16) & ~uint32_t(kStripRows - 1)), kStripRows, sink);
    }
    __syncwarp();
    // sweep: lane covers row lane / 8, columns (lane % 8) * 4 .. + 3 of the slot
    const int prow = lane >> 3;
    uint32_t covers = 0;                       // bit j: slot j hides everything before its command
    for (int j = 0; j < nk; j++) {
      const uint2 mt = meta[j];
      const uint32_t flags = mt.x >> 16, alpha = mt.x & 0xFFFFu;
      uint4* cell4 = reinterpret_cast<uint4*>(&cells[j][lane * 4]);
      const uint4 cv4 = *cell4;
      *cell4 = make_uint4(0u, 0u, 0u, 0u);
      const uint32_t s4 = cv4.x + cv4.y + cv4.z + cv4.w;
      uint32_t inc = s4;
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        uint32_t v = __shfl_up_sync(0xFFFFFFFFu, inc, o, 8);
        if ((lane & 7) >= o) inc += v;
      }
      uint32_t cov = (256u << 9) + bd[j][prow] + inc - s4;
      const uint32_t rule = (flags & 2u) ? 0x1FFu : 0xFFFFFFFFu;
      uint32_t m;
      cov += cv4.x; m = px::calc_mask(cov, rule, alpha);
      cov += cv4.y; m |= px::calc_mask(cov, rule, alpha) << 8;
      cov += cv4.z; m |= px::calc_mask(cov, rule, alpha) << 16;
      cov += cv4.w; m |= px::calc_mask(cov, rule, alpha) << 24;
      reinterpret_cast<uint32_t*>(f.masks + size_t(m0 + uint32_t(j)) * kSlotPixels)[lane] = m;
      if (occlusion && (flags & 1u) && alpha == 255u) {
        // an opaque SrcCopy command that covers every pixel of the slot on the canvas: none before it
        // shows there (what the occlusion pass could not see without the masks)
        const uint32_t o = org[j];
        const int cols = int(o & uint32_t(kTileW - 1)) + 1 - (lane & 7) * 4;          // of the lane's four
        const uint32_t on = prow > int((o >> 16) & uint32_t(kStripRows - 1)) || cols <= 0 ? 0u
                          : cols >= 4 ? 0xFFFFFFFFu : (1u << (8 * cols)) - 1u;
        if (__all_sync(0xFFFFFFFFu, (m | ~on) == 0xFFFFFFFFu)) covers |= 1u << j;
      }
    }
    if (lane < nk && ((covers >> lane) & 1u)) {      // a lane per covering slot: one latency for all of them
      const uint32_t o = org[lane], cmd = meta[lane].y, sr = (o >> 16) >> kStripShift;
      const DevCanvas& cv = f.canvases[f.cmds[cmd].canvas];
      const uint32_t tile = cv.tile_base + (sr >> (kTileShift - kStripShift)) * uint32_t(cv.tiles_x) + ((o & 0xFFFFu) >> kTileShift);
      atomicMax(&f.strip_cmd[tile * kStripsPerTile + (sr & (kStripsPerTile - 1u))], cmd);
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------------------------
// K3b - composite, persistent. The work unit is a strip of kStripRows x kTileW pixels (one warp,
// 4 pixels per lane held in registers from one 128-bit load to one 128-bit store). Warps pull
// strips from an atomic queue and never wait on each other; the commands of the strip's tile row
// that overlap the strip are applied in painter's order: analytic commands read their 4 masks per
// lane from the coverage pass, box fills compute theirs, then fetch + SrcOver/SrcCopy.
// ---------------------------------------------------------------------------------------------

// Masks of the lane's PX pixels (from xp on) as bytes of a word, for a command without stored masks:
// boxes from their rectangles.
template<int PX>
__device__ __forceinline__ uint32_t box_masks(const FrameView& f, uint32_t kind, uint32_t ci, uint32_t alpha, uint32_t xr,
                                              uint32_t yr, int xp, int y) {
  uint32_t w = 0;
  if (kind == kFillBoxA) {           // the pixel box is the command's own columns and rows
    const int x0 = int(xr & 0xFFFFu), x1 = int(xr >> 16);
    if (y >= int(yr & 0xFFFFu) && y <= int(yr >> 16)) {
#pragma unroll
      for (int k = 0; k < PX; k++) w |= (xp + k >= x0 && xp + k <= x1) ? alpha << (8 * k) : 0u;
    }
    return w;
  }
  const DevCmd& cmd = f.cmds[ci];
  if (kind == kFillMaskA) {
    // FillMask_Base's vmask spans (fillgeneric_p.h:67-162, compopgeneric_p.h:165-183): the mask
    // byte, times the fill alpha below 255 (udiv255)
    const bool in_y = y >= cmd.box[1] && y < cmd.box[3];
    const uint8_t* row = reinterpret_cast<const uint8_t*>(f.images) +
                         ((uint64_t(cmd.xform) << 32) | cmd.geom_first) + int64_t(y - cmd.box[1]) * cmd.geom_count;
#pragma unroll
    for (int k = 0; k < PX; k++) {
      if (in_y && xp + k >= cmd.box[0] && xp + k < cmd.box[2]) {
        uint32_t v = __ldg(row + (xp + k - cmd.box[0]));
        if (alpha < 255u) v = ((v * alpha + 0x80u) * 0x101u) >> 16;
        w |= v << (8 * k);
      }
    }
    return w;
  }
#pragma unroll
  for (int k = 0; k < PX; k++) w |= px::box_u_mask(cmd.box, alpha, xp + k, y) << (8 * k);
  return w;
}

// A word of four equal mask bytes for a slot no segment reaches: every pixel of a row has the row's
// carried-in coverage `bd`.
__device__ __forceinline__ uint32_t uniform_mask(uint32_t bd, uint32_t flags, uint32_t alpha) {
  return px::calc_mask((256u << 9) + bd, (flags & 2u) ? 0x1FFu : 0xFFFFFFFFu, alpha);
}

// Slot of an analytic command in strip row `strip_row`, tile column tx, from its list records
// (first slot, tx0 | columns << 16, rows y0 | y1 << 16), and its mask index + 1 (0: no segment
// reaches it).
__device__ __forceinline__ uint32_t strip_slot(const FrameView& f, uint32_t slot0, uint32_t tcols, uint32_t yr,
                                               uint32_t strip_row, int tx, uint32_t& nseg) {
  const uint32_t slot = slot0 + (strip_row - ((yr & 0xFFFFu) >> kStripShift)) * (tcols >> 16) + (uint32_t(tx) - (tcols & 0xFFFFu));
  nseg = f.slot_mask[slot];
  return slot;
}

// The bytes of a lane's mask word whose PX pixels lie on the canvas.
template<int PX>
__device__ __forceinline__ uint32_t pixels_on_canvas(int xp, int y, const DevCanvas& cv) {
  const int n = y < cv.h ? min(max(cv.w - xp, 0), PX) : 0;
  return n == 4 ? 0xFFFFFFFFu : (1u << (8 * n)) - 1u;
}

// Occlusion, per strip: a SrcCopy command whose mask is 255 on every pixel of the strip writes its
// source there whatever is below (CompOp_SrcCopy with m = 255 gives the source exactly), so nothing
// before the last such command of the strip's list shows: slot_compact_kernel gives the slots before it no
// masks and the composite starts at it. Such a command is found before any mask is rasterized: a box
// that covers the strip, or a path in whose slot no segment lies and whose carried-in coverage is full.
// (A path with segments in the slot that cover it all the same shows in its masks: coverage_kernel
// raises strip_cmd for the composite.)
//
// One warp per tile looks through the tile's list from the end, 32 entries at a time, for opaque SrcCopy
// commands over all its columns, and tests four of them on all eight strips at once, until every strip
// has one; in rows with SrcCopy commands besides a first clear. Bound: the latency of the list reads and
// slot look-ups. One warp per strip, one candidate at a time, took 1.19 ms on 512 canvases of the batch
// (0.43 this way), and after the coverage pass, so that every slot had masks: coverage kernel 3.6 -> 2.4
// ms there, and 1.0 -> 0.06 ms for 20,000 pattern quads on 4096x4096, where the pass itself went from 0.08
// to 0.26.
__global__ void __launch_bounds__(kFineThreads) cull_kernel(FrameView f) {
  const int lane = threadIdx.x & 31;
  if (frame_skipped(f)) return;
  const uint32_t num_tiles = f.counts[kCntTiles];
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  const uint32_t row_log2 = kTileShift - f.list_shift;           // list rows per tile
  const int strips = kStripsPerTile >> row_log2;                  // strips per list row
  for (uint32_t tile = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); tile < num_tiles; tile += warps) {
    const DevCanvas cv = f.canvases[f.tile_canvas[tile]];
    const uint32_t local = tile - cv.tile_base;
    const int tx = int(local % uint32_t(cv.tiles_x)), ty = int(local / uint32_t(cv.tiles_x));
    const uint32_t x0 = uint32_t(tx) << kTileShift, x1 = uint32_t(min(int(x0) + kTileW, cv.w) - 1);
    const int s = lane & 7, q = lane >> 3;                        // strip of the list row, candidate of four
    for (uint32_t lr = 0; lr < (1u << row_log2); lr++) {
      const uint32_t row_id = ((cv.row_base + uint32_t(ty)) << row_log2) + lr;
      const int top = (ty << kTileShift) + int(lr << f.list_shift);     // the list row's first pixel row
      const int sy0 = top + s * kStripRows, sy1 = min(sy0 + kStripRows, cv.h) - 1;
      const bool real = s < strips && sy0 < cv.h;
      uint32_t open = __ballot_sync(0xFFFFFFFFu, real) & 0xFFu;   // strips still without a covering command
      uint32_t start = 0, start_cmd = 0;                          // of strip `lane`, for lanes below `strips`
      if (top >= cv.h || f.row_copies[row_id] < 2) open = 0;
      const uint32_t list_first = open ? f.row_offsets[row_id] : 0u, list_count = open ? f.row_counts[row_id] : 0u;
      for (int cb = int((list_count - 1u) & ~31u); open && cb >= 0; cb -= 32) {
        uint4 ra = make_uint4(0u, 0u, 0u, 0u), rb = ra;
        bool cand = false;
        if (uint32_t(cb + lane) < list_count) {
          // the box first; the records only for commands over all columns
          const uint2 bb = f.row_box[list_first + uint32_t(cb + lane)];
          cand = (bb.x & 0xFFFFu) <= x0 && (bb.x >> 16) >= x1;
          if (cand) {
            const uint4* rec = f.row_recs + 2u * (list_first + uint32_t(cb + lane));
            ra = rec[0];
            rb = rec[1];
            cand = ((ra.w >> 2) & 1u) && ((ra.w >> 4) & 0xFFu) == 255u && (ra.w & 3u) != kFillMaskA;
          }
        }
        uint32_t todo = __ballot_sync(0xFFFFFFFFu, cand);
        while (todo && open) {
          // the next four candidates, the last one of the list first
          int at = -1;
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const int bit = 31 - __clz(todo);                     // -1 when there is none left
            if (q == j) at = bit;
            if (bit >= 0) todo &= ~(1u << bit);
          }
          const int from = at < 0 ? 0 : at;
          const uint32_t ci = __shfl_sync(0xFFFFFFFFu, ra.x, from), yr = __shfl_sync(0xFFFFFFFFu, ra.z, from);
          const uint32_t meta = __shfl_sync(0xFFFFFFFFu, ra.w, from);
          const uint32_t slot0 = __shfl_sync(0xFFFFFFFFu, rb.x, from), tcols = __shfl_sync(0xFFFFFFFFu, rb.y, from);
          bool full = at >= 0 && ((open >> s) & 1u) && int(yr & 0xFFFFu) <= sy0 && int(yr >> 16) >= sy1;
          if (full && (meta & 3u) == kFillAnalytic) {
            uint32_t nseg = 0;
            const uint32_t slot = strip_slot(f, slot0, tcols, yr, uint32_t(sy0) >> kStripShift, tx, nseg);
            full = nseg == 0u;
            if (full) {
              const uint4 bd = *reinterpret_cast<const uint4*>(f.backdrop + size_t(slot) * kStripRows);
              const uint32_t rows[4] = {bd.x, bd.y, bd.z, bd.w};
#pragma unroll
              for (int r = 0; r < 4; r++)
                full &= sy0 + r > sy1 || uniform_mask(rows[r], (meta >> 2) & 3u, 255u) == 255u;
            }
          }
          else if (full && (meta & 3u) == kFillBoxU) {
            // fractional borders thin only the box's first and last columns and rows: the strip's corners tell
            const int32_t* box = f.cmds[ci].box;
            full = px::box_u_mask(box, 255u, int(x0), sy0) == 255u && px::box_u_mask(box, 255u, int(x1), sy0) == 255u &&
                   px::box_u_mask(box, 255u, int(x0), sy1) == 255u && px::box_u_mask(box, 255u, int(x1), sy1) == 255u;
          }
          const uint32_t found = __ballot_sync(0xFFFFFFFFu, full);
          const uint32_t mine = (found >> s) & 0x01010101u;       // the candidates that cover strip s
          const int first = mine ? (__ffs(mine) - 1) >> 3 : 0;
          const int hit_at = __shfl_sync(0xFFFFFFFFu, at, first * 8);
          const uint32_t hit_cmd = __shfl_sync(0xFFFFFFFFu, ci, first * 8);
          if (mine && ((open >> s) & 1u)) { start = uint32_t(cb + hit_at); start_cmd = hit_cmd; }
          open &= ~((found | (found >> 8) | (found >> 16) | (found >> 24)) & 0xFFu);
        }
      }
      if (lane < strips) {
        const uint32_t unit = tile * kStripsPerTile + lr * uint32_t(strips) + uint32_t(lane);
        if (f.strip_start) f.strip_start[unit] = start;
        f.strip_cmd[unit] = start_cmd;
      }
    }
  }
}

// The PX pixels of a lane composited with their sources and mask bytes. A zero mask byte leaves
// its pixel as it is (SrcOver: the scaled source is 0 and d * 255 / 255 gives d; SrcCopy likewise),
// so no pixel needs a branch.
template<int PX>
__device__ __forceinline__ void composite(uint32_t pix[PX], const uint32_t sv[PX], uint32_t mw, bool src_copy) {
  if (src_copy) {
#pragma unroll
    for (int k = 0; k < PX; k++) pix[k] = px::src_copy(pix[k], sv[k], __byte_perm(mw, 0u, 0x4440u + k));
  }
  else {
#pragma unroll
    for (int k = 0; k < PX; k++) pix[k] = px::src_over(pix[k], sv[k], __byte_perm(mw, 0u, 0x4440u + k));
  }
}

// Sources of the lane's PX pixels (those with a mask byte) for a gradient style.
template<int PX>
__device__ __forceinline__ void gradient_sources(const FrameView& f, uint32_t style, uint32_t fetch, bool dither, uint32_t row_state,
                                          int xp, int y, uint32_t mw, uint32_t sv[PX]) {
  const DevStyle& st = f.styles[style];
  const uint4 common = *reinterpret_cast<const uint4*>(&st.maxi);      // maxi, rori, con_maxi, con_rori
  const uint32_t* lut = f.luts + st.lut_offset;
  uint32_t idx[PX];
  if (fetch <= kFetchLinearRoR) {
    const uint64_t dt = st.lin_dt;
    uint64_t pt = st.lin_pt0 + uint64_t(uint32_t(y)) * st.lin_dy + uint64_t(uint32_t(xp)) * dt;
#pragma unroll
    for (int k = 0; k < PX; k++, pt += dt) idx[k] = px::grad_index(uint32_t(pt >> 32), fetch == kFetchLinearPad, common.x, common.y);
  }
  else {
    const float4 rs = f.row_states[row_state];
    if (fetch <= kFetchRadialRoR) {
      const float2 r = *reinterpret_cast<const float2*>(&st.rad_bd);   // bd, ddd
#pragma unroll
      for (int k = 0; k < PX; k++) idx[k] = px::radial_index(r.x, r.y, rs.x, rs.y, rs.z, xp + k, fetch == kFetchRadialPad, common.x, common.y);
    }
    else {
      const float4 q = *reinterpret_cast<const float4*>(st.con_q);
      const float4 n = *reinterpret_cast<const float4*>(&st.con_n1);   // n1, n2, n4, offset
      const float xx = st.con_xx;
#pragma unroll
      for (int k = 0; k < PX; k++) idx[k] = px::conic_index(q, n, xx, rs.x, rs.y, rs.z, xp + k, int32_t(common.z), common.w);
    }
  }
  if (!dither) {
#pragma unroll
    for (int k = 0; k < PX; k++) sv[k] = (mw >> (8 * k)) & 0xFFu ? __ldg(lut + idx[k]) : 0u;
  }
  else {
    // 64-bit entries (lut_offset is even) + the ordered-dither threshold of each pixel
    uint2 e[PX];
#pragma unroll
    for (int k = 0; k < PX; k++)
      e[k] = (mw >> (8 * k)) & 0xFFu ? __ldg(reinterpret_cast<const uint2*>(lut) + idx[k]) : make_uint2(0u, 0u);
#pragma unroll
    for (int k = 0; k < PX; k++) sv[k] = px::dither_pixel(e[k], px::dither_threshold(xp + k, y));
  }
}

__device__ __forceinline__ void prefetch_l1(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// 32-entry chunks of the strip's command list: every lane tests one command's box and gathers what
// the strip needs of it - a stored mask's index, or the four row masks of a slot no segment reaches, which
// drops the command when they are all zero - so the loop over the chunk's commands, in painter's order,
// only broadcasts, and has the stored masks, the style and the row states it will read brought to the
// L1 (composite of 512 canvases of the batch 5.07 -> 4.44 ms: a load from the L2 is as long as a command's
// arithmetic). The loop is pipelined by one command: a command's source loads are under way while the
// one before it is composited. Bound: instruction issue on full grids, and the latency of a strip's
// chain of commands where few strips have long lists. The whole composite (with the cull pass), against
// per-pixel branches, one command at a time and masks found in the loop: 512 canvases of the batch 8.4
// -> 6.0 ms, 20,000 curve paths on 1920x1080 0.66 -> 0.46, 32 requests of up to 1024x1024 0.95 -> 0.56.
// Four blocks per SM (64 registers): three (80) 6.6 ms on the batch, five (48, spilling) 6.2.
//
// A warp takes a strip, four pixels a lane. With a tail launch to follow (kSpill), a warp that has come
// through kSpillHits commands while no strip is left to start, and has a good part of its list before it,
// writes its pixels back and leaves the rest to four warps of that launch (kTail), a row of the strip
// and one pixel a lane each, so that a few strips with long lists do not run alone. That pays where
// strips differ, in frames of several canvases: composite of 512 canvases of the batch 4.44 -> 4.07 ms, 32
// requests of up to 1024x1024 0.45 -> 0.43; on one canvas the strips' lists are alike and the launch costs 6 to 14
// us (20,000 curve paths 0.451 -> 0.465). Rows from the start, for frames of few strips, were slower (2,000
// polygons on 512x512 0.041 -> 0.055): a command costs a warp nearly as much for 32 pixels as for 128.
enum FineMode : int { kStrips = 0, kSpill = 1, kTail = 2 };
constexpr uint32_t kSpillHits = 64, kSpillLeft = 64;

template<int kMode>
__global__ void __launch_bounds__(kFineThreads, kFineBlocksPerSM) fine_kernel(FrameView f) {
  constexpr int PX = kMode == kTail ? 1 : 4;
  const int lane = threadIdx.x & 31;
  const int pcol = PX == 4 ? (lane & 7) * 4 : lane;     // first of this lane's columns
  uint32_t ops = 0, pat_ops = 0;         // composited pixels of this lane (all strips)
  if (frame_skipped(f)) return;
  const uint32_t num_strips = f.counts[kCntTiles] * kStripsPerTile;
  const uint32_t num_units = kMode == kTail ? f.work_counter[kSpilled] * kStripRows : num_strips;

  for (;;) {
    uint32_t unit = 0;
    if (lane == 0) unit = atomicAdd(f.work_counter + (kMode == kTail ? kSpillQueue : 0), 1u);
    unit = __shfl_sync(0xFFFFFFFFu, unit, 0);
    if (unit >= num_units) break;
    const int prow = kMode == kTail ? int(unit % kStripRows) : lane >> 3;     // row within the strip
    if (kMode == kTail) unit = f.spilled[unit / kStripRows];
    const uint32_t tile = unit / kStripsPerTile;
    int strip = int(unit % kStripsPerTile);
    const DevCanvas cv = f.canvases[f.tile_canvas[tile]];
    uint32_t local = tile - cv.tile_base;
    int tx = int(local % uint32_t(cv.tiles_x)), ty = int(local / uint32_t(cv.tiles_x));
    int x_base = tx * kTileW;
    int row0 = ty * kTileH + strip * kStripRows;
    if (row0 >= cv.h) continue;
    const uint32_t strip_row = uint32_t(row0) >> kStripShift;
    int row1 = min(row0 + kStripRows, cv.h) - 1;     // last row of the strip inside the canvas
    const int y = row0 + prow, xp = x_base + pcol;
    const uint32_t on_canvas = pixels_on_canvas<PX>(xp, y, cv);
    if (kMode == kTail && y >= cv.h) continue;
    uint32_t* dst = cv.pixels + int64_t(y) * cv.stride + xp;
    // an A8 canvas: one byte per pixel, composited as the alpha byte of a 32-bit pixel (the
    // reference's P8_Alpha operators are its P32 operators' alpha lane); rows start at 16-byte
    // boundaries and xp is a multiple of 4, so 4 pixels are one aligned word
    uint8_t* dst8 = reinterpret_cast<uint8_t*>(cv.pixels) + int64_t(y) * cv.stride + xp;

    uint32_t pix[PX];
    const bool full = PX == 4 && on_canvas == 0xFFFFFFFFu;
    if (cv.a8) {
      if (full) {
        const uint32_t v = *reinterpret_cast<const uint32_t*>(dst8);
#pragma unroll
        for (int k = 0; k < PX; k++) pix[k] = ((v >> (8 * k)) & 0xFFu) << 24;
      }
      else {
#pragma unroll
        for (int k = 0; k < PX; k++) pix[k] = ((on_canvas >> (8 * k)) & 1u) ? uint32_t(dst8[k]) << 24 : 0u;
      }
    }
    else if (full) {
      uint4 v = *reinterpret_cast<const uint4*>(dst);
      pix[0] = v.x; pix[1 % PX] = v.y; pix[2 % PX] = v.z; pix[3 % PX] = v.w;
    }
    else {
#pragma unroll
      for (int k = 0; k < PX; k++) pix[k] = ((on_canvas >> (8 * k)) & 1u) ? dst[k] : 0u;
    }

    const uint32_t row_id = (cv.row_base << (kTileShift - f.list_shift)) + (uint32_t(row0) >> f.list_shift);
    uint32_t list_first = f.row_offsets[row_id];
    uint32_t list_count = f.row_counts[row_id];
    const uint32_t strip_y = uint32_t(row0) | (uint32_t(row1) << 16);
    const uint32_t strip_x = uint32_t(x_base) | (uint32_t(min(x_base + kTileW, cv.w) - 1) << 16);

    const uint32_t start = f.strip_start ? f.strip_start[tile * kStripsPerTile + uint32_t(strip)] : 0u;   // cull_kernel
    const uint32_t cover = f.strip_cmd[tile * kStripsPerTile + uint32_t(strip)];        // ... and coverage_kernel
    uint32_t pend_mw = 0, pend[PX] = {};   // the command to composite next
    bool pend_copy = false;
    uint32_t done = 0;                               // commands composited

    for (uint32_t base = start & ~31u; base < list_count; base += 32) {
      if (kMode == kSpill && done >= kSpillHits && list_count - base >= kSpillLeft &&
          *reinterpret_cast<volatile const uint32_t*>(f.work_counter) >= num_units) {
        // no strip is waiting to be started: the rest of this one's list goes to four warps
        if (lane == 0) {
          f.strip_start[tile * kStripsPerTile + uint32_t(strip)] = base;
          f.spilled[atomicAdd(f.work_counter + kSpilled, 1u)] = unit;
        }
        break;
      }
      // commands of this chunk whose pixel bbox overlaps the strip, in painter's order: one pair
      // of list records per lane holds everything the tests and the slot lookup need
      uint4 ra = make_uint4(0u, 0u, 0u, 0u), rb = ra;
      bool hit = false, stored = false;
      uint32_t masks = 0;                            // index of the stored masks, or a mask byte per row
      if (base + lane < list_count && base + lane >= start) {
        // 8 bytes per entry to find the commands over the strip; their records only for those
        const uint2 bb = f.row_box[list_first + base + lane];
        hit = (bb.x & 0xFFFFu) <= (strip_x >> 16) && (bb.x >> 16) >= (strip_x & 0xFFFFu) &&
              (bb.y & 0xFFFFu) <= (strip_y >> 16) && (bb.y >> 16) >= (strip_y & 0xFFFFu);
        if (hit) {
          const uint4* rec = f.row_recs + 2u * (list_first + base + lane);
          ra = rec[0];
          rb = rec[1];
          hit = ra.x >= cover;
          if (hit && (ra.w & 3u) == kFillAnalytic) {
            uint32_t nseg = 0;
            const uint32_t slot = strip_slot(f, rb.x, rb.y, ra.z, strip_row, tx, nseg);
            stored = nseg != 0u;
            masks = nseg - 1u;
            if (stored) {
              prefetch_l1(f.masks + size_t(masks) * kSlotPixels);
            }
            else {
              const uint4 bd = *reinterpret_cast<const uint4*>(f.backdrop + size_t(slot) * kStripRows);
              const uint32_t flags = (ra.w >> 2) & 3u, alpha = (ra.w >> 4) & 0xFFu;
              masks = uniform_mask(bd.x, flags, alpha) | (uniform_mask(bd.y, flags, alpha) << 8) |
                      (uniform_mask(bd.z, flags, alpha) << 16) | (uniform_mask(bd.w, flags, alpha) << 24);
              hit = masks != 0u;
            }
          }
          if (hit && !(rb.z & kRecSolid)) {
            // what the loop will read of the style, while the other commands' turns last
            const char* st = reinterpret_cast<const char*>(f.styles + rb.z);
            prefetch_l1(st);
            prefetch_l1(st + 64);
            const uint32_t fetch = (ra.w >> kRecFetchShift) & 15u;
            if (fetch >= kFetchPatAlignedPad) { prefetch_l1(st + 192); prefetch_l1(st + 256); }
            else if (px::has_row_table(fetch)) {
              prefetch_l1(st + 128);
              prefetch_l1(f.row_states + rb.w + (max(uint32_t(row0), ra.z & 0xFFFFu) - (ra.z & 0xFFFFu)));
            }
          }
        }
      }
      uint32_t todo = __ballot_sync(0xFFFFFFFFu, hit);
      if (!todo) continue;
      const uint32_t stored_set = __ballot_sync(0xFFFFFFFFu, stored);
      // the first command's mask word, then each next one's while the current one is under way
      auto load_masks = [&](int from) -> uint32_t {
        const uint32_t v = __shfl_sync(0xFFFFFFFFu, masks, from);
        if (PX == 1)
          return (stored_set >> from) & 1u ? f.masks[size_t(v) * kSlotPixels + uint32_t(prow) * kTileW + uint32_t(lane)]
                                           : (v >> (8 * prow)) & 0xFFu;
        return (stored_set >> from) & 1u ? reinterpret_cast<const uint32_t*>(f.masks + size_t(v) * kSlotPixels)[lane]
                                         : __byte_perm(v, 0u, 0x1111u * uint32_t(prow));
      };
      int bit = __ffs(todo) - 1;
      uint32_t next_mw = load_masks(bit);
      done += uint32_t(__popc(todo));
      while (todo) {
        todo &= todo - 1;
        const uint32_t info = __shfl_sync(0xFFFFFFFFu, ra.w, bit);
        const uint32_t style = __shfl_sync(0xFFFFFFFFu, rb.z, bit);
        const uint32_t extra = __shfl_sync(0xFFFFFFFFu, rb.w, bit);      // colour, or first row state
        const uint32_t yr = __shfl_sync(0xFFFFFFFFu, ra.z, bit);
        uint32_t mw = next_mw;
        if ((info & 3u) != kFillAnalytic)
          mw = box_masks<PX>(f, info & 3u, __shfl_sync(0xFFFFFFFFu, ra.x, bit), (info >> 4) & 0xFFu,
                         __shfl_sync(0xFFFFFFFFu, ra.y, bit), yr, xp, y);
        if (todo) {
          bit = __ffs(todo) - 1;
          next_mw = load_masks(bit);
        }
        mw &= on_canvas;
        if (!__any_sync(0xFFFFFFFFu, mw != 0u)) continue;
        const uint32_t n = uint32_t(__popc((((mw & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | mw) & 0x80808080u));   // nonzero bytes
        ops += n;
        uint32_t sv[PX] = {};
        const uint32_t fetch = (info >> kRecFetchShift) & 15u;
        if (style & kRecSolid) {
#pragma unroll
          for (int k = 0; k < PX; k++) sv[k] = extra;
        }
        else if (fetch <= kFetchConic) {
          // a lane without masks may lie outside the command's rows: it reads no row state
          if (mw) gradient_sources<PX>(f, style, fetch, info & kRecDither, extra + uint32_t(y) - (yr & 0xFFFFu), xp, y, mw, sv);
        }
        else {
          pat_ops += n;
          // one copy of the fetch code: the 4 pixels rotate through the last place
          const DevStyle& st = f.styles[style];
          const px::RowState rs = px::row_state(st, y);
          uint32_t m = mw;
#pragma unroll 1
          for (int k = 0; k < PX; k++, m >>= 8) {
            uint32_t v = 0;
            if (m & 0xFFu) v = px::fetch(st, rs, xp + k, f.luts, f.images) | st.src_or;
            for (int j = 0; j + 1 < PX; j++) sv[j] = sv[j + 1];
            sv[PX - 1] = v;
          }
        }
        composite<PX>(pix, pend, pend_mw, pend_copy);
        pend_mw = mw;
        pend_copy = (info >> 2) & 1u;
#pragma unroll
        for (int k = 0; k < PX; k++) pend[k] = sv[k];
      }
    }
    composite<PX>(pix, pend, pend_mw, pend_copy);

    if (cv.a8) {
      if (full) {
        *reinterpret_cast<uint32_t*>(dst8) = (pix[0] >> 24) | ((pix[1 % PX] >> 24) << 8) | ((pix[2 % PX] >> 24) << 16) |
                                             (pix[3 % PX] & 0xFF000000u);
      }
      else {
#pragma unroll
        for (int k = 0; k < PX; k++) if ((on_canvas >> (8 * k)) & 1u) dst8[k] = uint8_t(pix[k] >> 24);
      }
    }
    else if (full) {
      *reinterpret_cast<uint4*>(dst) = make_uint4(pix[0], pix[1 % PX], pix[2 % PX], pix[3 % PX]);
    }
    else {
#pragma unroll
      for (int k = 0; k < PX; k++) if ((on_canvas >> (8 * k)) & 1u) dst[k] = pix[k];
    }
  }

  ops = __reduce_add_sync(0xFFFFFFFFu, ops);
  pat_ops = __reduce_add_sync(0xFFFFFFFFu, pat_ops);
  if (lane == 0 && ops) {
    atomicAdd(&f.pixel_ops[0], (unsigned long long)ops);
    if (pat_ops) atomicAdd(&f.pixel_ops[1], (unsigned long long)pat_ops);
  }
}

// Radial row values: one thread per (command, row) of every radial/conic command's bbox.
__global__ void row_state_kernel(FrameView f) {
  if (frame_skipped(f)) return;
  const uint32_t total = min(f.totals[4], f.num_row_states);
  uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  uint32_t lo = 0, hi = f.counts[kCntCmds] - 1;       // last command whose first row state is <= t
  while (lo < hi) { uint32_t mid = (lo + hi + 1) >> 1; if (f.rs_base[mid] <= t) lo = mid; else hi = mid - 1; }
  const uint32_t c = lo;
  const DevStyle& st = f.styles[f.cmds[c].style];
  if (st.fetch == kFetchConic) return;            // conic_rows_kernel
  f.row_states[t] = px::radial_row(st, int(f.cmd_yr[c] & 0xFFFFu) + int(t - f.rs_base[c]));
}

// Conic row values, one thread per run of rows sharing a fetcher start: the reference steps the
// fetcher's FP64 position row by row from there, so a run is one sequential chain (a thread per
// row would repeat the chain's prefix in every row; the FP64 pipe is the scarce one).
__global__ void conic_rows_kernel(FrameView f) {
  if (frame_skipped(f)) return;
  const uint32_t total = min(f.totals[6], f.num_row_runs);
  uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  uint32_t lo = 0, hi = f.counts[kCntCmds] - 1;       // last command whose first run is <= t
  while (lo < hi) { uint32_t mid = (lo + hi + 1) >> 1; if (f.rb_base[mid] <= t) lo = mid; else hi = mid - 1; }
  const uint32_t c = lo;
  const DevCmd& cmd = f.cmds[c];
  const DevCanvas& cv = f.canvases[cmd.canvas];
  const DevStyle& st = f.styles[cmd.style];
  const int y0 = int(f.cmd_yr[c] & 0xFFFFu), y1 = int(f.cmd_yr[c] >> 16);
  int ya = y0, yb = y1, fs = cmd.fetch_y0;
  if (cmd.kind == kFillAnalytic) {
    const int band = y0 / cv.band_height + int(t - f.rb_base[c]);
    ya = max(y0, band * cv.band_height);
    yb = min(y1, band * cv.band_height + cv.band_height - 1);
    fs = max(cmd.box[1], band * cv.band_height);
  }
  double tx = st.con_tx + st.con_yx * double(fs);
  double ty = st.con_ty + st.con_yy * double(fs);
  int cur = fs;
  float4* out = f.row_states + f.rs_base[c] + uint32_t(ya - y0);
  for (int y = ya; y <= yb; y++) {
    for (; cur < y; cur++) { tx += st.con_yx; ty += st.con_yy; }
    const float ay = float(ty);
    const uint32_t byb = uint32_t(int32_t(__float_as_uint(ay)) >> 31) & __float_as_uint(st.con_n1);
    *out++ = make_float4(float(tx), fabsf(ay), __uint_as_float(byb), 0.0f);
  }
}

}  // namespace blgpu

// =============================================================================================
// Host-side pipeline orchestration
// =============================================================================================

#include "launch.h"

namespace blgpu {

static inline uint32_t cdiv(uint64_t a, uint64_t b) { return uint32_t((a + b - 1) / b); }

// Exclusive scan of `n` u32 (in may equal out). `tmp` must hold scan_temp_words(n) words.
int exclusive_scan(const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* tmp, cudaStream_t st) {
  if (n == 0) return 0;
  uint32_t blocks = cdiv(n, kScanTile);
  if (blocks == 1) {
    scan_tiles_kernel<<<1, kScanThreads, 0, st>>>(in, out, nullptr, n);
    return 1;
  }
  uint32_t* sums = tmp;
  scan_tiles_kernel<<<blocks, kScanThreads, 0, st>>>(in, out, sums, n);
  int k = exclusive_scan(sums, sums, blocks, tmp + blocks, st);
  scan_add_kernel<<<blocks, kScanThreads, 0, st>>>(out, sums, n);
  return k + 2;
}

uint32_t scan_temp_words(uint32_t n) {
  uint32_t words = 0;
  while (n > uint32_t(kScanTile)) { n = cdiv(n, kScanTile); words += n; }
  return words + 16;
}

__global__ void total_kernel(const uint32_t* counts, const uint32_t* offsets, uint32_t n, uint32_t* total) {
  if (threadIdx.x == 0 && blockIdx.x == 0) *total = n ? offsets[n - 1] + counts[n - 1] : 0u;
}

int launch_total(const uint32_t* counts, const uint32_t* offsets, uint32_t n, uint32_t* total, cudaStream_t st) {
  total_kernel<<<1, 32, 0, st>>>(counts, offsets, n, total);
  return 1;
}

int launch_lut(const FrameView& f, cudaStream_t st) {
  if (!f.num_lut_jobs) return 0;
  lut_kernel<<<cdiv(f.num_lut_jobs, kLutWarps), 32 * kLutWarps, 0, st>>>(f.lut_jobs, f.stops, f.luts, f.counts);
  return 1;
}

template<typename K>
static int max_blocks_per_sm(K kernel, int threads, size_t dyn_smem = 0) {
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, dyn_smem);
  return n > 0 ? n : 1;
}

int launch_edges(const FrameView& f, const LaunchConfig& cfg, cudaStream_t st) {
  if (!f.num_cmds) return 0;
  const int sms = device_sms();
  static const int max_per_sm = max_blocks_per_sm(edge_pieces_kernel, kCurveThreads);
  const int few_per_sm = cfg.cubic_blocks_per_sm > 0 && cfg.cubic_blocks_per_sm < max_per_sm ? cfg.cubic_blocks_per_sm : max_per_sm;
  const uint32_t eb = cfg.edge_block == 64 || cfg.edge_block == 256 ? uint32_t(cfg.edge_block) : 128u;
  // four commands a warp once one each would be more than a wave of blocks
  const uint32_t per_warp = f.num_cmds > uint32_t(sms) * 8u * kClassifyWarps ? kClassifyMax : 1u;
  classify_kernel<<<cdiv(f.num_cmds, kClassifyWarps * per_warp), 32 * kClassifyWarps, 0, st>>>(f, per_warp);
  edge_items_kernel<<<cdiv(f.item_capacity ? f.item_capacity : 1, eb), eb, 0, st>>>(f);
  // every curve kernel has twice the blocks of one kind of curve (the first half cubic, the second quadratic)
  const uint32_t split_grid = min(cdiv(f.item_capacity ? f.item_capacity : 1, kSplitWarps * 4), uint32_t(sms) * kSplitBlocksPerSM);
  curve_split_kernel<<<2 * split_grid, 32 * kSplitWarps, 0, st>>>(f);
  // as many warps as there may be pieces, up to the grids' limits
  const uint32_t pgrid = cdiv(f.piece_capacity ? f.piece_capacity : 1, kCurveThreads / 32);
  edge_pieces_kernel<<<2 * min(pgrid, uint32_t(sms * max_per_sm)), kCurveThreads, 0, st>>>(
      f, min(pgrid, uint32_t(sms * few_per_sm)));
  edge_tree_kernel<<<2 * min(pgrid, uint32_t(sms * kTreeBlocksPerSM)), kCurveThreads, 0, st>>>(f);
  return 5;
}

int launch_cmd_tiles(const FrameView& f, uint32_t* cmdrow_counts_per_cmd, uint32_t* row_canvas, cudaStream_t st) {
  const uint32_t list_rows = f.num_rows << (kTileShift - f.list_shift);
  const uint32_t n = max(f.num_cmds, max(f.num_tiles, list_rows));
  if (!n) return 0;
  cmd_tiles_kernel<<<cdiv(n, 256), 256, 0, st>>>(f, cmdrow_counts_per_cmd, f.row_counts, row_canvas);
  return 1;
}

uint32_t frame_scan_words(uint32_t n) { return 4u * (cdiv(n, kScanTile) + 1u); }

int launch_frame_scans(const FrameView& f, const uint32_t* cmdrow_per_cmd, uint32_t* tmp, cudaStream_t st) {
  const uint32_t list_rows = f.num_rows << (kTileShift - f.list_shift);
  const uint32_t longest = max(f.num_cmds, list_rows), tiles = cdiv(longest, kScanTile);
  const ScanJobs j{{cmdrow_per_cmd, f.row_counts, f.rs_count, f.rb_count},
                   {f.cmdrow_base, f.row_offsets, f.rs_base, f.rb_base},
                   {f.totals + 2, f.totals + 3, f.totals + 4, f.totals + 6},
                   {tmp, tmp + tiles, tmp + 2 * tiles, tmp + 3 * tiles},
                   {f.num_cmds, list_rows, f.num_cmds, f.num_cmds}};
  if (longest <= kScanSmall) {
    scan_arrays_kernel<<<4, kScanWide, 0, st>>>(j, 0);
    return 1;
  }
  scan_arrays_tiles_kernel<<<dim3(tiles, 4), kScanThreads, 0, st>>>(j);
  scan_arrays_kernel<<<4, kScanWide, 0, st>>>(j, 1);
  scan_arrays_add_kernel<<<dim3(tiles, 4), kScanThreads, 0, st>>>(j);
  return 3;
}

template<bool kScatter>
static int launch_seg_bin(const FrameView& f, cudaStream_t st) {
  if (!f.num_segs) return 0;
  const uint32_t per_warp = f.num_segs < uint32_t(device_sms()) * 32u * 32u ? 8u : 32u;
  seg_bin_kernel<kScatter><<<cdiv(f.num_segs, per_warp * kBinWarps), 32 * kBinWarps, 0, st>>>(f, per_warp);
  return 1;
}
int launch_bin_count(const FrameView& f, cudaStream_t st) { return launch_seg_bin<false>(f, st); }

int launch_rows(const FrameView& f, uint32_t* row_canvas, cudaStream_t st) {
  const uint32_t list_rows = f.num_rows << (kTileShift - f.list_shift);
  if (!list_rows) return 0;
  row_fill_kernel<<<list_rows, 512, 0, st>>>(f, row_canvas);
  return 1;
}

template<int kMode>
static int fine_grid_size(int blocks_per_sm) {
  const int sms = device_sms();
  static const int max_per_sm = max_blocks_per_sm(fine_kernel<kMode>, kFineThreads);
  return sms * (blocks_per_sm > 0 && blocks_per_sm < max_per_sm ? blocks_per_sm : max_per_sm);
}

// Coverage pass: backdrop prefixes, occlusion, masks and work items of the slots that show, rasterize and
// sweep. Called after the binning count pass and the command lists.
int launch_coverage(const FrameView& f, const LaunchConfig& cfg, cudaStream_t st) {
  const int sms = device_sms();
  int k = 0;
  const uint32_t layout_grid = cdiv(f.num_cmdrows, kLayoutWarps * kLayoutSlots);
  if (f.num_cmdrows) {
    backdrop_prefix_kernel<<<cdiv(f.num_cmdrows, kLayoutWarps * kPrefixSlots), 32 * kLayoutWarps, 0, st>>>(f);
    k++;
  }
  if (cfg.no_occlusion_cull) {
    if (f.strip_start) cudaMemsetAsync(f.strip_start, 0, sizeof(uint32_t) * size_t(f.num_tiles) * kStripsPerTile, st);
    cudaMemsetAsync(f.strip_cmd, 0, sizeof(uint32_t) * size_t(f.num_tiles) * kStripsPerTile, st);
  }
  else if (f.num_tiles) {
    cull_kernel<<<min(uint32_t(sms) * kCullBlocksPerSM, cdiv(f.num_tiles, kFineWarps)), kFineThreads, 0, st>>>(f);
    k++;
  }
  if (!f.num_cmdrows) return k;
  slot_compact_kernel<<<layout_grid, 32 * kLayoutWarps, 0, st>>>(f);
  k += 1 + launch_seg_bin<true>(f, st);
  const int slots = cover_slots_of(cfg);       // no block without a group
  const bool occlusion = !cfg.no_occlusion_cull;
  const int grid = int(min(uint32_t(sms * cover_blocks_of(cfg)), cdiv(f.mask_capacity, uint32_t(slots))));
  if (slots == 16) coverage_kernel<16 / kCoverWarps><<<grid, 32 * kCoverWarps, 0, st>>>(f, occlusion);
  else if (slots == 64) coverage_kernel<64 / kCoverWarps><<<grid, 32 * kCoverWarps, 0, st>>>(f, occlusion);
  else coverage_kernel<32 / kCoverWarps><<<grid, 32 * kCoverWarps, 0, st>>>(f, occlusion);
  return k + 1;
}

int launch_row_states(const FrameView& f, cudaStream_t st) {
  if (!f.num_row_states) return 0;
  row_state_kernel<<<cdiv(f.num_row_states, 128), 128, 0, st>>>(f);
  if (!f.num_row_runs) return 1;
  conic_rows_kernel<<<cdiv(f.num_row_runs, 64), 64, 0, st>>>(f);
  return 2;
}

// work_counter must be zero on entry.
int launch_fine(const FrameView& f, const LaunchConfig& cfg, cudaStream_t st) {
  if (!f.num_tiles) return 0;
  const uint32_t strips = f.num_tiles * kStripsPerTile;
  const uint32_t needed = cdiv(strips, kFineWarps);
  if (f.several_canvases) {
    fine_kernel<kSpill><<<min(uint32_t(fine_grid_size<kSpill>(cfg.fine_blocks_per_sm)), needed), kFineThreads, 0, st>>>(f);
    fine_kernel<kTail><<<min(uint32_t(fine_grid_size<kTail>(cfg.fine_blocks_per_sm)), needed * kStripRows), kFineThreads, 0, st>>>(f);
    return 2;
  }
  fine_kernel<kStrips><<<min(uint32_t(fine_grid_size<kStrips>(cfg.fine_blocks_per_sm)), needed), kFineThreads, 0, st>>>(f);
  return 1;
}

}  // namespace blgpu
