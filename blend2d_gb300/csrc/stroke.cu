// Device stroking, in five kernels:
//   list    one thread per figure lists the figure's curve commands;
//   curves  one thread per curve offsets it to both sides (nearly all of the stroker's FP64 work) and
//           stores the quads in chunks from a pool;
//   count   one thread per figure runs the stroker over its lines, joins and caps, taking the stored
//           curves as blocks of known size, and counts the outline's vertices; an exclusive scan then
//           places the figures' outlines after the frame's recorded vertices;
//   emit    the same stroker again writes the vertices around the curves and notes where each curve's
//           quads go;
//   place   eight lanes per curve copy its quads there.
// A curve's offset depends on the curve alone, but for the stroker's current point, which is the
// previous vertex unless a degenerate command left it behind: a stored curve is taken only where the
// stroker stands on its start, bit for bit, and any other one is offset by the figure's thread. The
// stroke command then reads its outline like any analytic fill's path.
//
// Bound: the FP64 pipe in the curves kernel (82 % of its cycles, with 14 of 32 lanes active), latency in
// the others. 10,000 open paths of 2 to 6 cubics, 1920x1080: curves 0.73 ms, count 0.15, emit 0.18, place
// 0.03, list 0.01. One thread per figure, stroking everything once to
// count (3.7 ms) and once to write (3.8 ms), left two warps to an SM.
#include "blgpu_internal.h"
#include "launch.h"
#include "stroke_core.h"
#include "stroke_pool.h"

namespace blgpu {

namespace {

constexpr int kStrokeThreads = 64;

__device__ __forceinline__ const sk::V* stroke_vertices(const FrameView& f) { return reinterpret_cast<const sk::V*>(f.stroke_xy); }

__device__ __forceinline__ sk::Params stroke_params(const FrameView& f, uint32_t param) {
  const DevStrokeParams dp = f.stroke_params[param];
  return sk::Params{dp.width, dp.miter_limit, dp.join, dp.start_cap, dp.end_cap, 0u};
}

// The curves of a figure as the stroker's kernels find them, and where emit puts them.
struct StoredCurves {
  const uint32_t* at;                // vertex -> its curve's index; null: no curve is stored
  const sk::CurveRec* recs;
  const sk::OffsetQuad* pool;
  DevCurveDest* dests;               // emit only
  uint32_t a_first, b_end;           // where side A's vertex 0 goes; where side B's vertex 0 would
  uint32_t b_size;
  uint32_t flags;                    // DevCurveDest's, without kDestLast

  __device__ const sk::CurveRec* find(uint32_t i, sk::V p0) const {
    if (!at) return nullptr;
    const sk::CurveRec* r = recs + at[i];
    return r->count && sk::same_bits(r->from, p0) ? r : nullptr;
  }
  __device__ const sk::OffsetQuad& first_quad(const sk::CurveRec& r) const { return pool[size_t(r.chunk) * kStrokeChunk]; }
  __device__ void place(const sk::CurveRec& r, uint32_t ia, uint32_t ib) {
    if (!dests) return;
    DevCurveDest d;
    d.a = a_first + ia;
    d.b = b_end - ib;
    d.count = r.count;
    d.flags = flags | (ib + 2u * r.count == b_size ? kDestLast : 0u);
    dests[&r - recs] = d;
  }
};

__global__ void __launch_bounds__(kStrokeThreads) stroke_list_kernel(FrameView f) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= f.counts[kCntStrokeFigs]) return;
  const DevStrokeFig fg = f.stroke_figs[f.stroke_order[t]];
  uint32_t n = 0, at = 0;
  for (int pass = 0; pass < 2; pass++) {
    uint32_t i = fg.first + 1;
    while (i < fg.end) {
      const uint8_t c = f.stroke_cmds[i];
      if (c == sk::kOn) { i++; continue; }
      if (c != sk::kQuad && c != sk::kCubic) break;
      const uint32_t verts = c == sk::kQuad ? 2u : 3u;
      if (i + verts > fg.end) break;
      if (pass == 0) n++;
      else if (at < f.stroke_curve_cap) {
        f.stroke_curve_at[i] = at;
        f.stroke_curves[at++] = make_uint2(i, fg.param);
      }
      i += verts;
    }
    if (pass == 0) {
      if (!n) return;
      at = atomicAdd(f.stroke_counters + kStrokeCurves, n);
    }
  }
}

__global__ void __launch_bounds__(kStrokeThreads) stroke_curves_kernel(FrameView f) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= min(f.stroke_counters[kStrokeCurves], f.stroke_curve_cap)) return;
  const uint2 cv = f.stroke_curves[t];
  const sk::V* vtx = stroke_vertices(f);
  sk::Offsetter off;
  off.d = f.stroke_params[cv.y].width * 0.5;
  off.d2 = f.stroke_params[cv.y].width;
  sk::CurveRec& rec = static_cast<sk::CurveRec*>(f.stroke_recs)[t];
  sk::OffsetQuad* const pool = static_cast<sk::OffsetQuad*>(f.stroke_pool);
  uint32_t n = 0, chunk = 0;
  sk::V n_first{0.0, 0.0};
  if (sk::begin_curve_alone(f.stroke_cmds, vtx, cv.x, off, n_first)) {
    while (off.active()) {
      off.step([&](const sk::OffsetPiece& o) {
        if (n % kStrokeChunk == 0u) {
          const uint32_t c = atomicAdd(f.stroke_counters + kStrokeChunks, 1u);
          if (c < f.stroke_chunk_cap) {
            if (n) f.stroke_chunk_next[chunk] = c;
            else rec.chunk = c;
          }
          chunk = c;
        }
        if (chunk < f.stroke_chunk_cap) pool[size_t(chunk) * kStrokeChunk + n % kStrokeChunk] = o.q;
        rec.last = o;
        n++;
      });
      // the pool is used up: the figure's thread offsets this curve (StrokePool gives the next frame more)
      if (n && chunk >= f.stroke_chunk_cap) { n = 0; break; }
    }
  }
  rec.from = vtx[cv.x - 1];
  rec.n_first = n_first;
  rec.count = n;
  f.stroke_dests[t].count = 0u;      // until emit takes it
}

__device__ __forceinline__ StoredCurves stored_curves(const FrameView& f) {
  StoredCurves c{};
  c.at = f.stroke_curve_cap ? f.stroke_curve_at : nullptr;
  c.recs = static_cast<const sk::CurveRec*>(f.stroke_recs);
  c.pool = static_cast<const sk::OffsetQuad*>(f.stroke_pool);
  return c;
}

__global__ void __launch_bounds__(kStrokeThreads) stroke_count_kernel(FrameView f) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= f.counts[kCntStrokeFigs]) {
    if (t < f.num_stroke_figs) f.stroke_totals[t] = 0;   // beyond the frame's figures: nothing to scan
    return;
  }
  const uint32_t i = f.stroke_order[t];
  const DevStrokeFig fg = f.stroke_figs[i];
  const sk::Params p = stroke_params(f, fg.param);
  const sk::FigureCounts fc = sk::count_figure(f.stroke_cmds, stroke_vertices(f), fg.first, fg.end, p, stored_curves(f));
  f.stroke_counts[i] = make_uint4(fc.total(), fc.a, fc.b,
                                  fc.c | (fc.closed ? 1u << 30 : 0u) | (fc.b_ok ? 1u << 31 : 0u));
  f.stroke_totals[i] = fc.total();
}

__global__ void __launch_bounds__(kStrokeThreads) stroke_emit_kernel(FrameView f) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= f.counts[kCntStrokeFigs]) return;
  const uint32_t i = f.stroke_order[t];
  const DevStrokeFig fg = f.stroke_figs[i];
  const uint32_t off = f.stroke_offsets[i];
  const uint32_t vb = f.counts[kCntStrokeVertBase] + off;
  if (fg.cmd_figs) {
    DevCmd& c = f.cmds_rw[fg.cmd];
    c.geom_first = vb;
    c.geom_count = f.stroke_offsets[i + fg.cmd_figs] - off;
  }
  const uint4 cnt = f.stroke_counts[i];
  if (!cnt.x) return;
  sk::FigureCounts fc;
  fc.a = cnt.y;
  fc.b = cnt.z;
  fc.c = cnt.w & 0x3FFFFFFFu;
  fc.closed = (cnt.w >> 30) & 1u;
  fc.b_ok = (cnt.w >> 31) & 1u;
  const sk::Params p = stroke_params(f, fg.param);
  // the frame's vertex and command arrays are written here, before any kernel reads them
  uint8_t* out_cmd = const_cast<uint8_t*>(f.path_cmds) + vb;
  double* out_xy = const_cast<double*>(f.verts) + 2ull * vb;
  StoredCurves curves = stored_curves(f);
  curves.dests = f.stroke_dests;
  curves.a_first = vb;
  curves.b_end = vb + fc.a + fc.b - (fc.closed ? 1u : 2u);      // sk::ReverseSink's positions
  curves.b_size = fc.b;
  curves.flags = (fc.b_ok ? kDestSideB : 0u) | (fc.closed ? kDestClosed : 0u);
  sk::emit_figure(f.stroke_cmds, stroke_vertices(f), fg.first, fg.end, p, fc, out_cmd, out_xy, curves);
}

// Eight lanes per curve, a chunk at a time: lane 2q + s writes the two vertices of quad q on side s
// (A forward, B reversed as sk::ReverseSink writes it).
__global__ void __launch_bounds__(256) stroke_place_kernel(FrameView f) {
  const uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  if (t >= min(f.stroke_counters[kStrokeCurves], f.stroke_curve_cap)) return;
  const DevCurveDest d = f.stroke_dests[t];
  if (!d.count) return;
  const uint32_t lane = threadIdx.x & 7u, side = lane & 1u;
  if (side && !(d.flags & kDestSideB)) return;
  uint32_t chunk = static_cast<const sk::CurveRec*>(f.stroke_recs)[t].chunk;
  const sk::OffsetQuad* pool = static_cast<const sk::OffsetQuad*>(f.stroke_pool);
  uint8_t* cmds = const_cast<uint8_t*>(f.path_cmds);
  double2* verts = reinterpret_cast<double2*>(const_cast<double*>(f.verts));
  for (uint32_t k0 = 0; k0 < d.count; k0 += kStrokeChunk) {
    if (k0) chunk = f.stroke_chunk_next[chunk];
    const uint32_t k = k0 + (lane >> 1);
    if (k >= d.count) break;
    const sk::OffsetQuad& q = pool[size_t(chunk) * kStrokeChunk + (lane >> 1)];
    if (!side) {
      const uint32_t v = d.a + 2u * k;
      cmds[v] = sk::kQuad;
      cmds[v + 1] = sk::kOn;
      verts[v] = make_double2(q.a1.x, q.a1.y);
      verts[v + 1] = make_double2(q.a2.x, q.a2.y);
    }
    else {
      const uint32_t v = d.b - 2u * k;
      cmds[v] = sk::kQuad;
      verts[v] = make_double2(q.b1.x, q.b1.y);
      const bool last = k + 1u == d.count && (d.flags & kDestLast);
      if (last && !(d.flags & kDestClosed)) break;           // A's end cap ends there already
      cmds[v - 1] = last ? sk::kMove : sk::kOn;
      verts[v - 1] = make_double2(q.b2.x, q.b2.y);
    }
  }
}

}  // namespace

static_assert(sizeof(sk::CurveRec) <= kStrokeRecBytes && sizeof(sk::OffsetQuad) == kStrokeQuadBytes, "stroke records");

int launch_stroke_count(const FrameView& f, cudaStream_t st) {
  if (!f.num_stroke_figs) return 0;
  const uint32_t n = f.num_stroke_figs, grid = (n + kStrokeThreads - 1) / kStrokeThreads;
  int k = 1;
  cudaMemsetAsync(f.stroke_counters, 0, sizeof(uint32_t) * kStrokeCounters, st);
  if (f.stroke_curve_cap) {
    stroke_list_kernel<<<grid, kStrokeThreads, 0, st>>>(f);
    stroke_curves_kernel<<<(f.stroke_curve_cap + kStrokeThreads - 1) / kStrokeThreads, kStrokeThreads, 0, st>>>(f);
    k += 2;
  }
  stroke_count_kernel<<<grid, kStrokeThreads, 0, st>>>(f);
  k += exclusive_scan(f.stroke_totals, f.stroke_offsets, n, f.stroke_scan_tmp, st);
  k += launch_total(f.stroke_totals, f.stroke_offsets, n, f.stroke_offsets + n, st);
  return k;
}

int launch_stroke_emit(const FrameView& f, cudaStream_t st) {
  if (!f.num_stroke_figs) return 0;
  const uint32_t n = f.num_stroke_figs;
  stroke_emit_kernel<<<(n + kStrokeThreads - 1) / kStrokeThreads, kStrokeThreads, 0, st>>>(f);
  if (!f.stroke_curve_cap) return 1;
  stroke_place_kernel<<<(f.stroke_curve_cap + 31u) / 32u, 256, 0, st>>>(f);
  return 2;
}

}  // namespace blgpu
