// stroke_pool.h - how many chunks of offset quads a stroked frame's pool has (runtime.cpp, stroke.cu).
#pragma once

#include <stdint.h>

#include <algorithm>

namespace blgpu {

constexpr uint32_t kStrokeChunk = 4;                  // quads per chunk
constexpr uint32_t kStrokeQuadBytes = 64;             // sk::OffsetQuad
// A frame's pool holds this at most. Curves that find no room are offset by their figure's thread, so the
// limit costs time, not pixels: the 40,000 cubics of 10,000 paths get 62 MB.
constexpr uint64_t kStrokePoolBytes = uint64_t(1) << 30;
constexpr uint32_t kStrokeMaxChunks = uint32_t(kStrokePoolBytes / (kStrokeChunk * kStrokeQuadBytes + sizeof(uint32_t)));
// Chunks per curve of a frame: 24 quads, where curves of up to a few hundred pixels take 14 on average.
constexpr uint32_t kStrokeChunksPerCurve = 6;

// The size goes by the frame's own curves. Frames whose curves are longer than that run out, and the
// chunks such frames asked for are kept for the next ones: as a number of chunks, not per curve, so that
// a few long curves do not multiply what a large frame reserves, and less of it with every frame.
struct StrokePool {
  uint32_t recent = 0;

  uint32_t chunks(uint32_t curves) const {
    return curves ? uint32_t(std::min<uint64_t>(std::max<uint64_t>(uint64_t(curves) * kStrokeChunksPerCurve, recent), kStrokeMaxChunks)) : 0u;
  }
  // After a frame of `curves` curves whose pool had `had` chunks: `wanted` were asked for, by each curve
  // up to the first it did not get.
  void after(uint32_t curves, uint32_t had, uint32_t wanted) {
    const uint64_t need = wanted > had ? 2ull * wanted : uint64_t(wanted) + wanted / 4u;
    recent = recent / 4u * 3u;
    if (had && need > uint64_t(curves) * kStrokeChunksPerCurve)
      recent = std::max(recent, uint32_t(std::min<uint64_t>(need, kStrokeMaxChunks)));
  }
};

}  // namespace blgpu
