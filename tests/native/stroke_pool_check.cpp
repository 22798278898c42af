// Host check of the stroke pool's size (stroke_pool.h). Exit status 0 when every rule holds.
#include <cstdint>
#include <cstdio>

#include "stroke_pool.h"

using namespace blgpu;

static int g_bad = 0;
static void expect(bool ok, const char* what) {
  if (!ok) { printf("fails: %s\n", what); g_bad++; }
}

// A frame of `curves` curves that need `need` chunks, each curve the same: what the device counts when
// curves stop at the first chunk they do not get.
static uint32_t frame(StrokePool& p, uint32_t curves, uint64_t need) {
  const uint32_t had = p.chunks(curves);
  const uint64_t wanted = need <= had ? need : uint64_t(had) + curves;
  p.after(curves, had, uint32_t(wanted));
  return had;
}

int main() {
  expect(StrokePool{}.chunks(0) == 0, "no curves, no pool");
  expect(StrokePool{}.chunks(1) == kStrokeChunksPerCurve, "a first frame's pool goes by its curves");
  for (uint32_t curves : {1u, 7u, 40000u, 0x3FFFFFFFu})
    expect(uint64_t(StrokePool{}.chunks(curves)) * (kStrokeChunk * kStrokeQuadBytes + 4) <= kStrokePoolBytes, "the budget");
  {
    // long curves: the pool grows until they fit, and holds them while they come
    StrokePool p;
    uint32_t had = 0;
    int frames = 0;
    while (had < 12000u && frames < 20) { had = frame(p, 24, 12000); frames++; }
    expect(frames <= 9, "the pool doubles");
    for (int i = 0; i < 50; i++) had = frame(p, 24, 12000);
    expect(had >= 12000u && had <= 2u * 12000u, "the pool follows the frames' need");
    // a large frame after them asks for what its own curves need
    expect(p.chunks(100000) == StrokePool{}.chunks(100000), "a few long curves do not multiply a large frame's pool");
    // and once they have gone, so has their pool
    for (int i = 0; i < 60; i++) frame(p, 24, 30);
    expect(p.chunks(24) == StrokePool{}.chunks(24), "the pool shrinks again");
  }
  {
    // more than the budget, for ever
    StrokePool p;
    for (int i = 0; i < 200; i++) expect(frame(p, 1000, uint64_t(1) << 33) <= kStrokeMaxChunks, "the budget holds");
    expect(p.chunks(1) == kStrokeMaxChunks, "the budget is reached");
  }
  {
    // a frame without a pool (no memory for it) says nothing about its curves' need
    StrokePool p;
    p.after(1000, 0, 0);
    expect(p.recent == 0, "no pool, no need");
  }
  printf("failures %d\n", g_bad);
  return g_bad ? 1 : 0;
}
