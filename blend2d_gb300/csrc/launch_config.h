// launch_config.h - launch shapes of the pipeline and the values the autotuner tries for them.
#pragma once

#include <stdint.h>

namespace blgpu {

// Launch shapes the autotuner chooses between (0 = the default for that field).
struct LaunchConfig {
  int cover_slots = 0;            // slots with segments per coverage block (16, 32 or 64; 0 = 32)
  int cover_blocks_per_sm = 0;    // coverage grid: blocks per SM, more than fit at once (0 = 64)
  int fine_blocks_per_sm = 0;     // composite grid: blocks per SM (0 = as many as fit)
  int edge_block = 128;           // threads per block of the per-item edge builder (64/128/256)
  int cubic_blocks_per_sm = 3;    // clipped curve pieces' flattener: blocks per SM while they are few (0 = as many as fit)
  int no_occlusion_cull = 0;      // 1: the composite starts every strip at its first command
  int max_segments = 0;           // > 0: cap of the segment array (frames needing more fail)
  int graph_frames = 0;           // 1: frames run as a captured graph over capacity-sized arrays
  int list_rows = 32;             // pixel rows per command list (4, 8, 16 or 32)
  int device_order = 0;           // 1: pipelines of runtimes that set it run one after another on the device
};

// log2 of the list-row height a launch config selects.
inline uint32_t list_shift_of(const LaunchConfig& c) {
  return c.list_rows == 4 ? 2u : c.list_rows == 8 ? 3u : c.list_rows == 16 ? 4u : 5u;
}

// Slots per coverage block. Eight a warp: 16 (64 a block) leave less shared memory for other warps, 4
// fewer work items than lanes. The pass at 16, 32 and 64 slots a block: 5.44, 4.37 and 4.66 ms on 512
// canvases of the batch, 0.41, 0.36 and 0.41 on 20,000 curve paths.
inline int cover_slots_of(const LaunchConfig& c) { return c.cover_slots ? c.cover_slots : 32; }
// Coverage blocks per SM. Far more than fit at once, so that long groups even out (12, 16, 24, 32 and 64:
// 4.79, 4.34, 4.19, 4.16 and 4.01 ms on the batch's canvases).
inline int cover_blocks_of(const LaunchConfig& c) { return c.cover_blocks_per_sm > 0 ? c.cover_blocks_per_sm : 64; }

// What the autotuner tries, field by field in this order. No two values of a field are the same launch:
// the defaults stand as 0, and the coverage grid's neighbours as multiples of what fits.
struct LaunchField {
  int LaunchConfig::*field;
  int count;
  int values[4];
};
constexpr LaunchField kLaunchFields[] = {
    {&LaunchConfig::list_rows, 4, {32, 16, 8, 4}},
    {&LaunchConfig::cover_slots, 3, {0, 16, 64}},
    {&LaunchConfig::cover_blocks_per_sm, 4, {0, 16, 32, 128}},
    {&LaunchConfig::fine_blocks_per_sm, 4, {0, 1, 2, 3}},
    {&LaunchConfig::edge_block, 3, {64, 128, 256}},
    {&LaunchConfig::cubic_blocks_per_sm, 4, {0, 1, 2, 3}},
};

// Whether two configs launch the same kernels in the same shapes.
inline bool same_launches(const LaunchConfig& a, const LaunchConfig& b) {
  return cover_slots_of(a) == cover_slots_of(b) && cover_blocks_of(a) == cover_blocks_of(b) &&
         a.fine_blocks_per_sm == b.fine_blocks_per_sm && a.edge_block == b.edge_block &&
         a.cubic_blocks_per_sm == b.cubic_blocks_per_sm && a.no_occlusion_cull == b.no_occlusion_cull &&
         list_shift_of(a) == list_shift_of(b);
}

}  // namespace blgpu
