// launch.h - host entry points of the device pipeline (kernels.cu, stroke.cu). Each returns
// the number of kernels it launched on `st`.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "blgpu_internal.h"
#include "launch_config.h"

namespace blgpu {

int exclusive_scan(const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* tmp, cudaStream_t st);
uint32_t scan_temp_words(uint32_t n);
int launch_total(const uint32_t* counts, const uint32_t* offsets, uint32_t n, uint32_t* total, cudaStream_t st);

int launch_lut(const FrameView& f, cudaStream_t st);
int launch_edges(const FrameView& f, const LaunchConfig& cfg, cudaStream_t st);
int launch_cmd_tiles(const FrameView& f, uint32_t* cmdrow_counts_per_cmd, uint32_t* row_canvas, cudaStream_t st);
// The frame's scans and their totals; `tmp` holds frame_scan_words(longest array) words.
int launch_frame_scans(const FrameView& f, const uint32_t* cmdrow_per_cmd, uint32_t* tmp, cudaStream_t st);
uint32_t frame_scan_words(uint32_t n);
int launch_bin_count(const FrameView& f, cudaStream_t st);
int launch_rows(const FrameView& f, uint32_t* row_canvas, cudaStream_t st);
int launch_fine(const FrameView& f, const LaunchConfig& cfg, cudaStream_t st);
int launch_row_states(const FrameView& f, cudaStream_t st);
int launch_frame_gate(const FrameView& f, cudaStream_t st);
// Copies the `n` canvases of `xfers` (device memory) to their host images (to_host) or back.
int launch_canvas_copy(const DevXfer* xfers, uint32_t n, int to_host, cudaStream_t st);
int launch_coverage(const FrameView& f, const LaunchConfig& cfg, cudaStream_t st);
// Stroking: per-figure outline sizes and their exclusive scan (stroke_offsets), then the outlines.
int launch_stroke_count(const FrameView& f, cudaStream_t st);
int launch_stroke_emit(const FrameView& f, cudaStream_t st);

}  // namespace blgpu
