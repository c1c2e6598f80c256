// Interface of the warp (warp.cu) to the integration and the graphs
// (integrate.cu) and to the differentiable warp (adjoint.cu).
#pragma once

#include <vector>

#include "stack.cuh"

namespace gg {

// An in-place warp of some frames whose descriptors stay on the device, for
// captured graphs.  `items` is the caller's to free with cudaFree.
struct WarpBatch {
  void* items = nullptr;
  int64_t count = 0;
  std::vector<int64_t> forms;  // descriptors per launch form, in order
  int interp = 0;
  float clamp = -1.0f;
};
WarpBatch warp_batch_device(gg_stack* s, const int64_t* indices, int64_t count, const double* fwd, int interp,
                            float clamp);
// Only launches on the stack's stream (safe inside a stream capture).
void launch_warp_batch(gg_stack* s, const WarpBatch& batch, float fill);

// Fused warp (integrate_matrix_warped_*): a frame's samples come from its
// source pixels through the inverse of its matrix instead of from the stack.
struct FusedFrame {
  float m[9][2];  // inverse, float-float
  int affine;
  unsigned src_nonfinite;  // non-finite source pixels of the frame
  int pad[2];
};

// The spare slots hold the warped rows of a band: `per_slot` frames share one
// (one frame each, and a single band, while every frame has a spare slot).
struct BandLayout {
  int per_slot;      // frames per spare slot
  int64_t capacity;  // samples per frame, a multiple of 64
  int rows;          // rows per band; 0: less than a row per frame
};
BandLayout warp_band_layout(const gg_stack* s);

// Bytes of one frame's warp descriptor.
size_t warp_item_bytes();

// Fills the descriptors, the band base pointers and the non-finite counters;
// with more than one band also whether each frame has a non-finite sample.
// `own` (capacity samples per frame) takes the place of the spare slots.
void launch_warp_band_prepare(gg_stack* s, void* d_items, const FusedFrame* d_frames, int interp, float clamp,
                              const BandLayout& band, float* own, const float** base, unsigned* counts);

// Warps every frame into the band of rows [row0, row1) and writes the
// geometric coverage of those rows.  Both functions only launch on the
// stack's stream (safe inside a stream capture).
void launch_warp_band(gg_stack* s, void* d_items, int interp, float clamp, int row0, int row1, unsigned* counts,
                      float* geometric);

// Warp of one device image by inverse affine parameters; finite: the image is
// known to hold no non-finite sample.
void launch_affine_warp(const float* src, int height, int width, const double* theta, int interp, float fill,
                        bool finite, float* dst, cudaStream_t stream);

}  // namespace gg
