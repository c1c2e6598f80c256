// Matrix warps of resident frames: bilinear and Lanczos3, TMA-staged.
//
// Semantics (CPU oracle): output pixel (x, y) samples the source at
// M^-1 (x, y, 1) (float64 in the reference: engine/warp.py:155-227,
// tests/test_gpu_warp_vs_cpu.py:34-128; reference kernels
// warp_kernels.cu:206-777).
//   bilinear: valid iff 0 <= sx <= W-1 and 0 <= sy <= H-1; x1 = min(x0+1, W-1);
//             tx = float32(sx - x0); top/bottom/result in float32 arithmetic.
//   lanczos3: valid iff 2 <= sx < W-3 and 2 <= sy < H-3; 6x6 taps from
//             (x0-2, y0-2); w = sinc(d) sinc(d/3); non-finite taps are skipped
//             and the sum is renormalised; |sum w| <= 1e-12 -> invalid; an
//             optional clamp to [min - c*range, max + c*range] of the taps.
//   invalid pixels get `fill` and coverage 0.
//
// GB300 design
//   - source coordinates are evaluated in float-float (TwoProd/TwoSum) from
//     the float64 inverse, so floor/validity decisions agree with the float64
//     reference without float64 arithmetic on the device;
//   - each CTA owns a 64x48 output tile; its source footprint (an 80x64 box
//     for the small rotations registration produces) is copied to shared
//     memory by one cp.async.bulk.tensor (TMA) load, double-buffered against
//     the previous tile's compute.  Footprints that do not fit the box (large
//     rotation/scale) and image widths that TMA cannot describe (W % 4 != 0)
//     read the taps straight from global memory instead;
//   - output goes to a spare slot; a follow-up kernel swaps the frame->slot
//     table, so nothing is copied back (8 B/pixel instead of 16 B);
//   - Lanczos3 weights are paired even/odd polynomials in (t - 1/2)^2
//     (sampling.cuh); interior tiles of finite frames run a straight-line
//     form without per-pixel tests.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include <cudaTypedefs.h>

#include "async.cuh"
#include "sampling.cuh"
#include "stack.cuh"
#include "warp_band.cuh"

namespace gg {

constexpr int kTileW = 64;
constexpr int kTileH = 48;
constexpr int kWarpThreads = 256;  // 64 x 4; each thread covers kTileH / 4 rows
constexpr int kRowsPerThread = kTileH / 4;
// Affine source coordinates are stepped by 4 output rows in float-float and
// evaluated afresh every kFreshRows rows: at most three steps of rounding
// separate a coordinate from the float64-faithful evaluation, so floor and
// fraction decisions stay those of a direct evaluation.
constexpr int kFreshRows = 4;

struct WarpItem {
  int frame;
  int src_slot;     // filled on the device
  int dst_slot;     // filled on the device (-1: not a slot)
  unsigned src_nonfinite;
  int affine;
  int int_shift;  // inverse is an exact integer translation
  float* dst;     // first row of the output rows (filled on the device)
  float m[9][2];  // inverse matrix, float-float (hi, lo), row-major
};

struct WarpArgs {
  float* slots;
  unsigned* nonfinite;  // per frame: non-finite output samples are added
  WarpItem* items;
  int item_count;
  int64_t stride;
  int width;
  int height;
  int row0, row1;  // output rows [row0, row1); row0 is the first row at WarpItem::dst
  int tiles_x;
  int tiles_y;     // of those rows
  float fill;
  float clamp;
  int every_row;  // coordinates of tiles that are not interior afresh for every row
  float* coverage;  // optional accumulator (+1 per covered pixel)
  int* error;
};

// Register copy of one item's inverse matrix (loaded once per work item so
// that output stores cannot force re-reads of the descriptor).
struct Coef {
  float m[9][2];
  int affine;
};

__device__ __forceinline__ Coef load_coef(const WarpItem* p) {
  Coef c;
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    c.m[q][0] = __ldg(&p->m[q][0]);
    c.m[q][1] = __ldg(&p->m[q][1]);
  }
  c.affine = __ldg(&p->affine);
  return c;
}

// Tile plan: box origin for the source footprint of the output tile whose
// first pixel is (tile_x0, tile_y0).
struct TilePlan {
  int bx, by, fits, interior;
};

// interior: an affine map sends the whole tile at least one pixel inside the
// valid source range (valid_lo <= s <= valid_hi on both axes), so no pixel
// of the tile needs its own validity test.
__device__ __forceinline__ TilePlan plan_tile(const Coef& it, int tile_x0, int tile_y0, int radius, float valid_lo,
                                              float valid_hi_x, float valid_hi_y) {
  const float x0 = static_cast<float>(tile_x0), y0 = static_cast<float>(tile_y0);
  const float cx[4] = {x0, x0 + kTileW - 1, x0, x0 + kTileW - 1};
  const float cy[4] = {y0, y0, y0 + kTileH - 1, y0 + kTileH - 1};
  float minx = kInfF, maxx = -kInfF, miny = kInfF, maxy = -kInfF;
  bool ok = true;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    FFv sx, sy;
    ok &= source_coord(it, cx[c], cy[c], sx, sy);
    minx = fminf(minx, sx.hi);
    maxx = fmaxf(maxx, sx.hi);
    miny = fminf(miny, sy.hi);
    maxy = fmaxf(maxy, sy.hi);
  }
  TilePlan p{0, 0, 0, 0};
  if (!ok || !(maxx - minx < 1.0e6f) || !(maxy - miny < 1.0e6f) || fabsf(minx) > 1.0e8f || fabsf(miny) > 1.0e8f)
    return p;
  // taps span [floor(s) - (radius-1), floor(s) + radius]; one pixel of margin.
  const int lo_x = static_cast<int>(floorf(minx)) - radius;
  const int hi_x = static_cast<int>(floorf(maxx)) + radius + 1;  // inclusive
  const int lo_y = static_cast<int>(floorf(miny)) - radius;
  const int hi_y = static_cast<int>(floorf(maxy)) + radius + 1;
  p.bx = lo_x >= 0 ? (lo_x & ~3) : -((-lo_x + 3) & ~3);  // 16-byte aligned x (TMA rule)
  p.by = lo_y;
  p.fits = (hi_x - p.bx < kBoxW) && (hi_y - p.by < kBoxH);
  p.interior = it.affine && minx >= valid_lo + 1.0f && maxx <= valid_hi_x - 1.0f && miny >= valid_lo + 1.0f &&
               maxy <= valid_hi_y - 1.0f;
  return p;
}

// The output pixels of one thread in a 64 x 48 tile: column ox, rows oy0,
// oy0 + 4, ...; dst is the frame's output row 0.
// FINITE: the source frame holds no non-finite sample (every Lanczos3 window
// takes the plain normalised sum); returns the count of non-finite outputs.
template <int INTERP, bool FINITE>
__device__ __forceinline__ unsigned warp_tile_rows(const WarpArgs& a, const Coef& co, const TapSource& ts, float* dst,
                                                   int ox, int oy0, bool interior, bool int_shift) {
  constexpr int radius = (INTERP == GG_INTERP_LANCZOS3) ? 3 : 1;
  unsigned bad = 0;
  // Affine source coordinates step by 4 output rows: (sx, sy) += 4 (b, e)
  // in float-float (exact scaling by 4, one TwoSum per axis), with a fresh
  // evaluation every kFreshRows rows.
  FFv sx_row{0.0f, 0.0f}, sy_row{0.0f, 0.0f};
  bool row_ok = false;
  const float step_x_hi = 4.0f * co.m[1][0], step_x_lo = 4.0f * co.m[1][1];
  const float step_y_hi = 4.0f * co.m[4][0], step_y_lo = 4.0f * co.m[4][1];
#pragma unroll 1
  for (int r = 0; r < kRowsPerThread; ++r) {
    const int oy = oy0 + 4 * r;
    const bool inside = ox < a.width && oy < a.row1;
    bool valid = false;
    float value = a.fill;
    if (co.affine) {
      if (r % kFreshRows == 0 || a.every_row) {
        row_ok = source_coord(co, static_cast<float>(ox), static_cast<float>(oy), sx_row, sy_row);
      } else {
        sx_row = ff_add_ff(sx_row, step_x_hi, step_x_lo);
        sy_row = ff_add_ff(sy_row, step_y_hi, step_y_lo);
      }
    }
    if (inside) {
      FFv sx = sx_row, sy = sy_row;
      if (co.affine ? row_ok : source_coord(co, static_cast<float>(ox), static_cast<float>(oy), sx, sy)) {
        const float W = static_cast<float>(a.width), H = static_cast<float>(a.height);
        if (interior)
          valid = true;
        else if (INTERP != GG_INTERP_LANCZOS3)
          valid = ff_ge(sx, 0.0f) && ff_le(sx, W - 1.0f) && ff_ge(sy, 0.0f) && ff_le(sy, H - 1.0f);
        else
          valid = ff_ge(sx, 2.0f) && ff_lt(sx, W - 3.0f) && ff_ge(sy, 2.0f) && ff_lt(sy, H - 3.0f);
        if (valid) {
          int x0, y0;
          float tx, ty;
          ff_floor_frac(sx, x0, tx);
          ff_floor_frac(sy, y0, ty);
          if (INTERP == GG_INTERP_NEAREST) {
            // np.rint: round half to even (engine/warp.py:87-96).
            if (tx > 0.5f || (tx == 0.5f && (x0 & 1))) ++x0;
            if (ty > 0.5f || (ty == 0.5f && (y0 & 1))) ++y0;
          }
          TapSource src = ts;
          // Any tap outside the staged box reads global memory instead
          // (an affine tile that fits the box keeps every tap inside it).
          if (src.tile && !co.affine &&
              (x0 - (radius - 1) < src.bx || x0 + radius >= src.bx + kBoxW || y0 - (radius - 1) < src.by ||
               y0 + radius >= src.by + kBoxH))
            src.tile = nullptr;
          if (INTERP == GG_INTERP_NEAREST) {
            value = src.at(x0, y0);
          } else if (INTERP == GG_INTERP_BILINEAR) {
            value = sample_bilinear(src, x0, y0, tx, ty, a.width, a.height);
          } else if (int_shift) {
            // exact weights 0, 0, 1, 0, 0, 0: the source sample itself, or
            // no sample when it is not finite (nothing left to normalise)
            value = src.at(x0, y0);
            if (!isfinite(value)) {
              valid = false;
              value = a.fill;
            }
          } else {
            valid = FINITE ? sample_lanczos3_finite(src, x0, y0, tx, ty, a.clamp, value)
                           : sample_lanczos3(src, x0, y0, tx, ty, false, a.clamp, value);
            if (!valid) value = a.fill;
          }
        }
      }
      dst[static_cast<int64_t>(oy) * a.width + ox] = value;
      if (a.coverage && valid) atomicAdd(a.coverage + static_cast<int64_t>(oy) * a.width + ox, 1.0f);
      bad += isfinite(value) ? 0u : 1u;
    }
  }
  return bad;
}

// The common Lanczos3 tile in straight-line form: an affine map, the whole
// 64 x 48 tile inside the output and mapped at least one pixel inside the
// valid source range, its footprint staged in the shared-memory box, a source
// frame without non-finite samples, no clamp and no coverage map.  Every
// pixel is then valid and takes the plain normalised 6 x 6 sum, so the rows
// need no per-pixel tests (same arithmetic as the general path).
__device__ __forceinline__ unsigned warp_tile_rows_fast(const WarpArgs& a, const Coef& co, const float* box, int bx,
                                                        int by, float* dst, int ox, int oy0) {
  FFv sx, sy;
  const float step_x_hi = 4.0f * co.m[1][0], step_x_lo = 4.0f * co.m[1][1];
  const float step_y_hi = 4.0f * co.m[4][0], step_y_lo = 4.0f * co.m[4][1];
  float* out = dst + static_cast<int64_t>(oy0) * a.width + ox;
  const int64_t out_step = 4 * static_cast<int64_t>(a.width);
  unsigned bad = 0;
#pragma unroll 1
  for (int r = 0; r < kRowsPerThread; ++r) {
    if (r % kFreshRows == 0) {
      source_coord(co, static_cast<float>(ox), static_cast<float>(oy0 + 4 * r), sx, sy);
    } else {
      sx = ff_add_ff(sx, step_x_hi, step_x_lo);
      sy = ff_add_ff(sy, step_y_hi, step_y_lo);
    }
    int x0, y0;
    float tx, ty;
    ff_floor_frac(sx, x0, tx);
    ff_floor_frac(sy, y0, ty);
    float wx[6], wy[6];
    lanczos3_weights(tx, wx);
    lanczos3_weights(ty, wy);
    float swx = 0.0f, swy = 0.0f;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      swx += wx[i];
      swy += wy[i];
    }
    const float* r0 = box + (y0 - 2 - by) * kBoxW + (x0 - 2 - bx);
    float acc = 0.0f;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      float row = 0.0f;
#pragma unroll
      for (int i = 0; i < 6; ++i) row = __fmaf_rn(wx[i], r0[j * kBoxW + i], row);
      acc = __fmaf_rn(wy[j], row, acc);
    }
    const float wsum = swx * swy;
    const float value = fabsf(wsum) > 1.0e-12f ? __fdividef(acc, wsum) : a.fill;
    out[r * out_step] = value;
    bad += isfinite(value) ? 0u : 1u;
  }
  return bad;
}

template <int INTERP, bool USE_TMA>
__global__ void __launch_bounds__(kWarpThreads, 3) warp_tiles_kernel(const __grid_constant__ CUtensorMap tmap,
                                                                  WarpArgs a) {
  __shared__ alignas(128) float tile[2][kBoxH * kBoxW];
  __shared__ alignas(8) uint64_t bar[2];
  __shared__ int s_bx[2], s_by[2], s_fit[2], s_interior[2];
  __shared__ int s_abort;
  constexpr int radius = (INTERP == GG_INTERP_LANCZOS3) ? 3 : 1;
  const int tid = threadIdx.x;
  const int lx = tid & 63, ly = tid >> 6;
  const int tiles = a.tiles_x * a.tiles_y;
  const int items = a.item_count * tiles;
  if (tid == 0) {
    s_abort = 0;
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  auto issue = [&](int item, int buf) {
    // thread 0 only
    const WarpItem* ip = a.items + item / tiles;
    const int t = item % tiles;
    // validity ranges: bilinear 0 <= s <= W - 1; Lanczos3 2 <= s < W - 3
    const float vlo = INTERP == GG_INTERP_LANCZOS3 ? 2.0f : 0.0f;
    const float vhx = static_cast<float>(a.width) - (INTERP == GG_INTERP_LANCZOS3 ? 3.0f : 1.0f);
    const float vhy = static_cast<float>(a.height) - (INTERP == GG_INTERP_LANCZOS3 ? 3.0f : 1.0f);
    TilePlan p = plan_tile(load_coef(ip), t % a.tiles_x * kTileW, a.row0 + t / a.tiles_x * kTileH, radius, vlo, vhx,
                           vhy);
    if (!USE_TMA) p.fits = 0;
    s_interior[buf] = p.interior;
    s_bx[buf] = p.bx;
    s_by[buf] = p.by;
    s_fit[buf] = p.fits;
    if (p.fits) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_expect_tx(&bar[buf], kBoxW * kBoxH * 4);
      tma_load_3d(tile[buf], &tmap, p.bx, p.by, __ldg(&ip->src_slot), &bar[buf]);
    }
  };

  unsigned phase[2] = {0u, 0u};
  int item = blockIdx.x;
  if (tid == 0 && item < items) issue(item, 0);
  __syncthreads();
  for (int i = 0; item < items; ++i, item += gridDim.x) {
    const int buf = i & 1;
    const int next = item + gridDim.x;
    if (tid == 0 && next < items) issue(next, buf ^ 1);
    const int item_index = item / tiles;
    const WarpItem* ip = a.items + item_index;
    const Coef co = load_coef(ip);
    const int it_frame = __ldg(&ip->frame);
    const int it_src = __ldg(&ip->src_slot);
    float* const it_dst = ip->dst;
    const unsigned it_nonfinite = __ldg(&ip->src_nonfinite);
    const bool int_shift = __ldg(&ip->int_shift) != 0;
    const int t = item - item_index * tiles;
    const int tile_x0 = t % a.tiles_x * kTileW, tile_y0 = a.row0 + t / a.tiles_x * kTileH;
    const bool fit = s_fit[buf] != 0;
    const bool interior = s_interior[buf] != 0;
    if (fit) {
      // Bounded wait: on expiry flag the error, give the copy one more
      // bounded wait to land, finish this item (its output is discarded by
      // the host) and leave the loop with the whole CTA.
      if (!mbar_wait_bounded(&bar[buf], phase[buf], 1 << 24)) {
        atomicExch(a.error, 1);
        s_abort = 1;
        mbar_wait_bounded(&bar[buf], phase[buf], 1 << 24);
      }
      phase[buf] ^= 1u;
    }
    {
      TapSource ts;
      ts.tile = fit ? tile[buf] : nullptr;
      ts.src = a.slots + static_cast<int64_t>(it_src) * a.stride;
      ts.bx = s_bx[buf];
      ts.by = s_by[buf];
      ts.width = a.width;
      float* dst = it_dst - static_cast<int64_t>(a.row0) * a.width;
      // the renormalising path (and its out-of-line call) only for frames
      // that hold non-finite samples; the straight-line form for the common
      // interior tile
      const bool full_tile = tile_x0 + kTileW <= a.width && tile_y0 + kTileH <= a.row1;
      unsigned bad;
      if (INTERP == GG_INTERP_LANCZOS3 && fit && interior && co.affine && it_nonfinite == 0u && !int_shift &&
          a.clamp < 0.0f && a.coverage == nullptr && full_tile)
        bad = warp_tile_rows_fast(a, co, ts.tile, ts.bx, ts.by, dst, tile_x0 + lx, tile_y0 + ly);
      else if (INTERP == GG_INTERP_LANCZOS3 && it_nonfinite == 0u)
        bad = warp_tile_rows<INTERP, true>(a, co, ts, dst, tile_x0 + lx, tile_y0 + ly, interior, int_shift);
      else
        bad = warp_tile_rows<INTERP, false>(a, co, ts, dst, tile_x0 + lx, tile_y0 + ly, interior, int_shift);
      const unsigned warp_bad = __reduce_add_sync(0xffffffffu, bad);
      if ((tid & 31) == 0 && warp_bad) atomicAdd(a.nonfinite + it_frame, warp_bad);
    }
    __syncthreads();
    if (s_abort) {
      // Let the prefetch already issued for the next item land before exit.
      if (next < items && s_fit[buf ^ 1]) mbar_wait_bounded(&bar[buf ^ 1], phase[buf ^ 1], 1 << 24);
      break;
    }
  }
}

// Resolve slots for the batch and move the source non-finite counts aside.
__global__ void warp_prepare_kernel(WarpItem* items, int count, const int* slot_of_frame, const int* spare,
                                    unsigned* nonfinite, float* slots, int64_t stride) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count) return;
  const int f = items[k].frame;
  items[k].src_slot = slot_of_frame[f];
  items[k].dst_slot = spare[k];
  items[k].dst = slots + spare[k] * stride;
  items[k].src_nonfinite = nonfinite[f];
  nonfinite[f] = 0u;
}

// The warped frame now lives in the spare slot; the old slot becomes spare.
__global__ void warp_finish_kernel(const WarpItem* items, int count, int* slot_of_frame, int* spare) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count) return;
  slot_of_frame[items[k].frame] = items[k].dst_slot;
  spare[k] = items[k].src_slot;
}

__global__ void fill_kernel(float* p, int64_t n, float v) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    p[i] = v;
}

__global__ void add_scalar_kernel(float* p, int64_t n, float v) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    p[i] += v;
}

// ---- host side -------------------------------------------------------------------
static PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    else
      cudaGetLastError();
  }
  return fn;
}

bool make_slot_tensor_map(gg_stack* s, int box_w, int box_h) {
  auto fn = encode_fn();
  if (!fn) return false;
  if ((s->width * 4) % 16 != 0 || (s->stride * 4) % 16 != 0) return false;
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(s->width), static_cast<cuuint64_t>(s->height),
                              static_cast<cuuint64_t>(s->slots)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(s->width) * 4, static_cast<cuuint64_t>(s->stride) * 4};
  const cuuint32_t box[3] = {static_cast<cuuint32_t>(box_w), static_cast<cuuint32_t>(box_h), 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  std::memset(&s->slot_tmap, 0, sizeof(s->slot_tmap));
  const CUresult r = fn(&s->slot_tmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, s->d_slots, dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// float64 3x3 inverse (np.linalg.inv of the float32 matrix promoted to float64).
static void ensure_warp_items(gg_stack* s, int64_t count) {
  if (s->warp_item_capacity >= count) return;
  check_cuda(cudaStreamSynchronize(s->stream), "cudaStreamSynchronize(warp items)");
  if (s->d_warp_items) cudaFree(s->d_warp_items);
  if (s->h_warp_items) cudaFreeHost(s->h_warp_items);
  s->d_warp_items = nullptr;
  s->h_warp_items = nullptr;
  const size_t bytes = sizeof(WarpItem) * static_cast<size_t>(count);
  check_cuda(cudaMalloc(&s->d_warp_items, bytes), "cudaMalloc(warp items)");
  check_cuda(cudaHostAlloc(&s->h_warp_items, bytes, cudaHostAllocPortable), "cudaHostAlloc(warp items)");
  s->warp_item_capacity = count;
}

static void ensure_warp_coverage(gg_stack* s) {
  if (s->d_warp_coverage) return;
  check_cuda(cudaMalloc(reinterpret_cast<void**>(&s->d_warp_coverage), sizeof(float) * s->pixels),
             "cudaMalloc(warp coverage)");
  s->bytes_allocated += static_cast<int64_t>(sizeof(float) * s->pixels);
  check_cuda(cudaMemsetAsync(s->d_warp_coverage, 0, sizeof(float) * s->pixels, s->stream), "cudaMemsetAsync");
}

template <int INTERP>
static void launch_warp_tiles(gg_stack* s, const WarpArgs& args, bool use_tma) {
  int per_sm = 0;
  auto kern = use_tma ? warp_tiles_kernel<INTERP, true> : warp_tiles_kernel<INTERP, false>;
  check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kWarpThreads, 0), "occupancy(warp)");
  const int64_t items = static_cast<int64_t>(args.item_count) * args.tiles_x * args.tiles_y;
  const unsigned grid =
      static_cast<unsigned>(std::min<int64_t>(items, static_cast<int64_t>(sm_count()) * std::max(per_sm, 1)));
  note_launch();
  kern<<<grid, kWarpThreads, 0, s->stream>>>(s->slot_tmap, args);
  check_cuda(cudaGetLastError(), "warp kernel launch");
}

// Arguments of a launch over output rows [row0, row1) of `count` frames.
static WarpArgs warp_args(gg_stack* s, WarpItem* d_items, int count, int row0, int row1) {
  WarpArgs a{};
  a.slots = s->d_slots;
  a.items = d_items;
  a.item_count = count;
  a.stride = s->stride;
  a.width = static_cast<int>(s->width);
  a.height = static_cast<int>(s->height);
  a.row0 = row0;
  a.row1 = row1;
  a.tiles_x = (a.width + kTileW - 1) / kTileW;
  a.tiles_y = (row1 - row0 + kTileH - 1) / kTileH;
  a.error = s->d_error;
  return a;
}

static void launch_warp_rows(gg_stack* s, const WarpArgs& a, int interp) {
  const bool use_tma = s->has_slot_tmap;
  if (interp == GG_INTERP_NEAREST)
    launch_warp_tiles<GG_INTERP_NEAREST>(s, a, use_tma);
  else if (interp == GG_INTERP_BILINEAR)
    launch_warp_tiles<GG_INTERP_BILINEAR>(s, a, use_tma);
  else
    launch_warp_tiles<GG_INTERP_LANCZOS3>(s, a, use_tma);
}

// Host descriptors of a warp batch (validated; inverse coefficients).
static std::vector<WarpItem> warp_items_host(gg_stack* s, const int64_t* indices, int64_t count, const double* fwd) {
  std::vector<WarpItem> items(static_cast<size_t>(count));
  for (int64_t k = 0; k < count; ++k) {
    stack_require_loaded(s, indices[k], "warp");
    for (int64_t j = 0; j < k; ++j)
      if (indices[j] == indices[k]) fail(GG_ERR_INVALID_ARGUMENT, "frame indices of a warp batch must be unique");
    const double* m = fwd + 9 * k;
    for (int q = 0; q < 9; ++q)
      if (!std::isfinite(m[q])) fail(GG_ERR_INVALID_ARGUMENT, "warp matrix must be finite");
    WarpItem& it = items[static_cast<size_t>(k)];
    std::memset(&it, 0, sizeof(it));
    it.frame = static_cast<int>(indices[k]);
    if (!inverse_coefficients(m, it.m, it.affine)) fail(GG_ERR_INVALID_ARGUMENT, "warp matrix is singular");
    // an exact integer translation (identity linear part, integer shifts):
    // its inverse is one too and every source coordinate is an integer
    it.int_shift = (m[0] == 1.0 && m[1] == 0.0 && m[3] == 0.0 && m[4] == 1.0 && m[6] == 0.0 && m[7] == 0.0 &&
                    m[8] == 1.0 && m[2] == std::floor(m[2]) && m[5] == std::floor(m[5]) && std::fabs(m[2]) < 1.0e7 &&
                    std::fabs(m[5]) < 1.0e7)
                       ? 1
                       : 0;
  }
  return items;
}

// The kernels of a warp batch whose descriptors are already in device
// memory (d_items, `count` of them): per group of at most `spares` frames,
// resolve slots, warp into the spare slots, swap the slot table.  Only
// launches on the stack's stream (safe inside a stream capture).
static void launch_warp_items(gg_stack* s, WarpItem* d_items, int64_t count, int interp, float fill, float clamp,
                              bool track_coverage) {
  for (int64_t k0 = 0; k0 < count; k0 += s->spares) {
    const int nb = static_cast<int>(std::min<int64_t>(s->spares, count - k0));
    note_launch();
    warp_prepare_kernel<<<(nb + 127) / 128, 128, 0, s->stream>>>(d_items + k0, nb, s->d_slot_of_frame,
                                                                 s->d_spare_slot, s->d_frame_nonfinite, s->d_slots,
                                                                 s->stride);
    check_cuda(cudaGetLastError(), "warp_prepare launch");
    WarpArgs a = warp_args(s, d_items + k0, nb, 0, static_cast<int>(s->height));
    a.nonfinite = s->d_frame_nonfinite;
    a.fill = fill;
    a.clamp = clamp;
    a.coverage = track_coverage ? s->d_warp_coverage : nullptr;
    launch_warp_rows(s, a, interp);
    note_launch();
    warp_finish_kernel<<<(nb + 127) / 128, 128, 0, s->stream>>>(d_items + k0, nb, s->d_slot_of_frame,
                                                                s->d_spare_slot);
    check_cuda(cudaGetLastError(), "warp_finish launch");
  }
}

void warp_frames(gg_stack* s, const int64_t* indices, int64_t count, const double* fwd, int interp, float fill,
                 float clamp, bool track_coverage) {
  const std::vector<WarpItem> items = warp_items_host(s, indices, count, fwd);
  ensure_warp_items(s, std::max<int64_t>(count, s->spares));
  if (track_coverage) ensure_warp_coverage(s);
  // The staging buffer may still feed the previous call's copy.
  check_cuda(cudaEventSynchronize(s->warp_items_free), "cudaEventSynchronize(warp items)");
  std::memcpy(s->h_warp_items, items.data(), sizeof(WarpItem) * items.size());
  upload_params(s->stream, s->d_warp_items, s->h_warp_items, sizeof(WarpItem) * items.size(),
                "cudaMemcpyAsync(warp items)");
  check_cuda(cudaEventRecord(s->warp_items_free, s->stream), "cudaEventRecord(warp items)");
  launch_warp_items(s, static_cast<WarpItem*>(s->d_warp_items), count, interp, fill, clamp, track_coverage);
  if (track_coverage) s->warp_coverage_frames += count;
}

// Warp descriptors in a caller-owned device buffer (for captured graphs):
// returns the device pointer (cudaMalloc, the caller frees it with cudaFree)
// and their count through `count_out`.
void* warp_items_device(gg_stack* s, const int64_t* indices, int64_t count, const double* fwd) {
  const std::vector<WarpItem> items = warp_items_host(s, indices, count, fwd);
  void* d = nullptr;
  check_cuda(cudaMalloc(&d, sizeof(WarpItem) * items.size()), "cudaMalloc(graph warp items)");
  const cudaError_t err = cudaMemcpy(d, items.data(), sizeof(WarpItem) * items.size(), cudaMemcpyHostToDevice);
  if (err != cudaSuccess) {
    cudaFree(d);
    check_cuda(err, "cudaMemcpy(graph warp items)");
  }
  return d;
}

// ---- warp of every frame into a band of rows (fused warp + integration) --------
BandLayout warp_band_layout(const gg_stack* s) {
  BandLayout b;
  b.per_slot = static_cast<int>((s->frames + s->spares - 1) / s->spares);
  b.capacity = b.per_slot == 1 ? s->stride : s->stride / b.per_slot / 64 * 64;
  b.rows = static_cast<int>(std::min<int64_t>(s->height, b.capacity / s->width));
  // whole tile rows, so that only the last band has partial tiles
  if (b.rows < s->height && b.rows > kTileH) b.rows -= b.rows % kTileH;
  return b;
}

size_t warp_item_bytes() { return sizeof(WarpItem); }

// Descriptors and band buffers of every frame from its inverse coefficients.
// `own` (capacity samples per frame) takes the place of the spare slots when
// they hold less than a row per frame.
__global__ void warp_band_prepare_kernel(WarpItem* items, const FusedFrame* frames, int count,
                                         const int* slot_of_frame, const int* spare, const unsigned* nonfinite,
                                         float* slots, int64_t stride, int per_slot, int64_t capacity, float* own,
                                         const float** base, unsigned* counts) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count) return;
  WarpItem it{};
  it.frame = k;
  it.src_slot = slot_of_frame[k];
  it.dst_slot = -1;
  it.src_nonfinite = nonfinite[k];
  it.affine = frames[k].affine;
  it.dst = own ? own + k * capacity : slots + spare[k / per_slot] * stride + (k % per_slot) * capacity;
  for (int q = 0; q < 9; ++q) {
    it.m[q][0] = frames[k].m[q][0];
    it.m[q][1] = frames[k].m[q][1];
  }
  items[k] = it;
  base[k] = it.dst;
  counts[k] = 0u;
}

template <int INTERP>
__device__ __forceinline__ bool sample_valid(const Coef& co, int x, int y, int width, int height, FFv& sx, FFv& sy) {
  if (!source_coord(co, static_cast<float>(x), static_cast<float>(y), sx, sy)) return false;
  const float W = static_cast<float>(width), H = static_cast<float>(height);
  if (INTERP == GG_INTERP_LANCZOS3) return ff_ge(sx, 2.0f) && ff_lt(sx, W - 3.0f) && ff_ge(sy, 2.0f) && ff_lt(sy, H - 3.0f);
  return ff_ge(sx, 0.0f) && ff_le(sx, W - 1.0f) && ff_ge(sy, 0.0f) && ff_le(sy, H - 1.0f);
}

// Whether any sample of a frame's warp is non-finite, known before the first
// of several bands is integrated (one count is enough: it selects the
// integrator's all-valid formulas).  The valid source range is convex, so an
// affine map whose four corners are valid has only valid samples; the other
// frames have an invalid one.  What is left is scanned: projective maps, and
// frames that hold non-finite samples themselves.
template <int INTERP>
__global__ void __launch_bounds__(256) warp_nonfinite_kernel(WarpArgs a, unsigned* counts) {
  const WarpItem* ip = a.items + blockIdx.y;
  const Coef co = load_coef(ip);
  const unsigned src_nonfinite = ip->src_nonfinite;
  bool corners = true;
  FFv cx, cy;
#pragma unroll
  for (int c = 0; c < 4; ++c)
    corners = corners && sample_valid<INTERP>(co, (c & 1) ? a.width - 1 : 0, (c & 2) ? a.height - 1 : 0, a.width,
                                              a.height, cx, cy);
  if (!corners) {
    if (blockIdx.x == 0 && threadIdx.x == 0) counts[blockIdx.y] = 1u;
    return;
  }
  if (co.affine && src_nonfinite == 0u) return;
  TapSource ts;
  ts.tile = nullptr;
  ts.src = a.slots + static_cast<int64_t>(ip->src_slot) * a.stride;
  ts.bx = ts.by = 0;
  ts.width = a.width;
  const int64_t pixels = static_cast<int64_t>(a.width) * a.height;
  bool bad = false;
  for (int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; p < pixels && !bad;
       p += int64_t(gridDim.x) * blockDim.x) {
    const int y = static_cast<int>(p / a.width), x = static_cast<int>(p - static_cast<int64_t>(y) * a.width);
    FFv sx, sy;
    if (!sample_valid<INTERP>(co, x, y, a.width, a.height, sx, sy)) {
      bad = true;
      break;
    }
    int x0, y0;
    float tx, ty, v;
    ff_floor_frac(sx, x0, tx);
    ff_floor_frac(sy, y0, ty);
    if (INTERP == GG_INTERP_BILINEAR) v = sample_bilinear(ts, x0, y0, tx, ty, a.width, a.height);
    else if (!sample_lanczos3(ts, x0, y0, tx, ty, src_nonfinite == 0u, a.clamp, v)) v = __int_as_float(0x7fc00000);
    bad = !isfinite(v);
  }
  if (bad) counts[blockIdx.y] = 1u;
}

// Frames with a geometrically valid sample, per pixel of a band.  One CTA per
// 64 x 48 tile: a frame that maps the whole tile inside its valid range counts
// for every pixel without a test (all but the tiles along the border), the
// others are evaluated pixel by pixel.  Where a Lanczos3 frame holds
// non-finite samples, a window may have no weight left: its warped sample
// tells (NaN).
template <int INTERP>
__global__ void __launch_bounds__(kWarpThreads) warp_geometry_kernel(WarpArgs a, float* geometric) {
  __shared__ int s_inside, s_mixed;
  __shared__ int s_list[512];
  const int tile_x0 = blockIdx.x % a.tiles_x * kTileW, tile_y0 = a.row0 + blockIdx.x / a.tiles_x * kTileH;
  if (threadIdx.x == 0) s_inside = s_mixed = 0;
  __syncthreads();
  constexpr bool kLanczos = INTERP == GG_INTERP_LANCZOS3;
  const float vlo = kLanczos ? 2.0f : 0.0f, off = kLanczos ? 3.0f : 1.0f;
  for (int f = threadIdx.x; f < a.item_count; f += kWarpThreads) {
    const WarpItem* ip = a.items + f;
    const bool by_value = kLanczos && ip->src_nonfinite != 0u;
    const TilePlan p = plan_tile(load_coef(ip), tile_x0, tile_y0, kLanczos ? 3 : 1, vlo,
                                 static_cast<float>(a.width) - off, static_cast<float>(a.height) - off);
    if (p.interior && !by_value) atomicAdd(&s_inside, 1);
    else s_list[atomicAdd(&s_mixed, 1)] = f;
  }
  __syncthreads();
  const int ox = tile_x0 + (threadIdx.x & 63);
  if (ox >= a.width) return;
  int n[kRowsPerThread];
#pragma unroll
  for (int r = 0; r < kRowsPerThread; ++r) n[r] = s_inside;
  for (int i = 0; i < s_mixed; ++i) {
    const WarpItem* ip = a.items + s_list[i];
    const Coef co = load_coef(ip);
    const bool by_value = kLanczos && ip->src_nonfinite != 0u;
    const float* dst = ip->dst - static_cast<int64_t>(a.row0) * a.width;
    FFv sx, sy;
#pragma unroll
    for (int r = 0; r < kRowsPerThread; ++r) {
      const int oy = tile_y0 + (threadIdx.x >> 6) + 4 * r;
      if (oy >= a.row1) continue;
      if (by_value) n[r] += !isnan(dst[static_cast<int64_t>(oy) * a.width + ox]);
      else n[r] += sample_valid<INTERP>(co, ox, oy, a.width, a.height, sx, sy);
    }
  }
#pragma unroll
  for (int r = 0; r < kRowsPerThread; ++r) {
    const int oy = tile_y0 + (threadIdx.x >> 6) + 4 * r;
    if (oy < a.row1) geometric[static_cast<int64_t>(oy) * a.width + ox] = static_cast<float>(n[r]);
  }
}

void launch_warp_band(gg_stack* s, void* d_items, int interp, float clamp, int row0, int row1, unsigned* counts,
                      float* geometric) {
  WarpArgs a = warp_args(s, static_cast<WarpItem*>(d_items), static_cast<int>(s->frames), row0, row1);
  a.nonfinite = counts;
  a.fill = NAN;
  a.clamp = clamp;
  a.every_row = 1;  // the same validity as the geometric coverage below
  launch_warp_rows(s, a, interp);
  const unsigned tiles = static_cast<unsigned>(a.tiles_x) * static_cast<unsigned>(a.tiles_y);
  note_launch();
  if (interp == GG_INTERP_BILINEAR)
    warp_geometry_kernel<GG_INTERP_BILINEAR><<<tiles, kWarpThreads, 0, s->stream>>>(a, geometric);
  else
    warp_geometry_kernel<GG_INTERP_LANCZOS3><<<tiles, kWarpThreads, 0, s->stream>>>(a, geometric);
  check_cuda(cudaGetLastError(), "warp_geometry launch");
}

void launch_warp_band_prepare(gg_stack* s, void* d_items, const FusedFrame* d_frames, int interp, float clamp,
                              const BandLayout& band, float* own, const float** base, unsigned* counts) {
  const int n = static_cast<int>(s->frames);
  auto* items = static_cast<WarpItem*>(d_items);
  note_launch();
  warp_band_prepare_kernel<<<(n + 127) / 128, 128, 0, s->stream>>>(
      items, d_frames, n, s->d_slot_of_frame, s->d_spare_slot, s->d_frame_nonfinite, s->d_slots, s->stride,
      band.per_slot, band.capacity, own, base, counts);
  check_cuda(cudaGetLastError(), "warp_band_prepare launch");
  if (band.rows >= s->height) return;
  WarpArgs a = warp_args(s, items, n, 0, static_cast<int>(s->height));
  a.clamp = clamp;
  const dim3 grid(static_cast<unsigned>(std::max<int64_t>(
                      1, std::min<int64_t>((s->pixels + 255) / 256, sm_count() * 8 / n + 1))),
                  static_cast<unsigned>(n));
  note_launch();
  if (interp == GG_INTERP_BILINEAR)
    warp_nonfinite_kernel<GG_INTERP_BILINEAR><<<grid, 256, 0, s->stream>>>(a, counts);
  else
    warp_nonfinite_kernel<GG_INTERP_LANCZOS3><<<grid, 256, 0, s->stream>>>(a, counts);
  check_cuda(cudaGetLastError(), "warp_nonfinite launch");
}

void launch_warp_items_device(gg_stack* s, void* d_items, int64_t count, int interp, float fill, float clamp) {
  launch_warp_items(s, static_cast<WarpItem*>(d_items), count, interp, fill, clamp, false);
}

}  // namespace gg

using namespace gg;

extern "C" {

int gg_stack_warp_frames(gg_stack* s, const int64_t* indices, int64_t count, const double* host_matrices,
                         int interpolation, float fill, float clamping_threshold, int track_coverage) {
  GG_API_BEGIN
  require(s != nullptr && indices != nullptr && host_matrices != nullptr, "null argument");
  require(count > 0, "indices must contain at least one frame index");
  require(interpolation == GG_INTERP_NEAREST || interpolation == GG_INTERP_BILINEAR ||
              interpolation == GG_INTERP_LANCZOS3,
          "interpolation must be nearest, bilinear or lanczos3");
  require(s->width < (1 << 24) && s->height < (1 << 24), "frame too large for float coordinates");
  stack_activate(s);
  warp_frames(s, indices, count, host_matrices, interpolation, fill, clamping_threshold, track_coverage != 0);
  GG_API_END
}

int gg_stack_reset_warp_coverage(gg_stack* s) {
  GG_API_BEGIN
  require(s != nullptr, "stack is null");
  stack_activate(s);
  ensure_warp_coverage(s);
  check_cuda(cudaMemsetAsync(s->d_warp_coverage, 0, sizeof(float) * s->pixels, s->stream), "cudaMemsetAsync");
  s->warp_coverage_frames = 0;
  GG_API_END
}

int gg_stack_accumulate_full_warp_coverage_frame(gg_stack* s) {
  GG_API_BEGIN
  require(s != nullptr, "stack is null");
  stack_activate(s);
  ensure_warp_coverage(s);
  note_launch();
  add_scalar_kernel<<<grid_for(static_cast<size_t>(s->pixels), 256, 4), 256, 0, s->stream>>>(s->d_warp_coverage,
                                                                                            s->pixels, 1.0f);
  check_cuda(cudaGetLastError(), "add_scalar launch");
  s->warp_coverage_frames += 1;
  GG_API_END
}

int gg_stack_download_warp_coverage(gg_stack* s, float* host_out) {
  GG_API_BEGIN
  require(s != nullptr && host_out != nullptr, "null argument");
  stack_activate(s);
  ensure_warp_coverage(s);
  check_cuda(cudaMemcpyAsync(host_out, s->d_warp_coverage, sizeof(float) * s->pixels, cudaMemcpyDeviceToHost,
                             s->stream),
             "cudaMemcpyAsync(warp coverage)");
  check_cuda(cudaStreamSynchronize(s->stream), "cudaStreamSynchronize(warp coverage)");
  stack_check_device_error(s);
  GG_API_END
}

int gg_stack_tma_enabled(gg_stack* s, int* enabled) {
  GG_API_BEGIN
  require(s != nullptr && enabled != nullptr, "null argument");
  *enabled = s->has_slot_tmap ? 1 : 0;
  GG_API_END
}

int gg_warp_matrix_f32(const float* host_in, int64_t height, int64_t width, const double* host_matrix,
                       int interpolation, float fill, float clamping_threshold, float* host_out,
                       float* host_coverage) {
  GG_API_BEGIN
  require(host_in != nullptr && host_matrix != nullptr && host_out != nullptr, "null argument");
  gg_stack* s = nullptr;
  int rc = gg_stack_create(1, height, width, &s);
  if (rc != GG_OK) fail(rc, "temporary stack: create failed");
  struct Guard {
    gg_stack* s;
    ~Guard() { gg_stack_destroy(s); }
  } guard{s};
  rc = gg_stack_upload_frame(s, 0, host_in);
  if (rc != GG_OK) fail(rc, "temporary stack: upload failed");
  const int64_t idx = 0;
  if (host_coverage) {
    rc = gg_stack_reset_warp_coverage(s);
    if (rc != GG_OK) fail(rc, "temporary stack: coverage reset failed");
  }
  warp_frames(s, &idx, 1, host_matrix, interpolation, fill, clamping_threshold, host_coverage != nullptr);
  rc = gg_stack_download_frame_tile(s, 0, 0, 0, width, height, host_out);
  if (rc != GG_OK) fail(rc, "temporary stack: download failed");
  if (host_coverage) {
    rc = gg_stack_download_warp_coverage(s, host_coverage);
    if (rc != GG_OK) fail(rc, "temporary stack: coverage download failed");
  }
  GG_API_END
}

}  // extern "C"
