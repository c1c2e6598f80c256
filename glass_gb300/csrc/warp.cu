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
//   - each CTA takes 64x64 output tiles; a tile's source footprint (an 80x80
//     box for the small rotations registration produces) is copied to shared
//     memory by one cp.async.bulk.tensor (TMA) load while the SM's other CTAs
//     compute.  Larger rotations take shorter tiles, whose footprints fit the box
//     again; where none does (scale), and at image widths that TMA cannot describe
//     (W % 4 != 0), a launch without boxes reads the taps straight from global
//     memory (WarpForm);
//   - output goes to a spare slot; the launch's last CTA swaps the frame->slot
//     table, so nothing is copied back (8 B/pixel instead of 16 B);
//   - Lanczos3 weights are paired even/odd polynomials in (t - 1/2)^2
//     (sampling.cuh); tiles of affine maps run straight-line rows: two columns
//     per thread in packed float32, coordinates in fixed point, two output rows
//     from seven source rows.  Projective maps, the overshoot clamp, nearest
//     and very large footprints take the general path (warp_tile_rows).
//
// Bound: the FMA pipe (of 143 instructions per Lanczos3 pixel, the weights are
// 41 packed, the taps 21; 57 % of the pipe, 56 % of the issue slots at 16 warps
// per SM).  15 moving frames of 2048^2: Lanczos3 642 -> 438 us, bilinear 417 ->
// 159 us; frames with non-finite samples (23 of 512^2, Lanczos3) 275 -> 227 us.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <type_traits>
#include <vector>

#include <cudaTypedefs.h>

#include "async.cuh"
#include "sampling.cuh"
#include "stack.cuh"
#include "warp_band.cuh"

namespace gg {

constexpr int kTileW = 64;
constexpr int kTileH = 64;       // rows of a tile
constexpr int kMidTileH = 48;    // where a footprint of 64 rows does not fit the box
constexpr int kSmallTileH = 16;  // where one of 48 does not, or a launch has few tiles
constexpr int kWarpThreads = 128;
constexpr int kRowClasses = 4;  // rows y, y + 4, y + 8, ... of a tile share a chain of coordinates
// Affine source coordinates are stepped by 4 output rows in float-float and
// evaluated afresh every kFreshRows rows: at most three steps of rounding
// separate a coordinate from the float64-faithful evaluation, so floor and
// fraction decisions stay those of a direct evaluation.  Tile heights are
// multiples of 16 rows, so a row's chain does not depend on its tile.
constexpr int kFreshRows = 4;

struct WarpItem {
  int frame;
  int src_slot;     // filled on the device
  int dst_slot;     // filled on the device (-1: not a slot)
  unsigned src_nonfinite;
  int affine;
  int int_shift;  // inverse is an exact integer translation
  int form;       // WarpForm
  float* dst;     // first row of the output rows (filled on the device)
  float m[9][2];  // inverse matrix, float-float (hi, lo), row-major
  double inv[6];  // its first two rows
};

struct WarpArgs {
  float* slots;
  unsigned* nonfinite;  // per frame: non-finite output samples are added
  // in-place warp: the last CTA makes the output slots the frames' own
  int* slot_of_frame;  // nullptr: not an in-place warp
  int* spare;
  unsigned* ticket;
  WarpItem* items;
  int item_count;
  int64_t stride;
  int width;
  int height;
  int row0, row1;  // output rows [row0, row1); row0 is the first row at WarpItem::dst
  int tiles_x;
  int tiles_y;     // of those rows (set by the launch)
  float fill;
  float clamp;
  float* coverage;  // optional accumulator (+1 per covered pixel)
  int counted;      // whole tiles (counts_whole) are in it already
  int* error;
};

// How a launch takes its frames: staged boxes of tiles of 64, 48 or 16 rows, or
// windows straight from global memory, by straight-line rows or by the general
// path alone.
//
// Two boxes in each of four CTAs leave next to no L1, and a tile whose footprint
// misses its box reads its windows through it.  So the launch's form goes by the
// maps: the tallest tiles whose footprints fit (a shorter tile pays more for its
// plan and its box), else no boxes, and then the general path without the
// registers of the straight-line rows.  8 frames of 2048^2, us, boxes of 64 rows
// whatever the map -> by form:
//                        Lanczos3       Lanczos3, clamp  bilinear     nearest
//   turned by  7 degrees  376 -> 290       704 -> 502     98 -> 100   218 -> 218
//             20          986 -> 375      1026 -> 544    210 -> 163   329 -> 252
//             45         2123 -> 380      1259 -> 524    307 -> 161   313 -> 252
//   scaled by  1.15       421 -> 392       981 -> 621    182 -> 190   349 -> 276
//              2          415 -> 385       797 -> 487    188 -> 184   309 -> 223
// Without boxes at all (2048 x 2046): clamp 840 -> 660, nearest 308 -> 273.
enum WarpForm { kStaged64, kStaged48, kStaged16, kDirectRows, kDirectGeneral, kWarpForms };

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
  int grid;  // affine, and small enough for the fixed-point coordinates
};

// Source range of a tile: bounding box of its corners' source points; !ok: a
// corner has none.
struct TileRange {
  float minx, maxx, miny, maxy;
  bool ok;
};

// interior: an affine map sends the whole tile at least one pixel inside the
// valid source range (valid_lo <= s <= valid_hi on both axes), so no pixel
// of the tile needs its own validity test.
__device__ __forceinline__ TilePlan plan_of_range(const TileRange& s, bool affine, int radius, float valid_lo,
                                                  float valid_hi_x, float valid_hi_y) {
  TilePlan p{0, 0, 0, 0, 0};
  if (!s.ok || !(s.maxx - s.minx < 1.0e6f) || !(s.maxy - s.miny < 1.0e6f) || fabsf(s.minx) > 1.0e8f ||
      fabsf(s.miny) > 1.0e8f)
    return p;
  // taps span [floor(s) - (radius-1), floor(s) + radius]; one pixel of margin.
  const int lo_x = static_cast<int>(floorf(s.minx)) - radius;
  const int hi_x = static_cast<int>(floorf(s.maxx)) + radius + 1;  // inclusive
  const int lo_y = static_cast<int>(floorf(s.miny)) - radius;
  const int hi_y = static_cast<int>(floorf(s.maxy)) + radius + 1;
  p.bx = lo_x >= 0 ? (lo_x & ~3) : -((-lo_x + 3) & ~3);  // 16-byte aligned x (TMA rule)
  p.by = lo_y;
  p.fits = (hi_x - p.bx < kBoxW) && (hi_y - p.by < kBoxH);
  p.grid = affine && s.maxx - s.minx < 256.0f && s.maxy - s.miny < 256.0f;
  p.interior = affine && s.minx >= valid_lo + 1.0f && s.maxx <= valid_hi_x - 1.0f && s.miny >= valid_lo + 1.0f &&
               s.maxy <= valid_hi_y - 1.0f;
  return p;
}

template <int TH>
__device__ __forceinline__ TilePlan plan_tile(const Coef& it, int tile_x0, int tile_y0, int radius, float valid_lo,
                                              float valid_hi_x, float valid_hi_y) {
  TileRange s{kInfF, -kInfF, kInfF, -kInfF, true};
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    FFv sx, sy;
    s.ok &= source_coord(it, static_cast<float>(tile_x0 + (c & 1) * (kTileW - 1)),
                         static_cast<float>(tile_y0 + (c >> 1) * (TH - 1)), sx, sy);
    s.minx = fminf(s.minx, sx.hi);
    s.maxx = fmaxf(s.maxx, sx.hi);
    s.miny = fminf(s.miny, sy.hi);
    s.maxy = fmaxf(s.maxy, sy.hi);
  }
  return plan_of_range(s, it.affine != 0, radius, valid_lo, valid_hi_x, valid_hi_y);
}

// plan_tile by a whole warp, a corner per lane (the plan in every lane).
template <int TH>
__device__ __forceinline__ TilePlan plan_tile_warp(const Coef& it, int tile_x0, int tile_y0, int radius,
                                                   float valid_lo, float valid_hi_x, float valid_hi_y) {
  const int c = threadIdx.x & 3;
  FFv sx, sy;
  TileRange s;
  s.ok = __all_sync(0xffffffffu, source_coord(it, static_cast<float>(tile_x0 + (c & 1) * (kTileW - 1)),
                                              static_cast<float>(tile_y0 + (c >> 1) * (TH - 1)), sx, sy));
  s.minx = s.maxx = sx.hi;
  s.miny = s.maxy = sy.hi;
#pragma unroll
  for (int off = 1; off < 4; off <<= 1) {
    s.minx = fminf(s.minx, __shfl_xor_sync(0xffffffffu, s.minx, off));
    s.maxx = fmaxf(s.maxx, __shfl_xor_sync(0xffffffffu, s.maxx, off));
    s.miny = fminf(s.miny, __shfl_xor_sync(0xffffffffu, s.miny, off));
    s.maxy = fmaxf(s.maxy, __shfl_xor_sync(0xffffffffu, s.maxy, off));
  }
  return plan_of_range(s, it.affine != 0, radius, valid_lo, valid_hi_x, valid_hi_y);
}

// The output pixels of one column and row class of a tile: column ox, rows oy0,
// oy0 + 4, ...; dst is the frame's output row 0.
// FINITE: the source frame holds no non-finite sample (every Lanczos3 window
// takes the plain normalised sum); returns the count of non-finite outputs.
template <int INTERP, bool FINITE, int TH>
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
  for (int r = 0; r < TH / kRowClasses; ++r) {
    const int oy = oy0 + 4 * r;
    const bool inside = ox < a.width && oy < a.row1;
    bool valid = false;
    float value = a.fill;
    if (co.affine) {
      if (r % kFreshRows == 0) {
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

// ---- straight-line rows ---------------------------------------------------------
// Tiles of an affine map (Lanczos3: without clamp), with the arithmetic of
// the general path but for the coordinates' last bits.  A thread takes 16 (4 in
// small tiles) consecutive rows of two columns, x and x + 32, as the two lanes of
// packed float32.  Interior tiles (mapped at least one pixel inside the valid
// source range, whole inside the output) need no test per pixel; the others are
// masked.

// Source coordinates within a tile, in fixed point with 54 fraction bits
// relative to a whole origin (the staged box, or the tile's first source pixel):
// a step along a row or column is an exact integer add on the otherwise idle
// integer pipe, where the float-float step took 11 of the FMA pipe's operations
// per axis.  The tile's first coordinate is evaluated in float64, the steps'
// rounding moves a coordinate by at most 128 x 2^-55 pixels within a tile: as
// close to the float64 reference as its own rounding.
constexpr int kGridBits = 54;

struct TileGrid {
  long long x0, y0;  // source of the tile's first pixel, relative to (ox, oy)
  long long a, d, b, e;  // steps of x and y along a row, down a column
  int ox, oy;
};

// By a whole warp: lanes 0 to 5 make one value each.
__device__ __forceinline__ void tile_grid_warp(const double* inv, int tile_x0, int tile_y0, bool staged, int bx,
                                               int by, TileGrid& out) {
  const int lane = threadIdx.x & 31, axis = lane & 1;
  const double* row = inv + 3 * axis;
  constexpr double kOne = static_cast<double>(1ll << kGridBits);
  double v;
  int origin = 0;
  if (lane < 2) {
    v = fma(row[0], static_cast<double>(tile_x0), fma(row[1], static_cast<double>(tile_y0), row[2]));
    origin = staged ? (axis ? by : bx) : static_cast<int>(floor(v));
    v -= origin;
  } else {
    v = lane < 4 ? row[0] : row[1];
  }
  if (lane < 6) (&out.x0)[lane] = __double2ll_rn(v * kOne);
  if (lane < 2) (&out.ox)[lane] = origin;
}

constexpr float kTwoToMinus24 = 5.9604644775390625e-08f;

// The coordinates of a thread's two columns, x and x + 32, down its rows.
struct RowWalk {
  long long xa, xb, ya, yb;
  __device__ __forceinline__ RowWalk(const TileGrid& g, int lx, int ly) {
    xa = g.x0 + lx * g.a + ly * g.b;
    ya = g.y0 + lx * g.d + ly * g.e;
    xb = xa + 32 * g.a;
    yb = ya + 32 * g.d;
  }
  __device__ __forceinline__ void next(const TileGrid& g) {
    xa += g.b;
    xb += g.b;
    ya += g.e;
    yb += g.e;
  }
  static __device__ __forceinline__ int whole(long long v) { return static_cast<int>(v >> kGridBits); }
  // 2^24 times the fractions of both columns, rounded once to float32: two exact
  // halves of 24 bits and an FMA.
  static __device__ __forceinline__ F2 fraction24(long long p, long long q) {
    auto high = [](long long v) { return __uint2float_rn(static_cast<unsigned>(v >> (kGridBits - 24)) & 0xffffffu); };
    auto low = [](long long v) { return __uint2float_rn(static_cast<unsigned>(v >> (kGridBits - 48)) & 0xffffffu); };
    return f2_fma(f2(low(p), low(q)), f2(kTwoToMinus24), f2(high(p), high(q)));
  }
  __device__ __forceinline__ F2 x24() const { return fraction24(xa, xb); }
  __device__ __forceinline__ F2 y24() const { return fraction24(ya, yb); }
};

// Pixels of a masked tile: those inside the output (columns left of ncols, rows
// above nrows of the tile) are written, and valid where the source coordinate
// lies in [lo, hi) on both axes.
struct TileMask {
  long long lox, hix, loy, hiy;
  int ncols, nrows;
  float* coverage;  // optional: +1 per valid pixel, laid out like the output
};

__device__ __forceinline__ TileMask tile_mask(const TileGrid& g, bool lanczos, int width, int height, int tile_x0,
                                              int tile_y0, int row1, float* coverage) {
  auto fixed = [](int v) { return static_cast<long long>(min(max(v, -511), 511)) << kGridBits; };
  const int lo = lanczos ? 2 : 0, off = lanczos ? 3 : 1;
  TileMask m;
  m.lox = fixed(lo - g.ox);
  m.loy = fixed(lo - g.oy);
  // bilinear takes the last sample itself too
  m.hix = fixed(width - off - g.ox) + (lanczos ? 0 : 1);
  m.hiy = fixed(height - off - g.oy) + (lanczos ? 0 : 1);
  m.ncols = width - tile_x0;
  m.nrows = row1 - tile_y0;
  m.coverage = coverage;
  return m;
}

// Samples of the staged box (kBoxW columns) or of the frame itself, at positions
// relative to the grid's origin; (x0, y0) to (x1, y1) are the first and last that
// a window may start at.  CLAMP keeps the windows of invalid pixels inside the
// frame (the staged box holds them all).
template <bool STAGED>
struct Window {
  static constexpr bool kStaged = STAGED;
  using Index = std::conditional_t<STAGED, int, int64_t>;
  const float* data;
  int width;
  int x0, x1, y0, y1;
  __device__ __forceinline__ int pitch() const { return STAGED ? kBoxW : width; }
  template <bool CLAMP>
  __device__ __forceinline__ Index at(int x, int y) const {
    if constexpr (CLAMP && !STAGED) {
      x = min(max(x, x0), x1);
      y = min(max(y, y0), y1);
    }
    return static_cast<Index>(y) * pitch() + x;
  }
  __device__ __forceinline__ float load(Index i) const { return STAGED ? data[i] : __ldg(data + i); }
};

// Writes one pixel of a masked tile (`sampled`: its window has a value); returns
// whether it is non-finite.
__device__ __forceinline__ unsigned write_masked(const TileMask& m, float* out, int64_t at, int lx, int ly,
                                                 long long x, long long y, float value, float fill,
                                                 bool sampled = true) {
  const bool valid = sampled && x >= m.lox && x < m.hix && y >= m.loy && y < m.hiy;
  if (lx >= m.ncols || ly >= m.nrows) return 0u;
  const float v = valid ? value : fill;
  out[at] = v;
  if (m.coverage && valid) atomicAdd(m.coverage + at, 1.0f);
  return isfinite(v) ? 0u : 1u;
}

// Non-finite samples among those that a thread wrote (all finite but for
// overflow: counted only when their product with zero is not zero).
__device__ __forceinline__ unsigned count_nonfinite(F2 probe, const float* out, int64_t pitch, int rows) {
  if (f2_sum(probe) == 0.0f) return 0u;
  unsigned bad = 0;
  for (int r = 0; r < rows; ++r) {
    bad += isfinite(out[r * pitch]) ? 0u : 1u;
    bad += isfinite(out[r * pitch + 32]) ? 0u : 1u;
  }
  return bad;
}

// Sums of both columns' 6 x 6 windows at na, nb.
template <bool STAGED>
__device__ __forceinline__ F2 window_sum(const Window<STAGED>& win, typename Window<STAGED>::Index na,
                                         typename Window<STAGED>::Index nb, const F2 (&wx)[6], const F2 (&wy)[6]) {
  F2 acc;
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    F2 row;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const F2 v = f2(win.load(na + j * win.pitch() + i), win.load(nb + j * win.pitch() + i));
      row = i == 0 ? f2_mul(wx[0], v) : f2_fma(wx[i], v, row);
    }
    acc = j == 0 ? f2_mul(wy[0], row) : f2_fma(wy[j], row, acc);
  }
  return acc;
}

// Lanczos3, two rows at a time: where the second row's windows lie one source
// row below the first's (nearly always: scale and rotation move them by
// hundredths of a pixel per row), the seven source rows are loaded once for
// both, 21 loads per sample instead of 36.  (Windows kept in registers over all
// 16 rows need 6 loads, but a loop unrolled by 6 rows, and 30 KB of it starved
// the instruction cache: 843 us for five 4096^2 frames.)
template <int ROWS, bool STAGED, bool MASK>
__device__ __forceinline__ unsigned lanczos3_rows(const TileGrid& grid, const Window<STAGED> win,
                                                  const TileMask& mask, float fill, float* out, int64_t out_pitch,
                                                  int lx, int ly) {
  RowWalk at(grid, lx, ly);
  const int pitch = win.pitch();
  F2 probe;
  unsigned bad = 0;
#pragma unroll 1
  for (int r = 0; r < ROWS; r += 2) {
    typename Window<STAGED>::Index na[2], nb[2];
    F2 t[4], w[4][6], wsum[2];  // x and y of the first row, x and y of the second
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      t[2 * q] = at.x24();
      t[2 * q + 1] = at.y24();
      na[q] = win.template at<MASK>(RowWalk::whole(at.xa) - 2, RowWalk::whole(at.ya) - 2);
      nb[q] = win.template at<MASK>(RowWalk::whole(at.xb) - 2, RowWalk::whole(at.yb) - 2);
      at.next(grid);
    }
    lanczos3_weights2(t, w);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      F2 swx = w[2 * q][0], swy = w[2 * q + 1][0];
#pragma unroll
      for (int i = 1; i < 6; ++i) {
        swx = f2_add(swx, w[2 * q][i]);
        swy = f2_add(swy, w[2 * q + 1][i]);
      }
      wsum[q] = f2_mul(swx, swy);
    }
    F2 acc[2];
    if (__builtin_expect(__all_sync(0xffffffffu, na[1] == na[0] + pitch && nb[1] == nb[0] + pitch), 1)) {
#pragma unroll
      for (int j = 0; j < 7; ++j) {
        F2 v[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) v[i] = f2(win.load(na[0] + j * pitch + i), win.load(nb[0] + j * pitch + i));
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int k = j - q;  // row of this window
          if (k < 0 || k > 5) continue;
          F2 row = f2_mul(w[2 * q][0], v[0]);
#pragma unroll
          for (int i = 1; i < 6; ++i) row = f2_fma(w[2 * q][i], v[i], row);
          acc[q] = k == 0 ? f2_mul(w[2 * q + 1][0], row) : f2_fma(w[2 * q + 1][k], row, acc[q]);
        }
      }
    } else {
#pragma unroll
      for (int q = 0; q < 2; ++q) acc[q] = window_sum(win, na[q], nb[q], w[2 * q], w[2 * q + 1]);
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      float sa, sb, da, db;
      f2_split(acc[q], sa, sb);
      f2_split(wsum[q], da, db);
      // all taps count: the weights sum to 1 within a few per cent
      const float va = __fdividef(sa, da), vb = __fdividef(sb, db);
      if constexpr (MASK) {
        // the walk has moved on by two rows
        const long long k = 2 - q;
        bad += write_masked(mask, out, (r + q) * out_pitch, lx, ly + r + q, at.xa - k * grid.b, at.ya - k * grid.e,
                            va, fill);
        bad += write_masked(mask, out, (r + q) * out_pitch + 32, lx + 32, ly + r + q, at.xb - k * grid.b,
                            at.yb - k * grid.e, vb, fill);
      } else {
        out[(r + q) * out_pitch] = va;
        out[(r + q) * out_pitch + 32] = vb;
        probe = f2_fma(f2(va, vb), F2(), probe);
      }
    }
  }
  return MASK ? bad : count_nonfinite(probe, out, out_pitch, ROWS);
}

// Lanczos3 from a frame with non-finite samples: the float-float sums over the
// finite taps and their weights (lanczos3_nonfinite), where a tap that does not
// count adds an exact zero.
template <int ROWS, bool STAGED>
__device__ __forceinline__ unsigned lanczos3_renorm_rows(const TileGrid& grid, const Window<STAGED> win,
                                                         const TileMask& mask, float fill, float* out,
                                                         int64_t out_pitch, int lx, int ly) {
  RowWalk at(grid, lx, ly);
  const int pitch = win.pitch();
  unsigned bad = 0;
#pragma unroll 1
  for (int r = 0; r < ROWS; ++r) {
    float wxa[6], wxb[6], wya[6], wyb[6], ta, tb;
    f2_split(f2_mul(at.x24(), f2(kTwoToMinus24)), ta, tb);
    lanczos3_weights_trig(ta, wxa);
    lanczos3_weights_trig(tb, wxb);
    f2_split(f2_mul(at.y24(), f2(kTwoToMinus24)), ta, tb);
    lanczos3_weights_trig(ta, wya);
    lanczos3_weights_trig(tb, wyb);
    auto na = win.template at<true>(RowWalk::whole(at.xa) - 2, RowWalk::whole(at.ya) - 2);
    auto nb = win.template at<true>(RowWalk::whole(at.xb) - 2, RowWalk::whole(at.yb) - 2);
    FF2 sum, weight;
#pragma unroll 1
    for (int j = 0; j < 6; ++j, na += pitch, nb += pitch) {
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        const float a = win.load(na + i), b = win.load(nb + i);
        const bool fa = isfinite(a), fb = isfinite(b);
        const F2 v = f2(fa ? a : 0.0f, fb ? b : 0.0f);
        const F2 w = f2(fa ? wya[j] * wxa[i] : 0.0f, fb ? wyb[j] * wxb[i] : 0.0f);
        const F2 p = f2_mul(w, v);
        const F2 pe = f2_fma(w, v, f2_sub(F2(), p));
        sum.add(p);
        sum.lo = f2_add(sum.lo, pe);
        weight.add(w);
      }
    }
    float sh[2], sl[2], wh[2], wl[2];
    f2_split(sum.hi, sh[0], sh[1]);
    f2_split(sum.lo, sl[0], sl[1]);
    f2_split(weight.hi, wh[0], wh[1]);
    f2_split(weight.lo, wl[0], wl[1]);
    float value[2];
    bool sampled[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      sampled[k] = fabsf(__fadd_rn(wh[k], wl[k])) > 1.0e-12f;
      value[k] = ff_div_ff(sh[k], sl[k], wh[k], wl[k]);
    }
    bad += write_masked(mask, out, r * out_pitch, lx, ly + r, at.xa, at.ya, value[0], fill, sampled[0]);
    bad += write_masked(mask, out, r * out_pitch + 32, lx + 32, ly + r, at.xb, at.yb, value[1], fill, sampled[1]);
    at.next(grid);
  }
  return bad;
}

// Lanczos3 by a whole shift: the weights are exactly 0, 0, 1, 0, 0, 0, so each
// sample is the source's own, or none where that is not finite.
template <int ROWS, bool STAGED>
__device__ __forceinline__ unsigned shifted_rows(const TileGrid& grid, const Window<STAGED> win, const TileMask& mask,
                                                 float fill, float* out, int64_t out_pitch, int lx, int ly) {
  RowWalk at(grid, lx, ly);
  unsigned bad = 0;
#pragma unroll 4
  for (int r = 0; r < ROWS; ++r) {
    const auto na = win.template at<true>(RowWalk::whole(at.xa) - 2, RowWalk::whole(at.ya) - 2);
    const auto nb = win.template at<true>(RowWalk::whole(at.xb) - 2, RowWalk::whole(at.yb) - 2);
    const float a = win.load(na + 2 * win.pitch() + 2), b = win.load(nb + 2 * win.pitch() + 2);
    bad += write_masked(mask, out, r * out_pitch, lx, ly + r, at.xa, at.ya, a, fill, isfinite(a));
    bad += write_masked(mask, out, r * out_pitch + 32, lx + 32, ly + r, at.xb, at.yb, b, fill, isfinite(b));
    at.next(grid);
  }
  return bad;
}

// Sum of two packed products, lane by lane (each product rounded).
__device__ __forceinline__ F2 add_products(F2 a, F2 b) {
  float ax, ay, bx, by;
  f2_split(a, ax, ay);
  f2_split(b, bx, by);
  return f2(__fadd_rn(ax, bx), __fadd_rn(ay, by));
}

// Bilinear.
template <int ROWS, bool STAGED, bool MASK>
__device__ __forceinline__ unsigned bilinear_rows(const TileGrid& grid, const Window<STAGED> win,
                                                  const TileMask& mask, float fill, float* out, int64_t out_pitch,
                                                  int lx, int ly) {
  RowWalk at(grid, lx, ly);
  const int pitch = win.pitch();
  F2 probe;
  unsigned bad = 0;
#pragma unroll 4
  for (int r = 0; r < ROWS; ++r) {
    const F2 tx = f2_mul(at.x24(), f2(kTwoToMinus24)), ty = f2_mul(at.y24(), f2(kTwoToMinus24));
    const int xa = RowWalk::whole(at.xa), xb = RowWalk::whole(at.xb);
    const int ya = RowWalk::whole(at.ya), yb = RowWalk::whole(at.yb);
    const auto na = win.template at<MASK>(xa, ya), nb = win.template at<MASK>(xb, yb);
    // the last column's and row's right and lower neighbours are themselves, and so
    // are those of a position outside (its clamped place may be the last one: a
    // frame of one row or column has no other)
    auto step = [](int at_, int first, int last, int by) { return !MASK || (at_ >= first && at_ < last) ? by : 0; };
    const int ra = step(xa, win.x0, win.x1, 1), rb = step(xb, win.x0, win.x1, 1);
    const int da = step(ya, win.y0, win.y1, pitch), db = step(yb, win.y0, win.y1, pitch);
    const F2 v00 = f2(win.load(na), win.load(nb)), v01 = f2(win.load(na + ra), win.load(nb + rb));
    const F2 v10 = f2(win.load(na + da), win.load(nb + db));
    const F2 v11 = f2(win.load(na + da + ra), win.load(nb + db + rb));
    const F2 one = f2(1.0f), ox_ = f2_sub(one, tx), oy_ = f2_sub(one, ty);
    const F2 top = add_products(f2_mul(v00, ox_), f2_mul(v01, tx));
    const F2 bottom = add_products(f2_mul(v10, ox_), f2_mul(v11, tx));
    const F2 v = add_products(f2_mul(top, oy_), f2_mul(bottom, ty));
    float va, vb;
    f2_split(v, va, vb);
    if constexpr (MASK) {
      bad += write_masked(mask, out, r * out_pitch, lx, ly + r, at.xa, at.ya, va, fill);
      bad += write_masked(mask, out, r * out_pitch + 32, lx + 32, ly + r, at.xb, at.yb, vb, fill);
    } else {
      out[r * out_pitch] = va;
      out[r * out_pitch + 32] = vb;
      probe = f2_fma(v, F2(), probe);
    }
    at.next(grid);
  }
  return MASK ? bad : count_nonfinite(probe, out, out_pitch, ROWS);
}

// Whether every pixel of a tile is known to be valid: such tiles take the
// unmasked rows.
template <int INTERP, int TH>
__device__ __forceinline__ bool counts_whole(const WarpArgs& a, const TilePlan& p, bool finite, int tile_x0,
                                             int tile_y0) {
  const bool full_tile = tile_x0 + kTileW <= a.width && tile_y0 + TH <= a.row1;
  return p.interior && p.grid && full_tile && (INTERP != GG_INTERP_LANCZOS3 || (finite && a.clamp < 0.0f));
}

// Two box buffers: the next tile's copy is in flight while this one's rows are
// computed.
constexpr size_t kWarpTileBytes = size_t(2) * kBoxH * kBoxW * sizeof(float);

// GENERAL: the general path alone.
template <int INTERP, bool USE_TMA, int TH, bool GENERAL = false>
__global__ void __launch_bounds__(kWarpThreads, GENERAL ? 6 : 4)
    warp_tiles_kernel(const __grid_constant__ CUtensorMap tmap, WarpArgs a) {
  extern __shared__ __align__(128) float warp_boxes[];  // USE_TMA: [2][kBoxH * kBoxW]
  __shared__ alignas(8) uint64_t bar[2];
  __shared__ TilePlan s_plan[2];
  __shared__ TileGrid s_grid[2];
  __shared__ int s_abort;
  constexpr bool kLanczos = INTERP == GG_INTERP_LANCZOS3;
  const int tid = threadIdx.x;
  const int tiles = a.tiles_x * a.tiles_y;
  const int items = a.item_count * tiles;
  if (tid == 0) {
    s_abort = 0;
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  // Warp 0 plans a tile and starts its copy.
  auto issue = [&](int item, int buf) {
    const WarpItem* ip = a.items + item / tiles;
    const Coef co = load_coef(ip);
    const int t = item % tiles, tile_x0 = t % a.tiles_x * kTileW, tile_y0 = a.row0 + t / a.tiles_x * TH;
    // validity ranges: bilinear 0 <= s <= W - 1; Lanczos3 2 <= s < W - 3
    const float vlo = kLanczos ? 2.0f : 0.0f, off = kLanczos ? 3.0f : 1.0f;
    TilePlan p = plan_tile_warp<TH>(co, tile_x0, tile_y0, kLanczos ? 3 : 1, vlo, static_cast<float>(a.width) - off,
                                static_cast<float>(a.height) - off);
    if (!USE_TMA) p.fits = 0;
    if (INTERP != GG_INTERP_NEAREST && !GENERAL && p.grid)
      tile_grid_warp(ip->inv, tile_x0, tile_y0, p.fits != 0, p.bx, p.by, s_grid[buf]);
    if (tid != 0) return;
    s_plan[buf] = p;
    if (p.fits) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_expect_tx(&bar[buf], kBoxW * kBoxH * 4);
      tma_load_3d(warp_boxes + buf * (kBoxH * kBoxW), &tmap, p.bx, p.by, __ldg(&ip->src_slot), &bar[buf]);
    }
  };

  unsigned phase[2] = {0u, 0u};
  int item = blockIdx.x;
  if (tid < 32 && item < items) issue(item, 0);
  __syncthreads();
  for (int i = 0; item < items; ++i, item += gridDim.x) {
    const int buf = i & 1;
    const int next = item + gridDim.x;
    if (tid < 32 && next < items) issue(next, buf ^ 1);
    const TilePlan p = s_plan[buf];
    const float* tile = warp_boxes + buf * (kBoxH * kBoxW);
    const int item_index = item / tiles;
    const WarpItem* ip = a.items + item_index;
    const int it_frame = __ldg(&ip->frame);
    const float* src = a.slots + static_cast<int64_t>(__ldg(&ip->src_slot)) * a.stride;
    float* const dst = ip->dst - static_cast<int64_t>(a.row0) * a.width;
    const bool finite = __ldg(&ip->src_nonfinite) == 0u;
    const bool int_shift = __ldg(&ip->int_shift) != 0;
    const int t = item - item_index * tiles;
    const int tile_x0 = t % a.tiles_x * kTileW, tile_y0 = a.row0 + t / a.tiles_x * TH;
    if (p.fits) {
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
    const bool whole = counts_whole<INTERP, TH>(a, p, finite, tile_x0, tile_y0);
    unsigned bad = 0;
    if (INTERP != GG_INTERP_NEAREST && !GENERAL && p.grid && (!kLanczos || a.clamp < 0.0f) &&
        (p.fits || !kLanczos || (a.width >= 6 && a.height >= 6))) {
      const int lx = tid & 31, ly = (tid >> 5) * (TH / 4);
      const TileGrid& grid = s_grid[buf];
      const int64_t first = static_cast<int64_t>(tile_y0 + ly) * a.width + tile_x0 + lx;
      const TileMask mask = tile_mask(grid, kLanczos, a.width, a.height, tile_x0, tile_y0, a.row1,
                                      a.coverage ? a.coverage + first : nullptr);
      float* out = dst + first;
      auto rows = [&](auto win, auto masked) {
        constexpr bool kMask = decltype(masked)::value;
        if constexpr (kLanczos)
          return lanczos3_rows<TH / 4, decltype(win)::kStaged, kMask>(grid, win, mask, a.fill, out, a.width, lx, ly);
        else
          return bilinear_rows<TH / 4, decltype(win)::kStaged, kMask>(grid, win, mask, a.fill, out, a.width, lx, ly);
      };
      auto tile_rows = [&](auto win) {
        if constexpr (kLanczos) {
          constexpr bool kStaged = decltype(win)::kStaged;
          if (int_shift) return shifted_rows<TH / 4, kStaged>(grid, win, mask, a.fill, out, a.width, lx, ly);
          if (!finite) return lanczos3_renorm_rows<TH / 4, kStaged>(grid, win, mask, a.fill, out, a.width, lx, ly);
        }
        return whole && (a.coverage == nullptr || a.counted) ? rows(win, std::false_type{})
                                                            : rows(win, std::true_type{});
      };
      constexpr int kSpan = kLanczos ? 6 : 1;  // of a window's possible places
      const int x0 = -grid.ox, y0 = -grid.oy, x1 = a.width - kSpan + x0, y1 = a.height - kSpan + y0;
      if (USE_TMA && p.fits)
        bad = tile_rows(Window<true>{tile, kBoxW, x0, x1, y0, y1});
      else
        bad = tile_rows(Window<false>{src + static_cast<int64_t>(grid.oy) * a.width + grid.ox, a.width, x0, x1, y0, y1});
    } else {
      const Coef co = load_coef(ip);
      TapSource ts;
      ts.tile = p.fits ? tile : nullptr;
      ts.src = src;
      ts.bx = p.bx;
      ts.by = p.by;
      ts.width = a.width;
#pragma unroll 1
      for (int c = tid / kTileW; c < kRowClasses; c += kWarpThreads / kTileW) {
        const int ox = tile_x0 + tid % kTileW, oy0 = tile_y0 + c;
        if (kLanczos && finite)
          bad += warp_tile_rows<INTERP, true, TH>(a, co, ts, dst, ox, oy0, p.interior != 0, int_shift);
        else
          bad += warp_tile_rows<INTERP, false, TH>(a, co, ts, dst, ox, oy0, p.interior != 0, int_shift);
      }
    }
    const unsigned warp_bad = __reduce_add_sync(0xffffffffu, bad);
    if ((tid & 31) == 0 && warp_bad) atomicAdd(a.nonfinite + it_frame, warp_bad);
    __syncthreads();
    if (s_abort) {
      // Let the copy already issued for the next item land before exit.
      if (next < items && s_plan[buf ^ 1].fits) mbar_wait_bounded(&bar[buf ^ 1], phase[buf ^ 1], 1 << 24);
      break;
    }
  }
  if (a.slot_of_frame != nullptr && last_cta(a.ticket, gridDim.x)) {
    // the warped frame lives in the spare slot, and its old slot is spare
    for (int k = tid; k < a.item_count; k += kWarpThreads) {
      a.slot_of_frame[a.items[k].frame] = a.items[k].dst_slot;
      a.spare[k] = a.items[k].src_slot;
    }
  }
}

// Frames with a geometrically valid sample, per pixel of a band: this kernel
// writes each tile's frames that count for the whole tile (all but those whose
// border crosses it), the warp then adds the others' valid pixels.
template <int INTERP, int TH>
__global__ void __launch_bounds__(kWarpThreads) warp_geometry_kernel(WarpArgs a) {
  __shared__ int s_inside;
  const int tile_x0 = blockIdx.x % a.tiles_x * kTileW, tile_y0 = a.row0 + blockIdx.x / a.tiles_x * TH;
  if (threadIdx.x == 0) s_inside = 0;
  __syncthreads();
  constexpr bool kLanczos = INTERP == GG_INTERP_LANCZOS3;
  const float vlo = kLanczos ? 2.0f : 0.0f, off = kLanczos ? 3.0f : 1.0f;
  for (int f = threadIdx.x; f < a.item_count; f += kWarpThreads) {
    const WarpItem* ip = a.items + f;
    const TilePlan p = plan_tile<TH>(load_coef(ip), tile_x0, tile_y0, kLanczos ? 3 : 1, vlo,
                                     static_cast<float>(a.width) - off, static_cast<float>(a.height) - off);
    if (counts_whole<INTERP, TH>(a, p, ip->src_nonfinite == 0u, tile_x0, tile_y0)) atomicAdd(&s_inside, 1);
  }
  __syncthreads();
  const float n = static_cast<float>(s_inside);
  const int ox = tile_x0 + (threadIdx.x & 63);
  if (ox >= a.width) return;
  for (int oy = tile_y0 + (threadIdx.x >> 6); oy < min(tile_y0 + TH, a.row1); oy += kWarpThreads / kTileW)
    a.coverage[static_cast<int64_t>(oy) * a.width + ox] = n;
}

// One tile per CTA of an image's affine warp, windows from global memory.
template <int INTERP, int TH>
__global__ void __launch_bounds__(kWarpThreads, 4) affine_tiles_kernel(const __grid_constant__ WarpItem item,
                                                                    const float* src, float* dst, int finite,
                                                                    WarpArgs a) {
  __shared__ TilePlan s_plan;
  __shared__ TileGrid s_grid;
  constexpr bool kLanczos = INTERP == GG_INTERP_LANCZOS3;
  const int tid = threadIdx.x;
  const int tile_x0 = blockIdx.x % a.tiles_x * kTileW, tile_y0 = blockIdx.x / a.tiles_x * TH;
  Coef co;
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    co.m[q][0] = item.m[q][0];
    co.m[q][1] = item.m[q][1];
  }
  co.affine = item.affine;
  if (tid < 32) {
    const float off = kLanczos ? 3.0f : 1.0f;
    const TilePlan p = plan_tile_warp<TH>(co, tile_x0, tile_y0, kLanczos ? 3 : 1, kLanczos ? 2.0f : 0.0f,
                                          static_cast<float>(a.width) - off, static_cast<float>(a.height) - off);
    if (p.grid) tile_grid_warp(item.inv, tile_x0, tile_y0, false, 0, 0, s_grid);
    if (tid == 0) s_plan = p;
  }
  __syncthreads();
  const TilePlan p = s_plan;
  if (p.grid && (!kLanczos || (a.width >= 6 && a.height >= 6))) {
    const TileGrid& grid = s_grid;
    const int lx = tid & 31, ly = (tid >> 5) * (TH / 4);
    float* out = dst + static_cast<int64_t>(tile_y0 + ly) * a.width + tile_x0 + lx;
    const TileMask mask = tile_mask(grid, kLanczos, a.width, a.height, tile_x0, tile_y0, a.row1, nullptr);
    constexpr int kSpan = kLanczos ? 6 : 1;
    const int x0 = -grid.ox, y0 = -grid.oy;
    const Window<false> win{src + static_cast<int64_t>(grid.oy) * a.width + grid.ox, a.width, x0,
                            a.width - kSpan + x0, y0, a.height - kSpan + y0};
    const bool whole = counts_whole<INTERP, TH>(a, p, finite != 0, tile_x0, tile_y0);
    if constexpr (kLanczos) {
      if (!finite) lanczos3_renorm_rows<TH / 4, false>(grid, win, mask, a.fill, out, a.width, lx, ly);
      else if (whole) lanczos3_rows<TH / 4, false, false>(grid, win, mask, a.fill, out, a.width, lx, ly);
      else lanczos3_rows<TH / 4, false, true>(grid, win, mask, a.fill, out, a.width, lx, ly);
    } else {
      if (whole) bilinear_rows<TH / 4, false, false>(grid, win, mask, a.fill, out, a.width, lx, ly);
      else bilinear_rows<TH / 4, false, true>(grid, win, mask, a.fill, out, a.width, lx, ly);
    }
    return;
  }
  TapSource ts;
  ts.tile = nullptr;
  ts.src = src;
  ts.bx = ts.by = 0;
  ts.width = a.width;
#pragma unroll 1
  for (int c = tid / kTileW; c < kRowClasses; c += kWarpThreads / kTileW) {
    const int ox = tile_x0 + tid % kTileW, oy0 = tile_y0 + c;
    if (kLanczos && finite) warp_tile_rows<INTERP, true, TH>(a, co, ts, dst, ox, oy0, p.interior != 0, false);
    else warp_tile_rows<INTERP, false, TH>(a, co, ts, dst, ox, oy0, p.interior != 0, false);
  }
}

void launch_affine_warp(const float* src, int height, int width, const double* theta, int interp, float fill,
                        bool finite, float* dst, cudaStream_t stream) {
  WarpItem item{};
  item.affine = 1;
  for (int q = 0; q < 6; ++q) {
    item.inv[q] = theta[q];
    item.m[q][0] = static_cast<float>(theta[q]);
    item.m[q][1] = static_cast<float>(theta[q] - static_cast<double>(item.m[q][0]));
  }
  item.m[8][0] = 1.0f;
  WarpArgs a{};
  a.width = width;
  a.height = a.row1 = height;
  a.tiles_x = (width + kTileW - 1) / kTileW;
  a.fill = fill;
  a.clamp = -1.0f;
  auto launch = [&](auto kern, int th) {
    const int64_t tiles = static_cast<int64_t>(a.tiles_x) * ((height + th - 1) / th);
    note_launch();
    kern<<<static_cast<unsigned>(tiles), kWarpThreads, 0, stream>>>(item, src, dst, finite ? 1 : 0, a);
    check_cuda(cudaGetLastError(), "affine warp launch");
  };
  const bool small = static_cast<int64_t>(a.tiles_x) * ((height + kTileH - 1) / kTileH) < 2 * sm_count();
  if (interp == GG_INTERP_BILINEAR)
    small ? launch(affine_tiles_kernel<GG_INTERP_BILINEAR, kSmallTileH>, kSmallTileH)
          : launch(affine_tiles_kernel<GG_INTERP_BILINEAR, kTileH>, kTileH);
  else
    small ? launch(affine_tiles_kernel<GG_INTERP_LANCZOS3, kSmallTileH>, kSmallTileH)
          : launch(affine_tiles_kernel<GG_INTERP_LANCZOS3, kTileH>, kTileH);
}

// Resolve slots for the batch and move the source non-finite counts aside.
__device__ __forceinline__ void warp_prepare_item(WarpItem& it, int k, const int* slot_of_frame, const int* spare,
                                                  unsigned* nonfinite, float* slots, int64_t stride) {
  it.src_slot = slot_of_frame[it.frame];
  it.dst_slot = spare[k];
  it.dst = slots + spare[k] * stride;
  it.src_nonfinite = nonfinite[it.frame];
  nonfinite[it.frame] = 0u;
}

__global__ void warp_prepare_kernel(WarpItem* items, int count, const int* slot_of_frame, const int* spare,
                                    unsigned* nonfinite, float* slots, int64_t stride) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < count) warp_prepare_item(items[k], k, slot_of_frame, spare, nonfinite, slots, stride);
}

// The same with the descriptors in the launch parameters.
template <int CAP>
struct WarpItemBlock {
  WarpItem items[CAP];
};

template <int CAP>
__global__ void __launch_bounds__(128) warp_prepare_block_kernel(const __grid_constant__ WarpItemBlock<CAP> block,
                                                                 WarpItem* items, int count, const int* slot_of_frame,
                                                                 const int* spare, unsigned* nonfinite, float* slots,
                                                                 int64_t stride) {
  const int k = threadIdx.x;
  if (k >= count) return;
  WarpItem it = block.items[k];
  warp_prepare_item(it, k, slot_of_frame, spare, nonfinite, slots, stride);
  items[k] = it;
}

template <int CAP>
static void launch_prepare_block(gg_stack* s, WarpItem* d_items, const std::vector<WarpItem>& items) {
  WarpItemBlock<CAP> block;
  std::copy(items.begin(), items.end(), block.items);
  note_launch();
  warp_prepare_block_kernel<CAP><<<1, 128, 0, s->stream>>>(block, d_items, static_cast<int>(items.size()),
                                                          s->d_slot_of_frame, s->d_spare_slot, s->d_frame_nonfinite,
                                                          s->d_slots, s->stride);
  check_cuda(cudaGetLastError(), "warp_prepare launch");
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

template <int INTERP, int TH>
static void launch_warp_geometry(gg_stack* s, const WarpArgs& a) {
  note_launch();
  warp_geometry_kernel<INTERP, TH><<<static_cast<unsigned>(a.tiles_x * a.tiles_y), kWarpThreads, 0, s->stream>>>(a);
  check_cuda(cudaGetLastError(), "warp_geometry launch");
}

template <int INTERP, int TH, bool STAGED, bool GENERAL = false>
static void launch_warp_tiles(gg_stack* s, WarpArgs args) {
  args.tiles_y = (args.row1 - args.row0 + TH - 1) / TH;
  if constexpr (INTERP != GG_INTERP_NEAREST && TH != kMidTileH && !GENERAL)  // the bands' forms
    if (args.counted) launch_warp_geometry<INTERP, TH>(s, args);
  auto kern = warp_tiles_kernel<INTERP, STAGED, TH, GENERAL>;
  const size_t smem = STAGED ? kWarpTileBytes : 0;
  const int per_sm = kernel_ctas_per_sm(kern, kWarpThreads, smem, "warp launch shape");
  const int64_t items = static_cast<int64_t>(args.item_count) * args.tiles_x * args.tiles_y;
  unsigned grid =
      static_cast<unsigned>(std::min<int64_t>(items, static_cast<int64_t>(sm_count()) * per_sm));
  // A stride that shares no factor with the tiles of a row takes every CTA
  // through all tile columns: the slow border tiles of the first and last
  // column would fall to few CTAs otherwise.
  if (items > grid)
    while (std::gcd(grid, static_cast<unsigned>(args.tiles_x)) != 1) --grid;
  note_launch();
  kern<<<grid, kWarpThreads, smem, s->stream>>>(s->slot_tmap, args);
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
  a.error = s->d_error;
  return a;
}

template <int INTERP>
static void launch_warp_form(gg_stack* s, const WarpArgs& a, WarpForm form) {
  // With less than two 64-row tiles per SM the launch takes as long as a tile
  // does: 16-row tiles spread it over four times as many CTAs.
  const int64_t tiles = static_cast<int64_t>(a.item_count) * a.tiles_x * ((a.row1 - a.row0 + kTileH - 1) / kTileH);
  const bool small = tiles < 2 * sm_count() && INTERP != GG_INTERP_NEAREST;
  if constexpr (INTERP != GG_INTERP_NEAREST) {
    if (form == kDirectRows) {
      small ? launch_warp_tiles<INTERP, kSmallTileH, false>(s, a) : launch_warp_tiles<INTERP, kTileH, false>(s, a);
      return;
    }
  }
  if (form == kDirectGeneral)
    small ? launch_warp_tiles<INTERP, kSmallTileH, false, true>(s, a)
          : launch_warp_tiles<INTERP, kMidTileH, false, true>(s, a);
  else if (form == kStaged16 || small)
    launch_warp_tiles<INTERP, kSmallTileH, true>(s, a);
  else if (form == kStaged48)
    launch_warp_tiles<INTERP, kMidTileH, true>(s, a);
  else
    launch_warp_tiles<INTERP, kTileH, true>(s, a);
}

static void launch_warp_rows(gg_stack* s, const WarpArgs& a, int interp, WarpForm form) {
  if (interp == GG_INTERP_NEAREST)
    launch_warp_form<GG_INTERP_NEAREST>(s, a, form);
  else if (interp == GG_INTERP_BILINEAR)
    launch_warp_form<GG_INTERP_BILINEAR>(s, a, form);
  else
    launch_warp_form<GG_INTERP_LANCZOS3>(s, a, form);
}

// The form of a frame's warp.  Boxes where every tile's footprint fits one: an
// affine map takes a tile to source columns and rows that span |a| 63 + |b| (rows
// - 1) and |d| 63 + |e| (rows - 1), and a box holds the taps, the pixel of margin
// and the columns before its 16-byte boundary besides (plan_of_range).
static WarpForm warp_form(const gg_stack* s, const WarpItem& it, int interp, float clamp) {
  const bool lanczos = interp == GG_INTERP_LANCZOS3;
  const int radius = lanczos ? 3 : 1;
  if (s->has_slot_tmap) {
    auto fits = [&](int rows) {
      const double x = std::fabs(it.inv[0]) * (kTileW - 1) + std::fabs(it.inv[1]) * (rows - 1);
      const double y = std::fabs(it.inv[3]) * (kTileW - 1) + std::fabs(it.inv[4]) * (rows - 1);
      return x <= kBoxW - 5 - 2 * radius && y <= kBoxH - 2 - 2 * radius;
    };
    // a projective map's tiles are looked at one by one
    if (!it.affine || fits(kTileH)) return kStaged64;
    if (fits(kMidTileH)) return kStaged48;
    if (fits(kSmallTileH)) return kStaged16;
  }
  const bool straight = it.affine && interp != GG_INTERP_NEAREST && (!lanczos || clamp < 0.0f);
  return straight ? kDirectRows : kDirectGeneral;
}

// How many descriptors of a batch take each form (they stand in that order).
struct WarpForms {
  int64_t count[kWarpForms] = {};
};

// Host descriptors of a warp batch (validated; inverse coefficients), by form.
static std::vector<WarpItem> warp_items_host(gg_stack* s, const int64_t* indices, int64_t count, const double* fwd,
                                             int interp, float clamp, WarpForms& forms) {
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
    double inv[9];
    if (!inverse_coefficients(m, it.m, it.affine, inv)) fail(GG_ERR_INVALID_ARGUMENT, "warp matrix is singular");
    std::copy(inv, inv + 6, it.inv);
    // an exact integer translation (identity linear part, integer shifts):
    // its inverse is one too and every source coordinate is an integer
    it.int_shift = (m[0] == 1.0 && m[1] == 0.0 && m[3] == 0.0 && m[4] == 1.0 && m[6] == 0.0 && m[7] == 0.0 &&
                    m[8] == 1.0 && m[2] == std::floor(m[2]) && m[5] == std::floor(m[5]) && std::fabs(m[2]) < 1.0e7 &&
                    std::fabs(m[5]) < 1.0e7)
                       ? 1
                       : 0;
    it.form = warp_form(s, it, interp, clamp);
    ++forms.count[it.form];
  }
  if (forms.count[items[0].form] != count)
    std::stable_sort(items.begin(), items.end(), [](const WarpItem& a, const WarpItem& b) { return a.form < b.form; });
  return items;
}

// The kernels of a warp batch whose descriptors are already in device
// memory (d_items, `count` of them in the order of `forms`): per group of at most
// `spares` frames, resolve slots (unless that is done: `prepared`), warp into the
// spare slots, swap the slot table; a launch per form.  Only launches on the
// stack's stream (safe inside a stream capture).
static void launch_warp_items(gg_stack* s, WarpItem* d_items, int64_t count, const WarpForms& forms, int interp,
                              float fill, float clamp, bool track_coverage, bool prepared = false) {
  stack_slots_moved(s);
  int form = 0;
  int64_t form_end = forms.count[0];
  for (int64_t k0 = 0; k0 < count; k0 += s->spares) {
    const int nb = static_cast<int>(std::min<int64_t>(s->spares, count - k0));
    if (!prepared) {
      note_launch();
      warp_prepare_kernel<<<(nb + 127) / 128, 128, 0, s->stream>>>(d_items + k0, nb, s->d_slot_of_frame,
                                                                   s->d_spare_slot, s->d_frame_nonfinite, s->d_slots,
                                                                   s->stride);
      check_cuda(cudaGetLastError(), "warp_prepare launch");
    }
    for (int64_t k = k0; k < k0 + nb;) {
      while (k >= form_end) form_end += forms.count[++form];
      const int run = static_cast<int>(std::min<int64_t>(form_end, k0 + nb) - k);
      WarpArgs a = warp_args(s, d_items + k, run, 0, static_cast<int>(s->height));
      a.nonfinite = s->d_frame_nonfinite;
      a.fill = fill;
      a.clamp = clamp;
      a.coverage = track_coverage ? s->d_warp_coverage : nullptr;
      a.slot_of_frame = s->d_slot_of_frame;
      a.spare = s->d_spare_slot + (k - k0);
      a.ticket = s->d_tickets + s->frames;
      launch_warp_rows(s, a, interp, static_cast<WarpForm>(form));
      k += run;
    }
  }
}

void warp_frames(gg_stack* s, const int64_t* indices, int64_t count, const double* fwd, int interp, float fill,
                 float clamp, bool track_coverage) {
  WarpForms forms;
  const std::vector<WarpItem> items = warp_items_host(s, indices, count, fwd, interp, clamp, forms);
  ensure_warp_items(s, std::max<int64_t>(count, s->spares));
  if (track_coverage) ensure_warp_coverage(s);
  auto* d_items = static_cast<WarpItem*>(s->d_warp_items);
  // a batch that fits the launch parameters and the spare slots at once
  constexpr int kSmallBlock = 16, kLargeBlock = 96;
  static_assert(sizeof(WarpItemBlock<kLargeBlock>) <= 16384, "launch parameters");
  if (count <= std::min<int64_t>(s->spares, kLargeBlock)) {
    if (count <= kSmallBlock) launch_prepare_block<kSmallBlock>(s, d_items, items);
    else launch_prepare_block<kLargeBlock>(s, d_items, items);
    launch_warp_items(s, d_items, count, forms, interp, fill, clamp, track_coverage, true);
    if (track_coverage) s->warp_coverage_frames += count;
    return;
  }
  // The staging buffer may still feed the previous call's copy.
  check_cuda(cudaEventSynchronize(s->warp_items_free), "cudaEventSynchronize(warp items)");
  std::memcpy(s->h_warp_items, items.data(), sizeof(WarpItem) * items.size());
  upload_params(s->stream, s->d_warp_items, s->h_warp_items, sizeof(WarpItem) * items.size(),
                "cudaMemcpyAsync(warp items)");
  check_cuda(cudaEventRecord(s->warp_items_free, s->stream), "cudaEventRecord(warp items)");
  launch_warp_items(s, d_items, count, forms, interp, fill, clamp, track_coverage);
  if (track_coverage) s->warp_coverage_frames += count;
}

// Warp descriptors in a caller-owned device buffer (for captured graphs).
WarpBatch warp_batch_device(gg_stack* s, const int64_t* indices, int64_t count, const double* fwd, int interp,
                            float clamp) {
  WarpForms forms;
  const std::vector<WarpItem> items = warp_items_host(s, indices, count, fwd, interp, clamp, forms);
  WarpBatch batch;
  batch.count = count;
  batch.interp = interp;
  batch.clamp = clamp;
  batch.forms.assign(forms.count, forms.count + kWarpForms);
  check_cuda(cudaMalloc(&batch.items, sizeof(WarpItem) * items.size()), "cudaMalloc(graph warp items)");
  const cudaError_t err = cudaMemcpy(batch.items, items.data(), sizeof(WarpItem) * items.size(), cudaMemcpyHostToDevice);
  if (err != cudaSuccess) {
    cudaFree(batch.items);
    check_cuda(err, "cudaMemcpy(graph warp items)");
  }
  return batch;
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
    if (q < 6) it.inv[q] = static_cast<double>(it.m[q][0]) + static_cast<double>(it.m[q][1]);
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

void launch_warp_band(gg_stack* s, void* d_items, int interp, float clamp, int row0, int row1, unsigned* counts,
                      float* geometric) {
  WarpArgs a = warp_args(s, static_cast<WarpItem*>(d_items), static_cast<int>(s->frames), row0, row1);
  a.nonfinite = counts;
  a.fill = NAN;
  a.clamp = clamp;
  a.coverage = geometric;
  a.counted = 1;
  launch_warp_rows(s, a, interp, s->has_slot_tmap ? kStaged64 : kDirectRows);
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

void launch_warp_batch(gg_stack* s, const WarpBatch& batch, float fill) {
  WarpForms forms;
  std::copy(batch.forms.begin(), batch.forms.end(), forms.count);
  launch_warp_items(s, static_cast<WarpItem*>(batch.items), batch.count, forms, batch.interp, fill, batch.clamp, false);
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
