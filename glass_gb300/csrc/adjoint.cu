// Affine warp of one device image and its adjoint (reverse-mode derivative)
// with respect to the source image and the six affine parameters.
//
// The forward is the warp of warp.cu (engine/warp.py:99-152
// semantics; bilinear or Lanczos3 without the overshoot clamp): output pixel
// (x, y) samples the source at (sx, sy) = (t0 x + t1 y + t2, t3 x + t4 y + t5),
// where t are the parameters of the inverse (output -> source) map.
//
// Adjoint, per output pixel with incoming gradient g (zero where the sample
// is invalid or the loss ignores it):
//   bilinear   O = sum_ij wx_i wy_j S_ij, dO/dtx = (1-ty)(S01-S00) + ty(S11-S10),
//              dO/dty = ((1-tx)S10 + tx S11) - ((1-tx)S00 + tx S01);
//   Lanczos3   O = N / D over the finite taps, N = sum wx_i wy_j S_ij,
//              D = sum wx_i wy_j; dO/dtx = (N_x - O D_x) / D with N_x, D_x
//              the same sums with wx replaced by its derivative w'(t - k);
//   grad S_ij += g * wx_i wy_j / D            (cells per lane, float atomics);
//   grad t    += g * (dO/dsx (x, y, 1), dO/dsy (x, y, 1)).
// Weights and their derivatives are recomputed, never stored.
// w(d) = sinc(d) sinc(d/3), w'(d) = f'(d) g(d) + f(d) g'(d) with
// f(d) = sin(pi d)/(pi d), g(d) = f(d/3), f'(d) = pi (cos(pi d) pi d - sin(pi d)) / (pi d)^2.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "adjoint.cuh"
#include "stack.cuh"
#include "warp_band.cuh"

namespace gg {

struct AdjointArgs {
  const float* src;
  const float* grad_out;
  float* grad_src;
  double* partials;  // [blocks][6]
  AffineCoef coef;
  int width, height;
  int strip_rows;   // lanczos3_scatter_kernel
  double theta[6];  // lanczos3_scatter_kernel<true>
};

__device__ __forceinline__ bool sample_coords(const AdjointArgs& a, int x, int y, int interp, int& x0, int& y0,
                                              float& tx, float& ty) {
  FFv sx, sy;
  if (!source_coord(a.coef, static_cast<float>(x), static_cast<float>(y), sx, sy)) return false;
  const float W = static_cast<float>(a.width), H = static_cast<float>(a.height);
  const bool valid = interp == GG_INTERP_BILINEAR
                         ? (ff_ge(sx, 0.0f) && ff_le(sx, W - 1.0f) && ff_ge(sy, 0.0f) && ff_le(sy, H - 1.0f))
                         : (ff_ge(sx, 2.0f) && ff_lt(sx, W - 3.0f) && ff_ge(sy, 2.0f) && ff_lt(sy, H - 3.0f));
  if (!valid) return false;
  ff_floor_frac(sx, x0, tx);
  ff_floor_frac(sy, y0, ty);
  return true;
}

// Sample derivatives over the finite taps of a window (renormalised); with
// grad_src also the scatter of g to them.  False: no sample.
static __device__ __noinline__ bool lanczos3_adjoint_taps(const float* src, float* grad_src, int W, int x0, int y0,
                                                          float tx, float ty, float g, float& gsx, float& gsy) {
  float wx[6], wy[6], dwx[6], dwy[6];
  lanczos3_weights_grad(tx, wx, dwx);
  lanczos3_weights_grad(ty, wy, dwy);
  float N = 0.0f, D = 0.0f, Nx = 0.0f, Dx = 0.0f, Ny = 0.0f, Dy = 0.0f;
  for (int j = 0; j < 6; ++j) {
    const float* row = src + static_cast<int64_t>(y0 - 2 + j) * W + (x0 - 2);
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const float v = __ldg(row + i);
      if (!isfinite(v)) continue;
      const float w = wx[i] * wy[j], wxd = dwx[i] * wy[j], wyd = wx[i] * dwy[j];
      N = __fmaf_rn(w, v, N);
      D += w;
      Nx = __fmaf_rn(wxd, v, Nx);
      Dx += wxd;
      Ny = __fmaf_rn(wyd, v, Ny);
      Dy += wyd;
    }
  }
  if (!(fabsf(D) > 1.0e-12f)) return false;
  const float O = N / D;
  gsx = g * (Nx - O * Dx) / D;
  gsy = g * (Ny - O * Dy) / D;
  if (grad_src) {
    const float gd = g / D;
    for (int j = 0; j < 6; ++j) {
      float* grow = grad_src + static_cast<int64_t>(y0 - 2 + j) * W + (x0 - 2);
      const float* row = src + static_cast<int64_t>(y0 - 2 + j) * W + (x0 - 2);
#pragma unroll
      for (int i = 0; i < 6; ++i)
        if (isfinite(__ldg(row + i))) atomicAdd(grow + i, gd * wx[i] * wy[j]);
    }
  }
  return true;
}

// Per-CTA sums of the parameter gradient (float64), WARPS warps.
template <int WARPS>
__device__ __forceinline__ void reduce_theta(const double (&acc)[6], double* partials) {
  __shared__ double red[WARPS][6];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double d[6];
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    d[q] = acc[q];
    for (int off = 16; off > 0; off >>= 1) d[q] += __shfl_xor_sync(0xffffffffu, d[q], off);
  }
  if (lane == 0)
    for (int q = 0; q < 6; ++q) red[warp][q] = d[q];
  __syncthreads();
  if (threadIdx.x < 6) {
    double s = 0.0;
    for (int w = 0; w < WARPS; ++w) s += red[w][threadIdx.x];
    partials[static_cast<int64_t>(blockIdx.x) * 6 + threadIdx.x] = s;
  }
}

__device__ __forceinline__ void add_theta(float (&acc)[6], float gsx, float gsy, int x, int y) {
  const float xf = static_cast<float>(x), yf = static_cast<float>(y);
  acc[0] = __fmaf_rn(gsx, xf, acc[0]);
  acc[1] = __fmaf_rn(gsx, yf, acc[1]);
  acc[2] += gsx;
  acc[3] = __fmaf_rn(gsy, xf, acc[3]);
  acc[4] = __fmaf_rn(gsy, yf, acc[4]);
  acc[5] += gsy;
}

// ---- Lanczos3 adjoint with the image gradient --------------------------------
// A warp takes strips of 32 columns x strip_rows output rows.  Each lane keeps
// the 6 x 6 cells that its output pixel's window covers; where the next row's
// window lies one source row further down (scale and rotation move it by
// hundredths of a pixel per row) the window's first row is complete for this
// column: its six cells are summed with the neighbouring lanes' over shuffles,
// and one atomic per source pixel and strip (and a few along the strip's edge)
// takes the place of 36 per output pixel.  Any other step writes all six rows.
// Bound: latency at 12 warps per SM (168 registers), then issue (789
// instructions per pixel).  4096^2: 660 us, 1102 us with an atomic per tap.
constexpr int kScatterThreads = 128;

// Adds the cells of source row R, columns C .. C + 5 of every lane.
__device__ __forceinline__ void scatter_row(const AdjointArgs& a, const float (&v)[6], int R, int C) {
  const int lane = threadIdx.x & 31;
  const int R0 = __shfl_sync(0xffffffffu, R, 0), C0 = __shfl_sync(0xffffffffu, C, 0);
  float* row = a.grad_src + static_cast<int64_t>(R) * a.width;
  if (__all_sync(0xffffffffu, R == R0 && C - lane == C0)) {
    // column C is the own first cell and cell i of the lane i to the left
    float t = v[0];
#pragma unroll
    for (int i = 1; i < 6; ++i) {
      const float u = __shfl_up_sync(0xffffffffu, v[i], i);
      if (lane >= i) t += u;
    }
    if (R0 >= 0 && R0 < a.height && C0 >= 0 && C0 + 37 <= a.width) {
      row += C;
      atomicAdd(row, t);
#pragma unroll
      for (int i = 1; i < 6; ++i)
        if (lane > 31 - i) atomicAdd(row + i, v[i]);
      return;
    }
    if (R0 < 0 || R0 >= a.height) return;
    if (t != 0.0f && C >= 0 && C < a.width) atomicAdd(row + C, t);
#pragma unroll
    for (int i = 1; i < 6; ++i)
      if (lane > 31 - i && v[i] != 0.0f && C + i >= 0 && C + i < a.width) atomicAdd(row + C + i, v[i]);
    return;
  }
#pragma unroll
  for (int i = 0; i < 6; ++i)
    if (v[i] != 0.0f && R >= 0 && R < a.height && C + i >= 0 && C + i < a.width) atomicAdd(row + C + i, v[i]);
}

// FIXED: coordinates in fixed point down a strip (54 fraction bits, relative to
// the first row's pixel); for maps that move by at most 8 source pixels per row.
template <bool FIXED>
__global__ void __launch_bounds__(kScatterThreads) lanczos3_scatter_kernel(AdjointArgs a) {
  const int lane = threadIdx.x & 31;
  const int W = a.width;
  const int strips_x = (W + 31) / 32, strips_y = (a.height + a.strip_rows - 1) / a.strip_rows;
  const int strips = strips_x * strips_y;
  constexpr double kOne = static_cast<double>(1ll << 54);
  const long long step_x = FIXED ? __double2ll_rn(a.theta[1] * kOne) : 0;
  const long long step_y = FIXED ? __double2ll_rn(a.theta[4] * kOne) : 0;
  double acc[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  for (int s = blockIdx.x * (kScatterThreads / 32) + (threadIdx.x >> 5); s < strips;
       s += gridDim.x * (kScatterThreads / 32)) {
    const int x = s % strips_x * 32 + lane, ybase = s / strips_x * a.strip_rows;
    const int rows = min(a.strip_rows, a.height - ybase);
    float cell[6][6];
#pragma unroll
    for (int j = 0; j < 6; ++j)
#pragma unroll
      for (int i = 0; i < 6; ++i) cell[j][i] = 0.0f;
    int px = 0, py = 0, ox = 0, oy = 0;
    long long fx = 0, fy = 0;
    if (FIXED) {
      const double xd = x, yd = ybase;
      const double sx = fma(a.theta[0], xd, fma(a.theta[1], yd, a.theta[2]));
      const double sy = fma(a.theta[3], xd, fma(a.theta[4], yd, a.theta[5]));
      ox = static_cast<int>(floor(sx));
      oy = static_cast<int>(floor(sy));
      fx = __double2ll_rn((sx - ox) * kOne);
      fy = __double2ll_rn((sy - oy) * kOne);
    }
    // sums of g dO/dsx, g dO/dsy and of their products with the row
    float sum_x = 0.0f, sum_y = 0.0f, row_x = 0.0f, row_y = 0.0f;
#pragma unroll 1
    for (int r = 0; r < rows; ++r) {
      const int y = ybase + r;
      int x0, y0;
      CentredOffset tx, ty;
      if constexpr (FIXED) {
        // distance from the nearer tap: two exact halves of 24 bits, rounded once
        auto offset = [](long long v) {
          constexpr long long kMask = (1ll << 54) - 1;
          CentredOffset o;
          o.lower = ((v >> 53) & 1) == 0;
          const long long d = (o.lower ? v : -v) & kMask;
          const float high = __uint2float_rn(static_cast<unsigned>(d >> 30));
          const float low = __uint2float_rn(static_cast<unsigned>(d >> 6) & 0xffffffu);
          o.s = __fmul_rn(__fmaf_rn(low, 5.9604644775390625e-08f, high), 5.9604644775390625e-08f);
          return o;
        };
        x0 = ox + static_cast<int>(fx >> 54);
        y0 = oy + static_cast<int>(fy >> 54);
        tx = offset(fx);
        ty = offset(fy);
        fx += step_x;
        fy += step_y;
      } else {
        FFv sx, sy;
        source_coord(a.coef, static_cast<float>(x), static_cast<float>(y), sx, sy);
        // far outside: any position without a valid sample
        const bool near = fabsf(sx.hi) < 1.0e9f && fabsf(sy.hi) < 1.0e9f;
        auto offset = [](FFv v, int& whole) {
          float t;
          ff_floor_frac(v, whole, t);
          CentredOffset o;
          o.lower = t <= 0.5f;
          o.s = o.lower ? t : __fsub_rn(__fsub_rn(static_cast<float>(whole) + 1.0f, v.hi), v.lo);
          return o;
        };
        tx = offset(near ? sx : FFv{-100.0f, 0.0f}, x0);
        ty = offset(near ? sy : FFv{-100.0f, 0.0f}, y0);
      }
      // 2 <= s < size - 3 of the coordinate is that of its whole part
      const bool valid = x < W && x0 >= 2 && x0 < W - 3 && y0 >= 2 && y0 < a.height - 3;
      if (r > 0) {
        if (__all_sync(0xffffffffu, x0 == px && y0 == py + 1)) {
          scatter_row(a, cell[0], py - 2, px - 2);
#pragma unroll
          for (int j = 0; j < 5; ++j)
#pragma unroll
            for (int i = 0; i < 6; ++i) cell[j][i] = cell[j + 1][i];
#pragma unroll
          for (int i = 0; i < 6; ++i) cell[5][i] = 0.0f;
        } else {
#pragma unroll
          for (int j = 0; j < 6; ++j) {
            scatter_row(a, cell[j], py - 2 + j, px - 2);
#pragma unroll
            for (int i = 0; i < 6; ++i) cell[j][i] = 0.0f;
          }
        }
      }
      px = x0;
      py = y0;
      float g = valid ? a.grad_out[static_cast<int64_t>(y) * W + x] : 0.0f;
      if (!isfinite(g)) g = 0.0f;
      const bool live = g != 0.0f;
      if (!__any_sync(0xffffffffu, live)) continue;
      const LanczosAxis ax = lanczos3_axis_centred(tx), ay = lanczos3_axis_centred(ty);
      float N = 0.0f, Nx = 0.0f, Ny = 0.0f;
      // the other lanes read the image's first window (a live lane proves that
      // the image holds one)
      const float* at = a.src + (live ? static_cast<int64_t>(y0 - 2) * W + (x0 - 2) : 0);
      // taps relative to the middle one: the derivatives are the same, (Nx - O
      // Dx) / D for taps v + c equals that for v, without the rounding that a
      // background of many times its noise leaves in Nx
      const float middle = __ldg(at + 2 * static_cast<int64_t>(W) + 2);
#pragma unroll
      for (int j = 0; j < 6; ++j, at += W) {
        float rv = 0.0f, rd = 0.0f;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
          const float v = __fsub_rn(__ldg(at + i), middle);
          rv = __fmaf_rn(ax.w[i], v, rv);
          rd = __fmaf_rn(ax.dw[i], v, rd);
        }
        N = __fmaf_rn(ay.w[j], rv, N);
        Nx = __fmaf_rn(ay.w[j], rd, Nx);
        Ny = __fmaf_rn(ay.dw[j], rv, Ny);
      }
      float gd = 0.0f;
      if (live) {
        float gsx = 0.0f, gsy = 0.0f;
        if (isfinite(N) && isfinite(Nx) && isfinite(Ny)) {
          // a window of finite taps: its weights sum to 1 within a few per cent
          const float iD = __frcp_rn(ax.sum * ay.sum);
          const float O = N * iD;
          gd = g * iD;
          gsx = gd * (Nx - O * (ax.dsum * ay.sum));
          gsy = gd * (Ny - O * (ax.sum * ay.dsum));
        } else if (!lanczos3_adjoint_taps(a.src, a.grad_src, W, x0, y0, tx.t(), ty.t(), g, gsx, gsy)) {
          gsx = gsy = 0.0f;
        }
        const float rf = static_cast<float>(r);
        sum_x += gsx;
        sum_y += gsy;
        row_x = __fmaf_rn(gsx, rf, row_x);
        row_y = __fmaf_rn(gsy, rf, row_y);
      }
#pragma unroll
      for (int j = 0; j < 6; ++j) {
        const float gy = gd * ay.w[j];
#pragma unroll
        for (int i = 0; i < 6; ++i) cell[j][i] = __fmaf_rn(gy, ax.w[i], cell[j][i]);
      }
    }
    if (rows > 0) {
#pragma unroll
      for (int j = 0; j < 6; ++j) scatter_row(a, cell[j], py - 2 + j, px - 2);
    }
    acc[0] += static_cast<double>(sum_x) * x;
    acc[1] += static_cast<double>(sum_x) * ybase + row_x;
    acc[2] += sum_x;
    acc[3] += static_cast<double>(sum_y) * x;
    acc[4] += static_cast<double>(sum_y) * ybase + row_y;
    acc[5] += sum_y;
  }
  reduce_theta<kScatterThreads / 32>(acc, a.partials);
}

template <int INTERP>
__global__ void __launch_bounds__(256) affine_backward_kernel(AdjointArgs a) {
  const int64_t P = static_cast<int64_t>(a.width) * a.height;
  float acc[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
  const int W = a.width;
  for (int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; p < P; p += int64_t(gridDim.x) * blockDim.x) {
    const float g = a.grad_out[p];
    if (!(g != 0.0f) || !isfinite(g)) continue;
    const int y = static_cast<int>(p / W), x = static_cast<int>(p - static_cast<int64_t>(y) * W);
    int x0, y0;
    float tx, ty;
    if (!sample_coords(a, x, y, INTERP, x0, y0, tx, ty)) continue;
    float gsx = 0.0f, gsy = 0.0f;  // g * dO/dsx, g * dO/dsy
    if (INTERP == GG_INTERP_BILINEAR) {
      const int x1 = min(x0 + 1, W - 1), y1 = min(y0 + 1, a.height - 1);
      const float s00 = __ldg(a.src + static_cast<int64_t>(y0) * W + x0);
      const float s01 = __ldg(a.src + static_cast<int64_t>(y0) * W + x1);
      const float s10 = __ldg(a.src + static_cast<int64_t>(y1) * W + x0);
      const float s11 = __ldg(a.src + static_cast<int64_t>(y1) * W + x1);
      if (!(isfinite(s00) && isfinite(s01) && isfinite(s10) && isfinite(s11))) continue;  // NaN output
      const float ox = 1.0f - tx, oy = 1.0f - ty;
      gsx = g * (oy * (s01 - s00) + ty * (s11 - s10));
      gsy = g * ((ox * s10 + tx * s11) - (ox * s00 + tx * s01));
      if (a.grad_src) {
        atomicAdd(a.grad_src + static_cast<int64_t>(y0) * W + x0, g * ox * oy);
        atomicAdd(a.grad_src + static_cast<int64_t>(y0) * W + x1, g * tx * oy);
        atomicAdd(a.grad_src + static_cast<int64_t>(y1) * W + x0, g * ox * ty);
        atomicAdd(a.grad_src + static_cast<int64_t>(y1) * W + x1, g * tx * ty);
      }
    } else if (float Os, Osx, Osy; lanczos3_value_grad<true, false, true>(a.src, W, x0, y0, tx, ty, Os, Osx, Osy)) {
      // a window of finite taps: the separable sums with the warp's polynomial
      // weights and their exact derivatives
      gsx = g * Osx;
      gsy = g * Osy;
    } else if (!lanczos3_adjoint_taps(a.src, nullptr, W, x0, y0, tx, ty, g, gsx, gsy)) {
      continue;
    }
    add_theta(acc, gsx, gsy, x, y);
  }
  const double sums[6] = {acc[0], acc[1], acc[2], acc[3], acc[4], acc[5]};
  reduce_theta<8>(sums, a.partials);
}

// One warp per parameter.
__global__ void affine_reduce_kernel(const double* partials, int blocks, double* grad_theta) {
  const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double s = 0.0;
  for (int b = lane; b < blocks; b += 32) s += partials[static_cast<int64_t>(b) * 6 + q];
  for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if (lane == 0) grad_theta[q] = s;
}

static AffineCoef affine_coef(const double* theta) {
  for (int q = 0; q < 6; ++q) require(std::isfinite(theta[q]), "affine parameters must be finite");
  return affine_coef_from(theta);
}

static unsigned affine_grid(int64_t pixels) {
  return static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>((pixels + 255) / 256, sm_count() * 8)));
}

}  // namespace gg

using namespace gg;

extern "C" {

int gg_warp_affine_f32_device(const float* dev_src, int64_t height, int64_t width, const double* host_theta,
                              int interpolation, float fill, int src_all_finite, float* dev_out,
                              void* cuda_stream) {
  GG_API_BEGIN
  require(dev_src != nullptr && dev_out != nullptr && host_theta != nullptr, "null argument");
  require(height > 0 && width > 0 && height * width < (int64_t{1} << 31), "invalid image shape");
  require(interpolation == GG_INTERP_BILINEAR || interpolation == GG_INTERP_LANCZOS3,
          "interpolation must be bilinear or lanczos3");
  for (int q = 0; q < 6; ++q) require(std::isfinite(host_theta[q]), "affine parameters must be finite");
  launch_affine_warp(dev_src, static_cast<int>(height), static_cast<int>(width), host_theta, interpolation, fill,
                     src_all_finite != 0, dev_out, static_cast<cudaStream_t>(cuda_stream));
  GG_API_END
}

int gg_warp_affine_backward_f32_device(const float* dev_src, int64_t height, int64_t width, const double* host_theta,
                                       int interpolation, const float* dev_grad_out, float* dev_grad_src,
                                       double* dev_grad_theta, void* cuda_stream) {
  GG_API_BEGIN
  require(dev_src != nullptr && dev_grad_out != nullptr && host_theta != nullptr, "null argument");
  require(height > 0 && width > 0 && height * width < (int64_t{1} << 31), "invalid image shape");
  require(interpolation == GG_INTERP_BILINEAR || interpolation == GG_INTERP_LANCZOS3,
          "interpolation must be bilinear or lanczos3");
  AdjointArgs a{};
  a.src = dev_src;
  a.grad_out = dev_grad_out;
  a.grad_src = dev_grad_src;
  a.coef = affine_coef(host_theta);
  a.width = static_cast<int>(width);
  a.height = static_cast<int>(height);
  auto stream = static_cast<cudaStream_t>(cuda_stream);
  const unsigned blocks = affine_grid(height * width);
  double* partials = nullptr;
  check_cuda(cudaMallocAsync(reinterpret_cast<void**>(&partials), sizeof(double) * 6 * blocks, stream),
             "cudaMallocAsync(adjoint partials)");
  a.partials = partials;
  note_launch();
  if (interpolation == GG_INTERP_BILINEAR)
    affine_backward_kernel<GG_INTERP_BILINEAR><<<blocks, 256, 0, stream>>>(a);
  else if (dev_grad_src) {
    // long strips save edge atomics, short ones keep a small image's SMs busy
    a.strip_rows = 32;
    auto strips = [&] { return ((width + 31) / 32) * ((height + a.strip_rows - 1) / a.strip_rows); };
    while (a.strip_rows > 4 && strips() < sm_count() * 12) a.strip_rows /= 2;
    std::copy(host_theta, host_theta + 6, a.theta);
    const double reach = std::fabs(host_theta[2]) + std::fabs(host_theta[5]) +
                         (std::fabs(host_theta[0]) + std::fabs(host_theta[3])) * static_cast<double>(width) +
                         (std::fabs(host_theta[1]) + std::fabs(host_theta[4])) * static_cast<double>(height);
    if (std::fabs(host_theta[1]) <= 8.0 && std::fabs(host_theta[4]) <= 8.0 && reach < 1.0e9)
      lanczos3_scatter_kernel<true><<<blocks, kScatterThreads, 0, stream>>>(a);
    else
      lanczos3_scatter_kernel<false><<<blocks, kScatterThreads, 0, stream>>>(a);
  }
  else
    affine_backward_kernel<GG_INTERP_LANCZOS3><<<blocks, 256, 0, stream>>>(a);
  check_cuda(cudaGetLastError(), "affine_backward launch");
  if (dev_grad_theta) {
    note_launch();
    affine_reduce_kernel<<<1, 6 * 32, 0, stream>>>(partials, static_cast<int>(blocks), dev_grad_theta);
    check_cuda(cudaGetLastError(), "affine_reduce launch");
  }
  check_cuda(cudaFreeAsync(partials, stream), "cudaFreeAsync(adjoint partials)");
  GG_API_END
}

}  // extern "C"
