// Shared pieces of the integration kernels (integrate.cu, integrate_px.cuh):
// the launch arguments, the sorting network, the output writer and small
// per-pixel helpers.
#pragma once

#include "stack.cuh"
#include "warp_band.cuh"

namespace gg {

struct IntegrateArgs {
  const float* slots;
  const int* slot_of_frame;
  int64_t stride;
  const float* const* base;  // optional first sample of every frame (else its slot's)
  int64_t pixels;
  int frames;
  const float* weights;  // device [frames], raw values
  const unsigned* nonfinite;
  int rejection;
  float low_sigma;
  float high_sigma;
  int min_samples;
  float max_frac;
  int lfc_iterations;
  float* master;
  float* weight;
  void* coverage;
  void* low;
  void* high;
  int16_t* dq;
  int count_u16;
  const float* geometric;  // optional warp coverage (float32 per pixel)
  // fused warp only
  const FusedFrame* fused;
  int width, height;
  float clamp;
  float* geometric_out;  // frames with a geometrically valid sample, per pixel
  int tile_w, tile_h;    // fused path: 2-D pixel tiles (tile_w * tile_h == threads), 0 = rows
  int64_t tiles_x;       // tiles per image row
  int64_t tile_slots;    // tiles * threads
};

constexpr float kInf = __builtin_huge_valf();

// ---- sorting network (Batcher odd-even merge sort, fully unrolled) --------
// Loop counters are kept additive (log2 of p and k) so that nvcc unrolls the
// whole network and v[] stays in registers.  For an N that is no power of two
// it is the next larger network without the comparators that reach past N:
// with +inf there they would change nothing.
template <int N>
__device__ __forceinline__ void sort_network(float (&v)[N]) {
  constexpr int LOG2N = (N <= 1) ? 0 : (N <= 2) ? 1 : (N <= 4) ? 2 : (N <= 8) ? 3 : (N <= 16) ? 4 : (N <= 32) ? 5
                        : (N <= 64) ? 6 : 7;
  static_assert(N <= (1 << LOG2N), "sort_network sorts up to 128 values");
#pragma unroll
  for (int lp = 0; lp < LOG2N; ++lp) {
#pragma unroll
    for (int lk = lp; lk >= 0; --lk) {
#pragma unroll
      for (int a = 0; a < N; ++a) {
        // Comparator (a, a+k) of stage (p, k); all conditions fold at compile time.
        const int p = 1 << lp, k = 1 << lk, j0 = k % p;
        if (a >= j0 && a + k < N && ((a - j0) % (2 * k)) < k && (a / (2 * p)) == ((a + k) / (2 * p))) {
          const float lo = fminf(v[a], v[a + k]);
          const float hi = fmaxf(v[a], v[a + k]);
          v[a] = lo;
          v[a + k] = hi;
        }
      }
    }
  }
}

__device__ __forceinline__ float clipf(float x, float lo, float hi) { return fminf(fmaxf(x, lo), hi); }

// ---- output ---------------------------------------------------------------
// DQ bits: contracts.py:77-88; rules: resident_cuda.py:3110-3297.
__device__ __forceinline__ void write_outputs(const IntegrateArgs& a, int64_t p, float master, float weight, int cov,
                                              int nlow, int nhigh, int active_frames) {
  a.master[p] = master;
  a.weight[p] = weight;
  if (a.count_u16) {
    static_cast<uint16_t*>(a.coverage)[p] = static_cast<uint16_t>(min(cov, 65535));
    static_cast<uint16_t*>(a.low)[p] = static_cast<uint16_t>(min(nlow, 65535));
    static_cast<uint16_t*>(a.high)[p] = static_cast<uint16_t>(min(nhigh, 65535));
  } else {
    static_cast<float*>(a.coverage)[p] = static_cast<float>(cov);
    static_cast<float*>(a.low)[p] = static_cast<float>(nlow);
    static_cast<float*>(a.high)[p] = static_cast<float>(nhigh);
  }
  if (a.dq) {
    int bits = 0;
    bool invalid = !isfinite(master) || !isfinite(weight) || !(weight > 0.0f);
    if (cov <= 0) {
      bits |= 64;
      invalid = true;
    }
    if (a.geometric) {
      const float g = a.geometric[p];
      if (!isfinite(g) || g <= 0.5f) {
        bits |= 64;
        invalid = true;
      } else if (active_frames > 0 && g < static_cast<float>(active_frames) - 0.5f) {
        bits |= 64;
      }
    }
    if (invalid) bits |= 1;
    if (nlow > 0) bits |= 256;
    if (nhigh > 0) bits |= 512;
    a.dq[p] = static_cast<int16_t>(bits);
  }
}

struct CenterScale {
  float center;
  float scale;
};

__device__ __forceinline__ void ff_merge2(FF& a, const FF& b) {
  float s, e;
  two_sum(a.hi, b.hi, s, e);
  a.hi = s;
  a.lo = __fadd_rn(__fadd_rn(a.lo, b.lo), e);
}

// True when every value in [lo, hi] lies within a factor of two of c (same
// sign), so x - c is exact in float32 (Sterbenz).
__device__ __forceinline__ bool sterbenz_interval(float lo, float hi, float c) {
  if (c > 0.0f) return lo >= 0.5f * c && hi <= 2.0f * c;
  if (c < 0.0f) return hi <= 0.5f * c && lo >= 2.0f * c;
  return false;
}

// Number of sorted valid values < t (strict) or <= t.
__device__ __forceinline__ int count_below(const float* S, int T, int cnt, float t, bool inclusive) {
  int lo = 0, hi = cnt;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    const float v = S[mid * T];
    if (inclusive ? (v <= t) : (v < t)) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Integration of up to 256 resident frames, one thread per pixel
// (integrate_px.cuh): mean, sigma clip and winsorized sigma clip.
void launch_integrate_px(const IntegrateArgs& args, cudaStream_t stream);

}  // namespace gg
