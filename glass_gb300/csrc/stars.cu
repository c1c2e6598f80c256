// Star detection on resident frames: robust background, threshold,
// local-maximum candidates, windowed moments, flux-ordered de-duplication.
//
// Semantics: src/glass/cpu/star_detect.py:29-168 (detect_stars):
//   median / MAD of the finite pixels (exact order statistics; an even count
//   takes the float32 mean of the two middle values, as np.median does),
//   noise = 1.4826 * MAD (float64; falls back to the pixel std, then 1),
//   threshold = median + k * max(noise, 1e-6) (float64, compared against the
//   float32 pixels after rounding to float32 - NumPy's scalar promotion),
//   candidate = interior pixel, finite, > threshold, >= its 8 neighbours,
//   measurement in a (2r+1)^2 window clipped to the image with float64
//   moments of max(v - background, 0) (star_detect.py:45-100),
//   greedy de-duplication in flux order (stable: raster order breaks ties,
//   star_detect.py:103-118), then the brightest `max_stars`.
//
// GB300 layout:
//   - order statistics in one pass over the frame: a sample gives a key band
//     around the wanted ranks, the pass keeps the band's keys and a cluster per
//     frame selects among them; the MAD does the same with key |v - median|.
//     Frames whose band misses (heavily tied data) take a 3-pass radix select
//     (11+11+10 key bits, per-CTA histograms folded with global atomics);
//   - candidates are found chunk by chunk of a row; a prefix sum over the
//     chunks' counts puts them into raster order; flux and centroid one warp
//     per candidate; the flux-ordered de-duplication works on lists of the
//     brighter neighbours (centroids stay within the window of their peak);
//     one CTA per frame decides it and selects the brightest by an 8-bit radix
//     select on the flux bits; second moments (fwhm, eccentricity) and the
//     output order only for the selected stars;
//   - the first 80 selected stars (optionally only those passing a shape
//     filter) stay on the device as the frame's registration catalog.
#include <cmath>
#include <cstring>
#include <vector>

#include <cooperative_groups.h>
#include <math_constants.h>

#include "stack.cuh"

namespace gg {

constexpr int kSelBins = 2048;
constexpr int kMaxCandidates = 32768;  // per frame (15-bit indices)
constexpr int kMaxSelected = 4096;     // per frame: the largest max_stars

// Per-frame detection state on the device.
struct StarFrameState {
  unsigned count;        // valid (finite) pixels
  unsigned candidates;   // appended candidates (may exceed capacity)
  unsigned overflow;
  unsigned ticket;       // CTAs that have finished (zero between launches)
  unsigned prefix[2];    // radix-select prefix per requested rank
  unsigned residual[2];  // rank remaining inside the prefix bucket
  float median;
  float mad;
  double noise;
  double threshold;
  float threshold_f32;
  float background_f32;
  double background;
  int kept;      // output stars
  int selected;  // stars handed to the moments kernel (kept and ties at the last place)
  // sample-bracket selection (per mode: 0 median, 1 MAD)
  unsigned band_lo, band_hi;  // inclusive key band from the sample
  unsigned below;             // finite keys under band_lo
  unsigned inside;            // keys in the band (appended, may exceed capacity)
  int resolved[2];            // 1: the order statistic came from the band
};

__device__ __forceinline__ unsigned float_key(float v) {
  const unsigned b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_float(unsigned k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

struct SelectArgs {
  const float* slots;
  const int* slot_of_frame;
  int64_t stride;
  int64_t pixels;
  const int* frames;   // [count]
  StarFrameState* state;
  unsigned* hist;      // [count][2][kSelBins]
  int mode;            // 0: v, 1: |v - median|
};

// Locate each rank's bucket in the frame's complete histogram (a warp prefix
// scan over 32 runs of bins).  Pass 0 sets the ranks from the valid count
// (median of n: n//2 and n//2 - 1 when n is even, both n//2 when odd).
template <int PASS>
__device__ void select_digit(const SelectArgs& a, StarFrameState& st, const unsigned (*hs)[kSelBins]) {
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  const unsigned count = __ldcg(&st.count);
  constexpr int kBins = PASS == 2 ? 1024 : kSelBins;
  constexpr int kPer = kBins / 32;
  constexpr int kBits = PASS == 2 ? 10 : 11;
  unsigned prefix[2];
  for (int r = 0; r < 2; ++r) {
    const unsigned* hr = hs[PASS == 0 ? 0 : r];
    unsigned rem;
    if constexpr (PASS == 0) {
      const unsigned hi = count / 2;
      rem = r == 1 || (count & 1u) ? hi : (hi > 0 ? hi - 1 : 0);
    } else {
      rem = st.residual[r];
    }
    unsigned loc = 0;
    for (int b = 0; b < kPer; ++b) loc += hr[lane * kPer + b];
    unsigned incl = loc;
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned v = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += v;
    }
    const unsigned excl = incl - loc;
    const bool here = excl <= rem && rem < incl;
    unsigned bucket = static_cast<unsigned>(kBins - 1), left = 0u;  // empty frame (rank past the end)
    if (here) {
      left = rem - excl;
      int b = lane * kPer;
      while (left >= hr[b]) {
        left -= hr[b];
        ++b;
      }
      bucket = static_cast<unsigned>(b);
    }
    const unsigned owner = __ballot_sync(0xffffffffu, here);
    const int from = owner ? __ffs(owner) - 1 : 0;
    bucket = __shfl_sync(0xffffffffu, bucket, from);
    left = __shfl_sync(0xffffffffu, left, from);
    prefix[r] = ((PASS == 0 ? 0u : st.prefix[r]) << kBits) | bucket;
    __syncwarp();
    if (lane == 0) {
      st.prefix[r] = prefix[r];
      st.residual[r] = left;
    }
  }
  if (PASS == 2 && lane == 0) {
    // Both keys are complete: value = mean of the two middle values.
    const float med = count ? __fmul_rn(__fadd_rn(key_float(prefix[0]), key_float(prefix[1])), 0.5f) : 0.0f;
    if (a.mode == 0) st.median = med; else st.mad = med;
  }
}

// Histogram pass: digit of `pass` for keys matching each rank's prefix.
// Sky pixels share their leading digits, so each thread keeps a run-length
// counter per histogram (last digit, count) and only touches shared memory
// when the digit changes; four pixels per float4 load.  When both ranks
// share their prefix (the usual case: the two middle values of an even
// count lie in one bucket) only the first histogram is built and copied.
template <int PASS>
__global__ void __launch_bounds__(256) select_hist_kernel(SelectArgs a) {
  __shared__ unsigned h[2][kSelBins];
  __shared__ unsigned s_valid;
  const int k = blockIdx.y;
  if (a.state[k].resolved[a.mode]) return;  // the sample bracket found it
  for (int i = threadIdx.x; i < 2 * kSelBins; i += blockDim.x) (&h[0][0])[i] = 0u;
  if (threadIdx.x == 0) s_valid = 0;
  __syncthreads();
  const unsigned p0 = a.state[k].prefix[0], p1 = a.state[k].prefix[1];
  const bool shared_prefix = p0 == p1;
  const float median = a.state[k].median;
  const bool absdev = a.mode == 1;
  const float* src = a.slots + static_cast<int64_t>(a.slot_of_frame[a.frames[k]]) * a.stride;
  constexpr int kShift = PASS == 0 ? 21 : (PASS == 1 ? 10 : 0);
  constexpr unsigned kMask = PASS == 2 ? 1023u : 2047u;
  constexpr int kPrefixShift = PASS == 1 ? 21 : 10;
  unsigned valid = 0;
  unsigned d0 = 0xffffffffu, n0 = 0u, d1 = 0xffffffffu, n1 = 0u;
  auto add = [&](float v) {
    if (!isfinite(v)) return;
    ++valid;
    if (absdev) v = fabsf(__fsub_rn(v, median));
    const unsigned key = float_key(v);
    const unsigned digit = (key >> kShift) & kMask;
    bool in0 = true, in1 = false;
    if constexpr (PASS != 0) {
      const unsigned hp = key >> kPrefixShift;
      in0 = hp == p0;
      in1 = !shared_prefix && hp == p1;
    }
    if (in0) {
      if (digit == d0) {
        ++n0;
      } else {
        if (n0) atomicAdd(&h[0][d0], n0);
        d0 = digit;
        n0 = 1u;
      }
    }
    if (in1) {
      if (digit == d1) {
        ++n1;
      } else {
        if (n1) atomicAdd(&h[1][d1], n1);
        d1 = digit;
        n1 = 1u;
      }
    }
  };
  const int64_t gtid = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  const int64_t gstride = int64_t(gridDim.x) * blockDim.x;
  const int64_t n4 = a.pixels / 4;  // slots start on 256-byte boundaries
  const float4* src4 = reinterpret_cast<const float4*>(src);
  for (int64_t i = gtid; i < n4; i += gstride) {
    const float4 q = __ldg(src4 + i);
    add(q.x);
    add(q.y);
    add(q.z);
    add(q.w);
  }
  for (int64_t p = n4 * 4 + gtid; p < a.pixels; p += gstride) add(__ldg(src + p));
  if (n0) atomicAdd(&h[0][d0], n0);
  if (n1) atomicAdd(&h[1][d1], n1);
  if (PASS == 0) {
    valid = __reduce_add_sync(0xffffffffu, valid);
    if ((threadIdx.x & 31) == 0 && valid) atomicAdd(&s_valid, valid);
  }
  __syncthreads();
  unsigned* g = a.hist + static_cast<int64_t>(k) * 2 * kSelBins;
  const int nh = PASS == 0 ? 1 : 2;
  for (int i = threadIdx.x; i < nh * kSelBins; i += blockDim.x) {
    const unsigned v = (shared_prefix && i >= kSelBins) ? h[0][i - kSelBins] : (&h[0][0])[i];
    if (v) atomicAdd(g + i, v);
  }
  if (PASS == 0 && a.mode == 0 && threadIdx.x == 0 && s_valid) atomicAdd(&a.state[k].count, s_valid);
  // the frame's last CTA finds the digit and leaves the histogram zeroed
  if (!last_cta(&a.state[k].ticket, gridDim.x)) return;
  for (int i = threadIdx.x; i < nh * kSelBins; i += blockDim.x) {
    (&h[0][0])[i] = __ldcg(g + i);
    g[i] = 0u;
  }
  __syncthreads();
  select_digit<PASS>(a, a.state[k], h);
}

// ---- order statistics by a sample bracket ------------------------------------
// One pass over the frame instead of three: the middle ranks of
// kBracketSamples evenly spaced pixels give a key band that holds the wanted
// ranks (the middle ranks of the finite pixels) with a seven-sigma margin; the
// pass counts the finite keys below the band and copies the keys inside it to
// a per-frame buffer, where a radix select over the band's key range finds the
// exact order statistics.  A frame whose band misses the ranks or overflows
// the buffer (heavily tied data) keeps resolved = 0 and goes through the
// three-pass radix select above.
constexpr int kBracketSamples = 32768;
constexpr int kSampleThreads = 1024;
constexpr int kSampleCtas = 8;  // per frame: the scattered reads of the sample
constexpr unsigned kNoKey = 0xffffffffu;  // above every finite key

struct BracketArgs {
  const float* slots;
  const int* slot_of_frame;
  int64_t stride;
  int64_t pixels;
  const int* frames;
  StarFrameState* state;
  unsigned* band;      // [count][band_cap]; holds the sample's keys first (band_cap >= its size)
  int64_t band_cap;    // a multiple of 4
  int mode;            // 0: v, 1: |v - median|
};

__device__ __forceinline__ bool bracket_key(float v, int mode, float median, unsigned& key) {
  if (!isfinite(v)) return false;
  key = float_key(mode == 1 ? fabsf(__fsub_rn(v, median)) : v);
  return true;
}

// The sample's two band edges.  Several CTAs per frame read the scattered
// pixels; the last one holds the 32768 keys in registers and finds the two
// ranks bit by bit from the top, counting the keys below a trial prefix: 32
// rounds of register compares and one block sum each, whatever the values.
// The rounds bound it: 338 us as a bitonic sort of the sample in shared memory
// by one CTA per frame, 43 us here (8 frames of 4096^2).
__global__ void __launch_bounds__(kSampleThreads) bracket_sample_kernel(BracketArgs a) {
  const int k = blockIdx.y;
  StarFrameState& st = a.state[k];
  unsigned* keys = a.band + static_cast<int64_t>(k) * a.band_cap;
  const int n = static_cast<int>(a.pixels < kBracketSamples ? a.pixels : static_cast<int64_t>(kBracketSamples));
  {
    const float* src = a.slots + static_cast<int64_t>(a.slot_of_frame[a.frames[k]]) * a.stride;
    const float median = st.median;
    constexpr int kPer = kBracketSamples / (kSampleThreads * kSampleCtas);
    const int first = static_cast<int>(blockIdx.x) * kSampleThreads * kPer + static_cast<int>(threadIdx.x);
    float v[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int i = first + u * kSampleThreads;
      if (i < n) v[u] = __ldg(src + ((2 * static_cast<int64_t>(i) + 1) * a.pixels) / (2 * static_cast<int64_t>(n)));
    }
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int i = first + u * kSampleThreads;
      unsigned key = kNoKey;
      if (i < n) {
        bracket_key(v[u], a.mode, median, key);
        keys[i] = key;
      }
    }
  }
  if (!last_cta(&st.ticket, gridDim.x)) return;
  constexpr int kKeys = kBracketSamples / kSampleThreads;
  unsigned key[kKeys];
  int valid = 0;
#pragma unroll
  for (int u = 0; u < kKeys; ++u) {
    const int i = u * kSampleThreads + static_cast<int>(threadIdx.x);
    key[u] = i < n ? __ldcg(keys + i) : kNoKey;
  }
#pragma unroll
  for (int u = 0; u < kKeys; ++u) valid += key[u] != kNoKey ? 1 : 0;
  // sums of a round: both counts in one word (at most 32768 each); a slot is
  // cleared two rounds before it is added to
  __shared__ unsigned s_sum[4];
  __shared__ int s_valid;
  if (threadIdx.x < 4) s_sum[threadIdx.x] = 0u;
  if (threadIdx.x == 0) s_valid = 0;
  __syncthreads();
  valid = __reduce_add_sync(0xffffffffu, valid);
  if ((threadIdx.x & 31) == 0 && valid) atomicAdd(&s_valid, valid);
  __syncthreads();
  const int sv = s_valid;
  // middle of the finite samples +- 7 binomial sigma (+8 for small samples)
  const int margin = static_cast<int>(ceilf(3.5f * sqrtf(static_cast<float>(sv)))) + 8;
  const unsigned rank_lo = static_cast<unsigned>(max(0, sv / 2 - margin));
  const unsigned rank_hi = static_cast<unsigned>(max(0, min(sv - 1, sv / 2 + margin)));
  unsigned p_lo = 0u, p_hi = 0u;
  for (int bit = 31; bit >= 0; --bit) {
    const unsigned t_lo = p_lo | (1u << bit), t_hi = p_hi | (1u << bit);
    unsigned c_lo = 0u, c_hi = 0u;
#pragma unroll
    for (int u = 0; u < kKeys; ++u) c_lo += key[u] < t_lo ? 1u : 0u;
    if (t_hi != t_lo) {
#pragma unroll
      for (int u = 0; u < kKeys; ++u) c_hi += key[u] < t_hi ? 1u : 0u;
    } else {
      c_hi = c_lo;
    }
    const unsigned both = __reduce_add_sync(0xffffffffu, c_lo | (c_hi << 16));
    if ((threadIdx.x & 31) == 0) atomicAdd(&s_sum[bit & 3], both);
    if (threadIdx.x == 0) s_sum[(bit - 2) & 3] = 0u;
    __syncthreads();
    const unsigned sum = s_sum[bit & 3];
    if ((sum & 0xffffu) <= rank_lo) p_lo = t_lo;
    if ((sum >> 16) <= rank_hi) p_hi = t_hi;
  }
  if (threadIdx.x == 0) {
    st.band_lo = sv > 0 ? p_lo : 0u;
    st.band_hi = sv > 0 ? p_hi : 0u;
    st.below = 0u;
    st.inside = 0u;
    if (a.mode == 0) st.count = 0u;
  }
}

// One pass over a frame: the finite samples below the band and the band's
// keys (appended to the frame's band buffer in no particular order).  A warp
// takes 16 samples per lane at a time (four float4 loads issued first),
// collects its in-band keys in shared memory and hands them over in runs of
// kBandStage, coalesced and with one atomic each; no barrier in the loop.  The
// per-sample tests are unsigned range checks on the order-preserving keys: a
// finite float32 has a key in [0x00800000, 0xff7fffff] (float_key), so mode 0
// needs no separate isfinite; mode 1 (|v - median|) tests the sample itself.
// Bound by memory: 8 frames of 4096^2 in 107 us, 129 us with three barriers
// and one atomic per 4096 samples.
constexpr int kBracketThreads = 256;
constexpr int kBandStage = 256;

template <int MODE>
__global__ void __launch_bounds__(kBracketThreads) bracket_pass_kernel(BracketArgs a) {
  constexpr int kLoads = 4;
  constexpr int kSamples = 32 * 4 * kLoads;  // per warp and iteration
  __shared__ unsigned s_keys[kBracketThreads / 32][kBandStage + kSamples];
  const int k = blockIdx.y;
  StarFrameState& st = a.state[k];
  const unsigned lo = st.band_lo, hi = st.band_hi;
  const unsigned span = hi - lo;  // the band is [lo, lo + span]
  constexpr unsigned kFiniteLo = 0x00800000u, kFiniteSpan = 0xff7fffffu - 0x00800000u;
  // mode 0: key < lo for a finite key <=> (key - kFiniteLo) < (lo - kFiniteLo),
  // nothing is below a band that starts below the finite keys
  const unsigned lo_f = lo >= kFiniteLo ? lo - kFiniteLo : 0u;
  const float median = st.median;
  const float* src = a.slots + static_cast<int64_t>(a.slot_of_frame[a.frames[k]]) * a.stride;
  unsigned* band = a.band + static_cast<int64_t>(k) * a.band_cap;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned* stage = s_keys[warp];
  unsigned staged = 0;  // the same in every lane
  unsigned below = 0, valid = 0;
  auto flush = [&]() {
    __syncwarp();
    unsigned base = 0u;
    if (lane == 0) base = atomicAdd(&st.inside, staged);
    base = __shfl_sync(0xffffffffu, base, 0);
    for (unsigned i = lane; i < staged; i += 32)
      if (static_cast<int64_t>(base) + i < a.band_cap) band[static_cast<int64_t>(base) + i] = stage[i];
    __syncwarp();
    staged = 0u;
  };
  const int64_t n4 = a.pixels / 4;
  const float4* src4 = reinterpret_cast<const float4*>(src);
  const int64_t gstride = int64_t(gridDim.x) * (blockDim.x * kLoads);
  for (int64_t base = (int64_t(blockIdx.x) * (kBracketThreads / 32) + warp) * (32 * kLoads); base < n4;
       base += gstride) {
    float4 q[kLoads];
#pragma unroll
    for (int u = 0; u < kLoads; ++u) {
      const int64_t i = base + u * 32 + lane;
      q[u] = i < n4 ? __ldg(src4 + i) : make_float4(CUDART_INF_F, CUDART_INF_F, CUDART_INF_F, CUDART_INF_F);
    }
    unsigned key[4 * kLoads];
    unsigned in_mask = 0u;
#pragma unroll
    for (int u = 0; u < kLoads; ++u) {
      const float v4[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int j = 4 * u + c;
        bool fin;
        if constexpr (MODE == 0) {
          const unsigned bits = __float_as_uint(v4[c]);
          key[j] = bits ^ (static_cast<unsigned>(static_cast<int>(bits) >> 31) | 0x80000000u);  // float_key
          const unsigned kf = key[j] - kFiniteLo;
          fin = kf <= kFiniteSpan;
          valid += fin ? 1u : 0u;
          below += (kf < lo_f) ? 1u : 0u;  // implies finite
        } else {
          fin = (__float_as_uint(v4[c]) & 0x7f800000u) != 0x7f800000u;
          key[j] = __float_as_uint(fabsf(__fsub_rn(v4[c], median))) | 0x80000000u;  // float_key of a |d|
          below += (fin && key[j] < lo) ? 1u : 0u;
        }
        in_mask |= (fin && key[j] - lo <= span) ? (1u << j) : 0u;
      }
    }
    if (!__any_sync(0xffffffffu, in_mask != 0u)) continue;
    const unsigned mine = __popc(in_mask);
    unsigned incl = mine;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned n = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += n;
    }
    unsigned pos = staged + incl - mine;
#pragma unroll
    for (int j = 0; j < 4 * kLoads; ++j)
      if ((in_mask >> j) & 1u) stage[pos++] = key[j];
    staged += __shfl_sync(0xffffffffu, incl, 31);
    if (staged >= kBandStage) flush();
  }
  if (staged) flush();
  // the last pixels % 4 samples: one warp, one atomic per in-band sample
  if (blockIdx.x == 0 && threadIdx.x < 32) {
    for (int64_t p = n4 * 4 + threadIdx.x; p < a.pixels; p += 32) {
      unsigned key = 0u;
      const bool fin = bracket_key(__ldg(src + p), MODE, median, key);
      valid += fin ? 1u : 0u;
      below += (fin && key < lo) ? 1u : 0u;
      if (fin && key >= lo && key <= hi) {
        const unsigned at = atomicAdd(&st.inside, 1u);
        if (at < a.band_cap) band[at] = key;
      }
    }
  }
  below = __reduce_add_sync(0xffffffffu, below);
  valid = __reduce_add_sync(0xffffffffu, valid);
  if (lane == 0) {
    if (below) atomicAdd(&st.below, below);
    if (MODE == 0 && valid) atomicAdd(&st.count, valid);
  }
}

// The two middle ranks' keys inside the band by an MSB-first radix select
// over key - band_lo (8 bits per pass), then the median / MAD as the float32
// mean of the two middle values (np.median); no band select when the order
// statistics lie outside it: the radix fallback then takes the frame.  The
// band of a 9600 x 6422 frame holds ~1.6 M keys, so a cluster of CTAs shares
// it, one cluster barrier per pass: every CTA sums the cluster's histograms
// over distributed shared memory and finds the digits for itself.  Bound by
// the passes' latency: 36 us for 8 frames of 4096^2 (0.4 M keys each), 94 us
// as ten launches.
constexpr int kBandCtas = 8;
constexpr int kBandThreads = 512;

__global__ void __cluster_dims__(kBandCtas, 1, 1) __launch_bounds__(kBandThreads) bracket_band_kernel(BracketArgs a) {
  namespace cg = cooperative_groups;
  __shared__ unsigned hist[2][512];  // [pass parity][rank * 256 + digit]
  __shared__ unsigned total[512];
  __shared__ unsigned s_digit[2], s_rank[2];
  cg::cluster_group cluster = cg::this_cluster();
  const int k = blockIdx.y;
  StarFrameState& st = a.state[k];
  const unsigned n = st.count;
  const unsigned rhi = n / 2, rlo = (n & 1u) ? rhi : (rhi > 0 ? rhi - 1 : 0);
  const unsigned inside = st.inside, below = st.below;
  const unsigned lo = st.band_lo, range = st.band_hi - lo;
  const bool ok = n > 0 && static_cast<int64_t>(inside) <= a.band_cap && below <= rlo && rhi < below + inside;
  unsigned rank[2] = {rlo - below, rhi - below};
  unsigned prefix[2] = {0u, 0u};
  const int top = 32 - __clz(range);  // bits of the key range
  const unsigned* band = a.band + static_cast<int64_t>(k) * a.band_cap;
  const unsigned step = kBandCtas * kBandThreads;
  const unsigned first = cluster.block_rank() * kBandThreads + threadIdx.x;
  int parity = 0;
  if (ok) {  // the same in every CTA of the cluster
    for (int shift = ((top + 7) / 8) * 8 - 8; shift >= 0; shift -= 8, parity ^= 1) {
      unsigned* h = hist[parity];
      h[threadIdx.x] = 0u;
      __syncthreads();
      const bool split = prefix[0] != prefix[1];
      auto add = [&](unsigned key) {
        const unsigned d = key - lo;
        const unsigned hp = shift >= 24 ? 0u : (d >> (shift + 8));
        const unsigned digit = (d >> shift) & 255u;
        if (hp == prefix[0]) atomicAdd(&h[digit], 1u);
        if (split && hp == prefix[1]) atomicAdd(&h[256 + digit], 1u);
      };
      const uint4* band4 = reinterpret_cast<const uint4*>(band);
#pragma unroll 4
      for (unsigned i = first; i < inside / 4; i += step) {
        const uint4 q = band4[i];
        add(q.x);
        add(q.y);
        add(q.z);
        add(q.w);
      }
      if (first < (inside & 3u)) add(band[(inside & ~3u) + first]);
      cluster.sync();
      unsigned sum = 0u;
#pragma unroll
      for (int c = 0; c < kBandCtas; ++c) sum += cluster.map_shared_rank(h, c)[threadIdx.x];
      total[threadIdx.x] = sum;
      __syncthreads();
      if (threadIdx.x < 64) {
        const int r = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const unsigned* t = total + (split ? 256 * r : 0);
        unsigned loc = 0;
        for (int b = 0; b < 8; ++b) loc += t[lane * 8 + b];
        unsigned incl = loc;
        for (int off = 1; off < 32; off <<= 1) {
          const unsigned v = __shfl_up_sync(0xffffffffu, incl, off);
          if (lane >= off) incl += v;
        }
        const unsigned excl = incl - loc;
        if (excl <= rank[r] && rank[r] < incl) {
          unsigned left = rank[r] - excl;
          int b = lane * 8;
          while (left >= t[b]) {
            left -= t[b];
            ++b;
          }
          s_digit[r] = static_cast<unsigned>(b);
          s_rank[r] = left;
        }
      }
      __syncthreads();
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        prefix[r] = (prefix[r] << 8) | s_digit[r];
        rank[r] = s_rank[r];
      }
    }
  }
  // no CTA leaves while another may read its histogram, or before all have read the state
  cluster.sync();
  if (first != 0) return;
  st.resolved[a.mode] = ok ? 1 : 0;
  if (ok) {
    const float med = __fmul_rn(__fadd_rn(key_float(lo + prefix[0]), key_float(lo + prefix[1])), 0.5f);
    if (a.mode == 0) st.median = med; else st.mad = med;
  } else if (a.mode == 0) {
    st.count = 0u;  // the radix passes count the finite pixels again
  }
}

// Threshold from median / MAD (star_detect.py:29-43, 133-137).
__global__ void star_threshold_kernel(StarFrameState* state, int frames, float k_sigma, int has_background,
                                      float background, int has_noise, float noise, const double* rms) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= frames) return;
  StarFrameState& st = state[k];
  double med = st.count ? static_cast<double>(st.median) : 0.0;
  double nz = st.count ? 1.4826 * static_cast<double>(st.mad) : 1.0;
  if (st.count && !(nz > 0.0)) nz = rms ? rms[k] : 0.0;
  if (!(nz > 0.0)) nz = 1.0;
  if (has_background) med = static_cast<double>(background);
  if (has_noise) nz = static_cast<double>(noise);
  st.noise = nz;
  st.threshold = med + static_cast<double>(k_sigma) * fmax(nz, 1.0e-6);
  st.threshold_f32 = static_cast<float>(st.threshold);
  st.background_f32 = static_cast<float>(med);
  st.background = med;
}

// ---- background mesh (no reference counterpart) ------------------------------
// Cells of `cell` x `cell` pixels from the top-left corner (edge cells
// smaller).  Each cell's finite pixels give the float64 median (an even count
// takes 0.5 * (a + b) of the two middle values) and noise 1.4826 * MAD (1
// when the MAD is 0; NaN median and noise without finite pixels).  Values at
// a pixel interpolate bilinearly between cell centres, u = (x + 0.5) / cell -
// 0.5, clamped at the first and last centre, in float64 without fused
// multiply-adds (the oracle evaluates the same operations in NumPy).
constexpr int kMeshMaxCell = 64;
constexpr int kMeshElems = kMeshMaxCell * kMeshMaxCell;

struct MeshView {
  const double* bg;  // [count][ny * nx] or nullptr (global statistics)
  const double* nz;
  int cell, nx, ny;
};

__device__ __forceinline__ void mesh_axis(int coord, int cell, int n, int& i0, int& i1, double& f) {
  const double u = __dsub_rn(__ddiv_rn(__dadd_rn(static_cast<double>(coord), 0.5), static_cast<double>(cell)), 0.5);
  const double fl = floor(u);
  if (fl < 0.0) {
    i0 = 0;
    f = 0.0;
  } else if (fl >= static_cast<double>(n - 1)) {
    i0 = n - 1;
    f = 0.0;
  } else {
    i0 = static_cast<int>(fl);
    f = __dsub_rn(u, fl);
  }
  i1 = min(i0 + 1, n - 1);
}

__device__ __forceinline__ double mesh_lerp(const double* m, int nx, int i0, int i1, int j0, int j1, double fx,
                                            double fy) {
  const double gx = __dsub_rn(1.0, fx), gy = __dsub_rn(1.0, fy);
  const double top = __dadd_rn(__dmul_rn(gx, m[j0 * nx + i0]), __dmul_rn(fx, m[j0 * nx + i1]));
  const double bot = __dadd_rn(__dmul_rn(gx, m[j1 * nx + i0]), __dmul_rn(fx, m[j1 * nx + i1]));
  return __dadd_rn(__dmul_rn(gy, top), __dmul_rn(fy, bot));
}

// Interpolated background and noise of frame k at pixel (x, y).
__device__ __forceinline__ void mesh_at(const MeshView& m, int k, int x, int y, double& bg, double& nz) {
  int i0, i1, j0, j1;
  double fx, fy;
  mesh_axis(x, m.cell, m.nx, i0, i1, fx);
  mesh_axis(y, m.cell, m.ny, j0, j1, fy);
  const int64_t off = static_cast<int64_t>(k) * m.nx * m.ny;
  bg = mesh_lerp(m.bg + off, m.nx, i0, i1, j0, j1, fx, fy);
  nz = mesh_lerp(m.nz + off, m.nx, i0, i1, j0, j1, fx, fy);
}

__device__ void bitonic_sort_shared(double* v, int n) {
  for (int k = 2; k <= n; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int ixj = i ^ j;
        if (ixj > i) {
          const bool up = (i & k) == 0;
          const double a = v[i], b = v[ixj];
          if ((a > b) == up) {
            v[i] = b;
            v[ixj] = a;
          }
        }
      }
      __syncthreads();
    }
}

__device__ __forceinline__ double median_sorted(const double* v, int n) {
  const int m = n / 2;
  return (n & 1) ? v[m] : __dmul_rn(__dadd_rn(v[m - 1], v[m]), 0.5);
}

struct MeshArgs {
  const float* slots;
  const int* slot_of_frame;
  int64_t stride;
  int width, height;
  const int* frames;
  double* bg;
  double* nz;
  int cell, nx, ny;
};

// One CTA per (cell, frame): gather the finite pixels, sort, median; sort the
// absolute deviations, MAD.
__global__ void __launch_bounds__(1024) mesh_stats_kernel(MeshArgs a) {
  __shared__ double v[kMeshElems];
  __shared__ int s_n;
  __shared__ double s_med;
  const int c = blockIdx.x, k = blockIdx.y;
  const int cx = c % a.nx, cy = c / a.nx;
  const int x0 = cx * a.cell, y0 = cy * a.cell;
  const int w = min(a.cell, a.width - x0), h = min(a.cell, a.height - y0);
  const float* img = a.slots + static_cast<int64_t>(a.slot_of_frame[a.frames[k]]) * a.stride;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  for (int q = threadIdx.x; q < w * h; q += blockDim.x) {
    const float val = __ldg(img + static_cast<int64_t>(y0 + q / w) * a.width + x0 + q % w);
    if (isfinite(val)) v[atomicAdd(&s_n, 1)] = static_cast<double>(val);
  }
  __syncthreads();
  const int n = s_n;
  const int64_t out = static_cast<int64_t>(k) * a.nx * a.ny + c;
  if (n == 0) {
    if (threadIdx.x == 0) a.bg[out] = a.nz[out] = __longlong_as_double(0x7ff8000000000000LL);
    return;
  }
  int p2 = 1;
  while (p2 < n) p2 <<= 1;
  const double inf = __longlong_as_double(0x7ff0000000000000LL);
  for (int q = n + threadIdx.x; q < p2; q += blockDim.x) v[q] = inf;
  __syncthreads();
  bitonic_sort_shared(v, p2);
  if (threadIdx.x == 0) s_med = median_sorted(v, n);
  __syncthreads();
  const double med = s_med;
  for (int q = threadIdx.x; q < n; q += blockDim.x) v[q] = fabs(__dsub_rn(v[q], med));
  __syncthreads();
  bitonic_sort_shared(v, p2);
  if (threadIdx.x == 0) {
    const double mad = median_sorted(v, n);
    a.bg[out] = med;
    a.nz[out] = mad > 0.0 ? __dmul_rn(1.4826, mad) : 1.0;
  }
}

struct DetectArgs {
  const float* slots;
  const int* slot_of_frame;
  int64_t stride;
  int width, height;
  const int* frames;
  StarFrameState* state;
  unsigned* raw;     // [count][kMaxCandidates] raster indices, chunk by chunk
  unsigned* chunks;  // [count][chunk_stride] count << 16 | first of each chunk
  unsigned chunk_stride, chunk_count, chunks_per_row;
  MeshView mesh;
  double k_sigma;
};

// Local-maximum candidates (star_detect.py:142-151).  A warp takes a chunk of
// kChunk columns of a row, from the 16-byte boundary at or before the row's
// start: four float4 loads per lane, all issued first.  A chunk's candidates
// are appended in column order with one atomic and noted in the chunk table,
// so the raster order of the whole frame is a prefix sum over the table
// (star_order_kernel) and needs no sort.  Bound by issue slots (69 %), then
// the loads: 8 frames of 4096^2 in 121 us, 194 us with scalar loads.  MESH: per-pixel threshold from the
// background mesh (float64), else the frame's float32 threshold.
constexpr int kChunk = 512;

template <bool MESH>
__global__ void __launch_bounds__(256) star_detect_kernel(DetectArgs a) {
  const int k = blockIdx.y;
  const float* img = a.slots + static_cast<int64_t>(a.slot_of_frame[a.frames[k]]) * a.stride;
  const float thr = a.state[k].threshold_f32;
  const int W = a.width;
  unsigned* raw = a.raw + static_cast<int64_t>(k) * kMaxCandidates;
  unsigned* chunks = a.chunks + static_cast<int64_t>(k) * a.chunk_stride;
  const int lane = threadIdx.x & 31;
  const unsigned warps = gridDim.x * (blockDim.x >> 5);
  float4 next[4];
  // row and chunk of the row of the vectors in `next`, advanced without a division
  unsigned e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int next_y = 1 + static_cast<int>(e / a.chunks_per_row);
  unsigned next_c = e % a.chunks_per_row;
  const int step_y = static_cast<int>(warps / a.chunks_per_row);
  const unsigned step_c = warps % a.chunks_per_row;
  auto load = [&]() {
    const int64_t row_at = static_cast<int64_t>(next_y) * W;
    const int x0 = static_cast<int>(next_c) * kChunk - static_cast<int>(row_at & 3) + 4 * lane;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      // rows 1 .. H - 2: a vector that starts before the row or ends behind it stays inside the frame
      const int x = x0 + 128 * u;
      next[u] =
          x <= W - 2 ? __ldg(reinterpret_cast<const float4*>(img + row_at + x)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
  };
  if (e < a.chunk_count) load();
  for (; e < a.chunk_count; e += warps) {
    const int y = next_y;
    const int64_t row_at = static_cast<int64_t>(y) * W;
    const float* row = img + row_at;
    const int x0 = static_cast<int>(next_c) * kChunk - static_cast<int>(row_at & 3) + 4 * lane;  // lane's first column
    const float4 q[4] = {next[0], next[1], next[2], next[3]};
    next_y += step_y;
    next_c += step_c;
    if (next_c >= a.chunks_per_row) {
      next_c -= a.chunks_per_row;
      ++next_y;
    }
    if (e + warps < a.chunk_count) load();  // in flight while this chunk's candidates are tested
    // threshold first: most chunks hold no candidate
    if constexpr (!MESH) {
      float top = -CUDART_INF_F;  // NaN drops out
#pragma unroll
      for (int u = 0; u < 4; ++u) top = fmaxf(fmaxf(top, fmaxf(q[u].x, q[u].y)), fmaxf(q[u].z, q[u].w));
      if (!__any_sync(0xffffffffu, top > thr)) {
        if (lane == 0) chunks[e] = 0u;
        continue;
      }
    }
    unsigned bits = 0u;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float c[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        bool above;
        if constexpr (MESH) {
          const int x = x0 + 128 * u + j;
          above = false;
          if (x >= 1 && x <= W - 2) {  // the mesh is read inside the frame only
            double bg, nz;
            mesh_at(a.mesh, k, x, y, bg, nz);
            const double nzc = (nz >= 1.0e-6 || isnan(nz)) ? nz : 1.0e-6;  // np.maximum keeps NaN
            above = static_cast<double>(c[j]) > __dadd_rn(bg, __dmul_rn(a.k_sigma, nzc));
          }
        } else {
          above = c[j] > thr;
        }
        // a neighbour in the same vector that is not <= c (NaN included) settles it here
        above = above && (j == 0 || c[j] >= c[j > 0 ? j - 1 : 0]) && (j == 3 || c[j] >= c[j < 3 ? j + 1 : 3]);
        bits |= above ? (1u << (4 * u + j)) : 0u;
      }
    }
    if (!__any_sync(0xffffffffu, bits != 0u)) {
      if (lane == 0) chunks[e] = 0u;
      continue;
    }
    unsigned hits = 0u;
    while (bits) {
      const int b = __ffs(bits) - 1;
      bits &= bits - 1u;
      const int x = x0 + 128 * (b >> 2) + (b & 3);
      if (x < 1 || x > W - 2) continue;
      const float* p = row + x;
      const float c = __ldg(p);
      bool hit = c < CUDART_INF_F;
#pragma unroll
      for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx)
          if (dx || dy) hit &= (c >= __ldg(p + static_cast<int64_t>(dy) * W + dx));
      hits |= hit ? (1u << b) : 0u;
    }
    __syncwarp();
    // column order: vector u of every lane before vector u + 1; the four
    // prefixes in the bytes of one word (at most 128 each)
    unsigned mine = 0u;
#pragma unroll
    for (int u = 0; u < 4; ++u) mine |= static_cast<unsigned>(__popc((hits >> (4 * u)) & 15u)) << (8 * u);
    unsigned incl = mine;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned v = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += v;
    }
    const unsigned totals = __shfl_sync(0xffffffffu, incl, 31);
    const unsigned n = (totals & 255u) + ((totals >> 8) & 255u) + ((totals >> 16) & 255u) + (totals >> 24);
    unsigned base = 0u;
    if (lane == 0 && n) base = atomicAdd(&a.state[k].candidates, n);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (lane == 0) {
      const unsigned room = base < static_cast<unsigned>(kMaxCandidates) ? kMaxCandidates - base : 0u;
      const unsigned kept = min(n, room);
      chunks[e] = kept ? (kept << 16) | base : 0u;
    }
    const unsigned excl = incl - mine;
    unsigned start = base;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      unsigned pos = start + ((excl >> (8 * u)) & 255u);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if ((hits >> (4 * u + j)) & 1u) {
          if (pos < static_cast<unsigned>(kMaxCandidates))
            raw[pos] = static_cast<unsigned>(row_at + x0 + 128 * u + j);
          ++pos;
        }
      start += (totals >> (8 * u)) & 255u;
    }
  }
}

// Measured star (float64 fields as the CPU's Python floats).
// Float-float sum of the whole warp (TwoSum butterfly), in every lane.
__device__ __forceinline__ void ff_warp_sum(FF& s) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const float oh = __shfl_xor_sync(0xffffffffu, s.hi, off);
    const float ol = __shfl_xor_sync(0xffffffffu, s.lo, off);
    float h, e;
    two_sum(s.hi, oh, h, e);
    s.hi = h;
    s.lo = __fadd_rn(__fadd_rn(s.lo, ol), e);
  }
}

// (n.hi + n.lo) / (d.hi + d.lo) to about 46 bits, returned as a double.
__device__ __forceinline__ double ff_quotient_f64(const FF& n, const FF& d) {
  const float q = __fdiv_rn(n.hi, d.hi);
  float r = __fmaf_rn(-q, d.hi, n.hi);
  r = __fadd_rn(r, n.lo);
  r = __fmaf_rn(-q, d.lo, r);
  return static_cast<double>(q) + static_cast<double>(__fdiv_rn(r, d.hi));
}

struct StarRec {
  double x, y, flux, peak;
  int npix;
  int valid;
};

struct SelectedStar;

struct CatalogArgs {
  const float* slots;
  const int* slot_of_frame;
  int64_t stride;
  int width, height;
  const int* frames;
  StarFrameState* state;
  const unsigned* raw;           // [count][kMaxCandidates] candidates, chunk by chunk
  const unsigned* chunks;        // [count][chunk_stride] star_detect_kernel's chunk table
  unsigned* chunk_first;         // [count][chunk_stride] each chunk's first candidate in raster order
  unsigned chunk_stride, chunk_count, chunks_per_row;
  unsigned* cand;                // [count][kMaxCandidates] raster order
  StarRec* recs;                 // [count][kMaxCandidates]
  unsigned long long* keys;      // [count][kMaxCandidates] flux keys
  unsigned char* conflict_count; // [count][kMaxCandidates]
  unsigned short* conflicts;     // [count][kMaxCandidates][kConflicts]
  SelectedStar* selected;        // [count][kMaxSelected]
  gg_star_t* out;                // [count][max_stars]
  int max_stars;
  int radius;
  double min_sep;
  double* cat_xy;  // [frames][kCatalogPoints][2]: brightest stars, for registration
  int* cat_n;      // [frames]
  MeshView mesh;   // local background / noise per star when mesh.bg is set
};

// Sum of `v` over the block's earlier threads, and the block's total.
__device__ __forceinline__ unsigned block_exclusive_sum(unsigned v, unsigned& total) {
  __shared__ unsigned s_warp[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned incl = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned n = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += n;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  unsigned w = lane < static_cast<int>(blockDim.x >> 5) ? s_warp[lane] : 0u;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned n = __shfl_up_sync(0xffffffffu, w, off);
    if (lane >= off) w += n;
  }
  total = __shfl_sync(0xffffffffu, w, 31);
  const unsigned before = __shfl_sync(0xffffffffu, w, (warp + 31) & 31);
  __syncthreads();  // s_warp may be written again
  return incl - v + (warp ? before : 0u);
}

// Candidates into raster order: each chunk's place is the sum of the counts of
// the chunks before it (a few CTAs per frame, each of which sums the table up
// to its own part).  Also each chunk's first candidate, by which later kernels
// find a row.  8 us for 8 frames of 4096^2 with 13,000 candidates each, 142
// us as a bitonic sort by one CTA per frame.
constexpr int kOrderThreads = 1024;
constexpr int kOrderTile = 4 * kOrderThreads;
constexpr int kOrderCtas = 16;

__global__ void __launch_bounds__(kOrderThreads) star_order_kernel(CatalogArgs a) {
  const int k = blockIdx.y;
  StarFrameState& st = a.state[k];
  const unsigned* chunks = a.chunks + static_cast<int64_t>(k) * a.chunk_stride;
  unsigned* first = a.chunk_first + static_cast<int64_t>(k) * a.chunk_stride;
  const unsigned* raw = a.raw + static_cast<int64_t>(k) * kMaxCandidates;
  unsigned* cand = a.cand + static_cast<int64_t>(k) * kMaxCandidates;
  const unsigned tiles = (a.chunk_count + kOrderTile - 1) / kOrderTile;
  const unsigned per = (tiles + gridDim.x - 1) / gridDim.x;
  const unsigned tile0 = blockIdx.x * per, tile1 = min(tiles, tile0 + per);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st.overflow = st.candidates > static_cast<unsigned>(kMaxCandidates) ? 1u : 0u;
    first[a.chunk_count] = min(st.candidates, static_cast<unsigned>(kMaxCandidates));
  }
  if (tile0 >= tile1) return;
  unsigned sum = 0u, carry;
#pragma unroll 4
  for (unsigned i = 4 * threadIdx.x; i < tile0 * kOrderTile; i += kOrderTile) {
    const uint4 q = __ldg(reinterpret_cast<const uint4*>(chunks + i));
    sum += (q.x >> 16) + (q.y >> 16) + (q.z >> 16) + (q.w >> 16);
  }
  block_exclusive_sum(sum, carry);
  for (unsigned tile = tile0; tile < tile1; ++tile) {
    const unsigned i = tile * kOrderTile + 4 * threadIdx.x;
    unsigned e[4];
    unsigned c = 0u;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      e[j] = i + j < a.chunk_count ? __ldg(chunks + i + j) : 0u;
      c += e[j] >> 16;
    }
    unsigned total;
    unsigned at = carry + block_exclusive_sum(c, total);
    carry += total;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (i + j >= a.chunk_count) break;
      first[i + j] = at;
      const unsigned n = e[j] >> 16, from = e[j] & 0xffffu;
      for (unsigned m = 0; m < n; ++m) cand[at + m] = __ldg(raw + from + m);
      at += n;
    }
  }
}

__device__ __forceinline__ unsigned long long flux_key(double f) {
  return static_cast<unsigned long long>(__double_as_longlong(f));  // f > 0: bit order = value order
}

// One warp per candidate: windowed moments (star_detect.py:45-100).
__global__ void __launch_bounds__(256) star_measure_kernel(CatalogArgs a) {
  const int k = blockIdx.y;
  const StarFrameState& st = a.state[k];
  const int n = static_cast<int>(min(st.candidates, static_cast<unsigned>(kMaxCandidates)));
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const float* img = a.slots + static_cast<int64_t>(a.slot_of_frame[a.frames[k]]) * a.stride;
  const unsigned* cand = a.cand + static_cast<int64_t>(k) * kMaxCandidates;
  StarRec* recs = a.recs + static_cast<int64_t>(k) * kMaxCandidates;
  unsigned long long* keys = a.keys + static_cast<int64_t>(k) * kMaxCandidates;
  const int W = a.width, H = a.height, r = a.radius;
  for (int c = warp; c < n; c += nwarps) {
    const unsigned idx = cand[c];
    const int x = static_cast<int>(idx % static_cast<unsigned>(W));
    const int y = static_cast<int>(idx / static_cast<unsigned>(W));
    double bg = st.background, noise = st.noise;
    if (a.mesh.bg) mesh_at(a.mesh, k, x, y, bg, noise);
    const float bg32 = a.mesh.bg ? __double2float_rn(bg) : st.background_f32;
    (void)noise;
    const int x0 = max(0, x - r), x1 = min(W, x + r + 1);
    const int y0 = max(0, y - r), y1 = min(H, y + r + 1);
    const int ww = x1 - x0, npx = ww * (y1 - y0);
    // float-float sums (about 48 bits; the weights are float32 and the
    // coordinate products exact): float64 is scarce on this part
    FF f, sx, sy;
    int fin = 0, pos = 0;
    for (int q = lane; q < npx; q += 32) {
      const int row = q / ww;
      const int xx = x0 + (q - row * ww), yy = y0 + row;
      const float v = __ldg(img + static_cast<int64_t>(yy) * W + xx);
      if (!isfinite(v)) continue;
      ++fin;
      const float wv = fmaxf(__fsub_rn(v, bg32), 0.0f);
      pos += wv > 0.0f;
      f.add(wv);
      sx.add_prod(static_cast<float>(xx), wv);
      sy.add_prod(static_cast<float>(yy), wv);
    }
    ff_warp_sum(f);
    ff_warp_sum(sx);
    ff_warp_sum(sy);
    fin = __reduce_add_sync(0xffffffffu, fin);
    pos = __reduce_add_sync(0xffffffffu, pos);
    StarRec rec{};
    rec.valid = (fin > 0 && f.hi > 0.0f) ? 1 : 0;
    if (rec.valid && lane == 0) {
      // second moments, snr and sharpness: of the selected stars only (star_moments_kernel)
      rec.x = ff_quotient_f64(sx, f);
      rec.y = ff_quotient_f64(sy, f);
      rec.flux = static_cast<double>(f.hi) + static_cast<double>(f.lo);
      const float center = __ldg(img + static_cast<int64_t>(y) * W + x);
      rec.peak = fmax(static_cast<double>(center) - bg, 0.0);
      rec.npix = pos;
    }
    if (lane == 0) {
      recs[c] = rec;
      keys[c] = flux_key(rec.flux);
    }
  }
}

// Priority: higher flux first, then lower raster index (stable sort order).
__device__ __forceinline__ bool higher_priority(double fj, unsigned rj, double fi, unsigned ri) {
  return fj > fi || (fj == fi && rj < ri);
}

// The brighter neighbours of candidate i, in the rows that can hold one: a
// centroid stays within the window of its peak, so a conflict lies within
// `reach` rows and columns.
struct NeighbourRows {
  unsigned lo, hi;
  int px, reach;
  __device__ __forceinline__ NeighbourRows(const CatalogArgs& a, const unsigned* first, unsigned raster) {
    const double sep = fmin(ceil(a.min_sep), static_cast<double>(a.width) + a.height);
    reach = static_cast<int>(sep) + 2 * a.radius;
    const int py = static_cast<int>(raster / static_cast<unsigned>(a.width));
    px = static_cast<int>(raster % static_cast<unsigned>(a.width));
    lo = first[static_cast<unsigned>(max(1, py - reach) - 1) * a.chunks_per_row];
    hi = first[static_cast<unsigned>(min(a.height - 2, py + reach)) * a.chunks_per_row];
  }
};

__device__ __forceinline__ bool brighter_conflict(const CatalogArgs& a, const StarRec* recs, unsigned j, unsigned cj,
                                                  const StarRec& ri, unsigned ci) {
  const StarRec& rj = recs[j];
  if (!rj.valid || !higher_priority(rj.flux, cj, ri.flux, ci)) return false;
  const double dx = ri.x - rj.x, dy = ri.y - rj.y;
  return dx * dx + dy * dy < a.min_sep * a.min_sep;
}

// One warp per candidate: the list of its brighter conflicting neighbours, the
// only thing the de-duplication needs to know about positions.  A list that
// does not fit is marked and searched again when the star is decided.
constexpr int kConflicts = 8;
constexpr unsigned char kConflictsMany = kConflicts + 1;
constexpr unsigned char kConflictsDropped = 255;  // no measurable star

__global__ void __launch_bounds__(256) star_conflict_kernel(CatalogArgs a) {
  const int k = blockIdx.y;
  const int n = static_cast<int>(min(a.state[k].candidates, static_cast<unsigned>(kMaxCandidates)));
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const unsigned* cand = a.cand + static_cast<int64_t>(k) * kMaxCandidates;
  const unsigned* first = a.chunk_first + static_cast<int64_t>(k) * a.chunk_stride;
  const StarRec* recs = a.recs + static_cast<int64_t>(k) * kMaxCandidates;
  unsigned char* count = a.conflict_count + static_cast<int64_t>(k) * kMaxCandidates;
  unsigned short* list = a.conflicts + static_cast<int64_t>(k) * kMaxCandidates * kConflicts;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += nwarps) {
    const StarRec ri = recs[i];
    unsigned found = 0;
    if (ri.valid && a.min_sep > 0.0) {
      const unsigned ci = cand[i];
      const NeighbourRows rows(a, first, ci);
      for (unsigned base = rows.lo; base < rows.hi; base += 32) {
        const unsigned j = base + lane;
        bool conflict = false;
        if (j < rows.hi && j != static_cast<unsigned>(i)) {
          const unsigned cj = cand[j];
          conflict = abs(static_cast<int>(cj % static_cast<unsigned>(a.width)) - rows.px) <= rows.reach &&
                     brighter_conflict(a, recs, j, cj, ri, ci);
        }
        const unsigned mask = __ballot_sync(0xffffffffu, conflict);
        const unsigned pos = found + __popc(mask & ((1u << lane) - 1u));
        if (conflict && pos < kConflicts) list[i * kConflicts + pos] = static_cast<unsigned short>(j);
        found += __popc(mask);
      }
    }
    if (lane == 0)
      count[i] = ri.valid ? static_cast<unsigned char>(min(found, static_cast<unsigned>(kConflictsMany)))
                          : kConflictsDropped;
  }
}

// A selected star: priority (flux key, then raster), candidate, output place.
struct SelectedStar {
  unsigned long long key;
  unsigned raster;
  int idx;
  int rank;
  int pad;
};

// One CTA per frame: flux-ordered greedy de-duplication in rounds over the
// conflict lists (a star is kept when no brighter neighbour can be, dropped
// when one is), then the max_stars-th largest kept flux by a radix select; the
// selected stars are handed on in any order, star_rank_kernel finds their
// places.  Bound by the latency of its rounds: 29 us for 8 frames with 13,000
// candidates (the lists 37 us), 277 us with the neighbour search in the rounds and a sort of the
// result.
constexpr int kSelectThreads = 1024;

__global__ void __launch_bounds__(kSelectThreads) star_select_kernel(CatalogArgs a) {
  enum : unsigned char { kDropped = 0, kKept = 1, kOpen = 2 };
  __shared__ unsigned char states[kMaxCandidates];
  __shared__ unsigned long long s_min, s_max, s_prefix;
  __shared__ unsigned s_hist[256];
  __shared__ int s_count, s_rank, s_n;
  volatile unsigned char* state = states;
  const int k = blockIdx.x;
  StarFrameState& st = a.state[k];
  const int n = static_cast<int>(min(st.candidates, static_cast<unsigned>(kMaxCandidates)));
  const unsigned* cand = a.cand + static_cast<int64_t>(k) * kMaxCandidates;
  const unsigned* first = a.chunk_first + static_cast<int64_t>(k) * a.chunk_stride;
  const StarRec* recs = a.recs + static_cast<int64_t>(k) * kMaxCandidates;
  const unsigned long long* keys = a.keys + static_cast<int64_t>(k) * kMaxCandidates;
  const unsigned char* count = a.conflict_count + static_cast<int64_t>(k) * kMaxCandidates;
  const unsigned short* list = a.conflicts + static_cast<int64_t>(k) * kMaxCandidates * kConflicts;
  // 1) stars without a brighter neighbour are kept, invalid ones drop out
  if (threadIdx.x == 0) {
    s_min = ~0ull;
    s_max = 0ull;
    s_count = s_n = 0;
  }
  bool open = false;
  for (int i = threadIdx.x; i < n; i += kSelectThreads) {
    const unsigned char c = count[i];
    state[i] = c == kConflictsDropped ? kDropped : (c == 0 ? kKept : kOpen);
    open |= c != kConflictsDropped && c != 0;
  }
  // 2) rounds: the brightest open star is decided in each, so they end
  while (__syncthreads_or(open)) {
    open = false;
    for (int i = threadIdx.x; i < n; i += kSelectThreads) {
      if (state[i] != kOpen) continue;
      unsigned char verdict = kKept;
      const int c = count[i];
      if (c != kConflictsMany) {
        for (int q = 0; q < c; ++q) {
          const unsigned char sj = state[list[i * kConflicts + q]];
          if (sj == kKept) {
            verdict = kDropped;
            break;
          }
          if (sj == kOpen) verdict = kOpen;
        }
      } else {
        const StarRec ri = recs[i];
        const unsigned ci = cand[i];
        const NeighbourRows rows(a, first, ci);
        for (unsigned j = rows.lo; j < rows.hi; ++j) {
          const unsigned char sj = state[j];
          if (sj == kDropped || j == static_cast<unsigned>(i)) continue;
          const unsigned cj = cand[j];
          if (abs(static_cast<int>(cj % static_cast<unsigned>(a.width)) - rows.px) > rows.reach) continue;
          if (!brighter_conflict(a, recs, j, cj, ri, ci)) continue;
          if (sj == kKept) {
            verdict = kDropped;
            break;
          }
          verdict = kOpen;
        }
      }
      if (verdict == kOpen) open = true;
      else state[i] = verdict;
    }
  }
  // 3) the max_stars-th largest kept flux: radix select (8-bit digits, most
  //    significant first, from the first digit in which the keys differ) of
  //    rank total_kept - take in ascending key order
  {
    int c = 0;
    unsigned long long lo = ~0ull, hi = 0ull;
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += kSelectThreads)
      if (state[i] == kKept) {
        const unsigned long long key = keys[i];
        lo = min(lo, key);
        hi = max(hi, key);
        ++c;
      }
    for (int off = 16; off > 0; off >>= 1) {
      lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, off));
      hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, off));
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0 && c) {
      atomicMin(&s_min, lo);
      atomicMax(&s_max, hi);
      atomicAdd(&s_count, c);
    }
  }
  __syncthreads();
  const int total_kept = s_count;
  const int take = min(total_kept, a.max_stars);
  unsigned long long t = 0;  // keep fluxes with key > t, plus ties at t
  if (take < total_kept) {
    const unsigned long long diff = s_min ^ s_max;
    int shift = diff ? (63 - __clzll(static_cast<long long>(diff))) / 8 * 8 : -8;
    unsigned long long mask = shift + 8 >= 64 ? 0ull : ~0ull << (shift + 8);
    unsigned long long prefix = s_max & mask;
    int rank = total_kept - take;
    for (; shift >= 0; shift -= 8) {
      for (int i = threadIdx.x; i < 256; i += kSelectThreads) s_hist[i] = 0u;
      __syncthreads();
#pragma unroll 4
      for (int i = threadIdx.x; i < n; i += kSelectThreads) {
        if (state[i] != kKept) continue;
        const unsigned long long key = keys[i];
        if ((key & mask) == prefix) atomicAdd(&s_hist[(key >> shift) & 255u], 1u);
      }
      __syncthreads();
      if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        unsigned loc = 0;
        for (int b = 0; b < 8; ++b) loc += s_hist[lane * 8 + b];
        unsigned incl = loc;
        for (int off = 1; off < 32; off <<= 1) {
          const unsigned v = __shfl_up_sync(0xffffffffu, incl, off);
          if (lane >= off) incl += v;
        }
        const unsigned excl = incl - loc;
        if (excl <= static_cast<unsigned>(rank) && static_cast<unsigned>(rank) < incl) {
          unsigned r = static_cast<unsigned>(rank) - excl;
          int b = lane * 8;
          while (r >= s_hist[b]) {
            r -= s_hist[b];
            ++b;
          }
          s_prefix = prefix | (static_cast<unsigned long long>(b) << shift);
          s_rank = static_cast<int>(r);
        }
      }
      __syncthreads();
      prefix = s_prefix;
      rank = s_rank;
      mask |= 0xffull << shift;
      __syncthreads();
    }
    t = prefix;
  }
  // 4) the selected stars: key > t and all ties key == t; the first `take` by
  //    priority are the answer (ties at t come out in raster order)
  SelectedStar* sel = a.selected + static_cast<int64_t>(k) * kMaxSelected;
  for (int i = threadIdx.x; i < n; i += kSelectThreads) {
    if (state[i] == kKept && keys[i] >= t) {
      const int p = atomicAdd(&s_n, 1);
      if (p < kMaxSelected) sel[p] = {keys[i], cand[i], i, 0, 0};
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    st.selected = min(s_n, kMaxSelected);
    st.kept = min(take, st.selected);
  }
}

// Registration catalog of each frame: the first kCatalogPoints output stars
// (brightest first, cpu/registration.py:37-39) that pass the optional shape
// filter.  One warp per frame, order-preserving ballot compaction.
__global__ void star_catalog_kernel(CatalogArgs a, float min_fwhm, float max_ecc) {
  const int k = blockIdx.x;
  const int lane = threadIdx.x;
  const int nout = a.state[k].kept;
  const gg_star_t* out = a.out + static_cast<int64_t>(k) * a.max_stars;
  const int frame = a.frames[k];
  double* dst = a.cat_xy + static_cast<int64_t>(frame) * kCatalogPoints * 2;
  const bool test_fwhm = min_fwhm > 0.0f, test_ecc = max_ecc < 1.0f;
  int taken = 0;
  for (int base = 0; base < nout && taken < kCatalogPoints; base += 32) {
    const int i = base + lane;
    bool pass = false;
    double x = 0.0, y = 0.0;
    if (i < nout) {
      const gg_star_t s = out[i];
      pass = (!test_fwhm || s.fwhm >= static_cast<double>(min_fwhm)) &&
             (!test_ecc || s.eccentricity <= static_cast<double>(max_ecc));
      x = s.x;
      y = s.y;
    }
    const unsigned mask = __ballot_sync(0xffffffffu, pass);
    const int pos = taken + __popc(mask & ((1u << lane) - 1u));
    if (pass && pos < kCatalogPoints) {
      dst[2 * pos] = x;
      dst[2 * pos + 1] = y;
    }
    taken += __popc(mask);
  }
  if (lane == 0) a.cat_n[frame] = min(taken, kCatalogPoints);
}

// The output place of every selected star: how many come before it.  A CTA
// keeps the frame's keys in shared memory; four threads share a star's count.
constexpr int kRankThreads = 512;

__global__ void __launch_bounds__(kRankThreads) star_rank_kernel(CatalogArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned long long* keys = reinterpret_cast<unsigned long long*>(smem);  // [kMaxSelected]
  unsigned* raster = reinterpret_cast<unsigned*>(keys + kMaxSelected);     // [kMaxSelected]
  const int k = blockIdx.y;
  const int nsel = a.state[k].selected;
  const int i = static_cast<int>(blockIdx.x) * (kRankThreads / 4) + static_cast<int>(threadIdx.x >> 2);
  if (static_cast<int>(blockIdx.x) * (kRankThreads / 4) >= nsel) return;
  SelectedStar* sel = a.selected + static_cast<int64_t>(k) * kMaxSelected;
  for (int j = threadIdx.x; j < nsel; j += kRankThreads) {
    keys[j] = sel[j].key;
    raster[j] = sel[j].raster;
  }
  __syncthreads();
  int before = 0;
  if (i < nsel) {
    const unsigned long long key = keys[i];
    const unsigned own = raster[i];
#pragma unroll 8
    for (int j = threadIdx.x & 3; j < nsel; j += 4)
      before += (keys[j] > key || (keys[j] == key && raster[j] < own)) ? 1 : 0;
  }
  before += __shfl_xor_sync(0xffffffffu, before, 1);
  before += __shfl_xor_sync(0xffffffffu, before, 2);
  if (i < nsel && (threadIdx.x & 3) == 0) sel[i].rank = before;
}

// The output records: second moments of the selected stars (star_detect.py:83-99: intensity weighted about the centroid, fwhm from the
// mean of the principal variances, eccentricity from their ratio).  Bound by
// float64 operations, which a warp pays for whatever its active lanes, so:
// a lane per column of the window (3 stars of 9 columns in a warp), which
// needs only the column's sums of w, w dy and w dy^2; and after `rounds` such
// groups a lane per star adds up its columns and takes the quotients and roots.
// 45 us and the ranks 45 us for 8 x 2048 stars of radius 4, 150 us with a warp per
// star (and a sort of the selection).
constexpr int kMomentWarps = 4;
constexpr int kMomentRounds = 10;

__global__ void __launch_bounds__(32 * kMomentWarps) star_moments_kernel(CatalogArgs a, int rounds) {
  __shared__ double s_part[kMomentWarps][kMomentRounds][3][32];
  __shared__ __align__(16) double2 s_rows[kMomentWarps][33];  // (dy, dy^2) of each star's rows
  const int k = blockIdx.y;
  const StarFrameState& st = a.state[k];
  const int nsel = st.selected, nout = st.kept;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float* img = a.slots + static_cast<int64_t>(a.slot_of_frame[a.frames[k]]) * a.stride;
  const StarRec* recs = a.recs + static_cast<int64_t>(k) * kMaxCandidates;
  const SelectedStar* sel = a.selected + static_cast<int64_t>(k) * kMaxSelected;
  gg_star_t* out = a.out + static_cast<int64_t>(k) * a.max_stars;
  const int W = a.width, H = a.height, r = a.radius;
  const int side = 2 * r + 1;  // at most 33
  const int group = max(1, 32 / side);
  const int g = lane / side, col0 = lane - g * side;
  const int batch = group * rounds;  // stars of a warp, at most 32
  for (int first = (blockIdx.x * kMomentWarps + warp) * batch; first < nsel;
       first += gridDim.x * kMomentWarps * batch) {
    for (int round = 0; round < rounds; ++round) {
      const int i = first + round * group + g;
      double sxx = 0.0, syy = 0.0, sxy = 0.0, bx = 0.0;
      int ww = 0, hh = 0;
      float bg = 0.0f;
      const float* win = img;
      __syncwarp();
      if (g < group && i < nsel) {
        const SelectedStar s = sel[i];
        const int x = static_cast<int>(s.raster % static_cast<unsigned>(W));
        const int y = static_cast<int>(s.raster / static_cast<unsigned>(W));
        bg = st.background_f32;
        if (a.mesh.bg) {
          double mesh_bg, noise;
          mesh_at(a.mesh, k, x, y, mesh_bg, noise);
          bg = __double2float_rn(mesh_bg);
        }
        const int x0 = max(0, x - r), y0 = max(0, y - r);
        ww = min(W, x + r + 1) - x0;
        hh = min(H, y + r + 1) - y0;
        win = img + static_cast<int64_t>(y0) * W + x0;
        // differences of a centroid and a pixel near it are exact
        bx = static_cast<double>(x0) - recs[s.idx].x;
        const double by = static_cast<double>(y0) - recs[s.idx].y;
        for (int row = col0; row < side; row += 32) {
          const double dy = by + static_cast<double>(row);
          s_rows[warp][g * side + row] = make_double2(dy, dy * dy);
        }
      }
      __syncwarp();
      for (int col = col0; col < side; col += 32) {  // one trip but for radius 16
        double c0 = 0.0, c1 = 0.0, c2 = 0.0;
#pragma unroll 9  // all loads of a radius-4 window in flight
        for (int row = 0; row < side; ++row) {
          float w = 0.0f;
          if (row < hh && col < ww) {
            const float v = __ldg(win + static_cast<int64_t>(row) * W + col);
            w = isfinite(v) ? fmaxf(__fsub_rn(v, bg), 0.0f) : 0.0f;
          }
          const double wd = static_cast<double>(w);
          const double2 dy = s_rows[warp][min(g, group - 1) * side + row];
          c0 += wd;
          c1 += dy.x * wd;
          c2 += dy.y * wd;
        }
        if (col < ww) {
          const double dx = bx + static_cast<double>(col);
          sxx += dx * dx * c0;
          sxy += dx * c1;
          syy += c2;
        }
      }
      s_part[warp][round][0][lane] = sxx;
      s_part[warp][round][1][lane] = sxy;
      s_part[warp][round][2][lane] = syy;
    }
    __syncwarp();
    const int mine = first + lane;
    if (lane >= batch || mine >= nsel) continue;
    const SelectedStar s = sel[mine];
    if (s.rank >= nout) continue;  // ties at the last place beyond max_stars
    double mxx = 0.0, myy = 0.0, mxy = 0.0;
    const int round = lane / group, lane0 = (lane - round * group) * side;
    for (int c = 0; c < min(side, 32); ++c) {
      mxx += s_part[warp][round][0][lane0 + c];
      mxy += s_part[warp][round][1][lane0 + c];
      myy += s_part[warp][round][2][lane0 + c];
    }
    const StarRec rec = recs[s.idx];
    mxx /= rec.flux;
    myy /= rec.flux;
    mxy /= rec.flux;
    const double trace = fmax(mxx + myy, 0.0);
    const double det = fmax((mxx - myy) * (mxx - myy) + 4.0 * mxy * mxy, 0.0);
    const double root = sqrt(det);
    const double major = fmax((trace + root) / 2.0, 0.0);
    const double minor = fmax((trace - root) / 2.0, 0.0);
    const double mean_sigma = sqrt(fmax((major + minor) / 2.0, 0.0));
    double noise = st.noise;
    if (a.mesh.bg) {
      double bg_unused;
      mesh_at(a.mesh, k, static_cast<int>(s.raster % static_cast<unsigned>(W)),
              static_cast<int>(s.raster / static_cast<unsigned>(W)), bg_unused, noise);
    }
    gg_star_t o;
    o.x = rec.x;
    o.y = rec.y;
    o.flux = rec.flux;
    o.peak = rec.peak;
    o.fwhm = mean_sigma > 0.0 ? 2.354820045 * mean_sigma : nan("");
    o.eccentricity = major > 0.0 ? sqrt(fmax(0.0, 1.0 - minor / major)) : nan("");
    o.snr = rec.flux / fmax(noise * sqrt(static_cast<double>(max(rec.npix, 1))), 1.0e-6);
    o.sharpness = rec.peak / fmax(rec.flux, 1.0e-6);
    o.npix = rec.npix;
    o.pad = 0;
    out[s.rank] = o;
  }
}

// ---- np.std of the finite pixels, bit-exact (fallback noise, MAD == 0) -----
// NumPy sums a contiguous float32 array pairwise: blocks of <= 128 use eight
// interleaved accumulators, longer runs split at n/2 rounded down to a
// multiple of 8 (verified against np.sum).  np.std(finite) is
// sqrt(pairwise((x - m)^2) / n) with m = pairwise(x) / n, all float32.  The
// finite pixels form a compacted sequence; a per-1024-pixel finite-count
// prefix maps a compacted index back to raster order.  One CTA walks the
// frames of the batch in turn and only works on frames whose MAD is zero.
constexpr int kPwBlock = 1024;

struct PwArgs {
  const float* slots;
  const int* slot_of_frame;
  int64_t stride;
  int64_t pixels;
  const int* frames;
  int count;
  StarFrameState* state;
  double* rms;     // [count]
  int* prefix;     // [pixels / kPwBlock + 2]
  int2* leaves;    // [pixels / 64 + 2]
  float* leaf_sum; // [pixels / 64 + 2]
};

// Position of the `c`-th finite pixel (compacted index) in raster order.
__device__ int64_t finite_position(const float* src, const int* prefix, int nblocks, int64_t pixels, int64_t c,
                                   bool dense) {
  if (dense) return c;
  int lo = 0, hi = nblocks;  // last block with prefix <= c
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (prefix[mid] <= c) lo = mid; else hi = mid;
  }
  int64_t p = static_cast<int64_t>(lo) * kPwBlock;
  int64_t seen = prefix[lo];
  for (; p < pixels; ++p) {
    if (isfinite(src[p])) {
      if (seen == c) return p;
      ++seen;
    }
  }
  return pixels;
}

__device__ float pw_leaf(const float* src, const int* prefix, int nblocks, int64_t pixels, bool dense, int64_t off,
                         int len, bool square, float mean) {
  int64_t p = finite_position(src, prefix, nblocks, pixels, off, dense);
  auto next = [&]() -> float {
    while (!isfinite(src[p])) ++p;
    float v = src[p++];
    if (square) {
      const float d = __fsub_rn(v, mean);
      v = __fmul_rn(d, d);
    }
    return v;
  };
  if (len < 8) {
    float r = 0.0f;
    for (int i = 0; i < len; ++i) r = __fadd_rn(r, next());
    return r;
  }
  float r[8];
  for (int j = 0; j < 8; ++j) r[j] = next();
  int i = 8;
  for (; i < len - (len % 8); i += 8)
    for (int j = 0; j < 8; ++j) r[j] = __fadd_rn(r[j], next());
  float res = __fadd_rn(__fadd_rn(__fadd_rn(r[0], r[1]), __fadd_rn(r[2], r[3])),
                        __fadd_rn(__fadd_rn(r[4], r[5]), __fadd_rn(r[6], r[7])));
  for (; i < len; ++i) res = __fadd_rn(res, next());
  return res;
}

__device__ __forceinline__ int64_t pw_split(int64_t n) {
  int64_t n2 = n / 2;
  return n2 - n2 % 8;
}

// Thread 0: leaves of the pairwise tree in left-to-right order.
__device__ int pw_leaves(int64_t n, int2* leaves) {
  int64_t st_off[96], st_n[96];
  int top = 0, count = 0;
  st_off[0] = 0;
  st_n[0] = n;
  top = 1;
  while (top > 0) {
    --top;
    const int64_t off = st_off[top], m = st_n[top];
    if (m <= 128) {
      leaves[count++] = make_int2(static_cast<int>(off), static_cast<int>(m));
    } else {
      const int64_t m2 = pw_split(m);
      st_off[top] = off + m2;
      st_n[top] = m - m2;
      ++top;
      st_off[top] = off;
      st_n[top] = m2;
      ++top;
    }
  }
  return count;
}

// Thread 0: fold the leaf sums in the tree's order (left + right at each node).
__device__ float pw_fold(int64_t n, const float* leaf_sum) {
  int64_t node_n[96];
  int node_state[96];
  float vals[96];
  int top = 1, vtop = 0, next = 0;
  node_n[0] = n;
  node_state[0] = 0;
  while (top > 0) {
    const int64_t m = node_n[top - 1];
    if (m <= 128) {
      --top;
      vals[vtop++] = leaf_sum[next++];
    } else if (node_state[top - 1] == 0) {
      node_state[top - 1] = 1;
      const int64_t m2 = pw_split(m);
      node_n[top] = m - m2;
      node_state[top] = 0;
      ++top;
      node_n[top] = m2;
      node_state[top] = 0;
      ++top;
    } else {
      --top;
      const float b = vals[--vtop];
      const float a = vals[--vtop];
      vals[vtop++] = __fadd_rn(a, b);
    }
  }
  return vals[0];
}

__global__ void __launch_bounds__(1024) pairwise_std_kernel(PwArgs a) {
  __shared__ int s_leaves;
  __shared__ float s_mean;
  const int nblocks = static_cast<int>((a.pixels + kPwBlock - 1) / kPwBlock);
  bool wanted = false;
  for (int k = threadIdx.x; k < a.count; k += blockDim.x)
    wanted |= a.state[k].count != 0 && 1.4826 * static_cast<double>(a.state[k].mad) <= 0.0;
  if (!__syncthreads_or(wanted)) return;
  for (int k = 0; k < a.count; ++k) {
    const StarFrameState& st = a.state[k];
    if (st.count == 0 || !(1.4826 * static_cast<double>(st.mad) <= 0.0)) continue;  // uniform branch
    const float* src = a.slots + static_cast<int64_t>(a.slot_of_frame[a.frames[k]]) * a.stride;
    const bool dense = static_cast<int64_t>(st.count) == a.pixels;
    if (!dense) {
      // finite counts per block, then an exclusive prefix (thread 0)
      for (int b = threadIdx.x; b < nblocks; b += blockDim.x) {
        int c = 0;
        const int64_t p1 = min(a.pixels, static_cast<int64_t>(b + 1) * kPwBlock);
        for (int64_t p = static_cast<int64_t>(b) * kPwBlock; p < p1; ++p) c += isfinite(src[p]) ? 1 : 0;
        a.prefix[b + 1] = c;
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        a.prefix[0] = 0;
        for (int b = 1; b <= nblocks; ++b) a.prefix[b] += a.prefix[b - 1];
      }
    }
    const int64_t n = st.count;
    if (threadIdx.x == 0) s_leaves = pw_leaves(n, a.leaves);
    __syncthreads();
    const int L = s_leaves;
    for (int pass = 0; pass < 2; ++pass) {
      const float mean = pass ? s_mean : 0.0f;
      for (int l = threadIdx.x; l < L; l += blockDim.x) {
        const int2 lf = a.leaves[l];
        a.leaf_sum[l] = pw_leaf(src, a.prefix, nblocks, a.pixels, dense, lf.x, lf.y, pass == 1, mean);
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        const float total = pw_fold(n, a.leaf_sum);
        const float fn = static_cast<float>(n);
        if (pass == 0) {
          s_mean = __fdiv_rn(total, fn);
        } else {
          a.rms[k] = static_cast<double>(__fsqrt_rn(__fdiv_rn(total, fn)));
        }
      }
      __syncthreads();
    }
  }
}

// ---- host side -------------------------------------------------------------------
void ensure_catalog_storage(gg_stack* s) {
  if (s->d_cat_xy) return;
  check_cuda(cudaMalloc(&s->d_cat_xy, sizeof(double) * 2 * kCatalogPoints * s->frames), "cudaMalloc(catalogs)");
  check_cuda(cudaMalloc(&s->d_cat_n, sizeof(int) * s->frames), "cudaMalloc(catalog counts)");
  check_cuda(cudaMemsetAsync(s->d_cat_n, 0, sizeof(int) * s->frames, s->stream), "cudaMemsetAsync(catalogs)");
  s->bytes_allocated += static_cast<int64_t>(sizeof(double) * 2 * kCatalogPoints * s->frames + sizeof(int) * s->frames);
}

struct StarScratch {
  StarFrameState* state = nullptr;
  unsigned* hist = nullptr;
  unsigned* raw = nullptr;
  unsigned* chunks = nullptr;
  unsigned* chunk_first = nullptr;
  unsigned* cand = nullptr;
  StarRec* recs = nullptr;
  unsigned long long* keys = nullptr;
  unsigned char* conflict_count = nullptr;
  unsigned short* conflicts = nullptr;
  SelectedStar* selected = nullptr;
  gg_star_t* out = nullptr;
  int* frames = nullptr;
  double* rms = nullptr;
  int* pw_prefix = nullptr;
  int2* pw_leaves = nullptr;
  float* pw_sums = nullptr;
  int64_t pw_pixels = 0;
  int capacity_frames = 0;
  int max_stars = 0;
  double* mesh_bg = nullptr;  // [frames][cells]
  double* mesh_nz = nullptr;
  int64_t mesh_cap = 0;       // doubles per array
  unsigned* band = nullptr;   // sample-bracket key buffers
  int64_t band_elems = 0;
};

static void free_star_scratch(StarScratch& s) {
  void* ps[] = {s.state, s.hist,   s.raw, s.chunks,    s.chunk_first, s.cand,    s.recs,    s.keys, s.conflict_count,
                s.conflicts, s.selected, s.out, s.frames, s.rms, s.pw_prefix, s.pw_leaves, s.pw_sums, s.mesh_bg,
                s.mesh_nz,   s.band};
  for (void* p : ps)
    if (p) cudaFree(p);
  s = StarScratch{};
}

static void ensure_star_scratch(StarScratch& s, int frames, int max_stars, unsigned chunk_stride) {
  if (s.capacity_frames >= frames && s.max_stars >= max_stars) return;
  free_star_scratch(s);
  const size_t f = static_cast<size_t>(frames);
  check_cuda(cudaMalloc(&s.state, sizeof(StarFrameState) * f), "cudaMalloc(star state)");
  check_cuda(cudaMalloc(&s.hist, sizeof(unsigned) * f * 2 * kSelBins), "cudaMalloc(star hist)");
  check_cuda(cudaMalloc(&s.raw, sizeof(unsigned) * f * kMaxCandidates), "cudaMalloc(star candidates)");
  check_cuda(cudaMalloc(&s.chunks, sizeof(unsigned) * f * chunk_stride), "cudaMalloc(star chunks)");
  check_cuda(cudaMalloc(&s.chunk_first, sizeof(unsigned) * f * chunk_stride), "cudaMalloc(star chunks)");
  check_cuda(cudaMalloc(&s.cand, sizeof(unsigned) * f * kMaxCandidates), "cudaMalloc(star candidates)");
  check_cuda(cudaMalloc(&s.recs, sizeof(StarRec) * f * kMaxCandidates), "cudaMalloc(star records)");
  check_cuda(cudaMalloc(&s.keys, sizeof(unsigned long long) * f * kMaxCandidates), "cudaMalloc(star keys)");
  check_cuda(cudaMalloc(&s.conflict_count, f * kMaxCandidates), "cudaMalloc(star conflicts)");
  check_cuda(cudaMalloc(&s.conflicts, sizeof(unsigned short) * f * kMaxCandidates * kConflicts),
             "cudaMalloc(star conflicts)");
  check_cuda(cudaMalloc(&s.selected, sizeof(SelectedStar) * f * kMaxSelected), "cudaMalloc(star selection)");
  check_cuda(cudaMalloc(&s.out, sizeof(gg_star_t) * f * static_cast<size_t>(max_stars)), "cudaMalloc(star out)");
  check_cuda(cudaMalloc(&s.frames, sizeof(int) * f), "cudaMalloc(star frames)");
  check_cuda(cudaMalloc(&s.rms, sizeof(double) * f), "cudaMalloc(star rms)");
  s.capacity_frames = frames;
  s.max_stars = max_stars;
}

// Scratch lives with the stack (freed by gg_stack_destroy through the hook).
static StarScratch& star_scratch(gg_stack* s) {
  if (!s->star_scratch) {
    s->star_scratch = new StarScratch();
    s->star_scratch_free = [](void* p) {
      auto* sc = static_cast<StarScratch*>(p);
      free_star_scratch(*sc);
      delete sc;
    };
  }
  return *static_cast<StarScratch*>(s->star_scratch);
}

__global__ void star_rms_kernel(const double* partials, int blocks, int count, double* rms) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count) return;
  double s1 = 0.0, s2 = 0.0, n = 0.0;
  for (int b = 0; b < blocks; ++b) {
    const double* q = partials + (static_cast<int64_t>(k) * blocks + b) * 3;
    s1 += q[0];
    s2 += q[1];
    n += q[2];
  }
  const double mean = n > 0 ? s1 / n : 0.0;
  const double var = n > 0 ? fmax(s2 / n - mean * mean, 0.0) : 0.0;
  rms[k] = sqrt(var);
}

void launch_frame_stats_partials(gg_stack* s, const int* d_frames, int count, int blocks, double* partials);

void detect_stars(gg_stack* s, const int64_t* indices, int count, const gg_star_params_t& p) {
  StarScratch& sc = star_scratch(s);
  // chunks of the candidate search: a row's from the 16-byte boundary before it
  const unsigned chunks_per_row = static_cast<unsigned>((s->width + 3 + kChunk - 1) / kChunk);
  const unsigned chunk_count = chunks_per_row * static_cast<unsigned>(std::max<int64_t>(0, s->height - 2));
  const unsigned chunk_stride = (chunk_count + 1 + 3) / 4 * 4;
  ensure_star_scratch(sc, count, p.max_stars, chunk_stride);
  std::vector<int> frames(static_cast<size_t>(count));
  for (int k = 0; k < count; ++k) frames[static_cast<size_t>(k)] = static_cast<int>(indices[k]);
  upload_params(s->stream, sc.frames, frames.data(), sizeof(int) * count, "cudaMemcpyAsync(star frames)");
  check_cuda(cudaMemsetAsync(sc.state, 0, sizeof(StarFrameState) * count, s->stream), "cudaMemsetAsync(state)");
  const bool need_stats = !std::isfinite(p.background) || !std::isfinite(p.noise);
  SelectArgs sa{};
  sa.slots = s->d_slots;
  sa.slot_of_frame = s->d_slot_of_frame;
  sa.stride = s->stride;
  sa.pixels = s->pixels;
  sa.frames = sc.frames;
  sa.state = sc.state;
  sa.hist = sc.hist;
  const unsigned per_frame =
      std::max(1u, std::min<unsigned>(static_cast<unsigned>((s->pixels + 255) / 256),
                                      std::max(1u, static_cast<unsigned>(sm_count() * 8 / std::max(count, 1)))));
  double* rms = nullptr;
  if (need_stats) {
    // band buffers of the sample-bracket selection: a sixteenth of the frame
    // (the band holds ~2.5 % of a 9600 x 6422 frame's pixels)
    const int64_t band_cap =
        (std::min<int64_t>(s->pixels, std::max<int64_t>(65536, s->pixels / 16)) + 3) / 4 * 4;
    if (sc.band_elems < band_cap * count) {
      if (sc.band) cudaFree(sc.band);
      sc.band = nullptr;
      sc.band_elems = 0;
      check_cuda(cudaMalloc(&sc.band, sizeof(unsigned) * band_cap * count), "cudaMalloc(bracket band)");
      sc.band_elems = band_cap * count;
    }
    BracketArgs ba{s->d_slots, s->d_slot_of_frame, s->stride, s->pixels, sc.frames, sc.state, sc.band, band_cap, 0};
    const unsigned frames_y = static_cast<unsigned>(count);
    const unsigned sample_ctas = static_cast<unsigned>(
        std::max<int64_t>(1, std::min<int64_t>(kSampleCtas, (s->pixels + 4 * kSampleThreads - 1) / (4 * kSampleThreads))));
    check_cuda(cudaMemsetAsync(sc.hist, 0, sizeof(unsigned) * count * 2 * kSelBins, s->stream),
               "cudaMemsetAsync(hist)");
    for (int mode = 0; mode < 2; ++mode) {
      sa.mode = mode;
      ba.mode = mode;
      note_launch(3);
      bracket_sample_kernel<<<dim3(sample_ctas, frames_y), kSampleThreads, 0, s->stream>>>(ba);
      if (mode == 0)
        bracket_pass_kernel<0><<<dim3(per_frame, frames_y), kBracketThreads, 0, s->stream>>>(ba);
      else
        bracket_pass_kernel<1><<<dim3(per_frame, frames_y), kBracketThreads, 0, s->stream>>>(ba);
      bracket_band_kernel<<<dim3(kBandCtas, frames_y), kBandThreads, 0, s->stream>>>(ba);
      check_cuda(cudaGetLastError(), "bracket select launch");
      // frames the bracket could not settle: three-pass radix select
      note_launch(3);
      const dim3 hist_grid(per_frame, frames_y);
      select_hist_kernel<0><<<hist_grid, 256, 0, s->stream>>>(sa);
      select_hist_kernel<1><<<hist_grid, 256, 0, s->stream>>>(sa);
      select_hist_kernel<2><<<hist_grid, 256, 0, s->stream>>>(sa);
      check_cuda(cudaGetLastError(), "select_hist launch");
    }
    // np.std of the finite pixels, the fallback noise when the MAD is zero
    // (star_detect.py:35-41); computed only for such frames.
    if (sc.pw_pixels != s->pixels) {
      if (sc.pw_prefix) cudaFree(sc.pw_prefix);
      if (sc.pw_leaves) cudaFree(sc.pw_leaves);
      if (sc.pw_sums) cudaFree(sc.pw_sums);
      const size_t nb = static_cast<size_t>(s->pixels / kPwBlock + 2);
      // leaves hold >= 57 elements once n > 128 (split at n/2 rounded down to 8)
      const size_t nl = static_cast<size_t>(s->pixels / 32 + 2);
      check_cuda(cudaMalloc(&sc.pw_prefix, sizeof(int) * nb), "cudaMalloc(pairwise prefix)");
      check_cuda(cudaMalloc(&sc.pw_leaves, sizeof(int2) * nl), "cudaMalloc(pairwise leaves)");
      check_cuda(cudaMalloc(&sc.pw_sums, sizeof(float) * nl), "cudaMalloc(pairwise sums)");
      sc.pw_pixels = s->pixels;
    }
    PwArgs pa{};
    pa.slots = s->d_slots;
    pa.slot_of_frame = s->d_slot_of_frame;
    pa.stride = s->stride;
    pa.pixels = s->pixels;
    pa.frames = sc.frames;
    pa.count = count;
    pa.state = sc.state;
    pa.rms = sc.rms;
    pa.prefix = sc.pw_prefix;
    pa.leaves = sc.pw_leaves;
    pa.leaf_sum = sc.pw_sums;
    rms = sc.rms;
    note_launch();
    pairwise_std_kernel<<<1, 1024, 0, s->stream>>>(pa);
    check_cuda(cudaGetLastError(), "pairwise_std launch");
  }
  note_launch();
  star_threshold_kernel<<<(count + 127) / 128, 128, 0, s->stream>>>(
      sc.state, count, p.threshold_sigma, std::isfinite(p.background) ? 1 : 0, p.background,
      std::isfinite(p.noise) ? 1 : 0, p.noise, rms);
  check_cuda(cudaGetLastError(), "star_threshold launch");
  if (s->width < 3 || s->height < 3) return;  // no interior (star_detect.py:140-141)
  DetectArgs da{};
  da.slots = s->d_slots;
  da.slot_of_frame = s->d_slot_of_frame;
  da.stride = s->stride;
  da.width = static_cast<int>(s->width);
  da.height = static_cast<int>(s->height);
  da.frames = sc.frames;
  da.state = sc.state;
  da.raw = sc.raw;
  da.chunks = sc.chunks;
  da.chunk_stride = chunk_stride;
  da.chunk_count = chunk_count;
  da.chunks_per_row = chunks_per_row;
  da.k_sigma = static_cast<double>(p.threshold_sigma);
  if (p.mesh_cell > 0) {
    MeshArgs ma{};
    ma.cell = p.mesh_cell;
    ma.nx = static_cast<int>((s->width + p.mesh_cell - 1) / p.mesh_cell);
    ma.ny = static_cast<int>((s->height + p.mesh_cell - 1) / p.mesh_cell);
    const int64_t need = static_cast<int64_t>(ma.nx) * ma.ny * count;
    if (sc.mesh_cap < need) {
      if (sc.mesh_bg) cudaFree(sc.mesh_bg);
      if (sc.mesh_nz) cudaFree(sc.mesh_nz);
      sc.mesh_bg = sc.mesh_nz = nullptr;
      sc.mesh_cap = 0;
      check_cuda(cudaMalloc(&sc.mesh_bg, sizeof(double) * need), "cudaMalloc(background mesh)");
      check_cuda(cudaMalloc(&sc.mesh_nz, sizeof(double) * need), "cudaMalloc(noise mesh)");
      sc.mesh_cap = need;
    }
    ma.slots = s->d_slots;
    ma.slot_of_frame = s->d_slot_of_frame;
    ma.stride = s->stride;
    ma.width = static_cast<int>(s->width);
    ma.height = static_cast<int>(s->height);
    ma.frames = sc.frames;
    ma.bg = sc.mesh_bg;
    ma.nz = sc.mesh_nz;
    note_launch();
    mesh_stats_kernel<<<dim3(static_cast<unsigned>(ma.nx * ma.ny), static_cast<unsigned>(count)), 1024, 0,
                        s->stream>>>(ma);
    check_cuda(cudaGetLastError(), "mesh_stats launch");
    da.mesh = MeshView{sc.mesh_bg, sc.mesh_nz, ma.cell, ma.nx, ma.ny};
  }
  note_launch();
  const unsigned frames_y = static_cast<unsigned>(count);
  const unsigned detect_ctas =
      std::min((chunk_count + 7) / 8, static_cast<unsigned>(std::max(1, sm_count() * 8 / std::max(count, 1))));
  if (da.mesh.bg)
    star_detect_kernel<true><<<dim3(detect_ctas, frames_y), 256, 0, s->stream>>>(da);
  else
    star_detect_kernel<false><<<dim3(detect_ctas, frames_y), 256, 0, s->stream>>>(da);
  check_cuda(cudaGetLastError(), "star_detect launch");
  CatalogArgs ca{};
  ca.slots = s->d_slots;
  ca.slot_of_frame = s->d_slot_of_frame;
  ca.stride = s->stride;
  ca.width = da.width;
  ca.height = da.height;
  ca.frames = sc.frames;
  ca.state = sc.state;
  ca.cand = sc.cand;
  ca.recs = sc.recs;
  ca.raw = sc.raw;
  ca.chunks = sc.chunks;
  ca.chunk_first = sc.chunk_first;
  ca.chunk_stride = chunk_stride;
  ca.chunk_count = chunk_count;
  ca.chunks_per_row = chunks_per_row;
  ca.keys = sc.keys;
  ca.conflict_count = sc.conflict_count;
  ca.conflicts = sc.conflicts;
  ca.selected = sc.selected;
  ca.out = sc.out;
  ca.max_stars = p.max_stars;
  ca.radius = std::max(1, p.window_radius);
  ca.min_sep = p.min_separation_px;
  ensure_catalog_storage(s);
  ca.cat_xy = s->d_cat_xy;
  ca.cat_n = s->d_cat_n;
  ca.mesh = da.mesh;
  const unsigned order_ctas = std::min<unsigned>(kOrderCtas, (chunk_count + kOrderTile - 1) / kOrderTile);
  note_launch(6);
  star_order_kernel<<<dim3(order_ctas, frames_y), kOrderThreads, 0, s->stream>>>(ca);
  check_cuda(cudaGetLastError(), "star_order launch");
  star_measure_kernel<<<dim3(64, frames_y), 256, 0, s->stream>>>(ca);
  check_cuda(cudaGetLastError(), "star_measure launch");
  star_conflict_kernel<<<dim3(64, frames_y), 256, 0, s->stream>>>(ca);
  check_cuda(cudaGetLastError(), "star_conflict launch");
  star_select_kernel<<<frames_y, kSelectThreads, 0, s->stream>>>(ca);
  check_cuda(cudaGetLastError(), "star_select launch");
  const size_t rank_smem = (sizeof(unsigned long long) + sizeof(unsigned)) * kMaxSelected;
  check_cuda(cudaFuncSetAttribute(star_rank_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(rank_smem)),
             "cudaFuncSetAttribute(star rank)");
  // ties at the last place may select more stars than come out
  star_rank_kernel<<<dim3(kMaxSelected / (kRankThreads / 4), frames_y), kRankThreads, rank_smem, s->stream>>>(ca);
  check_cuda(cudaGetLastError(), "star_rank launch");
  // one round per warp until every SM has sixteen warps, then more stars per warp
  const int group = std::max(1, 32 / (2 * ca.radius + 1));
  const int64_t groups = (static_cast<int64_t>(p.max_stars) + group - 1) / group * count;
  const int rounds = static_cast<int>(std::max<int64_t>(
      1, std::min<int64_t>(std::min(kMomentRounds, 32 / group), groups / (int64_t{16} * sm_count()))));
  const unsigned mom_ctas =
      static_cast<unsigned>((p.max_stars + kMomentWarps * group * rounds - 1) / (kMomentWarps * group * rounds));
  star_moments_kernel<<<dim3(mom_ctas, frames_y), 32 * kMomentWarps, 0, s->stream>>>(ca, rounds);
  check_cuda(cudaGetLastError(), "star_moments launch");
  note_launch();
  star_catalog_kernel<<<static_cast<unsigned>(count), 32, 0, s->stream>>>(ca, p.catalog_min_fwhm,
                                                                           p.catalog_max_eccentricity);
  check_cuda(cudaGetLastError(), "star_catalog launch");
}

}  // namespace gg

using namespace gg;

extern "C" {

int gg_stack_detect_stars(gg_stack* s, const int64_t* indices, int64_t count, const gg_star_params_t* params,
                          gg_star_t* host_stars, int32_t* host_counts, gg_star_frame_info_t* host_info) {
  GG_API_BEGIN
  require(s != nullptr && indices != nullptr && params != nullptr, "null argument");
  require(count > 0 && count <= 65535, "frame count must be in [1, 65535]");
  const gg_star_params_t& p = *params;
  require(p.max_stars >= 1 && p.max_stars <= 4096, "max_stars must be in [1, 4096]");
  require(p.window_radius >= 0 && p.window_radius <= 16, "window_radius must be in [0, 16]");
  require(std::isfinite(p.threshold_sigma), "threshold_sigma must be finite");
  require(std::isfinite(p.min_separation_px), "min_separation_px must be finite");
  require(std::isfinite(p.catalog_min_fwhm) && std::isfinite(p.catalog_max_eccentricity),
          "catalog filter thresholds must be finite");
  require(p.mesh_cell == 0 || (p.mesh_cell >= 8 && p.mesh_cell <= kMeshMaxCell), "mesh_cell must be 0 or in [8, 64]");
  require(p.mesh_cell == 0 || (std::isnan(p.background) && std::isnan(p.noise)),
          "a background mesh estimates background and noise itself (pass NaN)");
  for (int64_t k = 0; k < count; ++k) stack_require_loaded(s, indices[k], "star detection");
  stack_activate(s);
  detect_stars(s, indices, static_cast<int>(count), p);
  StarScratch& sc = star_scratch(s);
  std::vector<StarFrameState> st(static_cast<size_t>(count));
  check_cuda(cudaMemcpyAsync(st.data(), sc.state, sizeof(StarFrameState) * count, cudaMemcpyDeviceToHost, s->stream),
             "cudaMemcpyAsync(star state)");
  if (host_stars) {
    check_cuda(cudaMemcpyAsync(host_stars, sc.out, sizeof(gg_star_t) * count * p.max_stars, cudaMemcpyDeviceToHost,
                               s->stream),
               "cudaMemcpyAsync(stars)");
  }
  check_cuda(cudaStreamSynchronize(s->stream), "cudaStreamSynchronize(stars)");
  stack_check_device_error(s);
  for (int64_t k = 0; k < count; ++k) {
    const StarFrameState& f = st[static_cast<size_t>(k)];
    if (f.overflow) fail(GG_ERR_RUNTIME, "more than 32768 star candidates in one frame; raise threshold_sigma");
    if (host_counts) host_counts[k] = (s->width < 3 || s->height < 3) ? 0 : f.kept;
    if (host_info) {
      host_info[k].median = f.median;
      host_info[k].mad = f.mad;
      host_info[k].noise = f.noise;
      host_info[k].threshold = f.threshold;
      host_info[k].candidates = static_cast<int64_t>(f.candidates);
      host_info[k].valid_pixels = static_cast<int64_t>(f.count);
    }
  }
  GG_API_END
}

}  // extern "C"

// ---- isolated cosmetic defects (source DQ) ------------------------------------
// cpu/cosmetic.py:97-307 on resident frames: a finite pixel is a hot (cold)
// candidate when it exceeds float32(median + k_hot sigma) (is below
// float32(median - k_cold sigma)) and its distance to the float32 median of
// its finite 8-neighbours (edge-clamped; float32 (a + b) / 2 for an even
// count; the global median without any) exceeds float32(k sigma); it is a
// defect when fewer than min_support neighbours pass float32(median -/+
// max(0, structure_sigma) sigma) on the same side; the protected variant
// keeps defects inside the radius of catalog stars with npix >= min_pixels
// and sharpness <= max_sharpness.  median and sigma are the frame's star-
// detection statistics (the same robust_background).  Defects become NaN
// (resident_source_dq.py:825-925: no replacement).
namespace gg {

struct CosmeticArgs {
  const float* slots;
  const int* slot_of_frame;
  int64_t stride;
  int width, height;
  const int* frames;
  const StarFrameState* state;
  const gg_star_t* stars;  // [count][max_stars] (protected variant)
  int max_stars;
  unsigned* hot_bits;      // [count][words]
  unsigned* cold_bits;
  int64_t words;
  unsigned long long* counts;  // [count][8]
  double hot_sigma, cold_sigma, support_sigma;
  int min_support;
  int protect;
  int min_pixels;
  double max_sharpness, radius_sq;
};

__device__ __forceinline__ bool star_protected(const CosmeticArgs& a, int k, int x, int y) {
  const int n = a.state[k].kept;
  const gg_star_t* st = a.stars + static_cast<int64_t>(k) * a.max_stars;
  for (int i = 0; i < n; ++i) {
    const gg_star_t s = st[i];
    if (s.npix < a.min_pixels || s.sharpness > a.max_sharpness) continue;
    if (!isfinite(s.x) || !isfinite(s.y)) continue;
    const double dx = static_cast<double>(x) - s.x, dy = static_cast<double>(y) - s.y;
    if (__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)) <= a.radius_sq) return true;
  }
  return false;
}

__global__ void __launch_bounds__(256) cosmetic_classify_kernel(CosmeticArgs a) {
  __shared__ unsigned long long s_counts[8];
  if (threadIdx.x < 8) s_counts[threadIdx.x] = 0;
  __syncthreads();
  const int k = blockIdx.y;
  const float* img = a.slots + static_cast<int64_t>(a.slot_of_frame[a.frames[k]]) * a.stride;
  const StarFrameState& st = a.state[k];
  const double med = static_cast<double>(st.median), sigma = st.noise;
  const float medf = st.median;
  const float hot_limit = __double2float_rn(__dadd_rn(med, __dmul_rn(a.hot_sigma, sigma)));
  const float cold_limit = __double2float_rn(__dsub_rn(med, __dmul_rn(a.cold_sigma, sigma)));
  const float hot_delta = __double2float_rn(__dmul_rn(a.hot_sigma, sigma));
  const float cold_delta = __double2float_rn(__dmul_rn(a.cold_sigma, sigma));
  const float sup_hi = __double2float_rn(__dadd_rn(med, __dmul_rn(a.support_sigma, sigma)));
  const float sup_lo = __double2float_rn(__dsub_rn(med, __dmul_rn(a.support_sigma, sigma)));
  const int W = a.width, H = a.height;
  const int64_t P = static_cast<int64_t>(W) * H;
  unsigned c_hot = 0, c_cold = 0, c_cand_hot = 0, c_cand_cold = 0, c_prot_hot = 0, c_prot_cold = 0;
  for (int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; p < P;
       p += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float v = __ldg(img + p);
    if (!isfinite(v) || !(v > hot_limit || v < cold_limit)) continue;  // only global outliers go on
    const int y = static_cast<int>(p / W), x = static_cast<int>(p - static_cast<int64_t>(y) * W);
    float nb[8];
    int n = 0, hs = 0, cs = 0;
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
      for (int dx = -1; dx <= 1; ++dx) {
        if (!dx && !dy) continue;
        const int yy = min(max(y + dy, 0), H - 1), xx = min(max(x + dx, 0), W - 1);
        const float u = __ldg(img + static_cast<int64_t>(yy) * W + xx);
        if (isfinite(u)) {
          nb[n++] = u;
          hs += u > sup_hi;
          cs += u < sup_lo;
        }
      }
    for (int i = 1; i < n; ++i) {  // insertion sort of <= 8 values
      const float t = nb[i];
      int j = i - 1;
      while (j >= 0 && nb[j] > t) {
        nb[j + 1] = nb[j];
        --j;
      }
      nb[j + 1] = t;
    }
    const float lmed = n == 0 ? medf : ((n & 1) ? nb[n / 2] : __fmul_rn(__fadd_rn(nb[n / 2 - 1], nb[n / 2]), 0.5f));
    const bool cand_hot = v > hot_limit && __fsub_rn(v, lmed) > hot_delta;
    const bool cand_cold = v < cold_limit && __fsub_rn(lmed, v) > cold_delta;
    c_cand_hot += cand_hot;
    c_cand_cold += cand_cold;
    bool hot = cand_hot && hs < a.min_support;
    bool cold = cand_cold && cs < a.min_support;
    if ((hot || cold) && a.protect && star_protected(a, k, x, y)) {
      c_prot_hot += hot;
      c_prot_cold += cold;
      hot = cold = false;
    }
    const int64_t word = static_cast<int64_t>(k) * a.words + (p >> 5);
    const unsigned bit = 1u << (p & 31);
    if (hot) {
      ++c_hot;
      atomicOr(a.hot_bits + word, bit);
    }
    if (cold) {
      ++c_cold;
      atomicOr(a.cold_bits + word, bit);
    }
  }
  const unsigned vals[6] = {c_hot, c_cold, c_cand_hot, c_cand_cold, c_prot_hot, c_prot_cold};
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    unsigned v = vals[i];
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&s_counts[i], static_cast<unsigned long long>(v));
  }
  __syncthreads();
  if (threadIdx.x < 6 && s_counts[threadIdx.x])
    atomicAdd(a.counts + static_cast<int64_t>(k) * 8 + threadIdx.x, s_counts[threadIdx.x]);
}

// Defects -> NaN; the frame's non-finite counter grows by the pixels set.
__global__ void __launch_bounds__(256) cosmetic_apply_kernel(CosmeticArgs a, unsigned* frame_nonfinite) {
  const int k = blockIdx.y;
  float* img = const_cast<float*>(a.slots) + static_cast<int64_t>(a.slot_of_frame[a.frames[k]]) * a.stride;
  const int64_t P = static_cast<int64_t>(a.width) * a.height;
  unsigned added = 0;
  for (int64_t w = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; w < a.words;
       w += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    unsigned bits = a.hot_bits[static_cast<int64_t>(k) * a.words + w] | a.cold_bits[static_cast<int64_t>(k) * a.words + w];
    while (bits) {
      const int b = __ffs(bits) - 1;
      bits &= bits - 1;
      const int64_t p = w * 32 + b;
      if (p < P) {
        img[p] = __int_as_float(0x7fc00000);
        ++added;
      }
    }
  }
  for (int off = 16; off > 0; off >>= 1) added += __shfl_xor_sync(0xffffffffu, added, off);
  if ((threadIdx.x & 31) == 0 && added) atomicAdd(frame_nonfinite + a.frames[k], added);
}

}  // namespace gg

extern "C" int gg_stack_cosmetic_mask(gg_stack* s, const int64_t* indices, int64_t count,
                                      const gg_cosmetic_params_t* params, gg_cosmetic_result_t* host_out) {
  using namespace gg;
  GG_API_BEGIN
  require(s != nullptr && indices != nullptr && params != nullptr, "null argument");
  require(count > 0 && count <= 65535, "frame count must be in [1, 65535]");
  const gg_cosmetic_params_t& p = *params;
  require(std::isfinite(p.hot_sigma) && std::isfinite(p.cold_sigma) && std::isfinite(p.structure_sigma),
          "cosmetic sigmas must be finite");
  require(!p.star_protection || (std::isfinite(p.star_protection_radius_px) && std::isfinite(p.star_threshold_sigma) &&
                                 std::isfinite(p.star_max_sharpness)),
          "star protection parameters must be finite");
  for (int64_t k = 0; k < count; ++k) stack_require_loaded(s, indices[k], "cosmetic defect detection");
  stack_activate(s);
  gg_star_params_t sp{};
  sp.threshold_sigma = p.star_threshold_sigma;
  sp.max_stars = 500;
  sp.window_radius = 4;
  sp.min_separation_px = std::max(2.0f, p.star_protection_radius_px * 0.5f);
  sp.background = std::nanf("");
  sp.noise = std::nanf("");
  sp.catalog_min_fwhm = 0.0f;
  sp.catalog_max_eccentricity = 1.0f;
  sp.mesh_cell = 0;
  detect_stars(s, indices, static_cast<int>(count), sp);
  StarScratch& sc = star_scratch(s);
  const int64_t words = (s->pixels + 31) / 32;
  unsigned* bits = nullptr;
  unsigned long long* counts = nullptr;
  check_cuda(cudaMallocAsync(reinterpret_cast<void**>(&bits), sizeof(unsigned) * words * count * 2, s->stream),
             "cudaMallocAsync(cosmetic bits)");
  check_cuda(cudaMallocAsync(reinterpret_cast<void**>(&counts), sizeof(unsigned long long) * 8 * count, s->stream),
             "cudaMallocAsync(cosmetic counts)");
  check_cuda(cudaMemsetAsync(bits, 0, sizeof(unsigned) * words * count * 2, s->stream), "cudaMemsetAsync(bits)");
  check_cuda(cudaMemsetAsync(counts, 0, sizeof(unsigned long long) * 8 * count, s->stream), "cudaMemsetAsync(counts)");
  CosmeticArgs a{};
  a.slots = s->d_slots;
  a.slot_of_frame = s->d_slot_of_frame;
  a.stride = s->stride;
  a.width = static_cast<int>(s->width);
  a.height = static_cast<int>(s->height);
  a.frames = sc.frames;
  a.state = sc.state;
  a.stars = sc.out;
  a.max_stars = sp.max_stars;
  a.hot_bits = bits;
  a.cold_bits = bits + words * count;
  a.words = words;
  a.counts = counts;
  a.hot_sigma = p.hot_sigma;
  a.cold_sigma = p.cold_sigma;
  a.support_sigma = std::max(0.0, static_cast<double>(p.structure_sigma));
  a.min_support = std::max(0, p.min_neighbor_support);
  a.protect = p.star_protection ? 1 : 0;
  a.min_pixels = p.star_min_pixels;
  a.max_sharpness = p.star_max_sharpness;
  const double r = std::max(0.0, static_cast<double>(p.star_protection_radius_px));
  a.radius_sq = r * r;
  if (!(r > 0.0)) a.protect = 0;
  const unsigned per_frame = grid_for(static_cast<size_t>(s->pixels), 256, std::max(1, 8 / static_cast<int>(std::min<int64_t>(count, 8))));
  note_launch();
  cosmetic_classify_kernel<<<dim3(per_frame, static_cast<unsigned>(count)), 256, 0, s->stream>>>(a);
  check_cuda(cudaGetLastError(), "cosmetic_classify launch");
  if (p.apply) {
    note_launch();
    cosmetic_apply_kernel<<<dim3(std::max(1u, static_cast<unsigned>(std::min<int64_t>((words + 255) / 256, 1024))),
                                 static_cast<unsigned>(count)), 256, 0, s->stream>>>(a, s->d_frame_nonfinite);
    check_cuda(cudaGetLastError(), "cosmetic_apply launch");
  }
  std::vector<unsigned long long> host(static_cast<size_t>(8 * count));
  std::vector<StarFrameState> states(static_cast<size_t>(count));
  check_cuda(cudaMemcpyAsync(host.data(), counts, sizeof(unsigned long long) * 8 * count, cudaMemcpyDeviceToHost,
                             s->stream),
             "cudaMemcpyAsync(cosmetic counts)");
  check_cuda(cudaMemcpyAsync(states.data(), sc.state, sizeof(StarFrameState) * count, cudaMemcpyDeviceToHost, s->stream),
             "cudaMemcpyAsync(cosmetic state)");
  check_cuda(cudaFreeAsync(bits, s->stream), "cudaFreeAsync(cosmetic bits)");
  check_cuda(cudaFreeAsync(counts, s->stream), "cudaFreeAsync(cosmetic counts)");
  check_cuda(cudaStreamSynchronize(s->stream), "cudaStreamSynchronize(cosmetic)");
  if (host_out) {
    for (int64_t k = 0; k < count; ++k) {
      gg_cosmetic_result_t& r = host_out[k];
      const unsigned long long* c = host.data() + 8 * k;
      r.hot_pixels = static_cast<int64_t>(c[0]);
      r.cold_pixels = static_cast<int64_t>(c[1]);
      r.candidate_hot_pixels = static_cast<int64_t>(c[2]);
      r.candidate_cold_pixels = static_cast<int64_t>(c[3]);
      r.star_protected_hot_pixels = static_cast<int64_t>(c[4]);
      r.star_protected_cold_pixels = static_cast<int64_t>(c[5]);
      r.median = static_cast<double>(states[static_cast<size_t>(k)].median);
      r.sigma = states[static_cast<size_t>(k)].noise;
      r.star_count = states[static_cast<size_t>(k)].kept;
      r.pad = 0;
    }
  }
  GG_API_END
}

namespace gg {

// Source-DQ invalid mask (glass_apply_invalid_mask_f32_kernel semantics):
// non-zero mask bytes make the sample NaN; the frame's non-finite counter
// counts the samples that were finite before.
__global__ void __launch_bounds__(256) invalid_mask_kernel(float* img, const unsigned char* mask, int64_t n,
                                                           unsigned* nonfinite) {
  unsigned added = 0;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    if (mask[i] && isfinite(img[i])) {
      img[i] = __int_as_float(0x7fc00000);
      ++added;
    }
  }
  for (int off = 16; off > 0; off >>= 1) added += __shfl_xor_sync(0xffffffffu, added, off);
  if ((threadIdx.x & 31) == 0 && added) atomicAdd(nonfinite, added);
}

}  // namespace gg

extern "C" int gg_stack_apply_invalid_mask(gg_stack* s, int64_t index, const uint8_t* host_mask,
                                           int64_t* host_invalid_samples) {
  using namespace gg;
  GG_API_BEGIN
  require(s != nullptr && host_mask != nullptr, "null argument");
  stack_require_loaded(s, index, "source-DQ invalid mask");
  stack_activate(s);
  std::vector<int> slots;
  stack_read_slots(s, slots);
  unsigned char* d_mask = nullptr;
  check_cuda(cudaMallocAsync(reinterpret_cast<void**>(&d_mask), static_cast<size_t>(s->pixels), s->stream),
             "cudaMallocAsync(invalid mask)");
  check_cuda(cudaMemcpyAsync(d_mask, host_mask, static_cast<size_t>(s->pixels), cudaMemcpyHostToDevice, s->stream),
             "cudaMemcpyAsync(invalid mask)");
  float* img = s->d_slots + static_cast<int64_t>(slots[static_cast<size_t>(index)]) * s->stride;
  note_launch();
  invalid_mask_kernel<<<grid_for(static_cast<size_t>(s->pixels), 256), 256, 0, s->stream>>>(
      img, d_mask, s->pixels, s->d_frame_nonfinite + index);
  check_cuda(cudaGetLastError(), "invalid_mask launch");
  check_cuda(cudaFreeAsync(d_mask, s->stream), "cudaFreeAsync(invalid mask)");
  check_cuda(cudaStreamSynchronize(s->stream), "cudaStreamSynchronize(invalid mask)");
  if (host_invalid_samples) {
    int64_t n = 0;
    for (int64_t i = 0; i < s->pixels; ++i) n += host_mask[i] != 0;
    *host_invalid_samples = n;
  }
  GG_API_END
}

namespace gg {

// Threshold-only cosmetic mask (apply / count_cosmetic_threshold_mask_frame(s)
// semantics, integration_kernels.cu:181-232, 266-330): per listed frame a
// sample is non-finite, hot (> high) or cold (< low), tested in that order;
// with `apply` all three become NaN and the frame's non-finite counter grows
// by the hot and cold samples (a non-finite sample was already counted).
// float4 grid-stride loop per frame (slots start 256-byte aligned), one
// store per quad that changed, counts folded per warp.
struct ThresholdFrame {
  int frame;
  float low, high;
  int pad;
};

__device__ __forceinline__ bool threshold_classify(float& x, float low, float high, bool apply, unsigned& hot,
                                                   unsigned& cold, unsigned& nonfinite) {
  bool hit = true;
  if (!isfinite(x)) ++nonfinite;
  else if (x > high) ++hot;
  else if (x < low) ++cold;
  else hit = false;
  if (hit && apply) x = __int_as_float(0x7fc00000);
  return hit && apply;
}

__global__ void __launch_bounds__(256) cosmetic_threshold_kernel(float* slots, const int* slot_of_frame, int64_t stride,
                                                                 int64_t pixels, const ThresholdFrame* frames,
                                                                 int apply, unsigned long long* counts,
                                                                 unsigned* frame_nonfinite) {
  const int k = blockIdx.y;
  const ThresholdFrame tf = frames[k];
  float* img = slots + static_cast<int64_t>(slot_of_frame[tf.frame]) * stride;
  const bool ap = apply != 0;
  unsigned hot = 0, cold = 0, nonf = 0;
  const int64_t quads = pixels / 4;
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x;
  float4* img4 = reinterpret_cast<float4*>(img);
  for (int64_t q = t0; q < quads; q += step) {
    float4 v = img4[q];
    bool changed = threshold_classify(v.x, tf.low, tf.high, ap, hot, cold, nonf);
    changed |= threshold_classify(v.y, tf.low, tf.high, ap, hot, cold, nonf);
    changed |= threshold_classify(v.z, tf.low, tf.high, ap, hot, cold, nonf);
    changed |= threshold_classify(v.w, tf.low, tf.high, ap, hot, cold, nonf);
    if (changed) img4[q] = v;
  }
  for (int64_t p = quads * 4 + t0; p < pixels; p += step) {
    float x = img[p];
    if (threshold_classify(x, tf.low, tf.high, ap, hot, cold, nonf)) img[p] = x;
  }
  for (int off = 16; off > 0; off >>= 1) {
    hot += __shfl_xor_sync(0xffffffffu, hot, off);
    cold += __shfl_xor_sync(0xffffffffu, cold, off);
    nonf += __shfl_xor_sync(0xffffffffu, nonf, off);
  }
  if ((threadIdx.x & 31) == 0) {
    unsigned long long* c = counts + static_cast<int64_t>(k) * 3;
    if (hot) atomicAdd(c, static_cast<unsigned long long>(hot));
    if (cold) atomicAdd(c + 1, static_cast<unsigned long long>(cold));
    if (nonf) atomicAdd(c + 2, static_cast<unsigned long long>(nonf));
    if (ap && hot + cold) atomicAdd(frame_nonfinite + tf.frame, hot + cold);
  }
}

}  // namespace gg

extern "C" int gg_stack_cosmetic_threshold(gg_stack* s, const int64_t* indices, int64_t count,
                                           const float* low_thresholds, const float* high_thresholds, int32_t apply,
                                           int64_t* host_counts) {
  using namespace gg;
  GG_API_BEGIN
  require(s != nullptr && indices != nullptr && low_thresholds != nullptr && high_thresholds != nullptr,
          "null argument");
  require(count > 0 && count <= 65535, "batch cosmetic threshold application supports at most 65535 frames per launch");
  std::vector<ThresholdFrame> frames(static_cast<size_t>(count));
  for (int64_t k = 0; k < count; ++k) {
    const float lo = low_thresholds[k], hi = high_thresholds[k];
    require(!std::isnan(lo) && !std::isnan(hi) && lo <= hi,
            "cosmetic thresholds must be finite-or-infinite values with low <= high");
    stack_require_loaded(s, indices[k], "source-DQ cosmetic threshold mask");
    frames[static_cast<size_t>(k)] = ThresholdFrame{static_cast<int>(indices[k]), lo, hi, 0};
  }
  stack_activate(s);
  const size_t count_bytes = sizeof(unsigned long long) * 3 * static_cast<size_t>(count);
  const size_t frame_bytes = sizeof(ThresholdFrame) * static_cast<size_t>(count);
  unsigned char* buf = nullptr;
  check_cuda(cudaMallocAsync(reinterpret_cast<void**>(&buf), count_bytes + frame_bytes, s->stream),
             "cudaMallocAsync(cosmetic threshold)");
  auto* d_counts = reinterpret_cast<unsigned long long*>(buf);
  auto* d_frames = reinterpret_cast<ThresholdFrame*>(buf + count_bytes);
  check_cuda(cudaMemsetAsync(d_counts, 0, count_bytes, s->stream), "cudaMemsetAsync(cosmetic threshold counts)");
  upload_params(s->stream, d_frames, frames.data(), frame_bytes, "cudaMemcpyAsync(cosmetic threshold frames)");
  const unsigned per_frame = grid_for(static_cast<size_t>((s->pixels + 3) / 4), 256,
                                      std::max(1, 8 / static_cast<int>(std::min<int64_t>(count, 8))));
  note_launch();
  cosmetic_threshold_kernel<<<dim3(per_frame, static_cast<unsigned>(count)), 256, 0, s->stream>>>(
      s->d_slots, s->d_slot_of_frame, s->stride, s->pixels, d_frames, apply ? 1 : 0, d_counts, s->d_frame_nonfinite);
  check_cuda(cudaGetLastError(), "cosmetic_threshold launch");
  std::vector<unsigned long long> host(3 * static_cast<size_t>(count));
  check_cuda(cudaMemcpyAsync(host.data(), d_counts, count_bytes, cudaMemcpyDeviceToHost, s->stream),
             "cudaMemcpyAsync(cosmetic threshold counts)");
  check_cuda(cudaFreeAsync(buf, s->stream), "cudaFreeAsync(cosmetic threshold)");
  check_cuda(cudaStreamSynchronize(s->stream), "cudaStreamSynchronize(cosmetic threshold)");
  if (host_counts)
    for (size_t i = 0; i < host.size(); ++i) host_counts[i] = static_cast<int64_t>(host[i]);
  GG_API_END
}
