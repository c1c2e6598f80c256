// Integration of up to 256 resident frames with one thread per pixel: mean,
// sigma clip and winsorized sigma clip (the rules of integrate.cu), for the
// frame counts and sizes that launch_integrate_args gives it.
//
// A warp owns tiles of 32 consecutive pixels.  A tile's rows (one per frame
// with a valid weight, 128 B each) come by cp.async into the warp's own shared
// memory, so a sample costs one shared-memory load and no address arithmetic
// (one bulk copy per row instead was slower: 26 clocks per 128-byte copy and
// SM).  Each lane keeps its pixel's column: it sorts it in one or two lists of
// NB registers (a Batcher network without branches or shuffles; one copy of it
// in the instruction cache), writes the lists back over the tile, finds the
// percentile ranks by a merge search over the two lists, and sums.  Nothing
// crosses lanes, so the per-pixel scalar work (percentiles, divisions, the
// square root) is paid once per 32 pixels.  The weighted sum needs the samples
// in frame order with their weights: the rows are copied a second time (they
// are in the L2 cache then), in chunks of 32 rows, and each chunk is refilled
// with the next tile's rows as soon as it is summed.
//
// Winsorized statistics are sums about the median m: S1 = sum d and
// S2 = sum d^2 of d = clip(x) - m in one pass, two samples per instruction; the
// mean is m + S1 / n and the squared deviations about a centre m + t are
// S2 - t (2 S1 - n t).  The weighted sum is taken about m too.
//
// Bound: latency at two warps per scheduler (a warp's tile takes 128 B x frames
// of shared memory), then the min / max pipe (64 lanes per clock and SM; the
// sort takes 22 per sample of the 60 instructions in all): half of the issue
// slots and of that pipe.  200 frames of 2400 x 1605, winsorized: 7.51 ms with a
// half-warp per pixel, 2.70 ms here (3.5 ps per sample); 40 frames of 3000 x
// 2000, sigma clip: 4.36 ms, 0.82 ms; 32 frames of 2048^2, winsorized: 0.81 ms with
// the column kernel, 0.39 ms here.  Samples around zero take the sums that round:
// 4.2 ps per sample for 200 frames; weights over three decades 4.0.
#pragma once

#include <algorithm>
#include <cfloat>

#include "async.cuh"
#include "f32x2.cuh"
#include "integrate.cuh"

namespace gg {

// Warps per CTA at most.
constexpr int px_max_warps(int nb) { return nb <= 32 ? 4 : 8; }
constexpr int kPxChunk = 16;  // row pairs per copy chunk: one row per lane

template <int NB, int L>
struct PxTable {
  float4 w[NB * L / 2];        // weights of a row pair: high parts, low parts
  const float* base[NB * L];   // frames with a valid weight, in order
  float total[2];              // sum of the weights
  float unit;                  // rounds a weight to its high part (0: no split)
  int narrow;                  // the parts' sums are exact (narrow_weights)
  int active;
  int allvalid;
};

// Exact sums without TwoSums.  Samples x of one sign that differ from a pivot
// m by at most their least magnitude are multiples of one unit u, and so is
// d = x - m: at most 2^24 u, hence exact.  Adding and subtracting `round`
// splits d into dh, a multiple of q with |dh| <= 2^8 q, and dl, |dl| <= q / 2.
// Of up to 256 samples sum dh, sum dl and sum dh^2 are exact in float32, and
// so are the products dh dl; their sum (signs at random, 2^-10 of sum dh^2)
// rounds by 2^-35 of sum d^2 at most where it exceeds 24 bits, the sum of dl^2
// by 2^-40.
struct Split {
  float round;
  bool ok;
};

__device__ __forceinline__ Split split_range(float least, float most, float m) {
  const float range = fmaxf(__fsub_rn(most, m), __fsub_rn(m, least));
  const float low = fminf(fabsf(least), fabsf(most));
  Split r;
  // 1.5 * 2^23 q with q = 2^(exponent of the range - 7): the range is below 2^8 q
  r.round = __int_as_float(__float_as_int(range) & 0x7f800000) * 98304.0f;
  r.ok = least > most || (range <= low && (least > 0.0f) == (most > 0.0f) && r.round < kInf);
  return r;
}

// Weights are split in two parts as well: w = wh + wl, wh a multiple of q with
// |wh| <= 2^9 q, |wl| <= q / 2.  A thread's sums over `pairs` row pairs of wh
// and of wh dh (2^17 units each) are exact in float32; those of wl are where the
// least weight's last place is at least pairs x q / 2^25.  Then the weight of a
// pixel is the frames' total minus the weights that do not count, exactly,
// whatever little is left of it.  Weights further apart (a ratio of 8 for 256
// frames, of 32 for 64), or at the ends of the float32 range, are not split: the
// weights that do count are added up in float-float.
__device__ __forceinline__ bool narrow_weights(float least, float most, int pairs) {
  const int low = max(__float_as_int(least) >> 23, 1), high = __float_as_int(most) >> 23;  // biased exponents
  return high >= 32 && high <= 127 + 110 && high - low <= 10 && (pairs << (high - low)) <= 1024;
}

__device__ __forceinline__ void split(F2 d, F2 round, F2& dh, F2& dl) {
  dh = f2_sub(f2_add(d, round), round);
  dl = f2_sub(d, dh);
}

// Sums of d = clip(x, lo, hi) - med and d^2 over a pixel's sorted lists.
struct DevSums {
  FF s1, s2;
};

template <int NB, int L>
struct PxColumn {
  static constexpr int kSteps = NB < 64 ? 6 : NB < 128 ? 7 : 8;  // of a search among NB + 1 places
  static_assert((1 << kSteps) > NB, "search steps");
  const float* col;  // this lane's column, rows 32 floats apart
  int na, nb;        // rows of the lists (warp-uniform)
  int ca, cb;        // valid samples of the lists

  __device__ __forceinline__ float a(int i) const { return col[i * 32]; }
  __device__ __forceinline__ float b(int i) const { return col[(NB + i) * 32]; }
  __device__ __forceinline__ int count() const { return ca + cb; }

  // Values of ranks k[q] and k[q] + 1 of both lists together (+inf past the
  // samples): the split of the merge that takes k + 1 samples.
  template <int Q>
  __device__ __forceinline__ void ranks(const int (&k)[Q], float (&v0)[Q], float (&v1)[Q]) const {
    if constexpr (L == 1) {
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        v0[q] = a(k[q]);
        v1[q] = k[q] + 1 < NB ? a(min(k[q] + 1, NB - 1)) : kInf;
      }
    } else {
      // i samples of list a and k + 1 - i of list b are taken: descend to the
      // largest i whose last sample is below the first untaken one of b
      int lo[Q], hi[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        lo[q] = max(0, k[q] + 1 - NB);
        hi[q] = min(k[q] + 1, NB);
      }
#pragma unroll
      for (int s = kSteps - 1; s >= 0; --s) {
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          const int i = lo[q] + (1 << s), m = max(min(i, hi[q]) - 1, 0);
          const float x = a(m), y = b(min(max(k[q] - m, 0), NB - 1));
          lo[q] = (i <= hi[q] && x < y) ? i : lo[q];
        }
      }
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int i = lo[q], j = k[q] + 1 - i;
        v0[q] = fmaxf(i > 0 ? a(i - 1) : -kInf, j > 0 ? b(j - 1) : -kInf);
        v1[q] = fminf(i < NB ? a(min(i, NB - 1)) : kInf, j < NB ? b(min(j, NB - 1)) : kInf);
      }
    }
  }

  // Valid samples below lt and above ht (binary searches side by side).
  __device__ __forceinline__ void outside(float lt, float ht, int& nl, int& nh) const {
    int n[2 * L];
#pragma unroll
    for (int q = 0; q < 2 * L; ++q) n[q] = 0;
#pragma unroll
    for (int s = kSteps - 1; s >= 0; --s) {
#pragma unroll
      for (int q = 0; q < 2 * L; ++q) {
        const int i = n[q] + (1 << s);
        const float v = col[((q / 2) * NB + min(i, NB) - 1) * 32];
        n[q] = (i <= (q < 2 ? ca : cb) && ((q & 1) ? !(v > ht) : v < lt)) ? i : n[q];
      }
    }
    nl = n[0] + (L == 2 ? n[2 * L - 2] : 0);
    nh = count() - n[1] - (L == 2 ? n[2 * L - 1] : 0);
  }

  // Smallest and largest valid sample (+inf, -inf without one).
  __device__ __forceinline__ float least() const { return L == 2 ? fminf(a(0), b(0)) : a(0); }
  __device__ __forceinline__ float most() const {
    return fmaxf(ca > 0 ? a(ca - 1) : -kInf, (L == 2 && cb > 0) ? b(cb - 1) : -kInf);
  }

  // `plain` (warp-uniform): every row is valid and `sp` splits its deviations.
  __device__ __forceinline__ DevSums deviations(float med, float lo, float hi, bool plain, Split sp) const {
    const F2 m = f2(med);
    const int pairs = L == 2 ? na : (na + 1) / 2;
    if (plain) {
      const F2 round = f2(sp.round);
      F2 sh, sl, hh, hl, ll;
      auto add = [&](float x, float y) {
        F2 dh, dl;
        split(f2_sub(f2(x, y), m), round, dh, dl);
        sh = f2_add(sh, dh);
        sl = f2_add(sl, dl);
        hh = f2_fma(dh, dh, hh);
        hl = f2_fma(dh, dl, hl);
        ll = f2_fma(dl, dl, ll);
      };
      const int full = L == 2 ? nb : na / 2;
#pragma unroll 8
      for (int k = 0; k < full; ++k)
        add(clipf(L == 2 ? a(k) : a(2 * k), lo, hi), clipf(L == 2 ? b(k) : a(2 * k + 1), lo, hi));
      if (full < pairs) add(clipf(L == 2 ? a(full) : a(2 * full), lo, hi), med);
      DevSums r;
      two_sum(f2_sum(sh), f2_sum(sl), r.s1.hi, r.s1.lo);
      two_sum(f2_sum(hh), 2.0f * f2_sum(hl), r.s2.hi, r.s2.lo);
      r.s2.lo = __fadd_rn(r.s2.lo, f2_sum(ll));
      return r;
    }
    FF2 s1, s2;
    F2 s2n;  // minus the rounding errors of the squares
#pragma unroll 2
    for (int k = 0; k < pairs; ++k) {
      const float x = L == 2 ? a(k) : a(2 * k), y = L == 2 ? b(k) : a(2 * k + 1);
      F2 d, e;
      f2_two_sum(f2(x < kInf ? clipf(x, lo, hi) : med, y < kInf ? clipf(y, lo, hi) : med), f2(-med), d, e);
      s1.add(d);
      s1.lo = f2_add(s1.lo, e);
      const F2 p = f2_mul(d, d);
      s2n = f2_add(s2n, f2_fma(d, f2_sub(F2(), d), p));
      s2.add(p);
      s2.lo = f2_fma(f2_add(d, d), e, s2.lo);
    }
    s2.lo = f2_sub(s2.lo, s2n);
    return {s1.merged(), s2.merged()};
  }

  // Mean and standard deviation of the valid samples clipped to [lo, hi]
  // (-+inf: not clipped).  With allvalid the deviations are taken from the
  // unrounded mean, else from the float32 mean (engine/rejection.py:219-349).
  __device__ __forceinline__ float clipped_std(float med, float lo, float hi, bool allvalid, bool finite,
                                               float& mean) const {
    const Split sp = split_range(clipf(least(), lo, hi), clipf(most(), lo, hi), med);
    const bool plain = __all_sync(0xffffffffu, finite && sp.ok);
    const DevSums s = deviations(med, lo, hi, plain, sp);
    const float n = static_cast<float>(count());
    float th, tl, c, ce;
    ff_div_pair(s.s1.hi, s.s1.lo, n, th, tl);
    two_sum(med, th, c, ce);
    mean = __fadd_rn(c, __fadd_rn(ce, tl));
    if (!allvalid) two_sum(mean, -med, th, tl);
    // S2 - t (2 S1 - n t) with t = (th, tl)
    const float nt = __fmul_rn(n, th);
    const float nte = __fmaf_rn(n, tl, __fmaf_rn(n, th, -nt));
    float uh, ul;
    two_sum(2.0f * s.s1.hi, -nt, uh, ul);
    ul = __fadd_rn(ul, __fsub_rn(2.0f * s.s1.lo, nte));
    const float q = __fmul_rn(th, uh);
    const float qe = __fmaf_rn(tl, uh, __fmaf_rn(th, ul, __fmaf_rn(th, uh, -q)));
    float vh, vl;
    two_sum(s.s2.hi, -q, vh, vl);
    vl = __fadd_rn(vl, __fsub_rn(s.s2.lo, qe));
    const float hi2 = __fadd_rn(vh, vl);
    if (hi2 < 0.0f) return 0.0f;
    float r, rl;
    ff_div_pair(hi2, __fsub_rn(vl, __fsub_rn(hi2, vh)), n, r, rl);
    return ff_sqrt_f32(r, rl);
  }
};

// NB registers per list, L lists (NB * L rows of shared memory per warp), the
// rejection MODE.
template <int NB, int L, int MODE>
__global__ void __launch_bounds__(32 * px_max_warps(NB), NB <= 32 ? 5 : NB <= 80 ? 2 : 1)
    integrate_px_kernel(IntegrateArgs a) {
  constexpr int ROWS = NB * L;
  constexpr int rejection = MODE;
  extern __shared__ __align__(128) float px_tiles[];  // [warps][ROWS][32]
  __shared__ PxTable<NB, L> tab;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  float* tile = px_tiles + static_cast<size_t>(warp) * ROWS * 32;

  // frames with a valid weight, in order; rows past them hold +inf
  if (warp == 0) {
    int rows = 0;
    unsigned bad = 0, invalid = 0;
    float least = kInf, most = 0.0f;
    FF total;
    for (int f0 = 0; f0 < a.frames; f0 += 32) {
      const int f = f0 + lane;
      const float w = f < a.frames ? (a.weights ? a.weights[f] : 1.0f) : 0.0f;
      const bool ok = f < a.frames && isfinite(w) && w > 0.0f;
      if (f < a.frames) {
        bad |= a.nonfinite[f];
        invalid |= ok ? 0u : 1u;
      }
      if (ok) {
        least = fminf(least, w);
        most = fmaxf(most, w);
        total.add(w);
      }
      const unsigned mask = __ballot_sync(0xffffffffu, ok);
      if (ok) tab.base[rows + __popc(mask & ((1u << lane) - 1u))] =
          a.base ? a.base[f] : a.slots + static_cast<int64_t>(a.slot_of_frame[f]) * a.stride;
      rows += __popc(mask);
    }
    bad = __reduce_or_sync(0xffffffffu, bad);
    invalid = __reduce_or_sync(0xffffffffu, invalid);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      least = fminf(least, __shfl_xor_sync(0xffffffffu, least, off));
      most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, off));
      FF o;
      o.hi = __shfl_xor_sync(0xffffffffu, total.hi, off);
      o.lo = __shfl_xor_sync(0xffffffffu, total.lo, off);
      ff_merge2(total, o);
    }
    if (lane == 0) {
      tab.total[0] = total.hi;
      tab.total[1] = total.lo;
      tab.narrow = narrow_weights(least, most, (rows + 1) / 2) ? 1 : 0;
      tab.unit = tab.narrow ? 0.5f * split_range(0.0f, most, 0.0f).round : 0.0f;
      tab.active = rows;
      tab.allvalid = (bad == 0u && invalid == 0u) ? 1 : 0;
    }
  }
  for (int i = threadIdx.x; i < ROWS / 2; i += blockDim.x) tab.w[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  for (int i = lane; i < ROWS * 32; i += 32) tile[i] = kInf;
  constexpr int kChunks = (ROWS / 2 + kPxChunk - 1) / kPxChunk;
  __syncthreads();
  const int rows = tab.active;
  const int na = L == 2 ? (rows + 1) / 2 : rows, nb = rows - na;
  if (warp == 0) {
    // weights by row pair: rows (k, NB + k) of two lists, (2k, 2k + 1) of one
    int r0 = 0;
    for (int f0 = 0; f0 < a.frames; f0 += 32) {
      const int f = f0 + lane;
      const float w = f < a.frames ? (a.weights ? a.weights[f] : 1.0f) : 0.0f;
      const bool ok = f < a.frames && isfinite(w) && w > 0.0f;
      const unsigned mask = __ballot_sync(0xffffffffu, ok);
      if (ok) {
        const int r = r0 + __popc(mask & ((1u << lane) - 1u));
        const int k = L == 2 ? (r < na ? r : r - na) : r / 2, half = L == 2 ? (r < na ? 0 : 1) : (r & 1);
        float* t = reinterpret_cast<float*>(&tab.w[k]);
        const float high = __fsub_rn(__fadd_rn(w, tab.unit), tab.unit);
        t[half] = high;
        t[2 + half] = __fsub_rn(w, high);
      }
      r0 += __popc(mask);
    }
  }
  __syncthreads();
  const bool allvalid = tab.allvalid != 0, narrow = tab.narrow != 0;
  const int pairs = L == 2 ? na : (na + 1) / 2;
  const int64_t P = a.pixels;
  const int64_t tiles = (P + 31) / 32;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * warps;
  const float ls = a.low_sigma, hs = a.high_sigma;

  // Copies of the 32 rows of chunk c of a tile (16 bytes per lane, four rows
  // per instruction), one group per chunk.  A tile's last row segment may
  // reach past the frame: slots are padded to a multiple of 64 samples, and
  // lanes past the frame write nothing.
  auto fetch = [&](int64_t t, int c) {
#pragma unroll
    for (int q = 0; q < 2 * kPxChunk / 4; ++q) {
      const int j = q * 4 + lane / 8, half = j / kPxChunk, k = c * kPxChunk + (j & (kPxChunk - 1));
      const int r = L == 2 ? (half ? na + k : k) : 2 * k + half;
      if (L == 2 ? k < (half ? nb : na) : r < rows)
        cp_async16(tile + (L == 2 ? half * NB + k : r) * 32 + (lane & 7) * 4,
                   tab.base[r] + t * 32 + (lane & 7) * 4);
    }
    cp_async_commit();
  };

  int64_t t = static_cast<int64_t>(blockIdx.x) * warps + warp;
  if (t < tiles)
    for (int c = 0; c < kChunks; ++c) fetch(t, c);
  for (; t < tiles; t += stride) {
    const int64_t p = t * 32 + lane;
    float lt = -FLT_MAX, ht = FLT_MAX;  // kept: finite samples in [lt, ht]
    int nl = 0, nh = 0, kept = 0;
    float pivot = 0.0f;  // the weighted sum is taken about it
    Split kept_split{0.0f, false};
    if (rejection != GG_REJECT_NONE) {
      cp_async_wait<0>();
      __syncwarp();
      PxColumn<NB, L> column;
      column.col = tile + lane;
      column.na = na;
      column.nb = nb;
      column.ca = column.cb = 0;
      bool finite = true;
      float sum = 0.0f;
#pragma unroll 1  // one copy of the network in the instruction cache
      for (int l = 0; l < L; ++l) {
        float* col = tile + lane + l * NB * 32;
        const int n = l ? nb : na;
        float v[NB];
#pragma unroll
        for (int k = 0; k < NB; ++k) v[k] = col[k * 32];
        // 0 * x is NaN for the samples that are not finite: of the n rows only, the
        // others hold +inf
        F2 probe;
#pragma unroll
        for (int k = 0; k < NB; k += 8)
          if (k + 8 <= n) {
#pragma unroll
            for (int q = k; q < k + 8; q += 2) probe = f2_fma(f2(v[q], v[q + 1]), F2(), probe);
          }
        float p0, p1;
        f2_split(probe, p0, p1);
#pragma unroll 1
        for (int k = n & ~7; k < n; ++k) p0 = __fmaf_rn(col[k * 32], 0.0f, p0);
        int valid = n;
        if (!__all_sync(0xffffffffu, p0 + p1 == 0.0f)) {
          valid = 0;
          finite = false;
#pragma unroll
          for (int k = 0; k < NB; ++k) {
            const bool is = fabsf(v[k]) < kInf;
            v[k] = is ? v[k] : kInf;
            valid += is ? 1 : 0;
          }
        }
        if (rejection == GG_REJECT_SIGMA_CLIP) {
          // float32 sum in frame order, as NumPy reduces over the frame axis
#pragma unroll
          for (int k = 0; k < NB; ++k) sum = __fadd_rn(sum, v[k] < kInf ? v[k] : 0.0f);
        }
        if (l == 0) column.ca = valid;
        else column.cb = valid;
        sort_network<NB>(v);
#pragma unroll
        for (int k = 0; k < NB; ++k) col[k * 32] = v[k];
      }
      const int cnt = column.count();
      const int c1 = max(cnt - 1, 0);
      CenterScale cs{0.0f, 0.0f};
      if (rejection == GG_REJECT_WINSORIZED) {
        // engine/rejection.py:299-321 (valid samples) and :352-366 (all valid)
        const float frac[3] = {0.5f, 0.25f, 0.75f};
        int k[3];
        float t3[3], v0[3], v1[3], pc[3];
        const float span = static_cast<float>(allvalid ? a.frames - 1 : c1);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const float pos = __fmul_rn(span, frac[q]);
          k[q] = static_cast<int>(floorf(pos));
          t3[q] = __fsub_rn(pos, static_cast<float>(k[q]));
        }
        column.ranks(k, v0, v1);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          if (allvalid) {
            pc[q] = t3[q] == 0.0f ? v0[q] : __fadd_rn(v0[q], __fmul_rn(__fsub_rn(v1[q], v0[q]), t3[q]));
          } else {
            const float up = k[q] < c1 ? v1[q] : v0[q];
            pc[q] = cnt > 0 ? __fadd_rn(__fmul_rn(v0[q], __fsub_rn(1.0f, t3[q])), __fmul_rn(up, t3[q])) : 0.0f;
          }
        }
        const float med = pc[0];
        pivot = med;
        float scale1 = __fdiv_rn(__fsub_rn(pc[2], pc[1]), 1.349f);
        const bool ok1 = allvalid ? (scale1 > 0.0f) : (scale1 > 0.0f && isfinite(scale1));
        if (__any_sync(0xffffffffu, !ok1 && cnt > 0)) {
          float unused;
          const float sd = column.clipped_std(med, -kInf, kInf, allvalid, finite, unused);
          if (!ok1) scale1 = sd;
        }
        const float lo1 = __fsub_rn(med, __fmul_rn(ls, scale1));
        const float hi1 = __fadd_rn(med, __fmul_rn(hs, scale1));
        const float scale = column.clipped_std(med, lo1, hi1, allvalid, finite, cs.center);
        const bool ok2 = allvalid ? (scale > 0.0f) : (scale > 0.0f && isfinite(scale));
        cs.scale = ok2 ? scale : scale1;
      } else {
        // NumPy nanmedian and float32 nanstd (engine/rejection.py:46-49)
        const int h = max(cnt, 1) / 2, l = (max(cnt, 1) & 1) ? h : h - 1;
        const int k[1] = {l};
        float v0[1], v1[1];
        column.ranks(k, v0, v1);
        const float n = static_cast<float>(cnt);
        const float mean = __fdiv_rn(sum, n);
        // the counts need the sorted lists, the variance the frame order:
        // the median's lists are kept until the thresholds are known by
        // reading the variance's samples from global memory
        float var = 0.0f;
        const bool inside = p < P;
#pragma unroll 8
        for (int r = 0; r < rows; ++r) {
          const float x = inside ? __ldg(tab.base[r] + p) : 0.0f;
          if (fabsf(x) < kInf) {
            const float d = __fsub_rn(x, mean);
            var = __fadd_rn(var, __fmul_rn(d, d));
          }
        }
        cs.center = cnt > 0 ? __fmul_rn(__fadd_rn(v0[0], h == l ? v0[0] : v1[0]), 0.5f) : 0.0f;
        pivot = cs.center;
        cs.scale = __fsqrt_rn(__fdiv_rn(var, n));
      }
      lt = __fsub_rn(cs.center, __fmul_rn(ls, cs.scale));
      ht = __fadd_rn(cs.center, __fmul_rn(hs, cs.scale));
      column.outside(lt, ht, nl, nh);
      const float least = column.least(), most = column.most();
      // the lists are done with: the rows again, in frame order
      __syncwarp();
      for (int c = 0; c < kChunks; ++c) fetch(t, c);
      if (nl + nh > 0) {
        // cpu/integration.py:85-99
        const int rej = nl + nh;
        const float frac = __fdiv_rn(static_cast<float>(rej), static_cast<float>(cnt));
        if (!((cnt - rej >= a.min_samples) && (frac <= a.max_frac))) nl = nh = 0;
      }
      kept = cnt - nl - nh;
      // nothing rejected: every finite sample is kept, whatever the thresholds
      lt = nl + nh > 0 ? fmaxf(lt, -FLT_MAX) : -FLT_MAX;
      ht = nl + nh > 0 ? fminf(ht, FLT_MAX) : FLT_MAX;
      // samples that span the float32 range have no finite difference from a
      // median, nor always a median
      if (!(fabsf(pivot) < kInf && __fsub_rn(most, least) < kInf)) pivot = 0.0f;
      kept_split = split_range(fmaxf(least, lt), fminf(most, ht), pivot);
    }
    // weighted sum over the kept samples, two rows at a time: pivot plus
    // split deviations by split weights where the kept samples and the weights
    // allow it
    const bool plain = __all_sync(0xffffffffu, narrow && kept_split.ok);
    const F2 m = f2(pivot), round = f2(kept_split.round);
    FF2 ws;
    F2 hh, hl, lh;
    F2 gone_h, gone_l;  // weights of the samples that do not count (narrow)
    FF2 counted;        // weights of those that do (else)
    int n2 = 0;
    const int64_t next = t + stride;
    for (int c = 0; c < kChunks; ++c) {
      // kChunks - 1 younger groups: this tile's later chunks and the next
      // tile's earlier ones
      cp_async_wait<kChunks - 1>();
      __syncwarp();
      const float* col = tile + lane + c * kPxChunk * (L == 2 ? 32 : 64);
      const float4* tw = tab.w + c * kPxChunk;
      auto row_pair = [&](int k, F2& v, F2& wh, F2& wl, F2& drop) {
        const float x = col[(L == 2 ? k : 2 * k) * 32], y = col[(L == 2 ? NB + k : 2 * k + 1) * 32];
        const float4 w = tw[k];
        const bool kx = x >= lt && x <= ht, ky = y >= lt && y <= ht;
        v = f2(kx ? x : pivot, ky ? y : pivot);
        wh = f2(w.x, w.y);
        wl = f2(w.z, w.w);
        drop = f2(kx ? 0.0f : 1.0f, ky ? 0.0f : 1.0f);
        gone_h = f2_fma(drop, wh, gone_h);
        gone_l = f2_fma(drop, wl, gone_l);
        if (rejection == GG_REJECT_NONE) n2 += (kx ? 1 : 0) + (ky ? 1 : 0);
      };
      auto add_split = [&](int k) {
        F2 v, wh, wl, drop, dh, dl;
        row_pair(k, v, wh, wl, drop);
        split(f2_sub(v, m), round, dh, dl);
        hh = f2_fma(wh, dh, hh);
        hl = f2_fma(wh, dl, hl);
        lh = f2_fma(wl, dh, f2_fma(wl, dl, lh));
      };
      auto add_rounded = [&](int k, F2& w, F2& drop) {
        F2 v, wh, wl, d, e;
        row_pair(k, v, wh, wl, drop);
        f2_two_sum(v, f2(-pivot), d, e);
        w = f2_add(wh, wl);
        const F2 prod = f2_mul(d, w);
        ws.lo = f2_add(ws.lo, f2_fma(w, e, f2_fma(d, w, f2_sub(F2(), prod))));
        ws.add(prod);
      };
      const int in_chunk = min(kPxChunk, pairs - c * kPxChunk);
      if (plain && in_chunk == kPxChunk) {
#pragma unroll
        for (int k = 0; k < kPxChunk; ++k) add_split(k);
      } else if (plain) {
#pragma unroll 1
        for (int k = 0; k < in_chunk; ++k) add_split(k);
      } else if (narrow) {
#pragma unroll 2
        for (int k = 0; k < in_chunk; ++k) {
          F2 w, drop;
          add_rounded(k, w, drop);
        }
      } else {
#pragma unroll 1
        for (int k = 0; k < in_chunk; ++k) {
          F2 w, drop;
          add_rounded(k, w, drop);
          counted.add(f2_fma(drop, f2_mul(w, f2(-1.0f)), w));
        }
      }
      __syncwarp();
      if (next < tiles) fetch(next, c);
      else cp_async_commit();
    }
    if (rejection == GG_REJECT_NONE) kept = n2;
    FF s, w;
    if (plain) {
      float e;
      two_sum(f2_sum(hh), f2_sum(hl), s.hi, s.lo);
      two_sum(s.hi, f2_sum(lh), s.hi, e);
      s.lo = __fadd_rn(s.lo, e);
    } else {
      s = ws.merged();
    }
    if (narrow) {
      w.hi = tab.total[0];
      w.lo = tab.total[1];
      float x, y, low, e;
      f2_split(gone_l, x, y);
      two_sum(x, y, low, e);
      FF gone;
      two_sum(-f2_sum(gone_h), -low, gone.hi, gone.lo);
      gone.lo = __fsub_rn(gone.lo, e);
      ff_merge2(w, gone);
    } else {
      w = counted.merged();
    }
    float master = 0.0f, weight = 0.0f;
    if (kept > 0 && w.hi > 0.0f) {
      // pivot + s / w
      const float q = __fdiv_rn(s.hi, w.hi);
      const float r = __fmaf_rn(-q, w.lo, __fadd_rn(__fmaf_rn(-q, w.hi, s.hi), s.lo));
      float mh, ml;
      two_sum(pivot, q, mh, ml);
      master = __fadd_rn(mh, __fadd_rn(ml, __fdiv_rn(r, w.hi)));
      weight = w.value_f32();
    }
    if (p < P) write_outputs(a, p, master, weight, kept, nl, nh, rows);
  }
}

// Warps per CTA.  A CTA's warps take turns on the SM's four schedulers, so the
// busiest one has ceil(w / 4) of each resident CTA; all warps have as many tiles,
// and that scheduler's run last.  A warp slows down by about one over the
// warps beside it, hence warps on the SM over 1 + warps on the busiest
// scheduler.  (The most warps alone picked two CTAs of five for 160 frames: 4.4
// ps per sample, 3.4 with one CTA of eight; 112 frames 4.0 and 3.2 with two of
// seven and three of four.)
template <int NB, int L, int MODE>
static int px_best_warps() {
  constexpr size_t kWarpBytes = size_t(NB) * L * 128;
  auto kern = integrate_px_kernel<NB, L, MODE>;
  double most = 0.0;
  int pick = 1;
  for (int w = px_max_warps(NB); w >= 2; --w) {
    if (kWarpBytes * w + sizeof(PxTable<NB, L>) > 227 * 1024) continue;
    const int per_sm = kernel_ctas_per_sm(kern, 32 * w, kWarpBytes * w, "launch shape (integrate_px)");
    const double score = static_cast<double>(per_sm * w) / (1 + per_sm * ((w + 3) / 4));
    if (score > most) {
      most = score;
      pick = w;
    }
  }
  return pick;
}

template <int NB, int L, int MODE>
static void launch_px(const IntegrateArgs& args, cudaStream_t stream) {
  constexpr size_t kWarpBytes = size_t(NB) * L * 128;
  auto kern = integrate_px_kernel<NB, L, MODE>;
  static const int best = px_best_warps<NB, L, MODE>();
  const int64_t tiles = (args.pixels + 31) / 32;
  // small frames: fewer warps per CTA, so that every SM has one
  const int warps = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(best, tiles / sm_count())));
  const size_t smem = kWarpBytes * warps;
  const int per_sm = kernel_ctas_per_sm(kern, 32 * warps, smem, "launch shape (integrate_px)");
  const int64_t ctas = std::min<int64_t>((tiles + warps - 1) / warps, int64_t(std::max(per_sm, 1)) * sm_count());
  note_launch();
  kern<<<static_cast<unsigned>(ctas), 32 * warps, smem, stream>>>(args);
  check_cuda(cudaGetLastError(), "integrate_px launch");
}

// A kernel for the rejection where it sorts: one for all of them shares its
// registers out by the most demanding (32 frames: 401 us with sigma clipping by
// itself, 436 beside winsorized in 122 registers), and which part of a kernel the
// compiler favours changes with any of its code.
// Short lists have those that small_stack_takes_tiles sends here.
template <int NB, int L>
static void launch_px_rule(const IntegrateArgs& a, cudaStream_t stream) {
  if (a.rejection == GG_REJECT_WINSORIZED) return launch_px<NB, L, GG_REJECT_WINSORIZED>(a, stream);
  if constexpr (NB * L > 16)
    if (a.rejection == GG_REJECT_SIGMA_CLIP) return launch_px<NB, L, GG_REJECT_SIGMA_CLIP>(a, stream);
  if constexpr (NB * L > 32)
    if (a.rejection == GG_REJECT_NONE) return launch_px<NB, L, GG_REJECT_NONE>(a, stream);
  fail(GG_ERR_INVALID_ARGUMENT, "no per-pixel integration kernel for this rejection and frame count");
}

// The kernel of `a.frames`, lists in steps of eight rows from NB to LAST.
template <int L, int NB, int LAST>
static void launch_px_list(const IntegrateArgs& a, cudaStream_t stream) {
  if constexpr (NB < LAST) {
    if (a.frames > NB * L) return launch_px_list<L, NB + 8, LAST>(a, stream);
  }
  launch_px_rule<NB, L>(a, stream);
}

// 65 to 256 frames (integrate_px2.cu).
void launch_integrate_px2(const IntegrateArgs& a, cudaStream_t stream);

}  // namespace gg
