// Triangle-asterism registration of star catalogs on the device.
//
// Semantics follow the reference's CPU estimator, src/glass/cpu/registration.py:
//   _local_triangle_descriptors  :273-303  k nearest neighbours per anchor
//        (stable distance order), every 3-subset in combination order, first
//        occurrence of each vertex set, area >= 2, area-descending stable
//        order, first max_descriptors
//   _ordered_triangle_by_sides   :242-270  vertex order from the side lengths,
//        descriptor (longest/middle, middle/shortest)
//   estimate_triangle_asterism_transform :361-475  matches within the
//        descriptor radius sorted by distance (stable), first max_candidates,
//        two reference orientations per match, best = most pairs then
//        smallest rms (first wins), three guarded refits
//   _fit_similarity_matrix       :140-162  Procrustes fit
//   _fit_affine_matrix           :106-119  least-squares affine fit (the
//        transform_model = "affine" estimator: 3-point affine hypotheses,
//        affine refits)
//   _greedy_pairs / _score_matrix :177-215 pairs within tolerance, greedy by
//        distance, rms of the residuals
// and, in descriptor-list mode, the reference's similarity-from-descriptors
// fallback (src/glass_cuda.py:2097-2140: every reference x moving descriptor
// pair within the radius in reference-major order, float32 descriptor
// distance, no truncation, no refit).
//
// The 2x2 SVD of the Procrustes fit is replaced by its closed form: rotation
// angle atan2(C01 - C10, C00 + C11) and sum of singular values max(E, F) with
// E = |(C00 + C11, C01 - C10)|, F = |(C00 - C11, C01 + C10)|.  Matrices agree
// with the reference to rounding; pair sets and inlier counts exactly.
//
// GB300 mapping: FP64 is scarce on this part, so every all-pairs loop filters
// in cheap arithmetic first (per-component descriptor bounds, float32
// transformed coordinates) and evaluates the float64 distance only for
// survivors.  One CTA per catalog builds descriptors in shared memory, several
// per frame pair find the descriptor matches and one selects among them, one
// warp per candidate transform fits it and counts its pairs in float32, the
// candidates that can still win get their float64 rms, and one CTA per frame
// pair picks the best and refits.
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "stack.cuh"

namespace gg {

constexpr int kRegPts = kCatalogPoints;  // points per catalog row (80)
constexpr int kMaxNeighbors = 6;
constexpr int kMaxCombos = 20;  // C(6, 3)
constexpr int kMaxTri = kRegPts * kMaxCombos;
constexpr int kMaxDesc = kMaxTri;
constexpr int kMaxSel = 2048;  // max_candidates ceiling of the estimator
constexpr int kPairCap = 512;  // point pairs within tolerance per candidate
constexpr int kStackMatchCap = 65536;
constexpr int kListMatchCap = 262144;

enum RegMode { kEstimator = 0, kDescriptorList = 1 };

struct Desc {
  double d0, d1, area;
  int v[3];
  int pad;
};

struct TriCand {
  double d0, d1, area;
  int packed;  // ordered vertices (7 bits each), bit 31 = has a descriptor
  int pad;
};

struct RegJob {
  int ref_row;
  int mov_row;
};

struct Cand {
  double m[6];
  double rms;
  long long order;
  int scored;  // rms: 0 not known, 1 the exact scorer's, 2 to rounding
  int pad;
};

// What a candidate is ranked by: its pair count (-1: no fit, or dropped;
// kConflictCount - c: at most c, the exact scorer's until it has run) and
// bounds of its rms.
constexpr int kConflictCount = -2;

struct CandRank {
  int count;
  float rms_lo, rms_hi;
};

struct RegResult {
  double m[9];
  double rms;
  long long best_order;
  int inliers;
  int status;
  int ndesc_ref;
  int ndesc_mov;
  int matches;
  int pad;
};

struct RegArgs {
  const double* pts;  // [rows][kRegPts][2]
  const int* npts;    // [rows]
  Desc* desc;         // [rows][kMaxDesc]
  int* ndesc;         // [rows]
  const RegJob* jobs;
  int* match_count;      // [jobs] matches found (may exceed match_cap)
  int* best_count;       // [jobs] most pairs of a candidate so far
  double* match_dist;    // [jobs][match_cap]
  int* match_key;        // [jobs][match_cap]
  int2* sel;             // [jobs][sel_cap]  (moving, reference) descriptor indices
  long long* sel_order;  // [jobs][sel_cap]
  int* nsel;             // [jobs]
  Cand* cands;           // [jobs][2 * sel_cap]
  CandRank* ranks;       // [jobs][2 * sel_cap]
  RegResult* out;        // [jobs]
  short2* pairs;         // [jobs][kRegPts]
  int* overflow;
  double tol;
  double radius;
  int match_cap;
  int sel_cap;
  int mode;
  int neighbors;
  int max_stars;
  int max_desc;
  int max_cand;
  int min_inliers;
  int model;  // GG_TRANSFORM_SIMILARITY or GG_TRANSFORM_AFFINE
};

// ---- float64 arithmetic rounded step by step like NumPy ---------------------
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
// sqrt(dx^2 + dy^2) as an elementwise square-and-sum (np.sum(d ** 2, axis=-1))
__device__ __forceinline__ double hyp_sum(double dx, double dy) { return sqrt(dadd(dmul(dx, dx), dmul(dy, dy))); }
// np.linalg.norm of a 2-vector: a dot product whose second term is fused
__device__ __forceinline__ double hyp_dot(double dx, double dy) { return sqrt(__fma_rn(dy, dy, dmul(dx, dx))); }
// Order-preserving bits of a non-negative double.
__device__ __forceinline__ unsigned long long dbits_of(double d) {
  return static_cast<unsigned long long>(__double_as_longlong(d));
}

// NumPy's pairwise sum of a contiguous float64 array (eight interleaved
// accumulators per block of <= 128, longer runs split at n/2 rounded down to
// a multiple of 8).
__device__ double pw_block(const double* v, int n) {
  if (n < 8) {
    double r = 0.0;
    for (int i = 0; i < n; ++i) r = dadd(r, v[i]);
    return r;
  }
  double r[8];
  for (int j = 0; j < 8; ++j) r[j] = v[j];
  int i = 8;
  for (; i < n - (n % 8); i += 8)
    for (int j = 0; j < 8; ++j) r[j] = dadd(r[j], v[i + j]);
  double res = dadd(dadd(dadd(r[0], r[1]), dadd(r[2], r[3])), dadd(dadd(r[4], r[5]), dadd(r[6], r[7])));
  for (; i < n; ++i) res = dadd(res, v[i]);
  return res;
}
__device__ double pw_sum(const double* v, int n) {
  if (n <= 128) return pw_block(v, n);
  int n2 = n / 2;
  n2 -= n2 % 8;
  return dadd(pw_block(v, n2), pw_block(v + n2, n - n2));  // n <= 160 here: both halves <= 128
}

// Similarity fit of n >= 2 point pairs (registration.py:140-162).  mx/my are
// moving coordinates, rx/ry reference; scratch holds 2n doubles.
__device__ bool fit_similarity(const double* mx, const double* my, const double* rx, const double* ry, int n,
                               double* scratch, double (&m)[6]) {
  if (n < 2) return false;
  double smx = 0.0, smy = 0.0, srx = 0.0, sry = 0.0;
  for (int i = 0; i < n; ++i) {  // np.mean(axis=0): rows added in order
    smx = dadd(smx, mx[i]);
    smy = dadd(smy, my[i]);
    srx = dadd(srx, rx[i]);
    sry = dadd(sry, ry[i]);
  }
  const double dn = static_cast<double>(n);
  const double mmx = __ddiv_rn(smx, dn), mmy = __ddiv_rn(smy, dn);
  const double mrx = __ddiv_rn(srx, dn), mry = __ddiv_rn(sry, dn);
  for (int i = 0; i < n; ++i) {
    const double cx = dsub(mx[i], mmx), cy = dsub(my[i], mmy);
    scratch[2 * i] = dmul(cx, cx);
    scratch[2 * i + 1] = dmul(cy, cy);
  }
  const double variance = pw_sum(scratch, 2 * n);
  if (!(variance > 1.0e-12)) return false;
  double c00 = 0.0, c01 = 0.0, c10 = 0.0, c11 = 0.0;
  for (int i = 0; i < n; ++i) {
    const double ax = dsub(mx[i], mmx), ay = dsub(my[i], mmy);
    const double bx = dsub(rx[i], mrx), by = dsub(ry[i], mry);
    c00 = dadd(c00, dmul(ax, bx));
    c01 = dadd(c01, dmul(ax, by));
    c10 = dadd(c10, dmul(ay, bx));
    c11 = dadd(c11, dmul(ay, by));
  }
  const double e = hyp_sum(dadd(c00, c11), dsub(c01, c10));
  const double f = hyp_sum(dsub(c00, c11), dadd(c01, c10));
  double cs = 1.0, sn = 0.0;
  if (e > 0.0) {
    cs = __ddiv_rn(dadd(c00, c11), e);
    sn = __ddiv_rn(dsub(c01, c10), e);
  }
  const double scale = __ddiv_rn(fmax(e, f), variance);
  const double l00 = dmul(scale, cs), l01 = dmul(scale, -sn), l10 = dmul(scale, sn), l11 = dmul(scale, cs);
  m[0] = l00;
  m[1] = l01;
  m[2] = dsub(mrx, dadd(dmul(mmx, l00), dmul(mmy, l01)));
  m[3] = l10;
  m[4] = l11;
  m[5] = dsub(mry, dadd(dmul(mmx, l10), dmul(mmy, l11)));
  return true;
}

// Affine fit of n >= 3 point pairs (registration.py:106-119: the least-squares
// solution of the 2n x 6 system).  The same solution from the normal
// equations about the means, which decouple the translation: with centred
// moving (a) and reference (b) coordinates,
//   [Sxx Sxy; Sxy Syy] (l00, l01) = (S(ax bx), S(ay bx)), likewise for row 1,
// solved by Cramer's rule; t = mean(b) - L mean(a).  False for fewer than 3
// pairs or a (numerically) singular system — collinear moving points, where
// the reference returns the minimum-norm solution instead; the descriptor
// filter (area >= 2 px^2) keeps those out of the 3-point fits.
struct AffineSums {
  double mmx, mmy, mrx, mry, sxx, sxy, syy, sxr, syr, sxs, sys;
};

__device__ __forceinline__ bool affine_from_sums(const AffineSums& q, double (&m)[6]) {
  const double det = dsub(dmul(q.sxx, q.syy), dmul(q.sxy, q.sxy));
  if (!(q.sxx > 0.0 && q.syy > 0.0 && det > dmul(1.0e-12, dmul(q.sxx, q.syy)))) return false;
  const double l00 = __ddiv_rn(dsub(dmul(q.sxr, q.syy), dmul(q.syr, q.sxy)), det);
  const double l01 = __ddiv_rn(dsub(dmul(q.syr, q.sxx), dmul(q.sxr, q.sxy)), det);
  const double l10 = __ddiv_rn(dsub(dmul(q.sxs, q.syy), dmul(q.sys, q.sxy)), det);
  const double l11 = __ddiv_rn(dsub(dmul(q.sys, q.sxx), dmul(q.sxs, q.sxy)), det);
  m[0] = l00;
  m[1] = l01;
  m[2] = dsub(q.mrx, dadd(dmul(l00, q.mmx), dmul(l01, q.mmy)));
  m[3] = l10;
  m[4] = l11;
  m[5] = dsub(q.mry, dadd(dmul(l10, q.mmx), dmul(l11, q.mmy)));
  return true;
}

__device__ bool fit_affine(const double* mx, const double* my, const double* rx, const double* ry, int n,
                           double (&m)[6]) {
  if (n < 3) return false;
  AffineSums q{};
  double smx = 0.0, smy = 0.0, srx = 0.0, sry = 0.0;
  for (int i = 0; i < n; ++i) {
    smx = dadd(smx, mx[i]);
    smy = dadd(smy, my[i]);
    srx = dadd(srx, rx[i]);
    sry = dadd(sry, ry[i]);
  }
  const double dn = static_cast<double>(n);
  q.mmx = __ddiv_rn(smx, dn);
  q.mmy = __ddiv_rn(smy, dn);
  q.mrx = __ddiv_rn(srx, dn);
  q.mry = __ddiv_rn(sry, dn);
  for (int i = 0; i < n; ++i) {
    const double ax = dsub(mx[i], q.mmx), ay = dsub(my[i], q.mmy);
    const double bx = dsub(rx[i], q.mrx), by = dsub(ry[i], q.mry);
    q.sxx = dadd(q.sxx, dmul(ax, ax));
    q.sxy = dadd(q.sxy, dmul(ax, ay));
    q.syy = dadd(q.syy, dmul(ay, ay));
    q.sxr = dadd(q.sxr, dmul(ax, bx));
    q.syr = dadd(q.syr, dmul(ay, bx));
    q.sxs = dadd(q.sxs, dmul(ax, by));
    q.sys = dadd(q.sys, dmul(ay, by));
  }
  return affine_from_sums(q, m);
}

// ---- point pairs of a transform (registration.py:177-215) ------------------------
// The reference catalog of a frame pair is bucketed into a uniform grid of at
// most 8 x 8 cells (at least 2 * (tol + 0.5) px wide), so a transformed
// moving star only visits the reference stars of <= 2 x 2 cells instead of
// all of them.
constexpr int kGrid = 8;

struct JobPoints {
  double mx[kRegPts], my[kRegPts], rx[kRegPts], ry[kRegPts];
  float mx32[kRegPts], my32[kRegPts], rx32[kRegPts], ry32[kRegPts];
  unsigned char cell_start[kGrid * kGrid + 1];
  unsigned char cell_pt[kRegPts];
  unsigned char cell_of[kRegPts];
  float gx0, gy0, ginv;
  int gnx, gny;
  float cmax;  // max |x| + |y| of the moving stars
  float rmax;  // max |x|, |y| of the reference stars
  int partners;  // most reference stars that can be in reach of one moving star
  int nm, nr;
};

constexpr int kNearCap = 256;

struct WarpScratch {
  double tx[kRegPts], ty[kRegPts];
  float tx32[kRegPts], ty32[kRegPts];
  unsigned long long key[kPairCap];  // distance bits of the pairs within tolerance
  int idx[kPairCap];                 // (moving << 8) | reference: row-major order
  int acc[kRegPts];                  // accepted entries in greedy order
  unsigned short near[kNearCap];     // pairs of the float32 test
  double res[kRegPts];
  unsigned used_r[3], used_m[3];
  int count;
  double rms;
};

// Reference stars within `r` of (x, y) in grid order; calls f(j).
template <class F>
__device__ __forceinline__ void grid_visit(const JobPoints& jp, float x, float y, float r, F&& f) {
  if (!(fabsf(x) < 3.0e38f && fabsf(y) < 3.0e38f) || jp.gnx == 0) return;
  const float fx0 = (x - r - jp.gx0) * jp.ginv, fx1 = (x + r - jp.gx0) * jp.ginv;
  const float fy0 = (y - r - jp.gy0) * jp.ginv, fy1 = (y + r - jp.gy0) * jp.ginv;
  if (fx1 < 0.0f || fy1 < 0.0f || fx0 >= static_cast<float>(jp.gnx) || fy0 >= static_cast<float>(jp.gny)) return;
  const int cx0 = max(0, static_cast<int>(floorf(fmaxf(fx0, -1.0f))));
  const int cx1 = min(jp.gnx - 1, static_cast<int>(floorf(fminf(fx1, static_cast<float>(jp.gnx)))));
  const int cy0 = max(0, static_cast<int>(floorf(fmaxf(fy0, -1.0f))));
  const int cy1 = min(jp.gny - 1, static_cast<int>(floorf(fminf(fy1, static_cast<float>(jp.gny)))));
  for (int cy = cy0; cy <= cy1; ++cy)
    for (int cx = cx0; cx <= cx1; ++cx) {
      const int c = cy * kGrid + cx;
      for (int k = jp.cell_start[c]; k < jp.cell_start[c + 1]; ++k) f(static_cast<int>(jp.cell_pt[k]));
    }
}

// NumPy pairwise sum of v[0..n) (n <= 128) by lanes 0..7 of the warp: lane j
// runs accumulator j; every lane returns the sum.
__device__ double warp_pw_sum(const double* v, int n) {
  const int lane = threadIdx.x & 31;
  double r = 0.0;
  if (n >= 8 && lane < 8) {
    r = v[lane];
    for (int i = lane + 8; i < n - (n % 8); i += 8) r = dadd(r, v[i]);
  }
  double out = 0.0;
  const double r1 = __shfl_down_sync(0xffffffffu, r, 1);
  const double r2 = __shfl_down_sync(0xffffffffu, r, 2);
  const double r3 = __shfl_down_sync(0xffffffffu, r, 3);
  const double r4 = __shfl_down_sync(0xffffffffu, r, 4);
  const double r5 = __shfl_down_sync(0xffffffffu, r, 5);
  const double r6 = __shfl_down_sync(0xffffffffu, r, 6);
  const double r7 = __shfl_down_sync(0xffffffffu, r, 7);
  if (lane == 0) {
    if (n < 8) {
      for (int i = 0; i < n; ++i) out = dadd(out, v[i]);
    } else {
      out = dadd(dadd(dadd(r, r1), dadd(r2, r3)), dadd(dadd(r4, r5), dadd(r6, r7)));
      for (int i = n - (n % 8); i < n; ++i) out = dadd(out, v[i]);
    }
  }
  return __shfl_sync(0xffffffffu, out, 0);
}

// The steps of the exact score, by a group of threads: `tid` of `threads`,
// `sync` their barrier.
struct WarpGroup {
  static constexpr int kThreads = 32;
  __device__ __forceinline__ static int tid() { return threadIdx.x & 31; }
  __device__ __forceinline__ static void sync() { __syncwarp(); }
  __device__ __forceinline__ static bool any(bool p) { return __any_sync(0xffffffffu, p); }
};
template <int THREADS>
struct CtaGroup {
  static constexpr int kThreads = THREADS;
  __device__ __forceinline__ static int tid() { return threadIdx.x; }
  __device__ __forceinline__ static void sync() { __syncthreads(); }
  __device__ __forceinline__ static bool any(bool p) { return __syncthreads_or(p) != 0; }
};

// The moving stars at their transformed places and the list of the pairs
// that pass the float32 test with a 0.5 px margin (w.near; the return value may
// exceed its capacity).
template <class G>
__device__ int near_pairs(const double (&m)[6], const JobPoints& jp, double tol, WarpScratch& w) {
  for (int i = G::tid(); i < jp.nm; i += G::kThreads) {
    const double x = dadd(dadd(dmul(jp.mx[i], m[0]), dmul(jp.my[i], m[1])), m[2]);
    const double y = dadd(dadd(dmul(jp.mx[i], m[3]), dmul(jp.my[i], m[4])), m[5]);
    w.tx[i] = x;
    w.ty[i] = y;
    w.tx32[i] = static_cast<float>(x);
    w.ty32[i] = static_cast<float>(y);
  }
  if (G::tid() == 0) w.count = 0;
  G::sync();
  const float r = static_cast<float>(tol + 0.5);
  const float pre = r * r;
  for (int i = G::tid(); i < jp.nm; i += G::kThreads) {
    const float x = w.tx32[i], y = w.ty32[i];
    grid_visit(jp, x, y, r, [&](int j) {
      const float fx = x - jp.rx32[j], fy = y - jp.ry32[j];
      if (fx * fx + fy * fy > pre) return;
      const int pos = atomicAdd(&w.count, 1);
      if (pos < kNearCap) w.near[pos] = static_cast<unsigned short>((i << 8) | j);
    });
  }
  G::sync();
  const int listed = w.count;
  G::sync();
  return listed;
}

__device__ __forceinline__ double pair_distance(const JobPoints& jp, const WarpScratch& w, int i, int j) {
  return hyp_sum(dsub(w.tx[i], jp.rx[j]), dsub(w.ty[i], jp.ry[j]));
}

// Exact scoring: every thread of the group returns the greedy pair count and
// rms (+inf without pairs); the pairs (moving, reference) go to `pairs` when
// not null.
template <class G>
__device__ void score_exact(const double (&m)[6], const JobPoints& jp, double tol, WarpScratch& w, int& npairs,
                            double& rms, short2* pairs, int* overflow) {
  const int listed = near_pairs<G>(m, jp, tol, w);
  if (G::tid() == 0) w.count = 0;
  G::sync();
  // the float64 distances, one pair per thread (a float64 operation costs a
  // warp the same for one lane as for all); any order, sorted below
  auto test = [&](int i, int j) {
    const double d = pair_distance(jp, w, i, j);
    if (!(d <= tol)) return;
    const int pos = atomicAdd(&w.count, 1);
    if (pos < kPairCap) {
      w.key[pos] = dbits_of(d);
      w.idx[pos] = (i << 8) | j;
    }
  };
  if (listed <= kNearCap) {
    for (int t = G::tid(); t < listed; t += G::kThreads) test(w.near[t] >> 8, w.near[t] & 255);
  } else {
    const float r = static_cast<float>(tol + 0.5);
    const float pre = r * r;
    for (int i = G::tid(); i < jp.nm; i += G::kThreads) {
      const float x = w.tx32[i], y = w.ty32[i];
      grid_visit(jp, x, y, r, [&](int j) {
        const float fx = x - jp.rx32[j], fy = y - jp.ry32[j];
        if (fx * fx + fy * fy <= pre) test(i, j);
      });
    }
  }
  G::sync();
  int L = w.count;
  if (L > kPairCap) {
    if (G::tid() == 0) atomicExch(overflow, 1);
    L = kPairCap;
  }
  // sort by (distance, row-major index), the stable distance sort of the
  // row-major candidate list: two threads count the entries before one
  constexpr int kHalf = G::kThreads / 2, kPer = kPairCap / kHalf;
  unsigned long long key[kPer];
  int idx[kPer], rank[kPer];
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    if (u * kHalf >= L) break;
    const int e = u * kHalf + (G::tid() >> 1);
    key[u] = e < L ? w.key[e] : ~0ull;
    idx[u] = e < L ? w.idx[e] : 0x7fffffff;
    int before = 0;
#pragma unroll 4
    for (int q = G::tid() & 1; q < L; q += 2) {
      const unsigned long long kq = w.key[q];
      before += (kq < key[u] || (kq == key[u] && w.idx[q] < idx[u])) ? 1 : 0;
    }
    rank[u] = before + __shfl_xor_sync(0xffffffffu, before, 1);
  }
  if (G::tid() < 3) w.used_r[G::tid()] = w.used_m[G::tid()] = 0u;
  G::sync();
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    if (u * kHalf >= L) break;
    if (u * kHalf + (G::tid() >> 1) < L && (G::tid() & 1) == 0) {
      w.key[rank[u]] = key[u];
      w.idx[rank[u]] = idx[u];
    }
  }
  G::sync();
  // greedy one-to-one pairing in distance order: every entry where no star
  // stands in two, else one after the other
  bool twice = false;
  for (int t = G::tid(); t < L; t += G::kThreads) {
    const int i = w.idx[t] >> 8, j = w.idx[t] & 255;
    const unsigned bi = 1u << (i & 31), bj = 1u << (j & 31);
    twice |= (atomicOr(&w.used_m[i >> 5], bi) & bi) != 0u;
    twice |= (atomicOr(&w.used_r[j >> 5], bj) & bj) != 0u;
    if (t < kRegPts) w.acc[t] = t;
  }
  int n = L;
  if (G::any(twice)) {
    if (G::tid() == 0) {
      n = 0;
      unsigned used_m[3] = {0u, 0u, 0u}, used_r[3] = {0u, 0u, 0u};
      for (int a = 0; a < L; ++a) {
        const int i = w.idx[a] >> 8, j = w.idx[a] & 255;
        if ((used_m[i >> 5] >> (i & 31)) & 1u) continue;
        if ((used_r[j >> 5] >> (j & 31)) & 1u) continue;
        used_m[i >> 5] |= 1u << (i & 31);
        used_r[j >> 5] |= 1u << (j & 31);
        w.acc[n++] = a;
      }
      w.count = n;
    }
    G::sync();
    n = w.count;
  }
  G::sync();
  for (int t = G::tid(); t < n; t += G::kThreads) {
    const int a = w.acc[t];
    const double d = __longlong_as_double(static_cast<long long>(w.key[a]));
    w.res[t] = dmul(d, d);
    if (pairs) pairs[t] = make_short2(static_cast<short>(w.idx[a] >> 8), static_cast<short>(w.idx[a] & 255));
  }
  G::sync();
  if (G::tid() < 32) {
    const double s = warp_pw_sum(w.res, n);
    if (G::tid() == 0)
      w.rms = n > 0 ? sqrt(__ddiv_rn(s, static_cast<double>(n))) : __longlong_as_double(0x7ff0000000000000ll);
  }
  G::sync();
  npairs = n;
  rms = w.rms;
  G::sync();
}

// Count and rms of a transform in which a few stars have two partners: every
// pair of two otherwise unpaired stars counts, and the greedy order is worked
// out among the others alone (at most 32).  False when there are more.
__device__ bool warp_resolve(const double (&m)[6], const JobPoints& jp, double tol, WarpScratch& w, int& npairs,
                             double& rms) {
  const int lane = threadIdx.x & 31;
  const int listed = near_pairs<WarpGroup>(m, jp, tol, w);
  if (listed > kNearCap) return false;
  int* with_m = w.acc;
  int* with_r = reinterpret_cast<int*>(w.res);
  for (int i = lane; i < kRegPts; i += 32) with_m[i] = with_r[i] = 0;
  __syncwarp();
  for (int t = lane; t < listed; t += 32) {
    const int i = w.near[t] >> 8, j = w.near[t] & 255;
    const double d = pair_distance(jp, w, i, j);
    w.key[t] = d <= tol ? dbits_of(d) : ~0ull;
    if (d <= tol) {
      atomicAdd(&with_m[i], 1);
      atomicAdd(&with_r[j], 1);
    }
  }
  __syncwarp();
  int n = 0, open = 0;
  double sum = 0.0;
  for (int t0 = 0; t0 < listed; t0 += 32) {
    const int t = t0 + lane;
    const unsigned long long key = t < listed ? w.key[t] : ~0ull;
    bool alone = false;
    if (key != ~0ull) alone = with_m[w.near[t] >> 8] == 1 && with_r[w.near[t] & 255] == 1;
    const unsigned rest = __ballot_sync(0xffffffffu, key != ~0ull && !alone);
    const int pos = open + __popc(rest & ((1u << lane) - 1u));
    if (key != ~0ull && !alone && pos < 32) w.idx[pos] = t;
    open += __popc(rest);
    n += __popc(__ballot_sync(0xffffffffu, alone));
    const double d = alone ? __longlong_as_double(static_cast<long long>(key)) : 0.0;
    sum = dadd(sum, dmul(d, d));
  }
  if (open > 32) return false;
  __syncwarp();
  const bool mine = lane < open;
  const unsigned long long key = mine ? w.key[w.idx[lane]] : ~0ull;
  const int pair = mine ? w.near[w.idx[lane]] : 0x7fffffff;
  int rank = 0;
  for (int q = 0; q < open; ++q) {
    const unsigned long long kq = __shfl_sync(0xffffffffu, key, q);
    const int pq = __shfl_sync(0xffffffffu, pair, q);
    rank += (kq < key || (kq == key && pq < pair)) ? 1 : 0;
  }
  bool free = mine, kept = false;
  for (int s = 0; s < open; ++s) {
    const int from = __ffs(__ballot_sync(0xffffffffu, mine && rank == s)) - 1;
    const int taken = __shfl_sync(0xffffffffu, free ? pair : -1, from);
    if (taken < 0) continue;
    if (lane == from) kept = true;
    if ((pair >> 8) == (taken >> 8) || (pair & 255) == (taken & 255)) free = false;
  }
  n += __popc(__ballot_sync(0xffffffffu, kept));
  const double d = kept ? __longlong_as_double(static_cast<long long>(key)) : 0.0;
  sum = dadd(sum, dmul(d, d));
  for (int off = 16; off > 0; off >>= 1) sum = dadd(sum, __shfl_xor_sync(0xffffffffu, sum, off));
  __syncwarp();
  npairs = n;
  rms = n > 0 ? sqrt(__ddiv_rn(sum, static_cast<double>(n))) : __longlong_as_double(0x7ff0000000000000ll);
  return true;
}

// float32 scoring of a transform: how far it can be off.
struct FastTransform {
  float m[6];
  float r;         // search radius
  float lo2, hi2;  // squared distance certainly inside / outside the tolerance
  float delta;     // bound of a pair distance's error
};

__device__ __forceinline__ FastTransform fast_transform(const double (&m)[6], const JobPoints& jp, double tol) {
  FastTransform t;
  for (int q = 0; q < 6; ++q) t.m[q] = static_cast<float>(m[q]);
  const double lin = fmax(fmax(fabs(m[0]), fabs(m[1])), fmax(fabs(m[3]), fabs(m[4])));
  const double trn = fmax(fabs(m[2]), fabs(m[5]));
  const double eps = 5.9604644775390625e-08;  // 2^-24
  const double delta = 2.0 * (1.5 * (6.0 * eps * (lin * jp.cmax + trn) + eps * jp.rmax) + 4.0 * eps * (tol + 1.0)) +
                       1.0e-6;
  const double lo = tol - delta;
  t.lo2 = lo > 0.0 ? static_cast<float>(lo * lo) : -1.0f;
  t.hi2 = static_cast<float>((tol + delta) * (tol + delta));
  t.r = static_cast<float>(tol + delta);
  t.delta = static_cast<float>(delta) * 1.000001f;
  return t;
}

// Whether candidates may be dropped unscored: the exact scorer reports more
// pairs than it holds, and no candidate that might do so is passed over.
__device__ __forceinline__ bool can_leave_early(const JobPoints& jp, double tol, float reach) {
  return jp.nm * jp.partners <= kPairCap && reach <= static_cast<float>(tol + 0.5);
}

// Pairs of a transform for ranking: the exact count when no moving or
// reference star has two partners within tolerance (then greedy pairing keeps
// every pair), and the float32 sum of squared residuals.  Membership is
// decided in float32 outside a band of +-delta around the tolerance (delta
// bounds the float32 transform error) and in float64 inside it.  `conflict`
// reports that the exact scorer is needed; the count is then the moving or the
// reference stars with a partner, whichever are fewer: the exact count cannot
// exceed either.
//
// `best`: a count that some candidate is known to reach; one that cannot reach
// it any more is left (count -1) after any 32 stars.
__device__ void warp_score_count(const FastTransform& t, const double* m, const JobPoints& jp, double tol, int best,
                                 unsigned* used_r, int& count, float& sum_d2, bool& conflict) {
  const int lane = threadIdx.x & 31;
  if (lane < 3) used_r[lane] = 0u;
  __syncwarp();
  int cnt = 0, paired = 0;
  float acc = 0.0f;
  bool conf = false;
  for (int i0 = 0; i0 < jp.nm; i0 += 32) {
    const int i = min(i0 + lane, jp.nm - 1);
    const bool real = i0 + lane < jp.nm;
    const float x = __fadd_rn(__fadd_rn(__fmul_rn(t.m[0], jp.mx32[i]), __fmul_rn(t.m[1], jp.my32[i])), t.m[2]);
    const float y = __fadd_rn(__fadd_rn(__fmul_rn(t.m[3], jp.mx32[i]), __fmul_rn(t.m[4], jp.my32[i])), t.m[5]);
    int hits = 0;
    if (real) grid_visit(jp, x, y, t.r, [&](int j) {
      const float fx = x - jp.rx32[j], fy = y - jp.ry32[j];
      const float d2 = fx * fx + fy * fy;
      if (d2 > t.hi2) return;
      if (!(d2 <= t.lo2)) {
        const double x64 = dadd(dadd(dmul(jp.mx[i], m[0]), dmul(jp.my[i], m[1])), m[2]);
        const double y64 = dadd(dadd(dmul(jp.mx[i], m[3]), dmul(jp.my[i], m[4])), m[5]);
        const double ex = dsub(x64, jp.rx[j]), ey = dsub(y64, jp.ry[j]);
        if (!(sqrt(dadd(dmul(ex, ex), dmul(ey, ey))) <= tol)) return;
      }
      ++hits;
      acc += d2;
      const unsigned bit = 1u << (j & 31);
      if (atomicOr(&used_r[j >> 5], bit) & bit) conf = true;
    });
    if (hits > 1) conf = true;
    cnt += hits;
    paired += __popc(__ballot_sync(0xffffffffu, hits > 0));
    if (paired + max(0, jp.nm - i0 - 32) < best) {
      count = -1;
      sum_d2 = 0.0f;
      conflict = false;
      __syncwarp();
      return;
    }
  }
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  conflict = __any_sync(0xffffffffu, conf);
  __syncwarp();
  count = conflict ? min(paired, __popc(used_r[0]) + __popc(used_r[1]) + __popc(used_r[2])) : cnt;
  sum_d2 = acc;
  __syncwarp();
}

// The same pairs (of a transform without conflicts) with float64 residuals:
// the sum of their squares in any order.
__device__ double warp_sum_d2(const double (&m)[6], const FastTransform& t, const JobPoints& jp, double tol) {
  const int lane = threadIdx.x & 31;
  double acc = 0.0;
  auto residual = [&](int i, int j) {
    const double x64 = dadd(dadd(dmul(jp.mx[i], m[0]), dmul(jp.my[i], m[1])), m[2]);
    const double y64 = dadd(dadd(dmul(jp.mx[i], m[3]), dmul(jp.my[i], m[4])), m[5]);
    const double ex = dsub(x64, jp.rx[j]), ey = dsub(y64, jp.ry[j]);
    return dadd(dmul(ex, ex), dmul(ey, ey));
  };
  for (int i0 = 0; i0 < jp.nm; i0 += 32) {
    const int i = i0 + lane;
    int partner = -1;  // at most one
    if (i < jp.nm) {
      const float x = __fadd_rn(__fadd_rn(__fmul_rn(t.m[0], jp.mx32[i]), __fmul_rn(t.m[1], jp.my32[i])), t.m[2]);
      const float y = __fadd_rn(__fadd_rn(__fmul_rn(t.m[3], jp.mx32[i]), __fmul_rn(t.m[4], jp.my32[i])), t.m[5]);
      grid_visit(jp, x, y, t.r, [&](int j) {
        const float fx = x - jp.rx32[j], fy = y - jp.ry32[j];
        const float d2 = fx * fx + fy * fy;
        if (d2 > t.hi2) return;
        if (!(d2 <= t.lo2) && !(sqrt(residual(i, j)) <= tol)) return;
        partner = j;
      });
    }
    __syncwarp();  // together: a float64 operation costs the warp the same for one lane as for all
    if (partner >= 0) acc = dadd(acc, residual(i, partner));
  }
  __syncwarp();
  for (int off = 16; off > 0; off >>= 1) acc = dadd(acc, __shfl_xor_sync(0xffffffffu, acc, off));
  return acc;
}

// Warp-cooperative similarity fit of n <= 80 pairs: the same arithmetic as
// fit_similarity with the independent sums on separate lanes.  Every lane
// returns the result.
__device__ bool warp_fit_similarity(const double* mx, const double* my, const double* rx, const double* ry, int n,
                                    double* sq, double (&m)[6]) {
  const int lane = threadIdx.x & 31;
  if (n < 2) return false;
  double s = 0.0;
  if (lane < 4) {
    const double* v = lane == 0 ? mx : (lane == 1 ? my : (lane == 2 ? rx : ry));
#pragma unroll 8
    for (int i = 0; i < n; ++i) s = dadd(s, v[i]);
  }
  s = __ddiv_rn(s, static_cast<double>(n));  // one quotient per lane costs as much as one
  const double mmx = __shfl_sync(0xffffffffu, s, 0), mmy = __shfl_sync(0xffffffffu, s, 1);
  const double mrx = __shfl_sync(0xffffffffu, s, 2), mry = __shfl_sync(0xffffffffu, s, 3);
  for (int i = lane; i < n; i += 32) {
    const double cx = dsub(mx[i], mmx), cy = dsub(my[i], mmy);
    sq[2 * i] = dmul(cx, cx);
    sq[2 * i + 1] = dmul(cy, cy);
  }
  __syncwarp();
  double variance;
  if (2 * n <= 128) {
    variance = warp_pw_sum(sq, 2 * n);
  } else {
    int n2 = n;  // (2n) / 2
    n2 -= n2 % 8;
    variance = dadd(warp_pw_sum(sq, n2), warp_pw_sum(sq + n2, 2 * n - n2));
  }
  if (!(variance > 1.0e-12)) return false;
  // the products by all lanes, then each sum in pair order by its own lane
  for (int i = lane; i < n; i += 32) {
    const double ax = dsub(mx[i], mmx), ay = dsub(my[i], mmy), bx = dsub(rx[i], mrx), by = dsub(ry[i], mry);
    sq[i] = dmul(ax, bx);
    sq[kRegPts + i] = dmul(ax, by);
    sq[2 * kRegPts + i] = dmul(ay, bx);
    sq[3 * kRegPts + i] = dmul(ay, by);
  }
  __syncwarp();
  double c = 0.0;
  if (lane < 4) {
#pragma unroll 8
    for (int i = 0; i < n; ++i) c = dadd(c, sq[lane * kRegPts + i]);
  }
  __syncwarp();
  const double c00 = __shfl_sync(0xffffffffu, c, 0), c01 = __shfl_sync(0xffffffffu, c, 1);
  const double c10 = __shfl_sync(0xffffffffu, c, 2), c11 = __shfl_sync(0xffffffffu, c, 3);
  const double u = lane == 1 ? dsub(c00, c11) : dadd(c00, c11);
  const double v = lane == 1 ? dadd(c01, c10) : dsub(c01, c10);
  const double norm = hyp_sum(u, v);
  const double e = __shfl_sync(0xffffffffu, norm, 0), f = __shfl_sync(0xffffffffu, norm, 1);
  const double quot = __ddiv_rn(lane == 0 ? u : (lane == 2 ? v : fmax(e, f)), lane == 3 ? variance : e);
  double cs = __shfl_sync(0xffffffffu, quot, 0), sn = __shfl_sync(0xffffffffu, quot, 2);
  if (!(e > 0.0)) {
    cs = 1.0;
    sn = 0.0;
  }
  const double scale = __shfl_sync(0xffffffffu, quot, 3);
  const double l00 = dmul(scale, cs), l01 = dmul(scale, -sn), l10 = dmul(scale, sn), l11 = dmul(scale, cs);
  m[0] = l00;
  m[1] = l01;
  m[2] = dsub(mrx, dadd(dmul(mmx, l00), dmul(mmy, l01)));
  m[3] = l10;
  m[4] = l11;
  m[5] = dsub(mry, dadd(dmul(mmx, l10), dmul(mmy, l11)));
  return true;
}

// Warp-cooperative affine fit of n <= 80 pairs: fit_affine's sums, one per
// lane (each in pair order).  Every lane returns the result.
__device__ bool warp_fit_affine(const double* mx, const double* my, const double* rx, const double* ry, int n,
                                double (&m)[6]) {
  const int lane = threadIdx.x & 31;
  if (n < 3) return false;
  double s = 0.0;
  if (lane < 4) {
    const double* v = lane == 0 ? mx : (lane == 1 ? my : (lane == 2 ? rx : ry));
    for (int i = 0; i < n; ++i) s = dadd(s, v[i]);
  }
  const double dn = static_cast<double>(n);
  AffineSums q{};
  q.mmx = __ddiv_rn(__shfl_sync(0xffffffffu, s, 0), dn);
  q.mmy = __ddiv_rn(__shfl_sync(0xffffffffu, s, 1), dn);
  q.mrx = __ddiv_rn(__shfl_sync(0xffffffffu, s, 2), dn);
  q.mry = __ddiv_rn(__shfl_sync(0xffffffffu, s, 3), dn);
  double c = 0.0;
  if (lane < 7) {
    // lane: 0 ax ax, 1 ax ay, 2 ay ay, 3 ax bx, 4 ay bx, 5 ax by, 6 ay by
    for (int i = 0; i < n; ++i) {
      const double ax = dsub(mx[i], q.mmx), ay = dsub(my[i], q.mmy);
      const double u = (lane == 0 || lane == 1 || lane == 3 || lane == 5) ? ax : ay;
      const double v = lane == 0 ? ax : (lane <= 2 ? ay : (lane <= 4 ? dsub(rx[i], q.mrx) : dsub(ry[i], q.mry)));
      c = dadd(c, dmul(u, v));
    }
  }
  q.sxx = __shfl_sync(0xffffffffu, c, 0);
  q.sxy = __shfl_sync(0xffffffffu, c, 1);
  q.syy = __shfl_sync(0xffffffffu, c, 2);
  q.sxr = __shfl_sync(0xffffffffu, c, 3);
  q.syr = __shfl_sync(0xffffffffu, c, 4);
  q.sxs = __shfl_sync(0xffffffffu, c, 5);
  q.sys = __shfl_sync(0xffffffffu, c, 6);
  return affine_from_sums(q, m);
}

// ---- K1: triangle descriptors, one CTA per catalog row ----------------------------------
__device__ __forceinline__ double row_x(const RegArgs& a, int row, int i) {
  return a.pts[(static_cast<int64_t>(row) * kRegPts + i) * 2];
}
__device__ __forceinline__ double row_y(const RegArgs& a, int row, int i) {
  return a.pts[(static_cast<int64_t>(row) * kRegPts + i) * 2 + 1];
}

// Bound by latency and, where float64 compares of the all-pairs loops were,
// by the float64 unit: those run on the order-preserving bits of the
// (non-negative) doubles, and all threads fill the distance matrix that the
// anchors search.  68 us for a catalog of 80 stars, 347 us before.
__global__ void __launch_bounds__(1024) reg_desc_kernel(RegArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  TriCand* tri = reinterpret_cast<TriCand*>(smem);
  unsigned long long* dist = reinterpret_cast<unsigned long long*>(smem);  // [n][n], before the triangles
  __shared__ double px[kRegPts], py[kRegPts];
  __shared__ int nb[kRegPts][kMaxNeighbors];
  __shared__ int combo[kMaxCombos][3];
  __shared__ __align__(16) int keys[kMaxTri];  // sorted vertex set, 7 bits per vertex
  __shared__ __align__(16) unsigned long long areas[kMaxTri];  // bits of a kept triangle's area, else 0
  __shared__ int s_kept;
  const int row = blockIdx.x;
  const int n = min(a.npts[row], a.max_stars);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    px[i] = row_x(a, row, i);
    py[i] = row_y(a, row, i);
  }
  const int k = min(n, max(3, a.neighbors));
  if (threadIdx.x == 0) {
    s_kept = 0;
    int c = 0;
    for (int i0 = 0; i0 < k; ++i0)
      for (int i1 = i0 + 1; i1 < k; ++i1)
        for (int i2 = i1 + 1; i2 < k; ++i2, ++c) {
          combo[c][0] = i0;
          combo[c][1] = i1;
          combo[c][2] = i2;
        }
  }
  __syncthreads();
  if (n < 3) {
    if (threadIdx.x == 0) a.ndesc[row] = 0;
    return;
  }
  for (int q = threadIdx.x; q < n * (n / 2 + 1); q += blockDim.x) {  // symmetric: j = i .. i + n / 2
    const int d = q / n, i = q - d * n, j = i + d < n ? i + d : i + d - n;
    const unsigned long long b = d == 0 ? 0ull : dbits_of(hyp_sum(dsub(px[j], px[i]), dsub(py[j], py[i])));
    dist[i * n + j] = b;
    dist[j * n + i] = b;
  }
  __syncthreads();
  // k nearest points of each anchor (the anchor itself first), index order on ties
  for (int an = threadIdx.x; an < n; an += blockDim.x) {
    unsigned long long bd[kMaxNeighbors];
    int bi[kMaxNeighbors];
#pragma unroll
    for (int q = 0; q < kMaxNeighbors; ++q) {
      bd[q] = ~0ull;
      bi[q] = 0;
    }
    for (int j = 0; j < n; ++j) {
      // insertion behind every entry that is not larger
      unsigned long long d = dist[an * n + j];
      int at = j;
      bool swap = false;
#pragma unroll
      for (int q = 0; q < kMaxNeighbors; ++q) {
        swap = swap || d < bd[q];
        const unsigned long long od = bd[q];
        const int oi = bi[q];
        bd[q] = swap ? d : od;
        bi[q] = swap ? at : oi;
        d = swap ? od : d;
        at = swap ? oi : at;
      }
    }
#pragma unroll
    for (int q = 0; q < kMaxNeighbors; ++q)
      if (q < k) nb[an][q] = bi[q];
  }
  __syncthreads();
  const int ncomb = k * (k - 1) * (k - 2) / 6;
  const int T = n * ncomb;
  for (int t = threadIdx.x; t < T; t += blockDim.x) {
    const int an = t / ncomb, c = t - (t / ncomb) * ncomb;
    const int r[3] = {nb[an][combo[c][0]], nb[an][combo[c][1]], nb[an][combo[c][2]]};
    int s0 = r[0], s1 = r[1], s2 = r[2];
    if (s0 > s1) { const int q = s0; s0 = s1; s1 = q; }
    if (s1 > s2) { const int q = s1; s1 = s2; s2 = q; }
    if (s0 > s1) { const int q = s0; s0 = s1; s1 = q; }
    TriCand tc;
    keys[t] = (s0 << 14) | (s1 << 7) | s2;
    tc.packed = 0;
    tc.d0 = tc.d1 = 0.0;
    const double ex = dsub(px[r[1]], px[r[0]]), ey = dsub(py[r[1]], py[r[0]]);
    const double fx = dsub(px[r[2]], px[r[0]]), fy = dsub(py[r[2]], py[r[0]]);
    tc.area = dmul(fabs(dsub(dmul(ex, fy), dmul(ey, fx))), 0.5);
    if (tc.area >= 2.0) {
      const int pa[3] = {0, 1, 2}, pb[3] = {1, 2, 0};
      double side[3];
      for (int q = 0; q < 3; ++q)
        side[q] = hyp_dot(dsub(px[r[pa[q]]], px[r[pb[q]]]), dsub(py[r[pa[q]]], py[r[pb[q]]]));
      double lo = side[0], mid = side[1], hi = side[2];
      if (lo > mid) { const double q = lo; lo = mid; mid = q; }
      if (mid > hi) { const double q = mid; mid = hi; hi = q; }
      if (lo > mid) { const double q = lo; lo = mid; mid = q; }
      if (lo > 1.0e-6 && mid > 1.0e-6) {
        int iarg = 0;  // first maximum
        for (int q = 1; q < 3; ++q)
          if (side[q] > side[iarg]) iarg = q;
        int first = pa[iarg], second = pb[iarg];
        const int third = 3 - first - second;
        const double dft = hyp_dot(dsub(px[r[first]], px[r[third]]), dsub(py[r[first]], py[r[third]]));
        const double dst = hyp_dot(dsub(px[r[second]], px[r[third]]), dsub(py[r[second]], py[r[third]]));
        if (dft < dst) {
          const int q = first;
          first = second;
          second = q;
        }
        tc.packed = static_cast<int>(0x80000000u |
                                     static_cast<unsigned>(r[first] | (r[second] << 7) | (r[third] << 14)));
        tc.d0 = __ddiv_rn(hi, mid);
        tc.d1 = __ddiv_rn(mid, lo);
      }
    }
    tri[t] = tc;
    areas[t] = 0ull;
  }
  __syncthreads();
  // keep the first occurrence of each vertex set (whatever its validity)
  for (int t = threadIdx.x; t < T; t += blockDim.x) {
    if (tri[t].packed >= 0) continue;
    const int key = keys[t];
    bool keep = true;
    int q = 0;
    for (; q + 4 <= t && keep; q += 4) {
      const int4 o = *reinterpret_cast<const int4*>(keys + q);
      keep = o.x != key && o.y != key && o.z != key && o.w != key;
    }
    for (; q < t && keep; ++q) keep = keys[q] != key;
    if (keep) areas[t] = dbits_of(tri[t].area);
  }
  __syncthreads();
  // stable area-descending rank
  for (int t = threadIdx.x; t < T; t += blockDim.x) {
    const unsigned long long ar = areas[t];
    if (ar == 0ull) continue;
    int rank = 0;
    int q = 0;
    for (; q + 2 <= t; q += 2) {
      const ulonglong2 o = *reinterpret_cast<const ulonglong2*>(areas + q);
      rank += (o.x >= ar ? 1 : 0) + (o.y >= ar ? 1 : 0);
    }
    if (q < t) rank += areas[q++] >= ar ? 1 : 0;
    for (; (q & 1) && q < T; ++q) rank += areas[q] > ar ? 1 : 0;
    for (; q + 2 <= T; q += 2) {
      const ulonglong2 o = *reinterpret_cast<const ulonglong2*>(areas + q);
      rank += (o.x > ar ? 1 : 0) + (o.y > ar ? 1 : 0);
    }
    if (q < T) rank += areas[q] > ar ? 1 : 0;
    if (rank < a.max_desc) {
      Desc d;
      d.d0 = tri[t].d0;
      d.d1 = tri[t].d1;
      d.area = tri[t].area;
      const int p = tri[t].packed;
      d.v[0] = p & 127;
      d.v[1] = (p >> 7) & 127;
      d.v[2] = (p >> 14) & 127;
      d.pad = 0;
      a.desc[static_cast<int64_t>(row) * kMaxDesc + rank] = d;
    }
    atomicAdd(&s_kept, 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) a.ndesc[row] = min(s_kept, a.max_desc);
}

// ---- K2: descriptor matches of a frame pair --------------------------------------------
// Descriptor distance of a moving and a reference descriptor; false when the
// pair is outside the radius.  `near` is the float32 bound per component
// (conversion error <= 2^-24 relative) that most pairs fail; a list compares
// the float32 distance itself.
struct MatchTest {
  double radius, bound;
  float radf;
  bool list_mode;
  __device__ __forceinline__ explicit MatchTest(const RegArgs& a)
      : radius(a.radius),
        bound(a.radius * 1.000001 + 1.0e-300),
        radf(static_cast<float>(a.radius) * 1.000001f + 1.0e-30f),
        list_mode(a.mode == kDescriptorList) {}
  __device__ __forceinline__ double list_distance(float2 rf, float2 mf) const {
    const float e0 = __fsub_rn(rf.x, mf.x);
    const float e1 = __fsub_rn(rf.y, mf.y);
    return static_cast<double>(sqrtf(__fadd_rn(__fmul_rn(e0, e0), __fmul_rn(e1, e1))));
  }
  __device__ __forceinline__ bool near(float2 rf, float2 mf) const {
    if (list_mode) return list_distance(rf, mf) <= radius;
    return !(fabsf(rf.x - mf.x) > radf + 3.0e-7f * (fabsf(rf.x) + fabsf(mf.x))) &&
           !(fabsf(rf.y - mf.y) > radf + 3.0e-7f * (fabsf(rf.y) + fabsf(mf.y)));
  }
  __device__ __forceinline__ bool within(double2 r, double2 m, double& d) const {
    if (list_mode) {
      d = list_distance(make_float2(static_cast<float>(r.x), static_cast<float>(r.y)),
                        make_float2(static_cast<float>(m.x), static_cast<float>(m.y)));
      return d <= radius;
    }
    const double e0 = dsub(r.x, m.x);
    if (fabs(e0) > bound) return false;
    const double e1 = dsub(r.y, m.y);
    if (fabs(e1) > bound) return false;
    d = hyp_sum(e0, e1);
    return d <= radius;
  }
};

__device__ __forceinline__ double2 desc_f64(const Desc& d) { return make_double2(d.d0, d.d1); }
__device__ __forceinline__ float2 desc_f32(const Desc& d) {
  return make_float2(static_cast<float>(d.d0), static_cast<float>(d.d1));
}

// All matches of a frame pair, several CTAs per pair: a warp per moving
// descriptor tests 32 reference descriptors at a time in float32 and collects
// the survivors, and evaluates the float64 distance when 32 of them are
// together: a warp pays for a float64 operation whether one lane or all need
// it, and a few per cent of the pairs survive.  Matches come in no order.
// Together with the selection 105 us for 32 pairs of about 500 descriptors,
// 606 us with one CTA per pair and the distance evaluated where the test
// passed.
constexpr int kPairWarps = 8;
constexpr int kPairCtas = 8;

__global__ void __launch_bounds__(32 * kPairWarps) reg_pairs_kernel(RegArgs a) {
  __shared__ float2 rdf[kMaxDesc];
  __shared__ int s_queue[kPairWarps][64];
  const int j = blockIdx.y;
  const RegJob job = a.jobs[j];
  const Desc* rd = a.desc + static_cast<int64_t>(job.ref_row) * kMaxDesc;
  const Desc* md = a.desc + static_cast<int64_t>(job.mov_row) * kMaxDesc;
  const int nr = a.ndesc[job.ref_row], nm = a.ndesc[job.mov_row];
  for (int i = threadIdx.x; i < nr; i += blockDim.x) rdf[i] = desc_f32(rd[i]);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int* queue = s_queue[warp];
  int queued = 0;  // the same in every lane
  const MatchTest test(a);
  double* mdist = a.match_dist + static_cast<int64_t>(j) * a.match_cap;
  int* mkey = a.match_key + static_cast<int64_t>(j) * a.match_cap;
  auto drain = [&](int n) {  // the first n <= 32 queued pairs
    const int q = lane < n ? queue[lane] : 0;
    double d = 0.0;
    const bool in = lane < n && test.within(desc_f64(rd[q % nr]), desc_f64(md[q / nr]), d);
    const unsigned mask = __ballot_sync(0xffffffffu, in);
    int base = 0;
    if (lane == 0 && mask) base = atomicAdd(a.match_count + j, __popc(mask));
    base = __shfl_sync(0xffffffffu, base, 0);
    const int pos = base + __popc(mask & ((1u << lane) - 1u));
    if (in && pos < a.match_cap) {
      mdist[pos] = d;
      mkey[pos] = q;
    }
  };
  for (int mi = blockIdx.x * kPairWarps + warp; mi < nm; mi += gridDim.x * kPairWarps) {
    const float2 mf = desc_f32(md[mi]);
    for (int base = 0; base < nr; base += 32) {
      const int ri = base + lane;
      const bool near = ri < nr && test.near(rdf[min(ri, nr - 1)], mf);
      const unsigned mask = __ballot_sync(0xffffffffu, near);
      if (near) queue[queued + __popc(mask & ((1u << lane) - 1u))] = mi * nr + ri;
      queued += __popc(mask);
      __syncwarp();
      if (queued >= 32) {
        drain(32);
        const int rest = queued > 32 + lane ? queue[32 + lane] : 0;
        __syncwarp();
        queue[lane] = rest;
        queued -= 32;
        __syncwarp();
      }
    }
  }
  if (queued) drain(queued);
}

struct SelEntry {
  unsigned long long d;  // order-preserving bits of the distance
  int key;
  int pad;
};

// The max_candidates best matches in order, one CTA per frame pair.
__global__ void __launch_bounds__(1024) reg_match_kernel(RegArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  double2* rdd = reinterpret_cast<double2*>(smem);         // [kMaxDesc] descriptors, for more matches than
  double2* mdd = rdd + kMaxDesc;                           // [kMaxDesc] the list holds
  float2* rdf = reinterpret_cast<float2*>(mdd + kMaxDesc); // [kMaxDesc]
  float2* mdf = rdf + kMaxDesc;                            // [kMaxDesc]
  __shared__ __align__(16) SelEntry sel[kMaxSel];
  __shared__ int s_c, s_n;
  __shared__ unsigned s_hist[256];
  __shared__ unsigned long long s_prefix;
  __shared__ int s_rank, s_eq;
  const int j = blockIdx.x;
  const RegJob job = a.jobs[j];
  const Desc* rd = a.desc + static_cast<int64_t>(job.ref_row) * kMaxDesc;
  const Desc* md = a.desc + static_cast<int64_t>(job.mov_row) * kMaxDesc;
  const int nr = a.ndesc[job.ref_row], nm = a.ndesc[job.mov_row];
  const double* mdist = a.match_dist + static_cast<int64_t>(j) * a.match_cap;
  const int* mkey = a.match_key + static_cast<int64_t>(j) * a.match_cap;
  const int total = nm * nr;
  const double radius = a.radius;
  const MatchTest test(a);
  auto match_dist = [&](int q, double& d) -> bool {
    const int mi = q / nr, ri = q - mi * nr;
    return test.near(rdf[ri], mdf[mi]) && test.within(rdd[ri], mdd[mi], d);
  };
  const int n = a.match_count[j];
  const bool stored_all = n <= a.match_cap;
  int2* out = a.sel + static_cast<int64_t>(j) * a.sel_cap;
  long long* out_order = a.sel_order + static_cast<int64_t>(j) * a.sel_cap;
  if (test.list_mode) {
    // every match is a candidate; order = reference-major enumeration index
    const bool fits = stored_all && n <= a.sel_cap;
    if (fits) {
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int q = mkey[i];
        const int mi = q / nr, ri = q - (q / nr) * nr;
        out[i] = make_int2(mi, ri);
        out_order[i] = static_cast<long long>(ri) * nm + mi;
      }
    }
    if (threadIdx.x == 0) {
      if (!fits) atomicExch(a.overflow, 1);
      a.nsel[j] = fits ? n : 0;
      a.out[j].matches = n;
      a.out[j].ndesc_ref = nr;
      a.out[j].ndesc_mov = nm;
    }
    return;
  }
  if (!stored_all) {
    for (int i = threadIdx.x; i < nr; i += blockDim.x) {
      rdd[i] = desc_f64(rd[i]);
      rdf[i] = desc_f32(rd[i]);
    }
    for (int i = threadIdx.x; i < nm; i += blockDim.x) {
      mdd[i] = desc_f64(md[i]);
      mdf[i] = desc_f32(md[i]);
    }
    __syncthreads();
  }
  // block-wide count of matches satisfying pred(distance bits, flat index)
  auto block_count = [&](auto pred) -> int {
    int c = 0;
    if (stored_all) {
      for (int q = threadIdx.x; q < n; q += blockDim.x) c += pred(dbits_of(mdist[q]), mkey[q]) ? 1 : 0;
    } else {
      for (int q = threadIdx.x; q < total; q += blockDim.x) {
        double d;
        if (match_dist(q, d)) c += pred(dbits_of(d), q) ? 1 : 0;
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) s_c = 0;
    __syncthreads();
    if (c) atomicAdd(&s_c, c);
    __syncthreads();
    const int r = s_c;
    __syncthreads();
    return r;
  };
  const int take = min(n, a.max_cand);
  // the take smallest (distance, index) pairs: distance threshold t, then the
  // index threshold K among the matches at exactly distance t
  unsigned long long t = dbits_of(radius);
  int K = total;
  if (take == 0) {
    t = 0ull;
    K = -1;  // keeps nothing: distances are never below +0
  } else if (take < n) {
    int need = 0, equal = 0;
    if (stored_all) {
      // radix select (8-bit digits, most significant first) of the
      // (take - 1)-th smallest distance among the stored matches
      unsigned long long prefix = 0ull, mask = 0ull;
      int rank = take - 1;
      for (int shift = 56; shift >= 0; shift -= 8) {
        for (int i = threadIdx.x; i < 256; i += blockDim.x) s_hist[i] = 0u;
        __syncthreads();
#pragma unroll 4
        for (int q = threadIdx.x; q < n; q += blockDim.x) {
          const unsigned long long k = dbits_of(mdist[q]);
          if ((k & mask) == prefix) atomicAdd(&s_hist[(k >> shift) & 255u], 1u);
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
          const bool here = excl <= static_cast<unsigned>(rank) && static_cast<unsigned>(rank) < incl;
          if (here) {
            unsigned r = static_cast<unsigned>(rank) - excl;
            int b = lane * 8;
            while (r >= s_hist[b]) {
              r -= s_hist[b];
              ++b;
            }
            s_prefix = prefix | (static_cast<unsigned long long>(b) << shift);
            s_rank = static_cast<int>(r);
            s_eq = static_cast<int>(s_hist[b]);
          }
        }
        __syncthreads();
        prefix = s_prefix;
        rank = s_rank;
        mask |= 0xffull << shift;
        __syncthreads();
      }
      t = prefix;
      need = rank + 1;  // entries at exactly distance t to keep
      equal = s_eq;     // entries at exactly distance t
    } else {
      unsigned long long lo = 0ull, hi = dbits_of(radius);
      while (lo < hi) {
        const unsigned long long mid = lo + (hi - lo) / 2;
        if (block_count([&](unsigned long long b, int) { return b <= mid; }) >= take) hi = mid;
        else lo = mid + 1;
      }
      t = lo;
      const int below = t == 0 ? 0 : block_count([&](unsigned long long b, int) { return b < t; });
      need = take - below;
      equal = block_count([&](unsigned long long b, int) { return b == t; });
    }
    if (need < equal) {  // ties at the cut: the smallest flat indices win
      int klo = 0, khi = total - 1;
      while (klo < khi) {
        const int mid = klo + (khi - klo) / 2;
        if (block_count([&](unsigned long long b, int q) { return b == t && q <= mid; }) >= need) khi = mid;
        else klo = mid + 1;
      }
      K = klo;
    }
  }
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  auto keep = [&](unsigned long long b, int q) { return b < t || (b == t && q <= K); };
  if (stored_all) {
    for (int q = threadIdx.x; q < n; q += blockDim.x) {
      if (keep(dbits_of(mdist[q]), mkey[q])) {
        const int p = atomicAdd(&s_n, 1);
        if (p < kMaxSel) sel[p] = {dbits_of(mdist[q]), mkey[q], 0};
      }
    }
  } else {
    for (int q = threadIdx.x; q < total; q += blockDim.x) {
      double d;
      if (match_dist(q, d) && keep(dbits_of(d), q)) {
        const int p = atomicAdd(&s_n, 1);
        if (p < kMaxSel) sel[p] = {dbits_of(d), q, 0};
      }
    }
  }
  __syncthreads();
  const int ns = min(s_n, kMaxSel);
  int m = 1;
  while (m < ns) m <<= 1;
  for (int i = ns + threadIdx.x; i < m; i += blockDim.x)
    sel[i] = {~0ull, 0x7fffffff, 0};
  __syncthreads();
  for (int size = 2; size <= m; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const int jj = i ^ stride;
        if (jj > i) {
          const bool up = (i & size) == 0;
          const SelEntry si = sel[i], sj = sel[jj];
          const bool gt = si.d > sj.d || (si.d == sj.d && si.key > sj.key);
          if (gt == up) {
            sel[i] = sj;
            sel[jj] = si;
          }
        }
      }
      __syncthreads();
    }
  }
  for (int i = threadIdx.x; i < ns; i += blockDim.x) {
    const int q = sel[i].key;
    out[i] = make_int2(q / nr, q - (q / nr) * nr);
    out_order[i] = i;
  }
  if (threadIdx.x == 0) {
    a.nsel[j] = ns;
    a.out[j].matches = ns;
    a.out[j].ndesc_ref = nr;
    a.out[j].ndesc_mov = nm;
  }
}

// ---- K3: candidate transforms ---------------------------------------------------------
// Loads the two catalogs of a job and buckets the reference stars (block-wide;
// the caller synchronises afterwards).
__device__ void load_job_points(const RegArgs& a, const RegJob& job, JobPoints& jp, double tol) {
  const int nm = min(a.npts[job.mov_row], a.max_stars);
  const int nr = min(a.npts[job.ref_row], a.max_stars);
  for (int i = threadIdx.x; i < kRegPts; i += blockDim.x) {
    if (i < nm) {
      jp.mx[i] = row_x(a, job.mov_row, i);
      jp.my[i] = row_y(a, job.mov_row, i);
      jp.mx32[i] = static_cast<float>(jp.mx[i]);
      jp.my32[i] = static_cast<float>(jp.my[i]);
    }
    if (i < nr) {
      jp.rx[i] = row_x(a, job.ref_row, i);
      jp.ry[i] = row_y(a, job.ref_row, i);
      jp.rx32[i] = static_cast<float>(jp.rx[i]);
      jp.ry32[i] = static_cast<float>(jp.ry[i]);
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) {  // extents, by one warp
    const int lane = threadIdx.x;
    float cmax = 0.0f, rmax = 0.0f;
    for (int i = lane; i < nm; i += 32) cmax = fmaxf(cmax, fabsf(jp.mx32[i]) + fabsf(jp.my32[i]));
    float x0 = 3.0e38f, x1 = -3.0e38f, y0 = 3.0e38f, y1 = -3.0e38f;
    for (int i = lane; i < nr; i += 32) {
      x0 = fminf(x0, jp.rx32[i]);
      x1 = fmaxf(x1, jp.rx32[i]);
      y0 = fminf(y0, jp.ry32[i]);
      y1 = fmaxf(y1, jp.ry32[i]);
      rmax = fmaxf(rmax, fmaxf(fabsf(jp.rx32[i]), fabsf(jp.ry32[i])));
    }
    for (int off = 16; off > 0; off >>= 1) {
      cmax = fmaxf(cmax, __shfl_xor_sync(0xffffffffu, cmax, off));
      rmax = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, off));
      x0 = fminf(x0, __shfl_xor_sync(0xffffffffu, x0, off));
      x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, off));
      y0 = fminf(y0, __shfl_xor_sync(0xffffffffu, y0, off));
      y1 = fmaxf(y1, __shfl_xor_sync(0xffffffffu, y1, off));
    }
    if (lane == 0) {
      jp.nm = nm;
      jp.nr = nr;
      jp.cmax = cmax * 1.0001f + 1.0f;
      jp.rmax = rmax * 1.0001f + 1.0f;
      jp.partners = 0;
      jp.gnx = jp.gny = 0;
      jp.gx0 = jp.gy0 = 0.0f;
      jp.ginv = 1.0f;
      if (nr > 0) {
        // cells at least 2 * (tol + 0.5) wide (> the widest search radius) so
        // a search touches <= 2 x 2 cells
        const float reach = static_cast<float>(2.0 * (tol + 0.5)) + 1.0f;
        const float cell = fmaxf(fmaxf(x1 - x0, y1 - y0) / static_cast<float>(kGrid), reach);
        jp.gx0 = x0;
        jp.gy0 = y0;
        if (cell < 1.0e30f) {
          jp.ginv = 1.0f / cell;
          jp.gnx = min(kGrid, static_cast<int>((x1 - x0) * jp.ginv) + 1);
          jp.gny = min(kGrid, static_cast<int>((y1 - y0) * jp.ginv) + 1);
        } else {  // one cell holding every star
          jp.ginv = 0.0f;
          jp.gnx = jp.gny = 1;
        }
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nr; i += blockDim.x) {
    const int cx = min(jp.gnx - 1, max(0, static_cast<int>((jp.rx32[i] - jp.gx0) * jp.ginv)));
    const int cy = min(jp.gny - 1, max(0, static_cast<int>((jp.ry32[i] - jp.gy0) * jp.ginv)));
    jp.cell_of[i] = static_cast<unsigned char>(cy * kGrid + cx);
  }
  __syncthreads();
  // counting sort by cell, in index order inside a cell; stars within reach of
  // one point are within twice the reach (tol + 0.5 at most, see
  // can_leave_early) of each other
  const float near = 2.0f * static_cast<float>(tol + 0.5) * 1.001f + 1.0e-6f * jp.rmax;
  for (int i = threadIdx.x; i < nr; i += blockDim.x) {
    const int cell = jp.cell_of[i];
    const float x = jp.rx32[i], y = jp.ry32[i];
    int pos = 0, close = 0;
    for (int q = 0; q < nr; ++q) {
      pos += (jp.cell_of[q] < cell || (jp.cell_of[q] == cell && q < i)) ? 1 : 0;
      close += (fabsf(jp.rx32[q] - x) <= near && fabsf(jp.ry32[q] - y) <= near) ? 1 : 0;
    }
    jp.cell_pt[pos] = static_cast<unsigned char>(i);
    atomicMax(&jp.partners, close);
  }
  for (int c = threadIdx.x; c <= kGrid * kGrid; c += blockDim.x) {
    int start = 0;
    for (int q = 0; q < nr; ++q) start += jp.cell_of[q] < c ? 1 : 0;
    jp.cell_start[c] = static_cast<unsigned char>(start);
  }
}

constexpr int kScoreWarps = 4;

// Fits one candidate per lane, then the warp counts the pairs of one after the
// other.  The float64 work is what a warp can do for 32 candidates at once (the
// fit, the error bounds) and what the float32 test leaves open; residuals in
// float64 are for the candidates that can still win (reg_rms_kernel), and a
// candidate that falls behind the best count known is dropped.  32 pairs
// of frames: 158 us, 114 us for the conflicts and 45 us for the residuals; 946 us
// with exact scores on the spot, float64 residuals
// and bounds for every candidate.
template <int MODEL>
__global__ void __launch_bounds__(32 * kScoreWarps) reg_score_kernel(RegArgs a) {
  __shared__ JobPoints jp;
  __shared__ unsigned used_r[kScoreWarps][3];
  __shared__ double cm[kScoreWarps][32][6];
  __shared__ FastTransform cf[kScoreWarps][32];
  __shared__ int cok[kScoreWarps][32];
  const int j = blockIdx.y;
  const RegJob job = a.jobs[j];
  load_job_points(a, job, jp, a.tol);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ncand = 2 * a.nsel[j];
  const Desc* rd = a.desc + static_cast<int64_t>(job.ref_row) * kMaxDesc;
  const Desc* md = a.desc + static_cast<int64_t>(job.mov_row) * kMaxDesc;
  const int2* sel = a.sel + static_cast<int64_t>(j) * a.sel_cap;
  const long long* order = a.sel_order + static_cast<int64_t>(j) * a.sel_cap;
  Cand* cands = a.cands + static_cast<int64_t>(j) * 2 * a.sel_cap;
  CandRank* ranks = a.ranks + static_cast<int64_t>(j) * 2 * a.sel_cap;
  for (int base = (blockIdx.x * kScoreWarps + warp) * 32; base < ncand; base += gridDim.x * kScoreWarps * 32) {
    // one 3-point fit per lane
    const int c = base + lane;
    int ok = 0;
    if (c < ncand) {
      const int2 s = sel[c >> 1];
      const Desc dm = md[s.x], dr = rd[s.y];
      int rv0 = dr.v[0], rv1 = dr.v[1];
      if (c & 1) {  // reference triangle in the order [1, 0, 2]
        const int q = rv0;
        rv0 = rv1;
        rv1 = q;
      }
      const double tmx[3] = {jp.mx[dm.v[0]], jp.mx[dm.v[1]], jp.mx[dm.v[2]]};
      const double tmy[3] = {jp.my[dm.v[0]], jp.my[dm.v[1]], jp.my[dm.v[2]]};
      const double trx[3] = {jp.rx[rv0], jp.rx[rv1], jp.rx[dr.v[2]]};
      const double try_[3] = {jp.ry[rv0], jp.ry[rv1], jp.ry[dr.v[2]]};
      double scratch[6];
      double m[6];
      if constexpr (MODEL == GG_TRANSFORM_AFFINE)
        ok = fit_affine(tmx, tmy, trx, try_, 3, m) ? 1 : 0;
      else
        ok = fit_similarity(tmx, tmy, trx, try_, 3, scratch, m) ? 1 : 0;
      Cand& cd = cands[c];
      for (int q = 0; q < 6; ++q) {
        cm[warp][lane][q] = ok ? m[q] : 0.0;
        cd.m[q] = ok ? m[q] : 0.0;
      }
      cd.order = 2 * order[c >> 1] + (c & 1);
      if (ok) cf[warp][lane] = fast_transform(m, jp, a.tol);
    }
    cok[warp][lane] = ok;
    __syncwarp();
    // score the chunk one candidate at a time with the whole warp
    const int nb = min(32, ncand - base);
    int my_count = -1;  // of the lane's candidate
    float my_sum = 0.0f;
    int best = __shfl_sync(0xffffffffu, __ldcg(a.best_count + j), 0);  // whatever other warps have found by now
    for (int t = 0; t < nb; ++t) {
      if (!cok[warp][t]) continue;
      int count;
      float sum;
      bool conflict;
      warp_score_count(cf[warp][t], cm[warp][t], jp, a.tol, can_leave_early(jp, a.tol, cf[warp][t].r) ? best : 0,
                       used_r[warp], count, sum, conflict);
      if (!conflict && count > best) {
        best = count;
        if (lane == 0) atomicMax(a.best_count + j, count);
      }
      if (lane == t) {
        my_count = conflict ? kConflictCount - count : count;
        my_sum = sum;
      }
    }
    if (c < ncand) {
      // bounds of the rms: every distance is known to delta, the sum to 80 roundings
      const float rms32 = sqrtf(my_sum / static_cast<float>(max(my_count, 1)));
      const float delta = ok ? cf[warp][lane].delta : 0.0f;
      ranks[c] = {my_count, (rms32 - delta) * 0.99999f, (rms32 + delta) * 1.00001f};
      cands[c].rms = __longlong_as_double(0x7ff0000000000000ll);
      cands[c].scored = 0;
    }
    __syncwarp();
  }
}

// ---- the candidates that can win ------------------------------------------------------
// The most pairs of any candidate and the smallest upper bound of an rms among
// those; block-wide, the same in every thread.
struct WinBound {
  int count;
  float rms;
};

__device__ WinBound win_bound(const CandRank* ranks, int ncand) {
  __shared__ int s_count;
  __shared__ int s_rms;  // non-negative floats compare as integers
  if (threadIdx.x == 0) {
    s_count = 0;
    s_rms = 0x7f800000;
  }
  __syncthreads();
  int bn = 0;
#pragma unroll 4
  for (int c = threadIdx.x; c < ncand; c += blockDim.x) bn = max(bn, ranks[c].count);
  bn = __reduce_max_sync(0xffffffffu, bn);
  if ((threadIdx.x & 31) == 0) atomicMax(&s_count, bn);
  __syncthreads();
  bn = s_count;
  int hi = 0x7f800000;
#pragma unroll 4
  for (int c = threadIdx.x; c < ncand; c += blockDim.x) {
    const CandRank r = ranks[c];
    if (r.count == bn && r.rms_hi >= 0.0f) hi = min(hi, __float_as_int(r.rms_hi));
  }
  hi = __reduce_min_sync(0xffffffffu, hi);
  if ((threadIdx.x & 31) == 0) atomicMin(&s_rms, hi);
  __syncthreads();
  return {bn, __int_as_float(s_rms)};
}

__device__ __forceinline__ bool can_win(const CandRank& r, const WinBound& b) {
  return b.count > 0 && r.count == b.count && !(r.rms_lo > b.rms);
}

// Counts of the candidates in which a star has two partners, where they may
// still reach the best count.  A kernel of its own: where two stars stand close
// together that is every good candidate of a frame pair, next to each other in
// the order of the candidates (the two orientations of a match take turns:
// the number of warps they are dealt to is odd).
constexpr int kRecheckCtas = 16;

__global__ void __launch_bounds__(32 * kScoreWarps) reg_exact_kernel(RegArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  WarpScratch* ws = reinterpret_cast<WarpScratch*>(smem);
  __shared__ JobPoints jp;
  const int j = blockIdx.y;
  const RegJob job = a.jobs[j];
  const int ncand = 2 * a.nsel[j];
  CandRank* ranks = a.ranks + static_cast<int64_t>(j) * 2 * a.sel_cap;
  Cand* cands = a.cands + static_cast<int64_t>(j) * 2 * a.sel_cap;
  load_job_points(a, job, jp, a.tol);
  __syncthreads();
  const int best = a.best_count[j];
  const int lane = threadIdx.x & 31, warp = blockIdx.x * kScoreWarps + (threadIdx.x >> 5);
  const int nwarps = static_cast<int>(gridDim.x * kScoreWarps - 1u) | 1;  // odd
  if (warp >= nwarps) return;
  for (int base = warp; base < ncand; base += 32 * nwarps) {
    const int c = base + lane * nwarps;
    const int count = c < ncand ? ranks[c].count : -1;
    bool check = count <= kConflictCount;
    if (check && kConflictCount - count < best) {
      double m[6];
      for (int q = 0; q < 6; ++q) m[q] = cands[c].m[q];
      check = !can_leave_early(jp, a.tol, fast_transform(m, jp, a.tol).r);
    }
    unsigned todo = __ballot_sync(0xffffffffu, check);
    while (todo) {
      const int t = base + (__ffs(todo) - 1) * nwarps;
      todo &= todo - 1u;
      double m[6];
      for (int q = 0; q < 6; ++q) m[q] = cands[t].m[q];
      int n;
      double rms;
      const bool resolved = warp_resolve(m, jp, a.tol, ws[threadIdx.x >> 5], n, rms);
      if (!resolved) score_exact<WarpGroup>(m, jp, a.tol, ws[threadIdx.x >> 5], n, rms, nullptr, a.overflow);
      if (lane == 0) {
        const float rms32 = static_cast<float>(rms);
        ranks[t] = {n, rms32 * 0.99999f, rms32 * 1.00001f};
        cands[t].rms = rms;
        cands[t].scored = resolved ? 2 : 1;
      }
    }
  }
}

// float64 rms of the candidates that can win (a warp takes every nwarps-th
// candidate: the likely ones stand together).
__global__ void __launch_bounds__(32 * kScoreWarps) reg_rms_kernel(RegArgs a) {
  __shared__ JobPoints jp;
  __shared__ double own_m[kScoreWarps][32][6];
  __shared__ FastTransform own_t[kScoreWarps][32];
  const int j = blockIdx.y;
  const RegJob job = a.jobs[j];
  const int ncand = 2 * a.nsel[j];
  const CandRank* ranks = a.ranks + static_cast<int64_t>(j) * 2 * a.sel_cap;
  Cand* cands = a.cands + static_cast<int64_t>(j) * 2 * a.sel_cap;
  load_job_points(a, job, jp, a.tol);
  const WinBound bound = win_bound(ranks, ncand);
  const int lane = threadIdx.x & 31, warp = blockIdx.x * kScoreWarps + (threadIdx.x >> 5);
  const int nwarps = gridDim.x * kScoreWarps;
  for (int base = warp; base < ncand; base += 32 * nwarps) {
    const int c = base + lane * nwarps;
    unsigned todo = __ballot_sync(0xffffffffu, c < ncand && can_win(ranks[min(c, ncand - 1)], bound) &&
                                                   cands[min(c, ncand - 1)].scored == 0);
    double own_sum = 0.0;
    const bool mine = (todo >> lane) & 1u;
    if (mine) {
      double m[6];
      for (int q = 0; q < 6; ++q) m[q] = cands[c].m[q];
      for (int q = 0; q < 6; ++q) own_m[threadIdx.x >> 5][lane][q] = m[q];
      own_t[threadIdx.x >> 5][lane] = fast_transform(m, jp, a.tol);
    }
    __syncwarp();
    while (todo) {
      const int t = __ffs(todo) - 1;
      todo &= todo - 1u;
      double m[6];
      for (int q = 0; q < 6; ++q) m[q] = own_m[threadIdx.x >> 5][t][q];
      const double sum = warp_sum_d2(m, own_t[threadIdx.x >> 5][t], jp, a.tol);
      if (lane == t) own_sum = sum;
    }
    if (mine) cands[c].rms = sqrt(__ddiv_rn(own_sum, static_cast<double>(bound.count)));
    __syncwarp();
  }
}

// ---- K4: best candidate and guarded refits, one CTA per frame pair ---------------------
// The reference keeps the first candidate with the most pairs and, among
// those, the smallest rms.  Counts are exact for every candidate; the fast
// rms differs from the exact one by < 1e-13 relative, so every candidate that
// can win lies in the window rms <= min * (1 + 1e-12) and only those are
// re-scored exactly (usually one).  Bound by the chain of scores and refits
// (float64 sums in NumPy's order): 134 us with the whole CTA on the search and
// the scores, 320 us by one warp.
constexpr int kWindowCap = 1024;
constexpr int kBestThreads = 256;

__global__ void __launch_bounds__(kBestThreads) reg_best_kernel(RegArgs a) {
  __shared__ JobPoints jp;
  __shared__ WarpScratch ws;
  __shared__ double fx[kRegPts], fy[kRegPts], gx[kRegPts], gy[kRegPts], buf[4 * kRegPts];
  __shared__ short2 prs[kRegPts], prs2[kRegPts];
  __shared__ int window[kWindowCap];
  __shared__ unsigned long long s_min;
  __shared__ double s_m[6];
  __shared__ int s_nw, s_fitted;
  const int j = blockIdx.x;
  const int lane = threadIdx.x;
  const RegJob job = a.jobs[j];
  load_job_points(a, job, jp, a.tol);
  const double inf = __longlong_as_double(0x7ff0000000000000ll);
  if (threadIdx.x == 0) {
    s_min = dbits_of(inf);
    s_nw = 0;
  }
  const int ncand = 2 * a.nsel[j];
  const Cand* cs = a.cands + static_cast<int64_t>(j) * 2 * a.sel_cap;
  const CandRank* ranks = a.ranks + static_cast<int64_t>(j) * 2 * a.sel_cap;
  const WinBound bound = win_bound(ranks, ncand);
  // smallest (fast) rms of the candidates with the most pairs
  for (int c = threadIdx.x; c < ncand; c += kBestThreads)
    if (can_win(ranks[c], bound) && cs[c].rms < inf) atomicMin(&s_min, dbits_of(cs[c].rms));
  __syncthreads();
  const double rmin = __longlong_as_double(static_cast<long long>(s_min));
  const double thr = rmin + rmin * 1.0e-12;
  // window members
  for (int c = threadIdx.x; c < ncand; c += kBestThreads)
    if (can_win(ranks[c], bound) && cs[c].rms <= thr) {
      const int pos = atomicAdd(&s_nw, 1);
      if (pos < kWindowCap) window[pos] = c;
    }
  __syncthreads();
  int nw = s_nw;
  if (nw > kWindowCap) {
    if (threadIdx.x == 0) atomicExch(a.overflow, 1);
    nw = kWindowCap;
  }
  using Cta = CtaGroup<kBestThreads>;
  // exact rms of the window members: smallest wins, earliest order on ties
  int bc = -1;
  double br = inf;
  long long bo = -1;
  for (int w = 0; w < nw; ++w) {
    const int c = window[w];
    double r = cs[c].rms;
    if (cs[c].scored != 1 && nw > 1) {  // a single member wins as it is
      double m[6];
      for (int q = 0; q < 6; ++q) m[q] = cs[c].m[q];
      int n;
      score_exact<Cta>(m, jp, a.tol, ws, n, r, nullptr, a.overflow);
    }
    const long long o = cs[c].order;
    if (bc < 0 || r < br || (r == br && o < bo)) {
      bc = c;
      br = r;
      bo = o;
    }
  }
  double best[6] = {1.0, 0.0, 0.0, 0.0, 1.0, 0.0};
  int best_n = 0;
  double best_rms = inf;
  if (bc >= 0) {
    for (int q = 0; q < 6; ++q) best[q] = cs[bc].m[q];
    score_exact<Cta>(best, jp, a.tol, ws, best_n, best_rms, prs, a.overflow);
  }
  const int iterations = a.mode == kEstimator ? 3 : 0;
  for (int it = 0; it < iterations; ++it) {
    if (best_n < 3) break;
    for (int q = threadIdx.x; q < best_n; q += kBestThreads) {
      fx[q] = jp.mx[prs[q].x];
      fy[q] = jp.my[prs[q].x];
      gx[q] = jp.rx[prs[q].y];
      gy[q] = jp.ry[prs[q].y];
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      double m[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
      const bool fitted = a.model == GG_TRANSFORM_AFFINE ? warp_fit_affine(fx, fy, gx, gy, best_n, m)
                                                         : warp_fit_similarity(fx, fy, gx, gy, best_n, buf, m);
      if (lane == 0) {
        s_fitted = fitted ? 1 : 0;
        for (int q = 0; q < 6; ++q) s_m[q] = m[q];
      }
    }
    __syncthreads();
    if (!s_fitted) break;
    double m[6];
    for (int q = 0; q < 6; ++q) m[q] = s_m[q];
    int n2;
    double r2;
    score_exact<Cta>(m, jp, a.tol, ws, n2, r2, prs2, a.overflow);
    if (n2 > best_n || (n2 == best_n && r2 <= best_rms)) {
      for (int q = 0; q < 6; ++q) best[q] = m[q];
      for (int q = threadIdx.x; q < n2; q += kBestThreads) prs[q] = prs2[q];
      best_n = n2;
      best_rms = r2;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    RegResult& r = a.out[j];
    for (int q = 0; q < 6; ++q) r.m[q] = best[q];
    r.m[6] = 0.0;
    r.m[7] = 0.0;
    r.m[8] = 1.0;
    r.rms = best_rms;
    r.best_order = bo;
    r.inliers = best_n;
    r.status = a.mode == kEstimator ? (best_n >= a.min_inliers ? 1 : 0) : (best_n > 0 ? 1 : 0);
  }
  for (int q = threadIdx.x; q < kRegPts; q += kBestThreads)
    a.pairs[static_cast<int64_t>(j) * kRegPts + q] = q < best_n ? prs[q] : make_short2(-1, -1);
}

__global__ void reg_copy_catalogs_kernel(const double* cat_xy, const int* cat_n, const int* row_frames, int rows,
                                         double* pts, int* npts) {
  const int row = blockIdx.x;
  if (row >= rows) return;
  const int f = row_frames[row];
  for (int i = threadIdx.x; i < kRegPts * 2; i += blockDim.x)
    pts[static_cast<int64_t>(row) * kRegPts * 2 + i] = cat_xy[static_cast<int64_t>(f) * kRegPts * 2 + i];
  if (threadIdx.x == 0) npts[row] = cat_n[f];
}

// ---- host side ------------------------------------------------------------------
struct RegScratch {
  double* pts = nullptr;
  int* npts = nullptr;
  Desc* desc = nullptr;
  int* ndesc = nullptr;
  RegJob* jobs = nullptr;
  int* row_frames = nullptr;
  int* match_count = nullptr;
  double* match_dist = nullptr;
  int* match_key = nullptr;
  int2* sel = nullptr;
  long long* sel_order = nullptr;
  int* nsel = nullptr;
  Cand* cands = nullptr;
  CandRank* ranks = nullptr;
  RegResult* out = nullptr;
  short2* pairs = nullptr;
  int* overflow = nullptr;
  int rows = 0;
  int jobs_cap = 0;
  int match_cap = 0;
  int sel_cap = 0;
  int device = -1;
};

static void reg_scratch_release(RegScratch& r) {
  void* ps[] = {r.pts, r.npts,      r.desc, r.ndesc, r.jobs,  r.row_frames, r.match_count, r.match_dist, r.match_key,
                r.sel, r.sel_order, r.nsel, r.cands, r.ranks, r.out,        r.pairs,       r.overflow};
  for (void* p : ps)
    if (p) cudaFree(p);
  r = RegScratch{};
}

static int64_t reg_scratch_bytes(const RegScratch& r) {
  if (r.device < 0) return 0;
  const int64_t R = r.rows, J = r.jobs_cap, M = r.match_cap, S = r.sel_cap;
  return R * (16 * kRegPts + 12 + static_cast<int64_t>(sizeof(Desc)) * kMaxDesc) +
         J * (8 + 8 + 12 * M + 16 * S + 4 + 2 * static_cast<int64_t>(sizeof(Cand) + sizeof(CandRank)) * S +
              static_cast<int64_t>(sizeof(RegResult)) + 4 * kRegPts) +
         4;
}

static void reg_scratch_ensure(RegScratch& r, int rows, int jobs, int match_cap, int sel_cap) {
  int dev = 0;
  check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
  if (r.device == dev && r.rows >= rows && r.jobs_cap >= jobs && r.match_cap >= match_cap && r.sel_cap >= sel_cap)
    return;
  if (r.device == dev) {
    rows = std::max(rows, r.rows);
    jobs = std::max(jobs, r.jobs_cap);
    match_cap = std::max(match_cap, r.match_cap);
    sel_cap = std::max(sel_cap, r.sel_cap);
  }
  reg_scratch_release(r);
  const size_t R = static_cast<size_t>(rows), J = static_cast<size_t>(jobs);
  const size_t M = static_cast<size_t>(match_cap), S = static_cast<size_t>(sel_cap);
  check_cuda(cudaMalloc(&r.pts, sizeof(double) * 2 * kRegPts * R), "cudaMalloc(registration points)");
  check_cuda(cudaMalloc(&r.npts, sizeof(int) * R), "cudaMalloc(registration counts)");
  check_cuda(cudaMalloc(&r.desc, sizeof(Desc) * kMaxDesc * R), "cudaMalloc(registration descriptors)");
  check_cuda(cudaMalloc(&r.ndesc, sizeof(int) * R), "cudaMalloc(registration descriptor counts)");
  check_cuda(cudaMalloc(&r.row_frames, sizeof(int) * R), "cudaMalloc(registration rows)");
  check_cuda(cudaMalloc(&r.jobs, sizeof(RegJob) * J), "cudaMalloc(registration jobs)");
  check_cuda(cudaMalloc(&r.match_count, sizeof(int) * 2 * J), "cudaMalloc(registration match counts)");
  check_cuda(cudaMalloc(&r.match_dist, sizeof(double) * M * J), "cudaMalloc(registration matches)");
  check_cuda(cudaMalloc(&r.match_key, sizeof(int) * M * J), "cudaMalloc(registration match keys)");
  check_cuda(cudaMalloc(&r.sel, sizeof(int2) * S * J), "cudaMalloc(registration selection)");
  check_cuda(cudaMalloc(&r.sel_order, sizeof(long long) * S * J), "cudaMalloc(registration order)");
  check_cuda(cudaMalloc(&r.nsel, sizeof(int) * J), "cudaMalloc(registration selection counts)");
  check_cuda(cudaMalloc(&r.cands, sizeof(Cand) * 2 * S * J), "cudaMalloc(registration candidates)");
  check_cuda(cudaMalloc(&r.ranks, sizeof(CandRank) * 2 * S * J), "cudaMalloc(registration ranks)");
  check_cuda(cudaMalloc(&r.out, sizeof(RegResult) * J), "cudaMalloc(registration results)");
  check_cuda(cudaMalloc(&r.pairs, sizeof(short2) * kRegPts * J), "cudaMalloc(registration pairs)");
  check_cuda(cudaMalloc(&r.overflow, sizeof(int)), "cudaMalloc(registration overflow)");
  r.rows = rows;
  r.jobs_cap = jobs;
  r.match_cap = match_cap;
  r.sel_cap = sel_cap;
  r.device = dev;
}

static void validate_reg(const gg_register_params_t& p) {
  require(p.transform_model == GG_TRANSFORM_SIMILARITY || p.transform_model == GG_TRANSFORM_AFFINE,
          "triangle asterism registration supports similarity or affine transforms");
  require(std::isfinite(p.tolerance_px) && p.tolerance_px >= 0.0, "tolerance_px must be non-negative");
  require(std::isfinite(p.descriptor_radius) && p.descriptor_radius >= 0.0, "descriptor_radius must be non-negative");
  require(p.neighbors <= kMaxNeighbors, "neighbors must be at most 6");
  require(p.max_stars >= 0 && p.max_stars <= kRegPts, "max_stars must be in [0, 80]");
  require(p.max_descriptors >= 0, "max_descriptors must be non-negative");
  require(p.max_candidates >= 0 && p.max_candidates <= kMaxSel, "max_candidates must be in [0, 2048]");
}

static RegArgs make_args(RegScratch& r, int mode, double tol, double radius) {
  RegArgs a{};
  a.pts = r.pts;
  a.npts = r.npts;
  a.desc = r.desc;
  a.ndesc = r.ndesc;
  a.jobs = r.jobs;
  a.match_count = r.match_count;
  a.best_count = r.match_count + r.jobs_cap;
  a.match_dist = r.match_dist;
  a.match_key = r.match_key;
  a.sel = r.sel;
  a.sel_order = r.sel_order;
  a.nsel = r.nsel;
  a.cands = r.cands;
  a.ranks = r.ranks;
  a.out = r.out;
  a.pairs = r.pairs;
  a.overflow = r.overflow;
  a.tol = tol;
  a.radius = radius;
  a.match_cap = r.match_cap;
  a.sel_cap = r.sel_cap;
  a.mode = mode;
  a.max_stars = kRegPts;
  a.neighbors = 5;
  a.max_desc = kMaxDesc;
  a.max_cand = kMaxSel;
  a.min_inliers = 0;
  a.model = GG_TRANSFORM_SIMILARITY;  // the descriptor-list fallback fits similarities
  return a;
}

static void apply_params(RegArgs& a, const gg_register_params_t& p) {
  a.max_stars = p.max_stars;
  a.neighbors = p.neighbors;
  a.max_desc = std::min(p.max_descriptors, kMaxDesc);
  a.max_cand = p.max_candidates;
  a.min_inliers = p.min_inliers;
  a.model = p.transform_model;
}

static void launch_desc(const RegArgs& a, int rows, cudaStream_t stream) {
  const size_t smem = sizeof(TriCand) * kMaxTri;
  check_cuda(cudaFuncSetAttribute(reg_desc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(smem)),
             "cudaFuncSetAttribute(reg_desc)");
  note_launch();
  reg_desc_kernel<<<rows, 1024, smem, stream>>>(a);
  check_cuda(cudaGetLastError(), "reg_desc launch");
}

static void launch_match_score_best(const RegArgs& a, int njobs, int64_t max_sel, cudaStream_t stream) {
  const size_t smem = (sizeof(double2) + sizeof(float2)) * 2 * kMaxDesc;
  check_cuda(cudaFuncSetAttribute(reg_match_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(smem)),
             "cudaFuncSetAttribute(reg_match)");
  check_cuda(cudaMemsetAsync(a.match_count, 0, sizeof(int) * (a.best_count - a.match_count + njobs), stream),
             "cudaMemsetAsync(match counts)");
  note_launch(2);
  reg_pairs_kernel<<<dim3(kPairCtas, static_cast<unsigned>(njobs)), 32 * kPairWarps, 0, stream>>>(a);
  check_cuda(cudaGetLastError(), "reg_pairs launch");
  reg_match_kernel<<<njobs, 1024, smem, stream>>>(a);
  check_cuda(cudaGetLastError(), "reg_match launch");
  const int64_t per_job = (2 * max_sel + 32 * kScoreWarps - 1) / (32 * kScoreWarps);
  const unsigned gx = static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>(per_job, 1024)));
  auto score = a.model == GG_TRANSFORM_AFFINE ? reg_score_kernel<GG_TRANSFORM_AFFINE>
                                              : reg_score_kernel<GG_TRANSFORM_SIMILARITY>;
  note_launch();
  score<<<dim3(gx, static_cast<unsigned>(njobs)), 32 * kScoreWarps, 0, stream>>>(a);
  check_cuda(cudaGetLastError(), "reg_score launch");
  const unsigned gr = std::min(gx, static_cast<unsigned>(kRecheckCtas));
  const size_t exact_smem = sizeof(WarpScratch) * kScoreWarps;
  check_cuda(cudaFuncSetAttribute(reg_exact_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(exact_smem)),
             "cudaFuncSetAttribute(reg_exact)");
  note_launch(3);
  reg_exact_kernel<<<dim3(gr, static_cast<unsigned>(njobs)), 32 * kScoreWarps, exact_smem, stream>>>(a);
  check_cuda(cudaGetLastError(), "reg_exact launch");
  reg_rms_kernel<<<dim3(gr, static_cast<unsigned>(njobs)), 32 * kScoreWarps, 0, stream>>>(a);
  check_cuda(cudaGetLastError(), "reg_rms launch");
  reg_best_kernel<<<njobs, kBestThreads, 0, stream>>>(a);
  check_cuda(cudaGetLastError(), "reg_best launch");
}

static void fill_result(const RegResult& q, gg_registration_t& o) {
  std::memcpy(o.matrix, q.m, sizeof(q.m));
  o.rms_px = std::isfinite(q.rms) ? q.rms : std::nan("");
  o.best_candidate = q.best_order;
  o.inliers = q.inliers;
  o.status = q.status;
  o.descriptors_reference = q.ndesc_ref;
  o.descriptors_moving = q.ndesc_mov;
  o.matches = q.matches;
  o.pad = 0;
}

static void copy_pairs(const RegScratch& r, int32_t* host_pairs) {
  if (!host_pairs) return;
  std::vector<short2> prs(kRegPts);
  check_cuda(cudaMemcpy(prs.data(), r.pairs, sizeof(short2) * kRegPts, cudaMemcpyDeviceToHost),
             "cudaMemcpy(registration pairs)");
  for (int i = 0; i < kRegPts; ++i) {
    host_pairs[2 * i] = prs[static_cast<size_t>(i)].x;
    host_pairs[2 * i + 1] = prs[static_cast<size_t>(i)].y;
  }
}

// Process-wide scratch for the point-list entry points (calls are serialised).
static std::mutex g_list_mu;
static RegScratch g_list_scratch;

static void require_device() {
  int devs = 0;
  if (cudaGetDeviceCount(&devs) != cudaSuccess || devs <= 0) {
    cudaGetLastError();
    fail(GG_ERR_NO_DEVICE, "no CUDA device is available");
  }
}

static void upload_points(RegScratch& r, int row, const double* xy, int n) {
  std::vector<double> pts(2 * kRegPts, 0.0);
  for (int i = 0; i < 2 * n; ++i) pts[static_cast<size_t>(i)] = xy[i];
  check_cuda(cudaMemcpy(r.pts + static_cast<size_t>(row) * 2 * kRegPts, pts.data(), sizeof(double) * pts.size(),
                        cudaMemcpyHostToDevice),
             "cudaMemcpy(points)");
  check_cuda(cudaMemcpy(r.npts + row, &n, sizeof(int), cudaMemcpyHostToDevice), "cudaMemcpy(point count)");
}

static void check_overflow(const RegScratch& r, cudaStream_t stream) {
  int overflow = 0;
  check_cuda(cudaMemcpyAsync(&overflow, r.overflow, sizeof(int), cudaMemcpyDeviceToHost, stream),
             "cudaMemcpyAsync(overflow)");
  check_cuda(cudaStreamSynchronize(stream), "cudaStreamSynchronize(registration)");
  if (overflow) fail(GG_ERR_RUNTIME, "registration buffers overflowed (too many descriptor matches or point pairs)");
}

// Pixel coordinates: finite and within +-1e15 (float32-representable with
// room for the transform error bound).
static void require_finite_points(const double* xy, int64_t n) {
  for (int64_t i = 0; i < 2 * n; ++i)
    require(std::isfinite(xy[i]) && std::fabs(xy[i]) <= 1.0e15, "star coordinates must be finite and within 1e15");
}

}  // namespace gg

using namespace gg;

extern "C" {

int gg_triangle_descriptors(const double* host_xy, int64_t n, int32_t max_stars, int32_t neighbors,
                            int32_t max_descriptors, double* host_descriptors, int32_t* host_indices,
                            double* host_areas, int64_t capacity, int64_t* count) {
  GG_API_BEGIN
  require(count != nullptr, "null count");
  require(n >= 0 && (n == 0 || host_xy != nullptr), "invalid point list");
  require(max_stars >= 0 && max_stars <= kRegPts, "max_stars must be in [0, 80]");
  require(neighbors <= kMaxNeighbors, "neighbors must be at most 6");
  require(max_descriptors >= 0, "max_descriptors must be non-negative");
  require(capacity >= 0, "capacity must be non-negative");
  const int np = static_cast<int>(std::min<int64_t>(n, max_stars));
  require_finite_points(host_xy, np);
  require_device();
  std::lock_guard<std::mutex> lock(g_list_mu);
  RegScratch& r = g_list_scratch;
  reg_scratch_ensure(r, 2, 1, kStackMatchCap, kMaxSel);
  upload_points(r, 0, host_xy, np);
  RegArgs a = make_args(r, kEstimator, 0.0, 0.0);
  a.max_stars = max_stars;
  a.neighbors = neighbors;
  a.max_desc = std::min(max_descriptors, kMaxDesc);
  launch_desc(a, 1, nullptr);
  int nd = 0;
  check_cuda(cudaMemcpy(&nd, r.ndesc, sizeof(int), cudaMemcpyDeviceToHost), "cudaMemcpy(descriptor count)");
  *count = nd;
  const bool want = host_descriptors || host_indices || host_areas;
  if (want && capacity < nd) fail(GG_ERR_OUT_OF_RANGE, "output capacity is smaller than the descriptor count");
  if (nd > 0 && want) {
    std::vector<Desc> d(static_cast<size_t>(nd));
    check_cuda(cudaMemcpy(d.data(), r.desc, sizeof(Desc) * nd, cudaMemcpyDeviceToHost), "cudaMemcpy(descriptors)");
    for (int i = 0; i < nd; ++i) {
      const Desc& q = d[static_cast<size_t>(i)];
      if (host_descriptors) {
        host_descriptors[2 * i] = q.d0;
        host_descriptors[2 * i + 1] = q.d1;
      }
      if (host_indices)
        for (int k = 0; k < 3; ++k) host_indices[3 * i + k] = q.v[k];
      if (host_areas) host_areas[i] = q.area;
    }
  }
  GG_API_END
}

int gg_register_star_lists(const double* host_ref_xy, int64_t n_ref, const double* host_mov_xy, int64_t n_mov,
                           const gg_register_params_t* params, gg_registration_t* host_out, int32_t* host_pairs) {
  GG_API_BEGIN
  require(params != nullptr && host_out != nullptr, "null argument");
  require(n_ref >= 0 && n_mov >= 0, "point counts must be non-negative");
  require((n_ref == 0 || host_ref_xy) && (n_mov == 0 || host_mov_xy), "null point list");
  validate_reg(*params);
  const int nr = static_cast<int>(std::min<int64_t>(n_ref, params->max_stars));
  const int nm = static_cast<int>(std::min<int64_t>(n_mov, params->max_stars));
  require_finite_points(host_ref_xy, nr);
  require_finite_points(host_mov_xy, nm);
  require_device();
  std::lock_guard<std::mutex> lock(g_list_mu);
  RegScratch& r = g_list_scratch;
  reg_scratch_ensure(r, 2, 1, kStackMatchCap, kMaxSel);
  upload_points(r, 0, host_ref_xy, nr);
  upload_points(r, 1, host_mov_xy, nm);
  const RegJob job{0, 1};
  check_cuda(cudaMemcpy(r.jobs, &job, sizeof(job), cudaMemcpyHostToDevice), "cudaMemcpy(job)");
  check_cuda(cudaMemset(r.overflow, 0, sizeof(int)), "cudaMemset(overflow)");
  RegArgs a = make_args(r, kEstimator, params->tolerance_px, params->descriptor_radius);
  apply_params(a, *params);
  launch_desc(a, 2, nullptr);
  launch_match_score_best(a, 1, params->max_candidates, nullptr);
  check_overflow(r, nullptr);
  RegResult res;
  check_cuda(cudaMemcpy(&res, r.out, sizeof(res), cudaMemcpyDeviceToHost), "cudaMemcpy(registration result)");
  fill_result(res, *host_out);
  if (nr < 3 || nm < 3) {
    host_out->descriptors_reference = 0;
    host_out->descriptors_moving = 0;
    host_out->matches = 0;
  }
  copy_pairs(r, host_pairs);
  GG_API_END
}

int gg_similarity_from_descriptors(const double* host_ref_xy, int64_t n_ref, const double* host_mov_xy,
                                   int64_t n_mov, const float* host_ref_desc, const int32_t* host_ref_idx,
                                   int64_t n_ref_desc, const float* host_mov_desc, const int32_t* host_mov_idx,
                                   int64_t n_mov_desc, double tolerance_px, double descriptor_radius,
                                   gg_registration_t* host_out, int32_t* host_pairs) {
  GG_API_BEGIN
  require(host_out != nullptr, "null output");
  require(std::isfinite(tolerance_px) && tolerance_px >= 0.0, "tolerance_px must be non-negative");
  require(std::isfinite(descriptor_radius) && descriptor_radius >= 0.0, "descriptor_radius must be non-negative");
  require(n_ref >= 0 && n_mov >= 0 && n_ref_desc >= 0 && n_mov_desc >= 0, "counts must be non-negative");
  if (n_ref > kRegPts || n_mov > kRegPts) fail(GG_ERR_OUT_OF_RANGE, "catalogs are limited to 80 stars");
  if (n_ref_desc > kMaxDesc || n_mov_desc > kMaxDesc)
    fail(GG_ERR_OUT_OF_RANGE, "descriptor lists are limited to 1600 rows");
  require((n_ref == 0 || host_ref_xy) && (n_mov == 0 || host_mov_xy), "null point list");
  require((n_ref_desc == 0 || (host_ref_desc && host_ref_idx)) && (n_mov_desc == 0 || (host_mov_desc && host_mov_idx)),
          "null descriptor list");
  for (int64_t i = 0; i < 3 * n_ref_desc; ++i)
    if (host_ref_idx[i] < 0 || host_ref_idx[i] >= n_ref)
      fail(GG_ERR_OUT_OF_RANGE, "reference triangle index out of range");
  for (int64_t i = 0; i < 3 * n_mov_desc; ++i)
    if (host_mov_idx[i] < 0 || host_mov_idx[i] >= n_mov) fail(GG_ERR_OUT_OF_RANGE, "moving triangle index out of range");
  require_finite_points(host_ref_xy, n_ref);
  require_finite_points(host_mov_xy, n_mov);
  require_device();
  std::lock_guard<std::mutex> lock(g_list_mu);
  RegScratch& r = g_list_scratch;
  reg_scratch_ensure(r, 2, 1, kListMatchCap, kListMatchCap);
  upload_points(r, 0, host_ref_xy, static_cast<int>(n_ref));
  upload_points(r, 1, host_mov_xy, static_cast<int>(n_mov));
  auto upload_desc = [&](int row, const float* dv, const int32_t* iv, int64_t nd) {
    std::vector<Desc> d(static_cast<size_t>(nd));
    for (int64_t i = 0; i < nd; ++i) {
      Desc& q = d[static_cast<size_t>(i)];
      q.d0 = dv[2 * i];
      q.d1 = dv[2 * i + 1];
      q.area = 0.0;
      for (int k = 0; k < 3; ++k) q.v[k] = iv[3 * i + k];
      q.pad = 0;
    }
    if (nd > 0)
      check_cuda(cudaMemcpy(r.desc + static_cast<size_t>(row) * kMaxDesc, d.data(), sizeof(Desc) * nd,
                            cudaMemcpyHostToDevice),
                 "cudaMemcpy(descriptors)");
    const int n32 = static_cast<int>(nd);
    check_cuda(cudaMemcpy(r.ndesc + row, &n32, sizeof(int), cudaMemcpyHostToDevice), "cudaMemcpy(descriptor count)");
  };
  upload_desc(0, host_ref_desc, host_ref_idx, n_ref_desc);
  upload_desc(1, host_mov_desc, host_mov_idx, n_mov_desc);
  const RegJob job{0, 1};
  check_cuda(cudaMemcpy(r.jobs, &job, sizeof(job), cudaMemcpyHostToDevice), "cudaMemcpy(job)");
  check_cuda(cudaMemset(r.overflow, 0, sizeof(int)), "cudaMemset(overflow)");
  RegArgs a = make_args(r, kDescriptorList, tolerance_px, descriptor_radius);
  const int64_t max_sel = std::max<int64_t>(1, std::min<int64_t>(n_ref_desc * n_mov_desc, kListMatchCap));
  launch_match_score_best(a, 1, max_sel, nullptr);
  check_overflow(r, nullptr);
  RegResult res;
  check_cuda(cudaMemcpy(&res, r.out, sizeof(res), cudaMemcpyDeviceToHost), "cudaMemcpy(registration result)");
  fill_result(res, *host_out);
  copy_pairs(r, host_pairs);
  GG_API_END
}

int gg_stack_register_frames(gg_stack* s, int64_t reference_index, const int64_t* indices, int64_t count,
                             const gg_register_params_t* params, gg_registration_t* host_out) {
  GG_API_BEGIN
  require(s != nullptr && indices != nullptr && params != nullptr && host_out != nullptr, "null argument");
  require(count > 0, "indices must contain at least one frame index");
  validate_reg(*params);
  stack_require_index(s, reference_index);
  for (int64_t k = 0; k < count; ++k) stack_require_index(s, indices[k]);
  if (!s->d_cat_xy) fail(GG_ERR_RUNTIME, "detect stars on the frames before registering them");
  stack_activate(s);
  if (!s->reg_scratch) {
    s->reg_scratch = new RegScratch();
    s->reg_scratch_free = [](void* q) {
      auto* r = static_cast<RegScratch*>(q);
      reg_scratch_release(*r);
      delete r;
    };
  }
  RegScratch& r = *static_cast<RegScratch*>(s->reg_scratch);
  const int64_t before = reg_scratch_bytes(r);
  const int rows = static_cast<int>(count) + 1;
  reg_scratch_ensure(r, rows, static_cast<int>(count), kStackMatchCap, kMaxSel);
  s->bytes_allocated += reg_scratch_bytes(r) - before;
  // row 0 = reference catalog, row k + 1 = moving catalog k; job k = (0, k + 1)
  std::vector<int> row_frames(static_cast<size_t>(rows));
  std::vector<RegJob> jobs(static_cast<size_t>(count));
  row_frames[0] = static_cast<int>(reference_index);
  for (int64_t k = 0; k < count; ++k) {
    row_frames[static_cast<size_t>(k + 1)] = static_cast<int>(indices[k]);
    jobs[static_cast<size_t>(k)] = RegJob{0, static_cast<int>(k + 1)};
  }
  upload_params(s->stream, r.row_frames, row_frames.data(), sizeof(int) * rows, "cudaMemcpyAsync(registration rows)");
  upload_params(s->stream, r.jobs, jobs.data(), sizeof(RegJob) * count, "cudaMemcpyAsync(registration jobs)");
  check_cuda(cudaMemsetAsync(r.overflow, 0, sizeof(int), s->stream), "cudaMemsetAsync(overflow)");
  note_launch();
  reg_copy_catalogs_kernel<<<rows, 128, 0, s->stream>>>(s->d_cat_xy, s->d_cat_n, r.row_frames, rows, r.pts, r.npts);
  check_cuda(cudaGetLastError(), "reg_copy_catalogs launch");
  RegArgs a = make_args(r, kEstimator, params->tolerance_px, params->descriptor_radius);
  apply_params(a, *params);
  launch_desc(a, rows, s->stream);
  launch_match_score_best(a, static_cast<int>(count), params->max_candidates, s->stream);
  std::vector<RegResult> res(static_cast<size_t>(count));
  check_cuda(cudaMemcpyAsync(res.data(), r.out, sizeof(RegResult) * count, cudaMemcpyDeviceToHost, s->stream),
             "cudaMemcpyAsync(registration results)");
  check_overflow(r, s->stream);  // synchronises the stack stream
  for (int64_t k = 0; k < count; ++k) fill_result(res[static_cast<size_t>(k)], host_out[k]);
  GG_API_END
}

}  // extern "C"
