// Grid local normalisation of registered frames to the reference frame (the
// resident grid_mean_std mode, tile 256 by default):
//
//   ln_pair_stats_kernel  one CTA per (tile, frame pair): sums of the source
//                         and reference pixels and their squares over the
//                         pixels finite in both (local_norm_kernels.cu:220-300),
//                         float-float per thread, float64 across the CTA;
//   ln_coeff_kernel       one thread per (pair, tile): mean = sum / n,
//                         std = sqrt(max(sum2 / n - mean^2, 0)) in float64,
//                         stored as float32 (native_bindings.cpp:10745-10760);
//                         coefficients (resident_cuda.py:1897-1927): empty
//                         tile scale 1 / offset 0; std <= eps on either side
//                         scale 1 / offset ref_mean - src_mean; else
//                         scale = ref_std / src_std, offset = ref_mean -
//                         src_mean * scale, float32 operations;
//   ln_apply_kernel       in place, v * scale + offset per tile (float32
//                         multiply, then add: cpu/local_norm.py:197-215).
//
// Traffic: the statistics read both frames of a pair (8 B per pixel), the
// apply reads and writes the source (8 B per pixel); both are HBM-bound
// streams (float-float accumulation keeps the statistics off the FP64 pipe).
#include <cmath>
#include <cstring>
#include <vector>

#include <math_constants.h>

#include "f32x2.cuh"
#include "stack.cuh"

namespace gg {

constexpr int kLnThreads = 256;

struct LnArgs {
  const float* slots;
  const int* slot_of_frame;
  int64_t stride;
  int width, height;
  int tile_w, tile_h, cols, rows;
  int ref_frame;
  const int* frames;         // [pairs] source frames
  double* sums;              // [pairs][tiles][4]
  unsigned long long* counts;  // [pairs][tiles]
  float* stats;              // [pairs][tiles][4]: src mean, src std, ref mean, ref std
  float* scales;             // [pairs][tiles]
  float* offsets;
  unsigned long long* totals;  // [pairs] paired finite pixels of the frame
  double eps;
};

// Bound by the packed arithmetic (17 instructions per pixel pair), then memory:
// 31 pairs of 2048^2 in 324 us, 452 us in scalar instructions with a division
// and a remainder per pixel.
constexpr int kLnLoads = 4;

__global__ void __launch_bounds__(kLnThreads) ln_pair_stats_kernel(LnArgs a) {
  __shared__ double red[kLnThreads / 32][4];
  __shared__ unsigned long long redn[kLnThreads / 32];
  const int tile = blockIdx.x, pair = blockIdx.y;
  const int tx = tile % a.cols, ty = tile / a.cols;
  const int x0 = tx * a.tile_w, y0 = ty * a.tile_h;
  const int w = min(a.tile_w, a.width - x0), h = min(a.tile_h, a.height - y0);
  const float* src = a.slots + static_cast<int64_t>(a.slot_of_frame[a.frames[pair]]) * a.stride;
  const float* ref = a.slots + static_cast<int64_t>(a.slot_of_frame[a.ref_frame]) * a.stride;
  F2Moments sums;  // lanes: source, reference; a pair that does not count adds zeros
  unsigned n = 0;
  const int npx = w * h;
  // pixels threadIdx.x, + kLnThreads, ...: the position follows by addition
  const int dx = kLnThreads % w, dy = kLnThreads / w;
  int x = static_cast<int>(threadIdx.x) % w, y = static_cast<int>(threadIdx.x) / w;
  for (int q = threadIdx.x; q < npx; q += kLnThreads * kLnLoads) {
    float s[kLnLoads], r[kLnLoads];
#pragma unroll
    for (int u = 0; u < kLnLoads; ++u) {
      s[u] = r[u] = CUDART_INF_F;
      if (q + u * kLnThreads < npx) {
        const int64_t p = static_cast<int64_t>(y0 + y) * a.width + x0 + x;
        s[u] = __ldcs(src + p);
        r[u] = __ldg(ref + p);
      }
      x += dx;
      y += dy;
      if (x >= w) {
        x -= w;
        ++y;
      }
    }
#pragma unroll
    for (int u = 0; u < kLnLoads; ++u) {
      const bool both = isfinite(s[u]) && isfinite(r[u]);
      sums.add(f2(both ? s[u] : 0.0f, both ? r[u] : 0.0f));
      n += both ? 1u : 0u;
    }
  }
  FF s1, s2, r1, r2;
  sums.split(s1, s2, r1, r2);
  double v[4] = {static_cast<double>(s1.hi) + static_cast<double>(s1.lo),
                 static_cast<double>(s2.hi) + static_cast<double>(s2.lo),
                 static_cast<double>(r1.hi) + static_cast<double>(r1.lo),
                 static_cast<double>(r2.hi) + static_cast<double>(r2.lo)};
  unsigned long long nn = n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], off);
    nn += __shfl_xor_sync(0xffffffffu, nn, off);
  }
  if (lane == 0) {
    for (int i = 0; i < 4; ++i) red[warp][i] = v[i];
    redn[warp] = nn;
  }
  __syncthreads();
  const int64_t t = static_cast<int64_t>(pair) * a.cols * a.rows + tile;
  if (threadIdx.x < 4) {
    double acc = 0.0;
    for (int k = 0; k < kLnThreads / 32; ++k) acc += red[k][threadIdx.x];
    a.sums[t * 4 + threadIdx.x] = acc;
  } else if (threadIdx.x == 4) {
    unsigned long long acc = 0;
    for (int k = 0; k < kLnThreads / 32; ++k) acc += redn[k];
    a.counts[t] = acc;
  }
}

__global__ void ln_coeff_kernel(LnArgs a, int pairs) {
  const int tiles = a.cols * a.rows;
  const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= static_cast<int64_t>(pairs) * tiles) return;
  const int pair = static_cast<int>(t / tiles);
  const unsigned long long c = a.counts[t];
  float sm = 0.0f, ss = 0.0f, rm = 0.0f, rs = 0.0f;
  float scale = 1.0f, offset = 0.0f;
  if (c > 0) {
    const double inv = 1.0 / static_cast<double>(c);
    const double* s = a.sums + t * 4;
    const double smd = s[0] * inv, rmd = s[2] * inv;
    const double sv = fmax(__dsub_rn(__dmul_rn(s[1], inv), __dmul_rn(smd, smd)), 0.0);
    const double rv = fmax(__dsub_rn(__dmul_rn(s[3], inv), __dmul_rn(rmd, rmd)), 0.0);
    sm = __double2float_rn(smd);
    ss = __double2float_rn(sqrt(sv));
    rm = __double2float_rn(rmd);
    rs = __double2float_rn(sqrt(rv));
    if (static_cast<double>(ss) <= a.eps || static_cast<double>(rs) <= a.eps) {
      offset = __fsub_rn(rm, sm);
    } else {
      scale = __fdiv_rn(rs, ss);
      offset = __fsub_rn(rm, __fmul_rn(sm, scale));
    }
    atomicAdd(a.totals + pair, c);
  }
  if (a.stats) {
    a.stats[t * 4 + 0] = sm;
    a.stats[t * 4 + 1] = ss;
    a.stats[t * 4 + 2] = rm;
    a.stats[t * 4 + 3] = rs;
  }
  a.scales[t] = scale;
  a.offsets[t] = offset;
}

// In place v * scale + offset for every pixel of each listed frame; frames
// whose pair had no finite pixel (totals == 0) are left as they are.  Groups of
// `lanes` threads take rows, threads the row's 16-byte vectors (the first and last
// may reach into the neighbouring rows: those go sample by sample).  Bound by
// memory: 31 frames of 2048^2 in 236 us, 483 us with a 64-bit division per
// sample; rows of less than 1024 columns share a CTA.
__global__ void __launch_bounds__(256) ln_apply_kernel(LnArgs a, int check_totals, int lanes) {
  const int pair = blockIdx.y;
  if (check_totals && a.totals[pair] == 0) return;
  float* img = const_cast<float*>(a.slots) + static_cast<int64_t>(a.slot_of_frame[a.frames[pair]]) * a.stride;
  const int W = a.width;
  const unsigned tile_w = static_cast<unsigned>(a.tile_w);
  const int rows = 256 / lanes, lane = static_cast<int>(threadIdx.x) % lanes;
  for (int y = blockIdx.x * rows + static_cast<int>(threadIdx.x) / lanes; y < a.height; y += gridDim.x * rows) {
    const int64_t at = static_cast<int64_t>(y) * W;
    const int64_t row_tile = (static_cast<int64_t>(pair) * a.rows + min(y / a.tile_h, a.rows - 1)) * a.cols;
    const float* sc = a.scales + row_tile;
    const float* of = a.offsets + row_tile;
    float* row = img + at;
    auto tile = [&](int x) { return min(static_cast<int>(static_cast<unsigned>(x) / tile_w), a.cols - 1); };
    auto apply = [&](float v, int t) { return __fadd_rn(__fmul_rn(v, __ldg(sc + t)), __ldg(of + t)); };
    for (int x = 4 * lane - static_cast<int>(at & 3); x < W; x += 4 * lanes) {
      if (x >= 0 && x + 3 < W) {
        float4 v = *reinterpret_cast<const float4*>(row + x);
        const int t0 = tile(x), t3 = tile(x + 3);
        const bool one = t0 == t3;
        v.x = apply(v.x, t0);
        v.y = apply(v.y, one ? t0 : tile(x + 1));
        v.z = apply(v.z, one ? t0 : tile(x + 2));
        v.w = apply(v.w, t3);
        *reinterpret_cast<float4*>(row + x) = v;
      } else {
        for (int i = max(x, 0); i < min(x + 4, W); ++i) row[i] = apply(row[i], tile(i));
      }
    }
  }
}

__global__ void ln_zero_weights_kernel(const unsigned long long* totals, const int* frames, int pairs,
                                       float* weights) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < pairs && totals[i] == 0) weights[frames[i]] = 0.0f;
}

struct LnScratch {
  double* sums = nullptr;
  unsigned long long* counts = nullptr;
  float* stats = nullptr;
  float* scales = nullptr;
  float* offsets = nullptr;
  unsigned long long* totals = nullptr;
  int* frames = nullptr;
  int* h_frames = nullptr;  // pinned
  int64_t tile_cap = 0;     // pairs * tiles
  int pair_cap = 0;
};

static void ln_release(LnScratch& g) {
  void* d[] = {g.sums, g.counts, g.stats, g.scales, g.offsets, g.totals, g.frames};
  for (void* p : d)
    if (p) cudaFree(p);
  if (g.h_frames) cudaFreeHost(g.h_frames);
  g = LnScratch{};
}

static LnScratch& ln_scratch(gg_stack* s, int pairs, int64_t tiles) {
  if (!s->ln_scratch) {
    s->ln_scratch = new LnScratch();
    s->ln_scratch_free = [](void* q) {
      auto* g = static_cast<LnScratch*>(q);
      ln_release(*g);
      delete g;
    };
  }
  LnScratch& g = *static_cast<LnScratch*>(s->ln_scratch);
  const int64_t need = static_cast<int64_t>(pairs) * tiles;
  if (g.tile_cap < need || g.pair_cap < pairs) {
    check_cuda(cudaStreamSynchronize(s->stream), "cudaStreamSynchronize(local norm scratch)");
    const int64_t tc = std::max(need, g.tile_cap);
    const int pc = std::max(pairs, g.pair_cap);
    ln_release(g);
    check_cuda(cudaMalloc(&g.sums, sizeof(double) * 4 * tc), "cudaMalloc(local norm sums)");
    check_cuda(cudaMalloc(&g.counts, sizeof(unsigned long long) * tc), "cudaMalloc(local norm counts)");
    check_cuda(cudaMalloc(&g.stats, sizeof(float) * 4 * tc), "cudaMalloc(local norm stats)");
    check_cuda(cudaMalloc(&g.scales, sizeof(float) * tc), "cudaMalloc(local norm scales)");
    check_cuda(cudaMalloc(&g.offsets, sizeof(float) * tc), "cudaMalloc(local norm offsets)");
    check_cuda(cudaMalloc(&g.totals, sizeof(unsigned long long) * pc), "cudaMalloc(local norm totals)");
    check_cuda(cudaMalloc(&g.frames, sizeof(int) * pc), "cudaMalloc(local norm frames)");
    check_cuda(cudaHostAlloc(reinterpret_cast<void**>(&g.h_frames), sizeof(int) * pc, cudaHostAllocDefault),
               "cudaHostAlloc(local norm frames)");
    g.tile_cap = tc;
    g.pair_cap = pc;
  }
  return g;
}

static LnArgs ln_args(gg_stack* s, int tile_h, int tile_w, int rows, int cols, int ref, LnScratch& g) {
  LnArgs a{};
  a.slots = s->d_slots;
  a.slot_of_frame = s->d_slot_of_frame;
  a.stride = s->stride;
  a.width = static_cast<int>(s->width);
  a.height = static_cast<int>(s->height);
  a.tile_w = tile_w;
  a.tile_h = tile_h;
  a.cols = cols;
  a.rows = rows;
  a.ref_frame = ref;
  a.frames = g.frames;
  a.sums = g.sums;
  a.counts = g.counts;
  a.stats = g.stats;
  a.scales = g.scales;
  a.offsets = g.offsets;
  a.totals = g.totals;
  return a;
}

static void upload_frames(gg_stack* s, LnScratch& g, const int64_t* idx, int64_t count) {
  for (int64_t k = 0; k < count; ++k) g.h_frames[k] = static_cast<int>(idx[k]);
  upload_params(s->stream, g.frames, g.h_frames, sizeof(int) * count, "cudaMemcpyAsync(local norm frames)");
}

static void launch_ln_apply(gg_stack* s, const LnArgs& a, int pairs, int check_totals) {
  int lanes = 8;  // of a row: its vectors, one more where it starts off a 16-byte boundary
  while (lanes < 256 && 4 * lanes < s->width + 3) lanes *= 2;
  const int64_t ctas = (s->height + 256 / lanes - 1) / (256 / lanes);
  const int64_t want = static_cast<int64_t>(sm_count()) * 8 / std::max(pairs, 1) + 1;
  note_launch();
  ln_apply_kernel<<<dim3(static_cast<unsigned>(std::min(ctas, want)), static_cast<unsigned>(pairs)), 256, 0,
                    s->stream>>>(a, check_totals, lanes);
  check_cuda(cudaGetLastError(), "ln_apply launch");
}

// statistics + coefficients (+ apply) for `count` source frames
static void ln_run(gg_stack* s, int64_t ref, const int64_t* sources, int64_t count, int tile_h, int tile_w, double eps,
                   bool apply, bool update_weights) {
  const int rows = static_cast<int>((s->height + tile_h - 1) / tile_h);
  const int cols = static_cast<int>((s->width + tile_w - 1) / tile_w);
  const int pairs = static_cast<int>(count);
  LnScratch& g = ln_scratch(s, pairs, static_cast<int64_t>(rows) * cols);
  upload_frames(s, g, sources, count);
  LnArgs a = ln_args(s, tile_h, tile_w, rows, cols, static_cast<int>(ref), g);
  a.eps = eps;
  check_cuda(cudaMemsetAsync(g.totals, 0, sizeof(unsigned long long) * pairs, s->stream), "cudaMemsetAsync(totals)");
  note_launch();
  ln_pair_stats_kernel<<<dim3(static_cast<unsigned>(rows * cols), static_cast<unsigned>(pairs)), kLnThreads, 0,
                         s->stream>>>(a);
  check_cuda(cudaGetLastError(), "ln_pair_stats launch");
  const int64_t tiles = static_cast<int64_t>(pairs) * rows * cols;
  note_launch();
  ln_coeff_kernel<<<static_cast<unsigned>((tiles + 255) / 256), 256, 0, s->stream>>>(a, pairs);
  check_cuda(cudaGetLastError(), "ln_coeff launch");
  if (apply) launch_ln_apply(s, a, pairs, 1);
  if (update_weights) {
    note_launch();
    ln_zero_weights_kernel<<<(pairs + 127) / 128, 128, 0, s->stream>>>(g.totals, g.frames, pairs, s->d_weights);
    check_cuda(cudaGetLastError(), "ln_zero_weights launch");
  }
}

static void validate_tiles(int tile_h, int tile_w) {
  require(tile_h > 0 && tile_w > 0, "tile dimensions must be positive");
}

}  // namespace gg

using namespace gg;

extern "C" {

int gg_stack_pair_grid_stats(gg_stack* s, int64_t reference_index, const int64_t* sources, int64_t count,
                             int32_t tile_h, int32_t tile_w, float* host_source_mean, float* host_source_std,
                             float* host_reference_mean, float* host_reference_std, uint64_t* host_valid) {
  GG_API_BEGIN
  require(s != nullptr && sources != nullptr, "null argument");
  require(count > 0 && count <= 65535, "source count must be in [1, 65535]");
  validate_tiles(tile_h, tile_w);
  stack_require_loaded(s, reference_index, "grid local normalization reference statistics");
  for (int64_t k = 0; k < count; ++k) stack_require_loaded(s, sources[k], "grid local normalization statistics");
  stack_activate(s);
  ln_run(s, reference_index, sources, count, tile_h, tile_w, 1.0e-6, false, false);
  const int rows = static_cast<int>((s->height + tile_h - 1) / tile_h);
  const int cols = static_cast<int>((s->width + tile_w - 1) / tile_w);
  const int64_t tiles = count * rows * cols;
  LnScratch& g = *static_cast<LnScratch*>(s->ln_scratch);
  std::vector<float> st(static_cast<size_t>(tiles) * 4);
  std::vector<unsigned long long> cn(static_cast<size_t>(tiles));
  check_cuda(cudaMemcpyAsync(st.data(), g.stats, sizeof(float) * 4 * tiles, cudaMemcpyDeviceToHost, s->stream),
             "cudaMemcpyAsync(local norm stats)");
  check_cuda(cudaMemcpyAsync(cn.data(), g.counts, sizeof(unsigned long long) * tiles, cudaMemcpyDeviceToHost,
                             s->stream),
             "cudaMemcpyAsync(local norm counts)");
  check_cuda(cudaStreamSynchronize(s->stream), "cudaStreamSynchronize(local norm stats)");
  for (int64_t t = 0; t < tiles; ++t) {
    if (host_source_mean) host_source_mean[t] = st[static_cast<size_t>(t) * 4 + 0];
    if (host_source_std) host_source_std[t] = st[static_cast<size_t>(t) * 4 + 1];
    if (host_reference_mean) host_reference_mean[t] = st[static_cast<size_t>(t) * 4 + 2];
    if (host_reference_std) host_reference_std[t] = st[static_cast<size_t>(t) * 4 + 3];
    if (host_valid) host_valid[t] = cn[static_cast<size_t>(t)];
  }
  GG_API_END
}

int gg_stack_apply_grid_normalization(gg_stack* s, const int64_t* indices, int64_t count, const float* host_scales,
                                      const float* host_offsets, int32_t grid_rows, int32_t grid_cols,
                                      int32_t tile_h, int32_t tile_w) {
  GG_API_BEGIN
  require(s != nullptr && indices != nullptr && host_scales != nullptr && host_offsets != nullptr, "null argument");
  require(count > 0 && count <= 65535, "frame count must be in [1, 65535]");
  validate_tiles(tile_h, tile_w);
  require(grid_rows > 0 && grid_cols > 0, "coefficient grid must not be empty");
  for (int64_t k = 0; k < count; ++k) stack_require_loaded(s, indices[k], "grid local normalization");
  stack_activate(s);
  const int64_t tiles = static_cast<int64_t>(grid_rows) * grid_cols;
  LnScratch& g = ln_scratch(s, static_cast<int>(count), tiles);
  upload_frames(s, g, indices, count);
  upload_params(s->stream, g.scales, host_scales, sizeof(float) * tiles * count, "cudaMemcpyAsync(local norm scales)");
  upload_params(s->stream, g.offsets, host_offsets, sizeof(float) * tiles * count,
                "cudaMemcpyAsync(local norm offsets)");
  LnArgs a = ln_args(s, tile_h, tile_w, grid_rows, grid_cols, 0, g);
  launch_ln_apply(s, a, static_cast<int>(count), 0);
  check_cuda(cudaStreamSynchronize(s->stream), "cudaStreamSynchronize(local norm apply)");
  GG_API_END
}

int gg_stack_local_normalize_grid(gg_stack* s, int64_t reference_index, const int64_t* sources, int64_t count,
                                  int32_t tile_h, int32_t tile_w, double eps, int update_weights, float* host_scales,
                                  float* host_offsets) {
  GG_API_BEGIN
  require(s != nullptr && sources != nullptr, "null argument");
  require(count > 0 && count <= 65535, "source count must be in [1, 65535]");
  validate_tiles(tile_h, tile_w);
  require(std::isfinite(eps) && eps >= 0.0, "eps must be finite and non-negative");
  stack_require_loaded(s, reference_index, "grid local normalization reference");
  for (int64_t k = 0; k < count; ++k) {
    stack_require_loaded(s, sources[k], "grid local normalization");
    require(sources[k] != reference_index, "the reference frame is not normalised to itself");
  }
  stack_activate(s);
  ln_run(s, reference_index, sources, count, tile_h, tile_w, eps, true, update_weights != 0);
  if (host_scales || host_offsets) {
    const int64_t tiles = count * ((s->height + tile_h - 1) / tile_h) * ((s->width + tile_w - 1) / tile_w);
    LnScratch& g = *static_cast<LnScratch*>(s->ln_scratch);
    if (host_scales)
      check_cuda(cudaMemcpyAsync(host_scales, g.scales, sizeof(float) * tiles, cudaMemcpyDeviceToHost, s->stream),
                 "cudaMemcpyAsync(local norm scales)");
    if (host_offsets)
      check_cuda(cudaMemcpyAsync(host_offsets, g.offsets, sizeof(float) * tiles, cudaMemcpyDeviceToHost, s->stream),
                 "cudaMemcpyAsync(local norm offsets)");
    check_cuda(cudaStreamSynchronize(s->stream), "cudaStreamSynchronize(local norm coefficients)");
  }
  GG_API_END
}

int gg_stack_apply_global_normalization(gg_stack* s, int64_t index, float scale, float offset) {
  GG_API_BEGIN
  require(s != nullptr, "null argument");
  stack_require_loaded(s, index, "global local normalization");
  stack_activate(s);
  LnScratch& g = ln_scratch(s, 1, 1);
  upload_frames(s, g, &index, 1);
  upload_params(s->stream, g.scales, &scale, sizeof(float), "cudaMemcpyAsync(global scale)");
  upload_params(s->stream, g.offsets, &offset, sizeof(float), "cudaMemcpyAsync(global offset)");
  LnArgs a = ln_args(s, static_cast<int>(s->height), static_cast<int>(s->width), 1, 1, 0, g);
  launch_ln_apply(s, a, 1, 0);
  check_cuda(cudaStreamSynchronize(s->stream), "cudaStreamSynchronize(global normalization)");
  GG_API_END
}

}  // extern "C"
