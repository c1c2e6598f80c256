// Fused uint16 decode + bias/dark/flat calibration into the resident stack.
//
// Semantics follow the CPU oracle cpu/calibration.py:51-76 (which the
// reference CUDA kernels calibration_kernels.cu:5-43 and :110-153 implement):
//   v = light
//   if dark:  v = v - dark * dark_scale ; if !dark_includes_bias and bias: v = v - bias
//   elif bias: v = v - bias
//   if flat:  v = v / max(flat, flat_floor)
//   if pedestal != 0: v = v + pedestal
// Every operation is rounded separately (no FMA), as NumPy does.
//
// GB300 design: one launch calibrates a batch of frames.  Each thread owns 8
// consecutive pixels, loads the masters for them once (16-byte vector loads) and
// then streams the batch's frames through registers, four frames' loads in
// flight: 16 B of uint16 in and 32 B of float32 out per frame, so the masters
// cost 12 B per pixel per batch instead of per frame.  Frames of a pixel count
// that is no multiple of 8 start at any 2-byte offset: their 16 bytes come out of
// two aligned loads.  The last CTA publishes the frames' non-finite counts.
// Raw frames arrive over PCIe/C2C on a copy stream into one of two lane buffers
// while the previous lane is being decoded (cudaEvent handshakes).
//
// Bound: HBM.  16 frames of 4096^2 in one launch 335 us, 5.4 TB/s of the
// algorithmic bytes (357 us in launches of 8 frames, which read the masters
// twice); 20 frames of 1537 x 2047 120 us (192 us one sample at a time).
#include <algorithm>
#include <vector>

#include "stack.cuh"

namespace gg {

struct CalibArgs {
  const uint16_t* raw;     // nframes * P (nullptr -> light_f32)
  const float* light_f32;  // P (single frame)
  const float* bias;
  const float* dark;
  const float* flat;
  float* slots;
  const int* slot_of_frame;
  unsigned* nonfinite;
  unsigned* counts;  // of this launch, zero before and after
  unsigned* ticket;
  int64_t stride;
  int64_t pixels;
  int nframes;
  int frame[GG_MAX_BATCH_FRAMES];
  int big_endian_bzero;
  int has_bias, has_dark, has_flat, dark_includes_bias;
  float dark_scale, flat_floor, pedestal;
};

__device__ __forceinline__ float calibrate_one(float v, float b, float d, float f, const CalibArgs& a) {
  if (a.has_dark) {
    v = __fsub_rn(v, __fmul_rn(d, a.dark_scale));
    if (!a.dark_includes_bias && a.has_bias) v = __fsub_rn(v, b);
  } else if (a.has_bias) {
    v = __fsub_rn(v, b);
  }
  if (a.has_flat) {
    // np.maximum(flat, floor): NaN propagates, anything below the floor is raised.
    v = __fdiv_rn(v, f < a.flat_floor ? a.flat_floor : f);
  }
  if (a.pedestal != 0.0f) v = __fadd_rn(v, a.pedestal);
  return v;
}

__device__ __forceinline__ float decode_u16(uint16_t raw, int big_endian_bzero) {
  if (big_endian_bzero) {
    const unsigned bits = ((static_cast<unsigned>(raw) & 0xffu) << 8) | (static_cast<unsigned>(raw) >> 8);
    return static_cast<float>(bits ^ 0x8000u);
  }
  return static_cast<float>(raw);
}

// 8 raw samples from any 2-byte aligned address.
struct Raw8 {
  unsigned w[4];
};

__device__ __forceinline__ Raw8 load_raw8(const uint16_t* p, const uint16_t* first, const uint16_t* last) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(p);
  const unsigned shift = static_cast<unsigned>(at) & 15u;  // the same in every thread of a frame
  Raw8 r;
  if (shift == 0) {
    const uint4 v = __ldcs(reinterpret_cast<const uint4*>(p));
    r.w[0] = v.x;
    r.w[1] = v.y;
    r.w[2] = v.z;
    r.w[3] = v.w;
    return r;
  }
  const auto* lo = reinterpret_cast<const uint4*>(at - shift);
  if (reinterpret_cast<const uint16_t*>(lo) < first || reinterpret_cast<const uint16_t*>(lo + 2) > last) {
    // the buffer's first and last samples
#pragma unroll
    for (int k = 0; k < 4; ++k) r.w[k] = p[2 * k] | static_cast<unsigned>(p[2 * k + 1]) << 16;
    return r;
  }
  const uint4 a = __ldg(lo), b = __ldg(lo + 1);
  const unsigned v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  unsigned s[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const unsigned q = shift >> 2;
    s[k] = q == 0 ? v[k] : q == 1 ? v[k + 1] : q == 2 ? v[k + 2] : v[min(k + 3, 7)];
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) r.w[k] = __funnelshift_r(s[k], s[k + 1], (shift & 2u) * 8u);
  return r;
}

// uint16 frames.  Thread t owns pixels [8t, 8t + 8); the last P % 8 pixels of
// every frame go one by one.
__global__ void __launch_bounds__(256) calibrate_u16_kernel(CalibArgs a) {
  const int64_t groups = a.pixels / 8;
  const uint16_t* last = a.raw + static_cast<int64_t>(a.nframes) * a.pixels;
  for (int64_t g = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; g < groups;
       g += int64_t(gridDim.x) * blockDim.x) {
    const int64_t p0 = g * 8;
    float b[8], d[8], f[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) b[k] = d[k] = f[k] = 0.0f;
    auto master = [&](const float* m, float (&v)[8]) {
      const float4 u = __ldg(reinterpret_cast<const float4*>(m + p0));
      const float4 w = __ldg(reinterpret_cast<const float4*>(m + p0) + 1);
      v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w; v[4] = w.x; v[5] = w.y; v[6] = w.z; v[7] = w.w;
    };
    if (a.has_bias) master(a.bias, b);
    if (a.has_dark) master(a.dark, d);
    if (a.has_flat) master(a.flat, f);
    constexpr int kAhead = 4;
    for (int f0 = 0; f0 < a.nframes; f0 += kAhead) {
      Raw8 r[kAhead];
#pragma unroll
      for (int q = 0; q < kAhead; ++q)
        if (f0 + q < a.nframes) r[q] = load_raw8(a.raw + (f0 + q) * a.pixels + p0, a.raw, last);
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        if (f0 + q >= a.nframes) break;
        const int frame = a.frame[f0 + q];
        float out[8];
        bool bad = false;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const auto raw = static_cast<uint16_t>(r[q].w[k / 2] >> (16 * (k & 1)));
          out[k] = calibrate_one(decode_u16(raw, a.big_endian_bzero), b[k], d[k], f[k], a);
          bad |= !isfinite(out[k]);
        }
        float* dst = a.slots + static_cast<int64_t>(a.slot_of_frame[frame]) * a.stride + p0;
        __stcs(reinterpret_cast<float4*>(dst), make_float4(out[0], out[1], out[2], out[3]));
        __stcs(reinterpret_cast<float4*>(dst) + 1, make_float4(out[4], out[5], out[6], out[7]));
        if (bad) {
          unsigned nbad = 0;
#pragma unroll
          for (int k = 0; k < 8; ++k) nbad += !isfinite(out[k]);
          atomicAdd(a.counts + frame, nbad);
        }
      }
    }
  }
  const int tail = static_cast<int>(a.pixels - groups * 8);
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < int64_t(tail) * a.nframes;
       i += int64_t(gridDim.x) * blockDim.x) {
    const int fi = static_cast<int>(i / tail), frame = a.frame[fi];
    const int64_t p = groups * 8 + (i - static_cast<int64_t>(fi) * tail);
    const float out = calibrate_one(decode_u16(a.raw[fi * a.pixels + p], a.big_endian_bzero), a.has_bias ? a.bias[p] : 0.0f,
                                    a.has_dark ? a.dark[p] : 0.0f, a.has_flat ? a.flat[p] : 0.0f, a);
    a.slots[static_cast<int64_t>(a.slot_of_frame[frame]) * a.stride + p] = out;
    if (!isfinite(out)) atomicAdd(a.counts + frame, 1u);
  }
  if (last_cta(a.ticket, gridDim.x))
    for (int i = threadIdx.x; i < a.nframes; i += blockDim.x)
      a.nonfinite[a.frame[i]] = atomicExch(a.counts + a.frame[i], 0u);
}

// One float32 light.
__global__ void __launch_bounds__(256) calibrate_f32_kernel(CalibArgs a) {
  const int frame = a.frame[0];
  float* dst = a.slots + static_cast<int64_t>(a.slot_of_frame[frame]) * a.stride;
  for (int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; p < a.pixels;
       p += int64_t(gridDim.x) * blockDim.x) {
    const float out = calibrate_one(a.light_f32[p], a.has_bias ? a.bias[p] : 0.0f, a.has_dark ? a.dark[p] : 0.0f,
                                    a.has_flat ? a.flat[p] : 0.0f, a);
    dst[p] = out;
    warp_count_add(a.counts + frame, !isfinite(out));
  }
  if (last_cta(a.ticket, gridDim.x) && threadIdx.x == 0)
    a.nonfinite[frame] = atomicExch(a.counts + frame, 0u);
}

__global__ void __launch_bounds__(256) count_nonfinite_kernel(const float* frame, int64_t n, unsigned* counter) {
  for (int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; p < n; p += int64_t(gridDim.x) * blockDim.x) {
    warp_count_add(counter, !isfinite(frame[p]));
  }
}

__global__ void __launch_bounds__(256) count_nonfinite_slot_kernel(const float* slots, const int* slot_of_frame,
                                                                   int64_t stride, int frame, int64_t n,
                                                                   unsigned* counters) {
  const float* src = slots + static_cast<int64_t>(slot_of_frame[frame]) * stride;
  for (int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; p < n; p += int64_t(gridDim.x) * blockDim.x) {
    warp_count_add(counters + frame, !isfinite(src[p]));
  }
}

static CalibArgs make_args(gg_stack* s, const gg_calib_params_t& p) {
  CalibArgs a{};
  a.bias = s->d_bias;
  a.dark = s->d_dark;
  a.flat = s->d_flat;
  a.slots = s->d_slots;
  a.slot_of_frame = s->d_slot_of_frame;
  a.nonfinite = s->d_frame_nonfinite;
  a.counts = s->d_count_acc;
  a.ticket = s->d_tickets + s->frames + 1;
  a.stride = s->stride;
  a.pixels = s->pixels;
  a.has_bias = s->has_bias;
  a.has_dark = s->has_dark;
  a.has_flat = s->has_flat;
  a.dark_includes_bias = p.master_dark_includes_bias;
  a.dark_scale = p.dark_scale;
  a.flat_floor = p.flat_floor;
  a.pedestal = p.pedestal;
  return a;
}

// A launch deals the last pixels of its frames to threads in no order and
// publishes one non-finite count per frame, so its frames are distinct: a frame
// that comes again starts another launch, and its last entry wins.
void launch_calibrate(gg_stack* s, const CalibLaunch& job, const gg_calib_params_t& p) {
  CalibArgs a = make_args(s, p);
  a.light_f32 = job.light_f32;
  a.big_endian_bzero = job.big_endian_bzero;
  for (int k = 0; k < job.nframes;) {
    if (job.raw != nullptr) a.raw = job.raw + static_cast<int64_t>(k) * s->pixels;
    a.nframes = 0;
    while (k < job.nframes && std::find(a.frame, a.frame + a.nframes, job.frame[k]) == a.frame + a.nframes)
      a.frame[a.nframes++] = job.frame[k++];
    note_launch();
    if (job.raw != nullptr)
      calibrate_u16_kernel<<<grid_for(static_cast<size_t>((s->pixels + 7) / 8), 256, 8), 256, 0, s->stream>>>(a);
    else
      calibrate_f32_kernel<<<grid_for(static_cast<size_t>(s->pixels), 256, 8), 256, 0, s->stream>>>(a);
    check_cuda(cudaGetLastError(), "calibrate kernel launch");
  }
}

void launch_count_nonfinite(gg_stack* s, int64_t frame) {
  check_cuda(cudaMemsetAsync(s->d_frame_nonfinite + frame, 0, sizeof(unsigned), s->stream), "cudaMemsetAsync");
  const unsigned grid = grid_for(static_cast<size_t>(s->pixels), 256, 4);
  note_launch();
  count_nonfinite_slot_kernel<<<grid, 256, 0, s->stream>>>(s->d_slots, s->d_slot_of_frame, s->stride,
                                                           static_cast<int>(frame), s->pixels, s->d_frame_nonfinite);
  check_cuda(cudaGetLastError(), "count_nonfinite kernel launch");
}

static void validate_calib(const gg_calib_params_t* p) {
  require(p != nullptr, "calibration parameters are null");
  require(std::isfinite(p->dark_scale), "dark_scale must be finite");
  require(std::isfinite(p->flat_floor), "flat_floor must be finite");
  require(std::isfinite(p->pedestal), "pedestal must be finite");
}

static void ensure_lanes(gg_stack* s) {
  if (s->d_raw_lane[0] != nullptr) return;
  s->lane_bytes = static_cast<size_t>(gg_stack::kLaneFrames) * static_cast<size_t>(s->pixels) * 2;
  for (int i = 0; i < gg_stack::kLanes; ++i) {
    void* d = nullptr;
    check_cuda(cudaMalloc(&d, s->lane_bytes), "cudaMalloc(raw lane)");
    s->d_raw_lane[i] = static_cast<uint16_t*>(d);
    s->bytes_allocated += static_cast<int64_t>(s->lane_bytes);
    check_cuda(cudaHostAlloc(&s->h_pinned_lane[i], s->lane_bytes, cudaHostAllocPortable), "cudaHostAlloc(raw lane)");
    s->host_pinned_bytes += static_cast<int64_t>(s->lane_bytes);
  }
}

static bool is_pinned(const void* p) {
  cudaPointerAttributes attr{};
  if (cudaPointerGetAttributes(&attr, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return attr.type == cudaMemoryTypeHost;
}

}  // namespace gg

using namespace gg;

extern "C" {

int gg_stack_calibrate_u16(gg_stack* s, const int64_t* indices, int64_t count, const void* host_raw,
                           int big_endian_bzero, const gg_calib_params_t* params) {
  GG_API_BEGIN
  require(s != nullptr && indices != nullptr && host_raw != nullptr, "null argument");
  require(count > 0, "indices must contain at least one frame index");
  validate_calib(params);
  for (int64_t k = 0; k < count; ++k) stack_require_index(s, indices[k]);
  stack_activate(s);
  ensure_lanes(s);
  const bool pinned = is_pinned(host_raw);
  const size_t frame_bytes = static_cast<size_t>(s->pixels) * 2;
  const auto* src = static_cast<const unsigned char*>(host_raw);
  int lane = s->next_lane;
  for (int64_t k0 = 0; k0 < count; k0 += gg_stack::kLaneFrames) {
    const int nb = static_cast<int>(std::min<int64_t>(gg_stack::kLaneFrames, count - k0));
    // The lane's previous decode must finish before its buffers are reused.
    check_cuda(cudaEventSynchronize(s->lane_free[lane]), "cudaEventSynchronize(lane)");
    const unsigned char* chunk = src + static_cast<size_t>(k0) * frame_bytes;
    const void* copy_src = chunk;
    if (!pinned) {
      std::memcpy(s->h_pinned_lane[lane], chunk, frame_bytes * nb);
      copy_src = s->h_pinned_lane[lane];
    }
    check_cuda(cudaStreamWaitEvent(s->copy_stream, s->lane_free[lane], 0), "cudaStreamWaitEvent");
    check_cuda(cudaMemcpyAsync(s->d_raw_lane[lane], copy_src, frame_bytes * nb, cudaMemcpyHostToDevice,
                               s->copy_stream),
               "cudaMemcpyAsync(raw lane)");
    check_cuda(cudaEventRecord(s->lane_ready[lane], s->copy_stream), "cudaEventRecord");
    check_cuda(cudaStreamWaitEvent(s->stream, s->lane_ready[lane], 0), "cudaStreamWaitEvent");
    CalibLaunch job{};
    job.raw = s->d_raw_lane[lane];
    job.big_endian_bzero = big_endian_bzero;
    job.nframes = nb;
    for (int i = 0; i < nb; ++i) job.frame[i] = static_cast<int>(indices[k0 + i]);
    launch_calibrate(s, job, *params);
    check_cuda(cudaEventRecord(s->lane_free[lane], s->stream), "cudaEventRecord");
    lane = (lane + 1) % gg_stack::kLanes;
  }
  s->next_lane = lane;
  for (int64_t k = 0; k < count; ++k) stack_mark_loaded(s, indices[k]);
  GG_API_END
}

// ---- staged ingest: uploads run ahead of the per-frame stages ---------------
// A device copy of every frame's raw uint16 samples (frames x P) filled from
// pinned host memory on the copy stream, one event per frame when its copy
// has landed and one when its calibration has read it: the caller enqueues
// the uploads of a whole stack at once and calibrates (and processes) the
// frames in chunks while later chunks are still in flight.
struct RawStage {
  uint16_t* d_raw = nullptr;
  std::vector<cudaEvent_t> ready;     // the frame's upload has landed
  std::vector<cudaEvent_t> consumed;  // the frame's calibration has read it
  std::vector<unsigned char> uploaded;
};

static void raw_stage_release(RawStage* r) {
  if (r->d_raw) cudaFree(r->d_raw);
  for (cudaEvent_t e : r->ready) cudaEventDestroy(e);
  for (cudaEvent_t e : r->consumed) cudaEventDestroy(e);
  delete r;
}

static RawStage& raw_stage(gg_stack* s) {
  if (!s->raw_stage) {
    auto* r = new RawStage();
    s->raw_stage = r;
    s->raw_stage_free = [](void* q) { raw_stage_release(static_cast<RawStage*>(q)); };
    const size_t bytes = static_cast<size_t>(s->frames) * static_cast<size_t>(s->pixels) * 2;
    check_cuda(cudaMalloc(&r->d_raw, bytes), "cudaMalloc(raw staging)");
    s->bytes_allocated += static_cast<int64_t>(bytes);
    r->ready.assign(static_cast<size_t>(s->frames), nullptr);
    r->consumed.assign(static_cast<size_t>(s->frames), nullptr);
    r->uploaded.assign(static_cast<size_t>(s->frames), 0);
    for (int64_t k = 0; k < s->frames; ++k) {
      check_cuda(cudaEventCreateWithFlags(&r->ready[k], cudaEventDisableTiming), "cudaEventCreate(raw ready)");
      check_cuda(cudaEventCreateWithFlags(&r->consumed[k], cudaEventDisableTiming), "cudaEventCreate(raw read)");
    }
  }
  return *static_cast<RawStage*>(s->raw_stage);
}

int gg_stack_calibrate_u16_device(gg_stack* s, const int64_t* indices, int64_t count, const void* dev_raw,
                                  int big_endian_bzero, const gg_calib_params_t* params) {
  GG_API_BEGIN
  require(s != nullptr && indices != nullptr && dev_raw != nullptr, "null argument");
  require(count > 0, "indices must contain at least one frame index");
  validate_calib(params);
  for (int64_t k = 0; k < count; ++k) stack_require_index(s, indices[k]);
  stack_activate(s);
  const auto* raw = static_cast<const uint16_t*>(dev_raw);
  for (int64_t k0 = 0; k0 < count;) {
    CalibLaunch job{};
    job.raw = raw + static_cast<size_t>(k0) * static_cast<size_t>(s->pixels);
    job.big_endian_bzero = big_endian_bzero;
    while (k0 < count && job.nframes < GG_MAX_BATCH_FRAMES) job.frame[job.nframes++] = static_cast<int>(indices[k0++]);
    launch_calibrate(s, job, *params);
  }
  for (int64_t k = 0; k < count; ++k) stack_mark_loaded(s, indices[k]);
  GG_API_END
}

int gg_stack_upload_raw_u16(gg_stack* s, const int64_t* indices, int64_t count, const void* host_raw) {
  GG_API_BEGIN
  require(s != nullptr && indices != nullptr && host_raw != nullptr, "null argument");
  require(count > 0, "indices must contain at least one frame index");
  for (int64_t k = 0; k < count; ++k) stack_require_index(s, indices[k]);
  require(is_pinned(host_raw), "staged uploads need page-locked (pinned) host memory");
  stack_activate(s);
  RawStage& r = raw_stage(s);
  const size_t frame_bytes = static_cast<size_t>(s->pixels) * 2;
  const auto* src = static_cast<const unsigned char*>(host_raw);
  for (int64_t k = 0; k < count; ++k) {
    const int64_t f = indices[k];
    // the previous calibration of this frame must have read its staged copy
    check_cuda(cudaStreamWaitEvent(s->copy_stream, r.consumed[f], 0), "cudaStreamWaitEvent(raw read)");
    check_cuda(cudaMemcpyAsync(reinterpret_cast<unsigned char*>(r.d_raw) + static_cast<size_t>(f) * frame_bytes,
                               src + static_cast<size_t>(k) * frame_bytes, frame_bytes, cudaMemcpyHostToDevice,
                               s->copy_stream),
               "cudaMemcpyAsync(raw staging)");
    check_cuda(cudaEventRecord(r.ready[f], s->copy_stream), "cudaEventRecord(raw ready)");
    r.uploaded[f] = 1;
  }
  GG_API_END
}

int gg_stack_calibrate_u16_staged(gg_stack* s, const int64_t* indices, int64_t count, int big_endian_bzero,
                                  const gg_calib_params_t* params) {
  GG_API_BEGIN
  require(s != nullptr && indices != nullptr, "null argument");
  require(count > 0, "indices must contain at least one frame index");
  validate_calib(params);
  for (int64_t k = 0; k < count; ++k) stack_require_index(s, indices[k]);
  require(s->raw_stage != nullptr, "no staged raw frames: call gg_stack_upload_raw_u16 first");
  RawStage& r = raw_stage(s);
  for (int64_t k = 0; k < count; ++k) require(r.uploaded[indices[k]] != 0, "frame has no staged raw samples");
  stack_activate(s);
  // runs of consecutive frame indices share one launch (their staged copies are
  // contiguous); short runs, as a launch waits for the uploads of all its frames
  constexpr int64_t kStagedBatch = 8;
  int64_t k0 = 0;
  while (k0 < count) {
    int64_t k1 = k0 + 1;
    while (k1 < count && k1 - k0 < kStagedBatch && indices[k1] == indices[k1 - 1] + 1) ++k1;
    for (int64_t k = k0; k < k1; ++k)
      check_cuda(cudaStreamWaitEvent(s->stream, r.ready[indices[k]], 0), "cudaStreamWaitEvent(raw ready)");
    CalibLaunch job{};
    job.raw = r.d_raw + static_cast<size_t>(indices[k0]) * static_cast<size_t>(s->pixels);
    job.big_endian_bzero = big_endian_bzero;
    job.nframes = static_cast<int>(k1 - k0);
    for (int64_t k = k0; k < k1; ++k) job.frame[k - k0] = static_cast<int>(indices[k]);
    launch_calibrate(s, job, *params);
    for (int64_t k = k0; k < k1; ++k)
      check_cuda(cudaEventRecord(r.consumed[indices[k]], s->stream), "cudaEventRecord(raw read)");
    k0 = k1;
  }
  for (int64_t k = 0; k < count; ++k) stack_mark_loaded(s, indices[k]);
  GG_API_END
}

int gg_stack_calibrate_f32(gg_stack* s, int64_t index, const float* host_light, const gg_calib_params_t* params) {
  GG_API_BEGIN
  require(s != nullptr && host_light != nullptr, "null argument");
  validate_calib(params);
  stack_require_index(s, index);
  stack_activate(s);
  // The float32 light is staged in stream-ordered pool memory.
  float* staging = nullptr;
  check_cuda(cudaMallocAsync(reinterpret_cast<void**>(&staging), static_cast<size_t>(s->pixels) * 4, s->stream),
             "cudaMallocAsync(light)");
  check_cuda(cudaMemcpyAsync(staging, host_light, static_cast<size_t>(s->pixels) * 4, cudaMemcpyHostToDevice,
                             s->stream),
             "cudaMemcpyAsync(light)");
  CalibLaunch job{};
  job.light_f32 = staging;
  job.nframes = 1;
  job.frame[0] = static_cast<int>(index);
  launch_calibrate(s, job, *params);
  check_cuda(cudaFreeAsync(staging, s->stream), "cudaFreeAsync(light)");
  check_cuda(cudaStreamSynchronize(s->stream), "cudaStreamSynchronize(calibrate)");
  stack_mark_loaded(s, index);
  GG_API_END
}

int gg_calibrate_tile_f32(const float* host_light, const float* host_bias, const float* host_dark,
                          const float* host_flat, int64_t n, const gg_calib_params_t* params, float* host_out) {
  GG_API_BEGIN
  require(host_light != nullptr && host_out != nullptr, "null argument");
  require(n >= 0, "n must be non-negative");
  validate_calib(params);
  if (n == 0) return GG_OK;
  int devs = 0;
  if (cudaGetDeviceCount(&devs) != cudaSuccess || devs <= 0) {
    cudaGetLastError();
    fail(GG_ERR_NO_DEVICE, "no CUDA device is available");
  }
  const size_t bytes = static_cast<size_t>(n) * 4;
  float* d[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
  unsigned* d_counter = nullptr;
  int* d_slot = nullptr;
  auto release = [&]() {
    for (float* p : d)
      if (p) cudaFree(p);
    if (d_counter) cudaFree(d_counter);
    if (d_slot) cudaFree(d_slot);
  };
  try {
    const float* srcs[4] = {host_light, host_bias, host_dark, host_flat};
    for (int i = 0; i < 4; ++i) {
      if (!srcs[i]) continue;
      check_cuda(cudaMalloc(&d[i], bytes), "cudaMalloc(calibrate tile)");
      check_cuda(cudaMemcpy(d[i], srcs[i], bytes, cudaMemcpyHostToDevice), "cudaMemcpy(calibrate tile)");
    }
    check_cuda(cudaMalloc(&d[4], bytes), "cudaMalloc(calibrate out)");
    check_cuda(cudaMalloc(&d_counter, 3 * sizeof(unsigned)), "cudaMalloc(counter)");
    check_cuda(cudaMalloc(&d_slot, sizeof(int)), "cudaMalloc(slot)");
    check_cuda(cudaMemset(d_counter, 0, 3 * sizeof(unsigned)), "cudaMemset");
    check_cuda(cudaMemset(d_slot, 0, sizeof(int)), "cudaMemset");
    CalibArgs a{};
    a.light_f32 = d[0];
    a.bias = d[1];
    a.dark = d[2];
    a.flat = d[3];
    a.slots = d[4];
    a.slot_of_frame = d_slot;
    a.nonfinite = d_counter;
    a.counts = d_counter + 1;
    a.ticket = d_counter + 2;
    a.stride = n;
    a.pixels = n;
    a.nframes = 1;
    a.frame[0] = 0;
    a.has_bias = host_bias != nullptr;
    a.has_dark = host_dark != nullptr;
    a.has_flat = host_flat != nullptr;
    a.dark_includes_bias = params->master_dark_includes_bias;
    a.dark_scale = params->dark_scale;
    a.flat_floor = params->flat_floor;
    a.pedestal = params->pedestal;
    note_launch();
    calibrate_f32_kernel<<<grid_for(static_cast<size_t>(n), 256, 4), 256>>>(a);
    check_cuda(cudaGetLastError(), "calibrate kernel launch");
    check_cuda(cudaMemcpy(host_out, d[4], bytes, cudaMemcpyDeviceToHost), "cudaMemcpy(calibrate out)");
  } catch (...) {
    release();
    throw;
  }
  release();
  GG_API_END
}

}  // extern "C"
