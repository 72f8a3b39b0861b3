// render_fp32.cu -- ray generation + compaction, the plain FP32 march
// (CUDA cores only), the occupancy-grid build and the FP16 table copy.
//
// These kernels stand in for the external instant-ngp-renderer that
// neserver reaches over TCP (src/server.cpp:161-194): a FrameRequest's
// camera becomes one ray per pixel, rays that miss the unit cube are dropped
// by a warp-ballot prefix sum, and the survivors are marched through the
// hash-grid field and composited into RGB and expected depth.
#include <cuda_fp16.h>

#include "kernels.h"
#include "ray_slot.cuh"
#include "tile32.cuh"

namespace nes {

namespace {

constexpr int kRaygenThreads = 256;
// Twelve warps of the march per SM: 185 KB of shared memory (weights, the
// warps' encodings and activations) and 168 registers a thread.  1080p: 8 warps
// 127 ms, 10 129, 11 125, 12 121; it is bound by the products' operand reads
// (a lane's 8 x 8 tile takes 64 bytes per 64 multiply-adds, 16 cycles of the
// SM's 128 bytes a cycle against 16 of its FMA lanes).
constexpr int kMarchWarps = 12;
constexpr int kMarchThreads = 32 * kMarchWarps;

// log2 of the steps of one ray that a warp takes at once: many where the rays
// are too few for the chip's 58,368 rows, fewer where that would evaluate
// steps behind an opaque surface or leave lanes without an occupied step.  The
// line lies at two rays for three rows, above which 32 steps gain nothing in a
// dense field and lose two thirds in a sparse one.  ms, 8 and 32 steps:
//               rays   seeded scene   opaque, sparse scene
//   64x48       0.9k   1.72, 0.54     0.53, 0.36
//   256x256     14k    3.35, 2.52     0.81, 1.01
//   400x300     33k    6.55, 5.76     1.45, 2.17
//   640x360     84k    14.2, 14.0     2.84, 4.73
//   853x481     149k   24.7, 24.8     4.81, 8.33
//   1920x1080   757k   121, 124       22.4, 41.5
__device__ __forceinline__ int march32_shift(uint32_t nrays, uint32_t rows) { return nrays <= rows / 3 * 2 ? 5 : 3; }

// Grid-stride over the batch's ray-generation threads (the loop bound is
// uniform per block, and every view's thread count is a multiple of 32, so
// each warp's ballot sees whole warps).
template <class Src>
__global__ void __launch_bounds__(kRaygenThreads)
raygen_kernel(const __grid_constant__ Src src, float4* __restrict__ ray_dt, RayMeta* __restrict__ ray_meta,
              uint32_t* __restrict__ counters, uint32_t max_rays) {
  const ViewBatch& vb = src.get();
  const uint32_t total = vb.total_pixels;
  for (uint32_t base = blockIdx.x * blockDim.x; base < total; base += gridDim.x * blockDim.x) {
    const uint32_t gid = base + threadIdx.x;
    const bool valid = gid < total;
    int v = 0;
    if (valid)
      while (v + 1 < vb.n && gid >= vb.v[v + 1].pix_offset) ++v;
    int n = 0, pix = 0;
    float3 o, d;
    float ts = 0.0f;
    if (valid) {
      const DevView& V = vb.v[v];
      const uint32_t local = gid - V.pix_offset;
      const uint32_t tile = local / (kTileW * kTileH), in = local % (kTileW * kTileH);
      const uint32_t tiles_x = (uint32_t)(V.W + kTileW - 1) / kTileW;
      int px, py;
      tile_pixel(in, &px, &py);
      px += (int)((tile % tiles_x) * kTileW);
      py += (int)((tile / tiles_x) * kTileH);
      if (px < V.W && py < V.H) {  // tile padding beyond the frame edge does nothing
        pix = py * V.W + px;
        n = ray_setup(V.M, V.W, V.H, V.focal, px, py, o, d, ts);
        if (n == 0) {  // miss: nothing to march, the pixel is black at depth 0
          if (V.rgb) {
            V.rgb[(size_t)pix * 3 + 0] = 0.0f;
            V.rgb[(size_t)pix * 3 + 1] = 0.0f;
            V.rgb[(size_t)pix * 3 + 2] = 0.0f;
          }
          if (V.depth) V.depth[pix] = 0.0f;
        }
      }
    }
    const unsigned lane = threadIdx.x & 31u;
    const unsigned mask = __ballot_sync(0xffffffffu, n > 0);
    if (mask == 0) continue;
    const int leader = __ffs(mask) - 1;
    uint32_t first = 0;
    if ((int)lane == leader) first = atomicAdd(counters + kCtrRays, (uint32_t)__popc(mask));
    first = __shfl_sync(0xffffffffu, first, leader);
    if (n > 0) {
      const uint32_t slot = first + (uint32_t)__popc(mask & ((1u << lane) - 1u));
      if (slot < max_rays) {
        ray_dt[slot] = make_float4(d.x, d.y, d.z, ts);
        ray_meta[slot] = RayMeta{v, pix, n, 0};
      }
    }
  }
}

// The march: one CTA per SM, its warps independent, each with 32 samples at a
// time: (32 >> kShift) rays with their next 1 << kShift occupied steps each.
// The warp encodes its lanes' samples into its shared-memory tile, evaluates
// the MLPs as matrix products over it (tile32.cuh) and composites each ray's
// samples in step order, by shuffle.
// While a tile is in the MLPs the next one is encoded, a level per eight
// inputs of the products, so the gathers run under the multiply-adds (1080p 138
// -> 128 ms, 256x256 2.9 -> 2.6 ms).
struct MarchSmem32 {
  TileWeights32 w;
  float enc[kMarchWarps][kEnc * 32];
  float act[kMarchWarps][kTileFloats];
};

// The encoding of the warp's next samples into its rows of E, level by level.
struct EncodeNext {
  const DevScene& sc;
  float* E;
  int lane;
  float3 x;
  bool has;
  LevelGather g;
  __device__ __forceinline__ void begin(int l) { g.begin(sc.table32, sc.T, sc.dense_mask, x, l, has); }
  __device__ __forceinline__ void finish(int l) {
    const float2 f = g.finish();
    const int at = (2 * l) * 32 + (lane ^ tile_swap(2 * l));  // rows 2 l and 2 l + 1 swap alike
    E[at] = has ? f.x : 0.0f;
    E[at + 32] = has ? f.y : 0.0f;
  }
};

template <int kShift>
__device__ __forceinline__ unsigned long long march_fp32_loop(const ViewBatch& vb, const DevScene& sc,
                                                              const DevScratch& s, uint32_t nrays,
                                                              const TileWeights32& W, float* E, float* X) {
  constexpr int kLanes = 1 << kShift;
  const int lane = threadIdx.x & 31, j = lane & (kLanes - 1), ray_lane = lane - j;
  Slot q;
  EncodeNext next{sc, E, lane, make_float3(0.0f, 0.0f, 0.0f), false, {}};
  float t_next = 0.0f;
  bool exhausted = false, first = false;
  // Rays and steps of the next tile; false when the warp is out of rays.
  auto take = [&]() -> bool {
    first = false;
    for (;;) {
      next_window<kShift>(sc, q, j);
      if (first && !q.live && j == 0) write_ray(vb, s, q.id, 0.0f, 0.0f, 0.0f, 0.0f);  // no occupied sample
      if (exhausted || __ballot_sync(0xffffffffu, q.live) != 0u) break;
      first = false;
      const uint32_t base = warp_claim(s.counters + kCtrCursor, 32u >> kShift);
      if (base >= nrays) {
        exhausted = true;
        break;
      }
      const uint32_t id = base + ((uint32_t)lane >> kShift);
      if (id < nrays) {
        q.start(vb, s, id);
        first = true;
      }
    }
    next.has = take_step<kShift>(q, j, ray_lane, &t_next);
    next.x = sample_pos(q.o, q.d, t_next);
    return __ballot_sync(0xffffffffu, q.live) != 0u;
  };

  constexpr uint32_t kNone = 0xFFFFFFFFu;
  uint32_t cur = kNone;  // ray being composited in this lane (none, or it has terminated)
  // Its transmittance, and by lane c of each four its channel c (red, green,
  // blue, expected depth).
  float T = 1.0f, acc = 0.0f;
  unsigned long long my_samples = 0;
  bool more = take();
  if (more)
#pragma unroll 1
    for (int l = 0; l < kLevels; ++l) {
      next.begin(l);
      next.finish(l);
    }
  while (more) {
    __syncwarp();
    // The tile that is encoded becomes the current one.
    const float t = t_next;
    const float3 d = q.d;
    const uint32_t have = __ballot_sync(0xffffffffu, next.has);
    if (first) {
      cur = q.id;
      T = 1.0f;
      acc = 0.0f;
    }
    more = take();
    float3 c;
    const float sigma = tile_mlp32(W, E, X, lane, d, &c, next);
    const float alpha_own = -expm1f(-sigma * kDt);
    float m[4] = {c.x, c.y, c.z, t};  // own sample's channels -> own channel of the four lanes' samples
    transpose4(m, lane);
    bool stop = false;
#pragma unroll
    for (int i = 0; i < kLanes; ++i) {
      const float alpha = __shfl_sync(0xffffffffu, alpha_own, ray_lane + i);
      const float vi = __shfl_sync(0xffffffffu, m[i & 3], ray_lane + (i & ~3) + (lane & 3));
      if (cur != kNone && !stop && ((have >> (ray_lane + i)) & 1u)) {
        ++my_samples;
        const float w = T * alpha;
        acc = fmaf(w, vi, acc);
        T -= w;
        stop = T < kTStop;
      }
    }
    // A ray is complete when it has terminated (the steps of it that are
    // already encoded are dropped) or its lanes turn to another or to none.
    if (cur != kNone && (stop || first || !q.live)) {
      if (stop && !first && q.live) q.live = next.has = false;
      if (j < 4) write_channel(vb, s, cur, j, acc);
      cur = kNone;
    }
  }
  return my_samples;
}

template <class Src>
__global__ void __launch_bounds__(kMarchThreads, 1)
march_fp32_kernel(const __grid_constant__ Src src, const DevScene sc, const DevScratch s) {
  const ViewBatch& vb = src.get();
  extern __shared__ float4 smem_raw[];
  MarchSmem32& S = *reinterpret_cast<MarchSmem32*>(smem_raw);
  load_tile_weights32(S.w, sc.weights);
  __syncthreads();
  const uint32_t nrays = min(s.counters[kCtrRays], s.max_rays);
  const uint32_t rows = gridDim.x * kMarchThreads;
  float* E = S.enc[threadIdx.x >> 5];
  float* X = S.act[threadIdx.x >> 5];
  unsigned long long my_samples;
  const int shift = march32_shift(nrays, rows);
  if (shift == 5) my_samples = march_fp32_loop<5>(vb, sc, s, nrays, S.w, E, X);
  else my_samples = march_fp32_loop<3>(vb, sc, s, nrays, S.w, E, X);
  // One 64-bit atomic per warp for the sample count, which each of a ray's
  // lanes has.
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) my_samples += __shfl_down_sync(0xffffffffu, my_samples, off);
  if ((threadIdx.x & 31u) == 0 && my_samples)
    atomicAdd(reinterpret_cast<unsigned long long*>(s.counters + kCtrSamples), my_samples >> shift);
}

// The density MLP per thread, its weights in shared memory laid out for
// broadcast float4 reads (the occupancy build).
struct DensityWeights32 {
  float dw1[kHid * kEnc];    // [j][k]
  float dw2t[kHid * kDOut];  // [j][m] (transposed)
};

__device__ inline void load_density_weights32(DensityWeights32& W, const float* __restrict__ g) {
  for (int i = threadIdx.x; i < kHid * kEnc; i += blockDim.x) W.dw1[i] = g[kOffDW1 + i];
  for (int i = threadIdx.x; i < kHid * kDOut; i += blockDim.x) {
    const int j = i / kDOut, m = i % kDOut;
    W.dw2t[i] = g[kOffDW2 + m * kHid + j];
  }
}

__device__ __forceinline__ float dot32(const float* __restrict__ w, const float in[32]) {
  const float4* w4 = reinterpret_cast<const float4*>(w);
  float a = 0.0f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float4 q = w4[k];
    a = fmaf(q.x, in[4 * k + 0], a);
    a = fmaf(q.y, in[4 * k + 1], a);
    a = fmaf(q.z, in[4 * k + 2], a);
    a = fmaf(q.w, in[4 * k + 3], a);
  }
  return a;
}

// Density MLP 32->64->16 (ReLU hidden), FP32.
__device__ __forceinline__ void density_mlp32(const DensityWeights32& W, const float enc[32], float out[16]) {
#pragma unroll
  for (int m = 0; m < kDOut; ++m) out[m] = 0.0f;
#pragma unroll 4
  for (int j = 0; j < kHid; ++j) {
    const float a = fmaxf(dot32(W.dw1 + j * kEnc, enc), 0.0f);
    const float4* w2 = reinterpret_cast<const float4*>(W.dw2t + j * kDOut);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float4 q = w2[k];
      out[4 * k + 0] = fmaf(q.x, a, out[4 * k + 0]);
      out[4 * k + 1] = fmaf(q.y, a, out[4 * k + 1]);
      out[4 * k + 2] = fmaf(q.z, a, out[4 * k + 2]);
      out[4 * k + 3] = fmaf(q.w, a, out[4 * k + 3]);
    }
  }
}

constexpr int kOccThreads = 128;

__global__ void __launch_bounds__(kOccThreads)
occupancy_kernel(const DevScene sc, float threshold, uint32_t* __restrict__ occ) {
  extern __shared__ float4 smem_raw[];
  DensityWeights32& W = *reinterpret_cast<DensityWeights32*>(smem_raw);
  load_density_weights32(W, sc.weights);
  __syncthreads();
  const uint32_t cell = blockIdx.x * blockDim.x + threadIdx.x;  // grid covers 128^3 exactly
  const uint32_t cx = cell % kOccRes, cy = (cell / kOccRes) % kOccRes, cz = cell / (kOccRes * kOccRes);
  const float3 x = make_float3(((float)cx + 0.5f) / kOccRes, ((float)cy + 0.5f) / kOccRes,
                               ((float)cz + 0.5f) / kOccRes);
  float enc[kEnc];
  encode_fp32(sc.table32, sc.T, sc.dense_mask, x, enc);
  float dout[kDOut];
  density_mlp32(W, enc, dout);
  const float sigma = expf(dout[0] - 1.0f);
  const unsigned bits = __ballot_sync(0xffffffffu, sigma > threshold);
  if ((threadIdx.x & 31u) == 0) occ[cell >> 5] = bits;
}

__global__ void table_to_fp16_kernel(const float2* __restrict__ src, __half2* __restrict__ dst, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    dst[i] = __float22half2_rn(src[i]);
}

}  // namespace

cudaError_t launch_raygen(const ViewBatch& views, const DevScratch& s, cudaStream_t stream) {
  if (views.total_pixels == 0) return cudaSuccess;
  const unsigned blocks = (views.total_pixels + kRaygenThreads - 1) / kRaygenThreads;
  raygen_kernel<<<blocks, kRaygenThreads, 0, stream>>>(InParam<ViewBatch>{views}, s.ray_dt, s.ray_meta, s.counters,
                                                       s.max_rays);
  return cudaGetLastError();
}

cudaError_t launch_raygen(const ViewBatch* views_dev, uint32_t max_pixels, int num_sms, const DevScratch& s,
                          cudaStream_t stream) {
  // Enough blocks for max_pixels in one pass, at most 8 per SM (grid-stride).
  const unsigned need = (max_pixels + kRaygenThreads - 1) / kRaygenThreads;
  const unsigned cap = (unsigned)num_sms * 8u;
  const unsigned blocks = need < cap ? (need ? need : 1u) : cap;
  raygen_kernel<<<blocks, kRaygenThreads, 0, stream>>>(InMemory<ViewBatch>{views_dev}, s.ray_dt, s.ray_meta,
                                                       s.counters, s.max_rays);
  return cudaGetLastError();
}

namespace {

template <class Src>
cudaError_t launch_march_fp32_src(const Src& src, const DevScene& scene, const DevScratch& s, int num_sms,
                                  cudaStream_t stream) {
  march_fp32_kernel<Src><<<num_sms, kMarchThreads, sizeof(MarchSmem32), stream>>>(src, scene, s);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_march_fp32(const ViewBatch& views, const DevScene& scene, const DevScratch& s,
                              int num_sms, cudaStream_t stream) {
  return launch_march_fp32_src(InParam<ViewBatch>{views}, scene, s, num_sms, stream);
}

cudaError_t launch_march_fp32(const ViewBatch* views_dev, const DevScene& scene, const DevScratch& s, int num_sms,
                              cudaStream_t stream) {
  return launch_march_fp32_src(InMemory<ViewBatch>{views_dev}, scene, s, num_sms, stream);
}

cudaError_t prepare_march_fp32() {
  const cudaFuncAttribute dynamic = cudaFuncAttributeMaxDynamicSharedMemorySize;
  const int smem = (int)sizeof(MarchSmem32);
  const cudaError_t e = cudaFuncSetAttribute(march_fp32_kernel<InParam<ViewBatch>>, dynamic, smem);
  return e != cudaSuccess ? e : cudaFuncSetAttribute(march_fp32_kernel<InMemory<ViewBatch>>, dynamic, smem);
}

cudaError_t launch_occupancy(const DevScene& scene, float threshold, uint32_t* occ_out, cudaStream_t stream) {
  const int smem = (int)sizeof(DensityWeights32);
  cudaError_t e = cudaFuncSetAttribute(occupancy_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const unsigned cells = kOccRes * kOccRes * kOccRes;
  occupancy_kernel<<<cells / kOccThreads, kOccThreads, smem, stream>>>(scene, threshold, occ_out);
  return cudaGetLastError();
}

cudaError_t launch_table_to_fp16(const float2* src, __half2* dst, size_t n, cudaStream_t stream) {
  table_to_fp16_kernel<<<1024, 256, 0, stream>>>(src, dst, n);
  return cudaGetLastError();
}

}  // namespace nes
