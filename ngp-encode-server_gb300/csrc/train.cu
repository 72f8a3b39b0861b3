// train.cu -- differentiation of the renderer and the Adam refit
// (nes_trainer_* in include/nes_gb300.h).  neserver itself only renders;
// this is the training form of the same field (refit configuration: teacher
// scene seed 1, student seed 2, 2^18 rays per step, L2 on RGB + 0.1 L2 on
// depth, Adam lr 1e-2, betas (0.9, 0.99), eps 1e-15).
//
// Per step:
//  1. rays: (view, pixel) pairs (drawn from the step seed or given) -> the
//     FP32 ray set-up of rendering, with the target colour and depth;
//  2. forward, as many rays at a time as the sample list holds: the rays'
//     occupied steps listed (warp per ray), each listed sample's hash-grid
//     encoding gathered (encode_kernel; kept for the backward), the MLPs
//     evaluated (by default on the tensor cores as 3xTF32, FP32-level;
//     exact_weight_grads = 1: FP32 on the CUDA cores), then each ray
//     composited with early termination (thread per ray), keeping each
//     evaluated sample's t, alpha, transmittance and colour at its place in
//     the list; loss; then walk the samples backwards carrying
//     A = dL/dT_k for each one's compositing adjoint
//        g_w = g_C . c_k + g_D t_k,   dL/dc_k = g_C w_k,
//        dL/dsigma_k = dt T_{k+1} (g_w - A_{k+1}),
//        A_k = g_w alpha_k + A_{k+1} (1 - alpha_k),   A_K = 0,
//     with g_C = 2 (C - C*)/B and g_D = 2 lambda (D - D*)/B, written as a
//     compact 32-byte record (position, place in the list, dsigma, dc).  The
//     backward sweep keeps every term proportional to T_{k+1}; the equivalent
//     forward form with suffix sums (C - prefix) cancels in FP32 late in
//     the ray;
//  3. backward (in chunks of the records): recompute both MLPs from the
//     kept encoding, backpropagate, and stage every layer's input activations
//     and output deltas.  By default the ten layer products of the recompute
//     and the backpropagation run on the tensor cores (backward_tc_kernel,
//     tcgen05 kind::tf32) and the staging is BF16; exact_weight_grads = 1
//     keeps the products and the staging in FP32, on the CUDA cores
//     (backward_kernel); scatter_kernel adds the encoding gradients into the
//     FP32 gradient table;
//  4. weight gradients: per layer dW[out][in] += sum_s delta[s][out] act[s][in]
//     over the chunk (by default dw_tc_kernel, tcgen05 kind::f16 with BF16
//     operands; exact: dw_kernel, register-tiled split-K reduction);
//  5. Adam on the table and the weights (bias-corrected); gradients zeroed.
// An FP64 variant of the loss evaluates the same function with one parameter
// perturbed, for central finite differences.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <new>
#include <vector>

#include "ctx_internal.h"
#include "kernels.h"
#include "nes_gb300.h"
#include "tc_ptx.cuh"
#include "tile32.cuh"

using namespace nes;

namespace {

struct TrainView {
  float M[12];
  int W, H;
  float focal;
  int pad;
  uint64_t offset;  // first pixel of this view in the concatenated targets
};

// The alignments of the three structs let them be read and written in 16-byte
// words; member by member (4 bytes, 32-byte stride per lane) compositing and
// the adjoint were bound by the load / store unit, 5 L1 sectors per record:
// 106.1 ms per 122 M sample step, 112.0 without.
struct alignas(16) TrainRay {
  float ox, oy, oz, ts;
  float dx, dy, dz;
  int n;                 // march steps (0: the ray misses the cube)
  float tr, tg, tb, td;  // target colour and depth
};

struct alignas(32) ScratchSample {  // state of one evaluated sample, at its place in the sample list
  float t, alpha, T, cr, cg, cb, pad0, pad1;  // T: transmittance before the sample
};

struct alignas(32) SampleRec {  // compacted sample with its compositing adjoint
  float x, y, z;
  uint32_t place;  // in the sample list
  float dsigma, dcr, dcg, dcb;
};

// Per-sample staging of the weight-gradient reductions, in 32-sample tiles.
// Strict mode: FP32, each tile of an F-wide array F rows (features) of 32
// samples.  The tensor-core mode stages BF16 operands, see stage8.
constexpr int kStageFloats = kEnc + kHid + kCIn + kHid + kHid  // activations: enc, h1, cin, g1, g2
                             + kHid + kDOut + kHid + kHid + 8;  // deltas: dh1, dout, dg1, dg2, dlogit(3)+zeros
struct Staging {
  float *enc, *h1, *cin, *g1, *g2;       // F = 32, 64, 32, 64, 64
  float *dh1, *dout, *dg1, *dg2, *dlog;  // F = 64, 16, 64, 64, 8 (features 3..7 zero)
};
constexpr int kFDlog = 8;

__device__ __forceinline__ float* stage_tile(float* a, int F, uint32_t tile) { return a + (size_t)tile * F * 32; }

constexpr uint32_t kErrBadRay = 2u, kErrOverflow = 3u;

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// Draw i of the step: view = low word mod nviews, pixel = high word mod W*H.
__global__ void sample_pairs_kernel(uint64_t seed, int n, const TrainView* __restrict__ views, int nviews,
                                    int2* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint64_t u = mix64(mix64(seed * 256ull + 7ull) + (uint64_t)(i + 1) * 0x9E3779B97F4A7C15ull);
  const int v = (int)((u & 0xffffffffull) % (uint64_t)nviews);
  const uint64_t px = (uint64_t)views[v].W * views[v].H;
  out[i] = make_int2(v, (int)((u >> 32) % px));
}

__global__ void make_rays_kernel(const int2* __restrict__ pairs, int n, const TrainView* __restrict__ views, int nviews,
                                 const float* __restrict__ trgb, const float* __restrict__ tdep,
                                 TrainRay* __restrict__ rays, uint32_t* __restrict__ err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int2 p = pairs[i];
  TrainRay r{};
  if (p.x < 0 || p.x >= nviews || p.y < 0 || (uint64_t)p.y >= (uint64_t)views[p.x].W * views[p.x].H) {
    atomicExch(err, kErrBadRay);
    rays[i] = r;
    return;
  }
  const TrainView& V = views[p.x];
  float3 o, d;
  float ts;
  r.n = ray_setup(V.M, V.W, V.H, V.focal, p.y % V.W, p.y / V.W, o, d, ts);
  r.ox = o.x; r.oy = o.y; r.oz = o.z; r.ts = ts;
  r.dx = d.x; r.dy = d.y; r.dz = d.z;
  const uint64_t q = V.offset + (uint64_t)p.y;
  r.tr = trgb[q * 3 + 0];
  r.tg = trgb[q * 3 + 1];
  r.tb = trgb[q * 3 + 2];
  r.td = tdep[q];
  rays[i] = r;
}

struct RayOut {  // composited result of one training ray
  float C0, C1, C2, D;
  int K;           // evaluated samples up to early termination
  uint32_t first;  // the ray's occupied steps in the sample list, from its block's first one (block_first)
  uint32_t count;
  int pad;
};

// Forward, in passes over the batch's samples, so that the per-sample work
// runs with every lane of a warp busy (marched one ray per thread, the lanes
// whose ray is at an empty step would idle while the others evaluate) or on
// the tensor cores in 128-sample tiles:
//  1. count_kernel and scan_kernel: the rays' occupied steps -- the march's
//     sample set before early termination -- counted, and their places in a
//     list of all of them, ray after ray;
// then for as many rays at a time as the list holds (trainer_sizes):
//  2. list_kernel, warp per ray: (ray, step) of each sample;
//  3. encode_kernel, thread per listed sample: the hash-grid encoding, kept
//     for the backward (a warp's samples are consecutive samples of one or two
//     rays: coherent gathers);
//  4. eval_kernel (FP32, warp per 32 listed samples) or eval_tc_kernel (the
//     MLP products on tcgen05 as 3xTF32, thread = TMEM lane per sample): the
//     MLPs at that sample, its t, alpha and colour written to the sample's
//     place;
//  5. composite_kernel, thread per ray: the ray's samples in order, composited
//     and stopped at T < kTStop exactly as a one-pass march composites, with
//     each sample's transmittance and the ray's RayOut filled in.
// With eval_kernel the per-sample arithmetic is the one-pass FP32 march's;
// only the samples after an early termination are evaluated and then left
// unused.
// Rays per block of the per-ray kernels: one warp, so that a small batch still
// reaches most SMs (4,001 rays in blocks of 256 ran on 16 of the 152: the four
// per-ray kernels took 1.21 of a strict gradient's 8.4 ms, 0.52 in single
// warps; of 2^18 rays the same).  Counting and listing have a warp per ray.
constexpr int kRayBlock = 32;

// A ray per thread left a small batch's walk serial over ~800 steps and its
// list entries scattered (counting and listing 4,001 rays: 65 + 71 us; 17 + 19
// so); a 122 M sample step is 1.0 ms shorter.
//
// Walks rays [first, first + kRayBlock) of n, a warp per ray, 32 steps at a
// time: visit(k, step, occ) for ray number k of the block, occ the
// occupied steps among step .. step + 31, lane by lane.
constexpr int kWalkThreads = 512;
template <class Visit>
__device__ __forceinline__ void walk_rays(const TrainRay* __restrict__ rays, int first, int n, const DevScene& sc,
                                          Visit&& visit) {
  const int lane = threadIdx.x & 31;
  for (int k = threadIdx.x >> 5; k < kRayBlock && first + k < n; k += kWalkThreads / 32) {
    const TrainRay r = rays[first + k];
    const float3 o = make_float3(r.ox, r.oy, r.oz), d = make_float3(r.dx, r.dy, r.dz);
    for (int step = 0; step < r.n; step += 32) {
      const int st = step + lane;
      const bool in = st < r.n && occupied(sc.occ, sample_pos(o, d, fmaf((float)st + 0.5f, kDt, r.ts)));
      visit(k, step, __ballot_sync(0xffffffffu, in));
    }
  }
}

__global__ void __launch_bounds__(kWalkThreads)
count_kernel(const TrainRay* __restrict__ rays, int n, const DevScene sc, RayOut* __restrict__ rout,
             uint32_t* __restrict__ block_count) {
  static_assert(kRayBlock == 32, "a lane per ray");
  __shared__ uint32_t count[kRayBlock];
  const int lane = threadIdx.x & 31, first = blockIdx.x * kRayBlock;
  if (threadIdx.x < kRayBlock) count[threadIdx.x] = 0;
  __syncthreads();
  walk_rays(rays, first, n, sc, [&](int k, int, uint32_t occ) {
    if (lane == 0) count[k] += __popc(occ);
  });
  __syncthreads();
  if (threadIdx.x >= 32) return;
  const uint32_t cnt = count[lane];
  uint32_t incl = cnt;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += v;
  }
  if (lane == 31) block_count[blockIdx.x] = incl;
  if (first + lane < n) {
    RayOut ro{};
    ro.first = incl - cnt;
    ro.count = cnt;
    rout[first + lane] = ro;
  }
}

// block_first[b] = samples of the blocks before b (one block of 1,024 threads;
// block_first[blocks] = all samples).
constexpr int kScanThreads = 1024, kScanItems = 33;
static_assert(((1 << 20) / kRayBlock + kScanThreads) / kScanThreads <= kScanItems, "one scan block covers the largest batch");
__global__ void __launch_bounds__(kScanThreads)
scan_kernel(const uint32_t* __restrict__ block_count, int blocks, uint32_t* __restrict__ block_first) {
  __shared__ uint32_t warp_sum[kScanThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = (blocks + kScanThreads) / kScanThreads;  // covers entry `blocks` too
  const int i0 = threadIdx.x * per;
  uint32_t v[kScanItems], sum = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = k < per && i0 + k < blocks ? block_count[i0 + k] : 0u;
    sum += v[k];
  }
  uint32_t incl = sum;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += u;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  uint32_t first = incl - sum;
  for (int w = 0; w < warp; ++w) first += warp_sum[w];
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (k < per && i0 + k <= blocks) block_first[i0 + k] = first;
    first += v[k];
  }
}

// The samples of rays [0, n) from list place 0 (the rays' blocks start at
// sample `base` of the batch).
__global__ void __launch_bounds__(kWalkThreads)
list_kernel(const TrainRay* __restrict__ rays, int n, const DevScene sc, const RayOut* __restrict__ rout,
            const uint32_t* __restrict__ block_first, uint32_t base, uint2* __restrict__ list) {
  const uint32_t lane = threadIdx.x & 31;
  const int first = blockIdx.x * kRayBlock;
  uint2* out = nullptr;
  walk_rays(rays, first, n, sc, [&](int k, int step, uint32_t occ) {
    if (step == 0) out = list + (block_first[blockIdx.x] - base + rout[first + k].first);
    if ((occ >> lane) & 1u) out[__popc(occ & ((1u << lane) - 1u))] = make_uint2((uint32_t)(first + k), step + lane);
    out += __popc(occ);
  });
}

// Encodings of the listed samples, FP32: 32-sample tiles of 8 chunks, a
// chunk four features (two levels) of the tile's samples, 16 bytes each.
constexpr int kEncTileFloats = kEnc * 32;
__device__ __forceinline__ float4* enc_chunk(float* enc, uint32_t sample, int chunk) {
  return reinterpret_cast<float4*>(enc + (size_t)(sample >> 5) * kEncTileFloats + chunk * 128 + (sample & 31u) * 4);
}
__device__ __forceinline__ float4 enc_chunk(const float* __restrict__ enc, uint32_t sample, int chunk) {
  return __ldg(reinterpret_cast<const float4*>(enc + (size_t)(sample >> 5) * kEncTileFloats + chunk * 128 + (sample & 31u) * 4));
}

// Gathering in a kernel of its own lets every SM hold as many samples as its
// registers allow and overlap their table reads; inside the MLP kernels only
// the 256 or 512 threads that TMEM has room for did, twice per sample: 58 of
// the backward phase's 161 ms and 16 of the forward's 50 ms at 122 M samples.
constexpr int kEncThreads = 256;
__global__ void __launch_bounds__(kEncThreads)
encode_kernel(const uint2* __restrict__ list, uint32_t m, const TrainRay* __restrict__ rays, const DevScene sc,
              float* __restrict__ enc) {
  const uint32_t j = blockIdx.x * kEncThreads + threadIdx.x;
  if (j >= m) return;
  const uint2 e = list[j];
  const TrainRay& r = rays[e.x];
  const float t = fmaf((float)e.y + 0.5f, kDt, r.ts);
  const float3 x = sample_pos(make_float3(r.ox, r.oy, r.oz), make_float3(r.dx, r.dy, r.dz), t);
#pragma unroll
  for (int c = 0; c < kEnc / 4; ++c) {
    float4 f;
    encode_level_fp32(sc.table32, sc.T, sc.dense_mask, x, 2 * c, f.x, f.y);
    encode_level_fp32(sc.table32, sc.T, sc.dense_mask, x, 2 * c + 1, f.z, f.w);
    *enc_chunk(enc, j, c) = f;
  }
}

// A warp's samples' features -> the rows of its shared-memory tile.
__device__ __forceinline__ void load_enc_tile(const float* __restrict__ enc, uint32_t sample, bool valid, float* E,
                                              int lane) {
#pragma unroll
  for (int c = 0; c < kEnc / 4; ++c) {
    const float4 v = valid ? enc_chunk(enc, sample, c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float* row = E + 4 * c * 32 + (lane ^ tile_swap(4 * c));  // the chunk's four rows swap alike
    row[0] = v.x;
    row[32] = v.y;
    row[64] = v.z;
    row[96] = v.w;
  }
  __syncwarp();
}

// All 32 features of a listed sample.
__device__ __forceinline__ void load_enc(const float* __restrict__ enc, uint32_t sample, float (&f)[kEnc]) {
#pragma unroll
  for (int c = 0; c < kEnc / 4; ++c) {
    const float4 v = enc_chunk(enc, sample, c);
    f[4 * c + 0] = v.x;
    f[4 * c + 1] = v.y;
    f[4 * c + 2] = v.z;
    f[4 * c + 3] = v.w;
  }
}

// The FP32 MLPs of the listed samples, a warp 32 at a time as matrix products
// (tile32.cuh), over the list in strides of the grid (1.88 M samples: 0.61 ms;
// one sample per thread with the weights broadcast, 1.01).
constexpr int kEvalWarps = 12;
struct EvalSmem {
  TileWeights32 w;
  float enc[kEvalWarps][kEnc * 32];
  float act[kEvalWarps][kTileFloats];
};

__global__ void __launch_bounds__(32 * kEvalWarps, 1)
eval_kernel(const uint2* __restrict__ list, uint32_t m, const TrainRay* __restrict__ rays, const DevScene sc,
            const float* __restrict__ encs, ScratchSample* __restrict__ scratch) {
  extern __shared__ float4 smem_raw[];
  EvalSmem& S = *reinterpret_cast<EvalSmem*>(smem_raw);
  load_tile_weights32(S.w, sc.weights);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* const E = S.enc[warp];
  NoOtherWork none;
  const uint32_t tiles = (m + 31u) / 32u;
  for (uint32_t tile = blockIdx.x * kEvalWarps + warp; tile < tiles; tile += gridDim.x * kEvalWarps) {
    const uint32_t j = tile * 32u + (uint32_t)lane;
    const bool valid = j < m;
    float t = 0.0f;
    float3 d = make_float3(0.0f, 0.0f, 1.0f);
    if (valid) {
      const uint2 e = list[j];
      const TrainRay& r = rays[e.x];
      d = make_float3(r.dx, r.dy, r.dz);
      t = fmaf((float)e.y + 0.5f, kDt, r.ts);
    }
    load_enc_tile(encs, j, valid, E, lane);
    float3 c;
    const float sigma = tile_mlp32(S.w, E, S.act[warp], lane, d, &c, none);
    if (valid) scratch[j] = ScratchSample{t, -expm1f(-sigma * kDt), 0.0f, c.x, c.y, c.z, 0.0f, 0.0f};
    __syncwarp();  // E is written again
  }
}

__global__ void __launch_bounds__(kRayBlock)
composite_kernel(int n, ScratchSample* __restrict__ scratch, const uint32_t* __restrict__ block_first, uint32_t base,
                 RayOut* __restrict__ rout) {
  const int i = blockIdx.x * kRayBlock + threadIdx.x;
  if (i >= n) return;
  RayOut ro = rout[i];
  ScratchSample* row = scratch + (block_first[blockIdx.x] - base + ro.first);
  float T = 1.0f, C0 = 0.0f, C1 = 0.0f, C2 = 0.0f, D = 0.0f;
  int K = 0;
  bool stop = false;
  // Rows in batches of kBatch, all loaded before the first is used: the
  // stop test of one sample no longer holds back the next sample's load.
  constexpr uint32_t kBatch = 8;
  for (uint32_t k0 = 0; k0 < ro.count && !stop; k0 += kBatch) {
    ScratchSample q[kBatch];
#pragma unroll
    for (uint32_t u = 0; u < kBatch; ++u)
      if (k0 + u < ro.count) q[u] = row[k0 + u];
#pragma unroll
    for (uint32_t u = 0; u < kBatch; ++u) {
      if (stop || k0 + u >= ro.count) break;
      const float w = T * q[u].alpha;
      row[k0 + u].T = T;
      ++K;
      C0 = fmaf(w, q[u].cr, C0);
      C1 = fmaf(w, q[u].cg, C1);
      C2 = fmaf(w, q[u].cb, C2);
      D = fmaf(w, q[u].t, D);
      T -= w;
      stop = T < kTStop;
    }
  }
  ro.C0 = C0;
  ro.C1 = C1;
  ro.C2 = C2;
  ro.D = D;
  ro.K = K;
  rout[i] = ro;
}

// Loss and compositing adjoint, thread per ray: the ray's samples are walked
// backwards carrying A = dL/dT (see the file comment) and written as compact
// records; one record-range atomic per warp (warp prefix sum of K).
__global__ void __launch_bounds__(kRayBlock)
adjoint_kernel(const TrainRay* __restrict__ rays, const RayOut* __restrict__ rout, int n,
               const ScratchSample* __restrict__ scratch, const uint32_t* __restrict__ block_first, uint32_t list_base,
               SampleRec* __restrict__ recs, uint32_t capacity,
               uint32_t* __restrict__ cursor, uint32_t* __restrict__ err, double* __restrict__ loss_sum,
               float depth_w, float inv_n) {
  const int i = blockIdx.x * kRayBlock + threadIdx.x;
  const unsigned lane = threadIdx.x & 31u;
  TrainRay r{};
  RayOut ro{};
  if (i < n) {
    r = rays[i];
    ro = rout[i];
  }
  const int K = i < n ? ro.K : 0;
  int incl = K;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, off);
    if ((int)lane >= off) incl += v;
  }
  uint32_t base = 0;
  if (lane == 31 && incl > 0) base = atomicAdd(cursor, (uint32_t)incl);
  base = __shfl_sync(0xffffffffu, base, 31) + (uint32_t)(incl - K);
  float my_loss = 0.0f;
  if (i < n) {
    const float ec0 = ro.C0 - r.tr, ec1 = ro.C1 - r.tg, ec2 = ro.C2 - r.tb, ed = ro.D - r.td;
    my_loss = (ec0 * ec0 + ec1 * ec1 + ec2 * ec2 + depth_w * ed * ed) * inv_n;
    if (K > 0 && base + (uint32_t)K > capacity) {
      atomicExch(err, kErrOverflow);
    } else if (K > 0) {
      const float gC0 = 2.0f * ec0 * inv_n, gC1 = 2.0f * ec1 * inv_n, gC2 = 2.0f * ec2 * inv_n;
      const float gD = 2.0f * depth_w * ed * inv_n;
      const float3 o = make_float3(r.ox, r.oy, r.oz), d = make_float3(r.dx, r.dy, r.dz);
      const uint32_t place = block_first[blockIdx.x] - list_base + ro.first;
      const ScratchSample* row = scratch + place;
      float A = 0.0f;
      // Rows in batches of kBatch from the back, all loaded before the
      // first is used (the loads do not wait on the sweep's arithmetic).
      constexpr int kBatch = 8;
      for (int k1 = K - 1; k1 >= 0; k1 -= kBatch) {
        ScratchSample qb[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
          if (k1 - u >= 0) qb[u] = row[k1 - u];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const int k = k1 - u;
          if (k < 0) break;
          const ScratchSample& q = qb[u];
          const float w = q.T * q.alpha;
          const float T1 = q.T - w;
          const float gw = fmaf(gC0, q.cr, fmaf(gC1, q.cg, fmaf(gC2, q.cb, gD * q.t)));
          const float dsig = kDt * T1 * (gw - A);
          const float3 x = sample_pos(o, d, q.t);
          recs[base + k] = SampleRec{x.x, x.y, x.z, place + (uint32_t)k, dsig, gC0 * w, gC1 * w, gC2 * w};
          A = fmaf(gw, q.alpha, A * (1.0f - q.alpha));
        }
      }
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) my_loss += __shfl_down_sync(0xffffffffu, my_loss, off);
  if (lane == 0 && my_loss != 0.0f) atomicAdd(loss_sum, (double)my_loss);
}

// Strict backward of the chunk [first, first + count), a warp 32 records at a
// time: both MLPs recomputed and backpropagated as matrix products over the
// warp's shared-memory tile (tile32.cuh), FP32 throughout, activations and
// deltas staged from the lanes' registers.  ReLU masks are 64 bits of a lane's
// own outputs: a layer's output and its delta lie in the same lanes.  Records
// past the chunk's end have zero adjoints, hence zero deltas.  One sample per
// thread with the weights broadcast from shared memory (L1 / shared-memory
// pipe 87 % busy) took 3.94 ms per 1.88 M records, scatter-add included; this
// 1.46 and scatter_kernel 0.43.
constexpr int kBwdWarps = 12;
struct BackwardSmem {
  TileWeights32 w;                 // [input][output]
  float dw1[kHid * kEnc];          // and as the products back want them: [output][input]
  float dw2[kDOut * kHid];
  float cw1[kHid * kCIn];
  float cw2[kHid * kHid];
  float act[kBwdWarps][kTileFloats];
  float dlog[kBwdWarps][3 * 32];
};

// v where the lane's i-th four mask bits are set, else 0.
__device__ __forceinline__ float4 masked4(const float4& v, uint64_t mask, int i) {
  const uint32_t m = (uint32_t)(mask >> (4 * i));
  return make_float4((m & 1u) ? v.x : 0.0f, (m & 2u) ? v.y : 0.0f, (m & 4u) ? v.z : 0.0f, (m & 8u) ? v.w : 0.0f);
}
__device__ __forceinline__ uint64_t positive4(const float4& v, int i) {
  return (uint64_t)((v.x > 0.0f ? 1u : 0u) | (v.y > 0.0f ? 2u : 0u) | (v.z > 0.0f ? 4u : 0u) | (v.w > 0.0f ? 8u : 0u))
         << (4 * i);
}

__global__ void __launch_bounds__(32 * kBwdWarps, 1)
backward_kernel(const SampleRec* __restrict__ recs, uint32_t first, uint32_t count, const uint2* __restrict__ list,
                const TrainRay* __restrict__ rays, const float* __restrict__ encs, const DevScene sc, Staging st,
                float* __restrict__ denc) {
  extern __shared__ float4 smem_raw[];
  BackwardSmem& S = *reinterpret_cast<BackwardSmem*>(smem_raw);
  load_tile_weights32(S.w, sc.weights);
  for (int i = threadIdx.x; i < kHid * kEnc; i += blockDim.x) S.dw1[i] = sc.weights[kOffDW1 + i];
  for (int i = threadIdx.x; i < kDOut * kHid; i += blockDim.x) S.dw2[i] = sc.weights[kOffDW2 + i];
  for (int i = threadIdx.x; i < kHid * kCIn; i += blockDim.x) S.cw1[i] = sc.weights[kOffCW1 + i];
  for (int i = threadIdx.x; i < kHid * kHid; i += blockDim.x) S.cw2[i] = sc.weights[kOffCW2 + i];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* const X = S.act[warp];
  float* const D = S.dlog[warp];
  NoOtherWork none;
  const uint32_t tiles = (count + 31u) / 32u;
  for (uint32_t tile = blockIdx.x * kBwdWarps + warp; tile < tiles; tile += gridDim.x * kBwdWarps) {
    const uint32_t s = tile * 32u + (uint32_t)lane;
    const bool valid = s < count;
    SampleRec q{};
    float3 dir = make_float3(0.0f, 0.0f, 1.0f);
    if (valid) {
      q = recs[first + s];
      const TrainRay& r = rays[list[q.place].x];
      dir = make_float3(r.dx, r.dy, r.dz);
    }
    // Stages and passes on a lane's four outputs of row `row`.
    auto put = [&](float* tile_rows, int row, int sample, const float4& v) {
      *reinterpret_cast<float4*>(tile_rows + row * 32 + sample) = v;
      return v;
    };
    // ---- forward recompute ----
    load_enc_tile(encs, q.place, valid, X, lane);
    {
      float* const rows = stage_tile(st.enc, kEnc, tile);
#pragma unroll
      for (int k = 0; k < kEnc; ++k) rows[k * 32 + lane] = X[k * 32 + (lane ^ tile_swap(k))];
    }
    uint64_t m_h1 = 0, m_g1 = 0, m_g2 = 0;
    float* rows = stage_tile(st.h1, kHid, tile);
    tile_layer64(S.w.dw1, kEnc, X, X, lane, none, 0, [&](int i, int row, int sample, const float4& v) {
      m_h1 |= positive4(v, i);
      return put(rows, row, sample, relu4(v));
    });
    float sh[16];
    const float sigma = expf(tile_colour_input(S.w.dw2, X, lane, dir, sh) - 1.0f);
    rows = stage_tile(st.cin, kCIn, tile);
#pragma unroll
    for (int k = 0; k < kCIn; ++k) rows[k * 32 + lane] = k < 16 ? sh[k] : X[k * 32 + (lane ^ tile_swap(k))];
    rows = stage_tile(st.g1, kHid, tile);
    tile_layer64(S.w.cw1, kCIn, X, X, lane, none, 0, [&](int i, int row, int sample, const float4& v) {
      m_g1 |= positive4(v, i);
      return put(rows, row, sample, relu4(v));
    });
    rows = stage_tile(st.g2, kHid, tile);
    tile_layer64(S.w.cw2, kHid, X, X, lane, none, 0, [&](int i, int row, int sample, const float4& v) {
      m_g2 |= positive4(v, i);
      return put(rows, row, sample, relu4(v));
    });
    const float3 lg = tile_logits(S.w.cw3, X, lane);
    // ---- backward ----
    {
      const float c0 = sigmoidf(lg.x), c1 = sigmoidf(lg.y), c2 = sigmoidf(lg.z);
      const float dl[3] = {q.dcr * c0 * (1.0f - c0), q.dcg * c1 * (1.0f - c1), q.dcb * c2 * (1.0f - c2)};
      rows = stage_tile(st.dlog, kFDlog, tile);
#pragma unroll
      for (int c = 0; c < kFDlog; ++c) rows[c * 32 + lane] = c < 3 ? dl[c] : 0.0f;
#pragma unroll
      for (int c = 0; c < 3; ++c) D[c * 32 + lane] = dl[c];
    }
    __syncwarp();
    rows = stage_tile(st.dg2, kHid, tile);
    {  // dg2 = (cW3^T dlogit) of the lane's outputs and samples, as tile_layer64 gives them
      const int sg = 4 * ((lane >> 1) & 3), og = 4 * ((lane & 1) | ((lane >> 2) & 6));
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float4 d[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) d[c] = *reinterpret_cast<const float4*>(D + c * 32 + sg + 16 * h);
#pragma unroll
        for (int o = 0; o < 8; ++o) {
          const int row = og + (o & 3) + (o >> 2) * 32;
          const float4 w = *reinterpret_cast<const float4*>(S.w.cw3 + row * 4);
          float4 v;
          v.x = fmaf(w.x, d[0].x, fmaf(w.y, d[1].x, w.z * d[2].x));
          v.y = fmaf(w.x, d[0].y, fmaf(w.y, d[1].y, w.z * d[2].y));
          v.z = fmaf(w.x, d[0].z, fmaf(w.y, d[1].z, w.z * d[2].z));
          v.w = fmaf(w.x, d[0].w, fmaf(w.y, d[1].w, w.z * d[2].w));
          *reinterpret_cast<float4*>(X + row * 32 + ((sg + 16 * h) ^ tile_swap(row))) =
              put(rows, row, sg + 16 * h, masked4(v, m_g2, 2 * o + h));
        }
      }
    }
    __syncwarp();
    rows = stage_tile(st.dg1, kHid, tile);
    tile_layer64(S.cw2, kHid, X, X, lane, none, 0, [&](int i, int row, int sample, const float4& v) {
      return put(rows, row, sample, masked4(v, m_g1, i));
    });
    rows = stage_tile(st.dout, kDOut, tile);
    tile_layer16<kHid, kCIn>(S.cw1 + 16, X, lane, [&](int m, int sample, const float4& v) {
      if (m == 15) return;  // the input's padding column
      *reinterpret_cast<float4*>(X + (1 + m) * 32 + (sample ^ tile_swap(1 + m))) = put(rows, 1 + m, sample, v);
    });
    X[lane] = rows[lane] = q.dsigma * sigma;  // row 0
    __syncwarp();
    rows = stage_tile(st.dh1, kHid, tile);
    tile_layer64(S.dw2, kDOut, X, X, lane, none, 0, [&](int i, int row, int sample, const float4& v) {
      return put(rows, row, sample, masked4(v, m_h1, i));
    });
    {  // the encoding's gradient: samples 4 sg + {0..3, 16..19}, features 4 og + {0..3}, a chunk of denc
      const int sg = 4 * ((lane >> 1) & 3), og = (lane & 1) | ((lane >> 2) & 6);
      float acc[4][8];
#pragma unroll
      for (int o = 0; o < 4; ++o)
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[o][k] = 0.0f;
#pragma unroll 1
      for (int k0 = 0; k0 < kHid; k0 += 8) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float* xr = X + (k0 + k) * 32;
          const float4 x0 = *reinterpret_cast<const float4*>(xr + (sg ^ tile_swap(k)));
          const float4 x1 = *reinterpret_cast<const float4*>(xr + ((sg + 16) ^ tile_swap(k)));
          const float4 w0 = *reinterpret_cast<const float4*>(S.dw1 + (k0 + k) * kEnc + 4 * og);
          const float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
          const float w[4] = {w0.x, w0.y, w0.z, w0.w};
#pragma unroll
          for (int o = 0; o < 4; ++o)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[o][i] = fmaf(w[o], x[i], acc[o][i]);
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
        *enc_chunk(denc, tile * 32u + (uint32_t)(sg + (i & 3) + (i >> 2) * 16), og) =
            make_float4(acc[0][i], acc[1][i], acc[2][i], acc[3][i]);
    }
    __syncwarp();  // X is written again
  }
}

// dW[o][i] += sum_s delta[s][o] * act[s][i] over `tiles` staged tiles of 32
// samples (IN activation features, LDD-wide delta tiles of which OUT are
// real).  A thread owns P x Q of dW, four samples at a time; when these are
// fewer than the block's threads, thread groups split the samples of a
// 64-sample smem tile.  Each block reduces a contiguous range of samples,
// the next tile's reads in flight during the current one's products, and adds
// its partial dW with one atomic per element and group.  All five per 1.88 M
// samples: 1.01 ms (3.5 GB read), 2.03 with 4 x 4 per thread, one sample at a
// time and a transposing copy.
constexpr int kDwThreads = 256;
constexpr int kDwSamples = 64;

template <int IN, int OUT, int LDD, int P, int Q>
__global__ void __launch_bounds__(kDwThreads)
dw_kernel(const float* __restrict__ act, const float* __restrict__ delta, uint32_t tiles, float* __restrict__ dw) {
  constexpr int TI = IN / P, TO = LDD / Q, THREADS = TI * TO;
  static_assert(TI == 8 && IN % P == 0 && LDD % Q == 0 && TO % 2 == 0 && OUT <= LDD && kDwThreads % THREADS == 0,
                "thread tiles");
  constexpr int G = kDwThreads / THREADS;  // sample groups
  static_assert(G <= kDwSamples / 4, "at least four samples per group");
  // Rows of 64 samples padded by 4 floats: eight neighbouring rows' 16-byte
  // reads fall into different banks.
  constexpr int kRow = kDwSamples + 4;
  __shared__ __align__(16) float sa[IN][kRow];
  __shared__ __align__(16) float sd[LDD][kRow];
  const int tid = threadIdx.x;
  // As in tile_layer64: lanes i and i ^ 1 share an activation row, i and i ^ 2
  // a delta row.
  const int ti = (tid >> 1) & 7, to = ((tid & 1) | ((tid >> 4) << 1)) % TO, grp = tid / THREADS;
  constexpr int NA = IN * kDwSamples / 4 / kDwThreads;                                // float4 per thread
  constexpr int ND = (LDD * kDwSamples / 4 + kDwThreads - 1) / kDwThreads;
  const uint32_t pairs = (tiles + 1u) / 2u;  // 64-sample tiles
  const uint32_t per = (pairs + gridDim.x - 1) / gridDim.x;
  const uint32_t lo = blockIdx.x * per, hi = min(pairs, lo + per);
  const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  // float4 e of a 64-sample tile of an F-wide array: staged tile e / (8 F),
  // feature e / 8 % F, samples 4 (e % 8) and on.
  auto read = [&](const float* a, int F, uint32_t pair, int e) {
    const uint32_t t = 2u * pair + (uint32_t)(e / (8 * F));
    return t < tiles ? __ldg(reinterpret_cast<const float4*>(a + (size_t)t * F * 32) + e % (8 * F)) : zero;
  };
  float4 pa[NA], pd[ND];
  auto fetch = [&](uint32_t pair) {
#pragma unroll
    for (int n = 0; n < NA; ++n) pa[n] = read(act, IN, pair, tid + n * kDwThreads);
#pragma unroll
    for (int n = 0; n < ND; ++n)
      if (tid + n * kDwThreads < LDD * kDwSamples / 4) pd[n] = read(delta, LDD, pair, tid + n * kDwThreads);
  };
  float acc[P][Q];
#pragma unroll
  for (int p = 0; p < P; ++p)
#pragma unroll
    for (int c = 0; c < Q; ++c) acc[p][c] = 0.0f;
  if (lo < hi) fetch(lo);
  for (uint32_t pair = lo; pair < hi; ++pair) {
#pragma unroll
    for (int n = 0; n < NA; ++n) {
      const int e = tid + n * kDwThreads;
      *reinterpret_cast<float4*>(&sa[e / 8 % IN][e / (8 * IN) * 32 + (e & 7) * 4]) = pa[n];
    }
#pragma unroll
    for (int n = 0; n < ND; ++n) {
      const int e = tid + n * kDwThreads;
      if (e < LDD * kDwSamples / 4) *reinterpret_cast<float4*>(&sd[e / 8 % LDD][e / (8 * LDD) * 32 + (e & 7) * 4]) = pd[n];
    }
    __syncthreads();
    if (pair + 1 < hi) fetch(pair + 1);
#pragma unroll 1
    for (int r = 4 * grp; r < kDwSamples; r += 4 * G) {
      float4 a[P];
#pragma unroll
      for (int p = 0; p < P; ++p) a[p] = *reinterpret_cast<const float4*>(&sa[ti + p * TI][r]);
#pragma unroll
      for (int c = 0; c < Q; ++c) {
        const float4 d = *reinterpret_cast<const float4*>(&sd[to + c * TO][r]);
#pragma unroll
        for (int p = 0; p < P; ++p)
          acc[p][c] = fmaf(d.w, a[p].w, fmaf(d.z, a[p].z, fmaf(d.y, a[p].y, fmaf(d.x, a[p].x, acc[p][c]))));
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int c = 0; c < Q; ++c) {
    const int o = to + c * TO;
    if (o < OUT)
#pragma unroll
      for (int p = 0; p < P; ++p)
        if (acc[p][c] != 0.0f) atomicAdd(dw + o * IN + ti + p * TI, acc[p][c]);
  }
}

// ---------------- weight gradients on the tensor cores (kind::f16, BF16 operands) ----------------
// The tensor-core backward stages its activations and deltas as BF16 (FP32's
// exponent range, 8-bit mantissa; FP16's range cannot hold the deltas) in the
// 16-bit operand layout of stage8: half the bytes of FP32 staging written by
// the backward and read back here, the round trip that bounds both kernels.
// Per 32-sample tile, two MMA groups, M = 128, K = 32 as two K = 16 steps:
//   D1[128 x 144] += [enc | cin | h1] (rows = features) x [dh1 | dg1 | dout]^T
//   D2[128 x  80] += [g1 | g2] x [dg2 | dlog | 0]^T
// whose diagonal blocks are the five dW^T (D1[enc][dh1] = DW1^T, D1[cin][dg1]
// = CW1^T, D1[h1][dout] = DW2^T, D2[g1][dg2] = CW2^T, D2[g2][dlog] = CW3^T);
// the off-diagonal products are discarded.  D stays in TMEM across all of a
// CTA's tiles and is added to dW once at the end.  One CTA per SM: warp 0
// lane 0 streams tiles into a 3-stage ring with bulk copies (one per array,
// the staging is already in the operand layout), warp 1 lane 0 issues the
// MMAs and releases stages by tcgen05.commit, warps 0 to 3 read D back.  dg2 is
// not staged: warps 4 to 7 make it, (dlog cW3) where g2 > 0, from the FP32 dlog
// and the BF16 g2 of the tile, with the operands of the backward chain's own
// product so that it is the same dg2.  The kernel is bound by reading the staging
// (26,112 B per tile, 7 TB/s; with dg2 staged 30,208, which also cost the
// backward, bound by writing it: 67.7 ms for both and the scatter-add at 122 M
// records, 65.3 so).
constexpr int kTcStages = 3;
// Operand tiles of 32 records, BF16 (64 bytes per feature row).
constexpr uint32_t kA1Bytes = 128 * 64, kB1Bytes = 144 * 64, kA2Bytes = 128 * 64, kB2Bytes = 80 * 64;
constexpr uint32_t kStageBytes = kA1Bytes + kB1Bytes + kA2Bytes + kB2Bytes;
constexpr uint32_t kTileTx = (kEnc + kCIn + kHid + kHid + kHid + kDOut + kHid + kHid) * 64 + 32 * 16;
constexpr uint32_t kD1Col = 0, kD2Col = 144, kTmemCols = 256;
constexpr int kDwTcThreads = 256, kDwDeltaThreads = 128;  // warps 4..7 compute dg2 and dlog
constexpr uint32_t kErrTimeout = 4u;

struct DwTcSmem {
  uint8_t stage[kTcStages][kStageBytes];
  float4 dlog[kTcStages][32];
  uint64_t full[kTcStages], ready[kTcStages], empty[kTcStages], done;
  uint32_t tmem_base;
};

// Two FP32 values -> packed BF16 (round to nearest even), lo in the low half.
__device__ __forceinline__ uint32_t bf16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// The TF32 operand that the tensor core reads of an FP32 value.
__device__ __forceinline__ float tf32_trunc(float v) { return __uint_as_float(__float_as_uint(v) & 0xffffe000u); }

__global__ void __launch_bounds__(kDwTcThreads, 1)
dw_tc_kernel(Staging st, const float* __restrict__ cw3, uint32_t ntiles, float* __restrict__ dw,
             uint32_t* __restrict__ err) {
  extern __shared__ __align__(128) uint8_t smem_dw[];
  DwTcSmem& S = *reinterpret_cast<DwTcSmem*>(smem_dw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t per = (ntiles + gridDim.x - 1) / gridDim.x;
  const uint32_t t0 = blockIdx.x * per, t1 = min(ntiles, t0 + per);
  if (t1 <= t0) return;  // uniform over the CTA, before any barrier or TMEM use
  const uint32_t my = t1 - t0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kTcStages; ++i) {
      tc::mbar_init(&S.full[i], 1);
      tc::mbar_init(&S.ready[i], kDwDeltaThreads);
      tc::mbar_init(&S.empty[i], 1);
    }
    tc::mbar_init(&S.done, 1);
    tc::fence_mbar_init();
  }
  // B2 rows 72..79 are never copied: zero in every stage.
  for (int i = threadIdx.x; i < kTcStages * 128; i += blockDim.x)
    reinterpret_cast<float*>(S.stage[i / 128] + kA1Bytes + kB1Bytes + kA2Bytes + 72 * 64)[i % 128] = 0.0f;
  tc::fence_async_smem();
  if (warp == 1) {
    tc::tmem_alloc(&S.tmem_base, kTmemCols);
    tc::tmem_relinquish();
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = S.tmem_base;
  if (warp == 0 && lane == 0) {  // producer
    uint32_t issued = 0;
    bool ok = true;
    for (uint32_t i = 0; i < my; ++i) {
      const int sidx = (int)(i % kTcStages);
      if (i >= (uint32_t)kTcStages && !tc::mbar_wait_sleep(&S.empty[sidx], ((i / kTcStages) & 1u) ^ 1u)) {
        ok = false;
        break;
      }
      uint8_t* a1 = S.stage[sidx];
      uint8_t* b1 = a1 + kA1Bytes;
      uint8_t* a2 = b1 + kB1Bytes;
      const size_t t = t0 + i;
      uint64_t* bar = &S.full[sidx];
      tc::mbar_arrive_expect_tx(bar, kTileTx);
      // Tile t of an F-wide BF16 array: F x 64 bytes at byte t x F x 64.
      auto tile = [&](const float* arr, int F) { return reinterpret_cast<const uint8_t*>(arr) + t * F * 64; };
      tc::bulk_g2s(a1, tile(st.enc, kEnc), kEnc * 64, bar);
      tc::bulk_g2s(a1 + kEnc * 64, tile(st.cin, kCIn), kCIn * 64, bar);
      tc::bulk_g2s(a1 + (kEnc + kCIn) * 64, tile(st.h1, kHid), kHid * 64, bar);
      tc::bulk_g2s(b1, tile(st.dh1, kHid), kHid * 64, bar);
      tc::bulk_g2s(b1 + kHid * 64, tile(st.dg1, kHid), kHid * 64, bar);
      tc::bulk_g2s(b1 + 2 * kHid * 64, tile(st.dout, kDOut), kDOut * 64, bar);
      tc::bulk_g2s(a2, tile(st.g1, kHid), kHid * 64, bar);
      tc::bulk_g2s(a2 + kHid * 64, tile(st.g2, kHid), kHid * 64, bar);
      tc::bulk_g2s(S.dlog[sidx], tile(st.dlog, 8), 32 * 16, bar);
      ++issued;
    }
    if (!ok) atomicExch(err, kErrTimeout);
    // Copies still in flight land before the CTA may exit: wait (bounded)
    // for the last issued tile of every stage.
    for (uint32_t k = 0; k < (uint32_t)kTcStages && k < issued; ++k) {
      const uint32_t i = issued - 1 - k;
      if (!tc::mbar_wait_sleep(&S.full[i % kTcStages], (i / kTcStages) & 1u)) atomicExch(err, kErrTimeout);
    }
  } else if (warp == 1 && lane == 0) {  // MMA issuer
    constexpr uint32_t id1 = tc::idesc_bf16_f32_mn(128, 144), id2 = tc::idesc_bf16_f32_mn(128, 80);
    for (uint32_t i = 0; i < my; ++i) {
      const int sidx = (int)(i % kTcStages);
      if (!tc::mbar_wait_sleep(&S.full[sidx], (i / kTcStages) & 1u) ||
          !tc::mbar_wait_sleep(&S.ready[sidx], (i / kTcStages) & 1u)) {
        atomicExch(err, kErrTimeout);
        break;
      }
      tc::fence_after();
      const uint32_t a1 = tc::smem_addr(S.stage[sidx]), b1 = a1 + kA1Bytes, a2 = b1 + kB1Bytes, b2 = a2 + kA2Bytes;
#pragma unroll
      for (uint32_t kk = 0; kk < 2; ++kk) {  // K = 32 records as two K = 16 steps
        const uint32_t acc = (i > 0 || kk > 0) ? 1u : 0u;
        tc::mma_f16(tmem + kD1Col, tc::sdesc(a1 + kk * 256, 128, 512), tc::sdesc(b1 + kk * 256, 128, 512), id1, acc);
        tc::mma_f16(tmem + kD2Col, tc::sdesc(a2 + kk * 256, 128, 512), tc::sdesc(b2 + kk * 256, 128, 512), id2, acc);
      }
      tc::mma_commit(&S.empty[sidx]);
    }
    tc::mma_commit(&S.done);
  } else if (warp >= 4) {  // dg2 = (dlog cW3) where g2 > 0, and dlog, as BF16 operands
    const int f0 = 2 * (warp - 4);  // this thread's record `lane`, features 8 f0 .. 8 f0 + 15
    float w[3][16];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int e = 0; e < 16; ++e) w[c][e] = tf32_trunc(__ldg(cw3 + c * kHid + 8 * f0 + e));
    for (uint32_t i = 0; i < my; ++i) {
      const int sidx = (int)(i % kTcStages);
      if (!tc::mbar_wait_sleep(&S.full[sidx], (i / kTcStages) & 1u)) {
        atomicExch(err, kErrTimeout);
        break;
      }
      const uint8_t* g2 = S.stage[sidx] + kA1Bytes + kB1Bytes + kHid * 64;
      uint8_t* b2 = S.stage[sidx] + kA1Bytes + kB1Bytes + kA2Bytes;
      const float4 dl = S.dlog[sidx][lane];
      const float d0 = tf32_trunc(dl.x), d1 = tf32_trunc(dl.y), d2 = tf32_trunc(dl.z);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int at = (f0 + h) * 512 + lane * 16;
        const uint4 g = *reinterpret_cast<const uint4*>(g2 + at);
        const uint32_t gw[4] = {g.x, g.y, g.z, g.w};
        uint32_t out[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          // g2 is never negative: its BF16 halves are positive or zero.
          const int k = 8 * h + 2 * e;
          const float a = fmaf(w[0][k], d0, fmaf(w[1][k], d1, w[2][k] * d2));
          const float b = fmaf(w[0][k + 1], d0, fmaf(w[1][k + 1], d1, w[2][k + 1] * d2));
          out[e] = bf16x2((gw[e] & 0x7fffu) ? a : 0.0f, (gw[e] & 0x7fff0000u) ? b : 0.0f);
        }
        *reinterpret_cast<uint4*>(b2 + at) = make_uint4(out[0], out[1], out[2], out[3]);
      }
      if (warp == 4)
        *reinterpret_cast<uint4*>(b2 + 8 * 512 + lane * 16) = make_uint4(bf16x2(dl.x, dl.y), bf16x2(dl.z, 0.0f), 0u, 0u);
      tc::fence_async_smem();
      tc::mbar_arrive(&S.ready[sidx]);
    }
  }
  __syncwarp();
  // Epilogue: warp w < 4 owns TMEM lanes 32w..32w+31 (rows of D1 and D2).
  const bool done = warp >= 4 || tc::mbar_wait_sleep(&S.done, 0);
  tc::fence_after();
  if (warp >= 4) {
  } else if (!done) {
    if (lane == 0) atomicExch(err, kErrTimeout);
  } else {
    const uint32_t lanes = tmem + ((uint32_t)(warp * 32) << 16);
    const int row = warp * 32 + lane;
    float v[32];
    if (warp == 0) {  // D1 rows 0..31: enc feature `row` x dh1 j -> DW1[j][row]
      for (int c = 0; c < 2; ++c) {
        tc::tmem_ld32(lanes + kD1Col + 32 * c, v);
        for (int j = 0; j < 32; ++j) atomicAdd(dw + kOffDW1 + (32 * c + j) * kEnc + row, v[j]);
      }
    } else if (warp == 1) {  // D1 rows 32..63: cin feature row-32 x dg1 j -> CW1[j][row-32]
      for (int c = 0; c < 2; ++c) {
        tc::tmem_ld32(lanes + kD1Col + 64 + 32 * c, v);
        for (int j = 0; j < 32; ++j) atomicAdd(dw + kOffCW1 + (32 * c + j) * kCIn + (row - 32), v[j]);
      }
    } else {  // D1 rows 64..127: h1 feature row-64 x dout m -> DW2[m][row-64]
      float u[16];
      tc::tmem_ld16(lanes + kD1Col + 128, u);
      for (int m = 0; m < kDOut; ++m) atomicAdd(dw + kOffDW2 + m * kHid + (row - 64), u[m]);
    }
    if (warp < 2) {  // D2 rows 0..63: g1 feature `row` x dg2 j -> CW2[j][row]
      for (int c = 0; c < 2; ++c) {
        tc::tmem_ld32(lanes + kD2Col + 32 * c, v);
        for (int j = 0; j < 32; ++j) atomicAdd(dw + kOffCW2 + (32 * c + j) * kHid + row, v[j]);
      }
    } else {  // D2 rows 64..127: g2 feature row-64 x dlog c -> CW3[c][row-64]
      float u[16];
      tc::tmem_ld16(lanes + kD2Col + 64, u);
      for (int c = 0; c < 3; ++c) atomicAdd(dw + kOffCW3 + c * kHid + (row - 64), u[c]);
    }
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 1) tc::tmem_dealloc(tmem, kTmemCols);
}

// ---------------- per-sample MLP recompute and backward on the tensor cores (kind::tf32) ----------------
// One CTA per SM, four independent groups of 4 warps; a group takes 128
// records at a time (thread = record = TMEM lane) and runs the 10 layer
// products of the recompute and the backward as tcgen05.mma kind::tf32 with
// the A operand (this layer's input, one FP32 element per TMEM column) in
// TMEM and B (a weight image, below) in shared memory, the FP32 product in
// TMEM.  Between products each thread reads its row back, applies the
// elementwise step (ReLU and its mask, exp, SH, sigmoid and their
// derivatives), stages activations and deltas for the weight-gradient GEMMs
// (same layout as backward_kernel) and writes the next A.  TF32 operands
// (10-bit mantissa, FP32 accumulation) put ~1e-3 relative error on the
// per-sample activations and deltas; backward_kernel is the FP32 form.
//   forward:  h1 = relu(enc dW1^T)  out = h1 dW2^T  g1 = relu(cin cW1^T)
//             g2 = relu(g1 cW2^T)   logit = g2 cW3^T
//   backward: dg2 = (dlog cW3) m2   dg1 = (dg2 cW2) m1   dgeo = dg1 cW1[:,16:32]
//             dh1 = (dout dW2) mh   denc = dh1 dW1
constexpr int kBtGroups = 4;
constexpr int kBtThreads = 128 * kBtGroups;
constexpr uint32_t kBtColsPerGroup = 128;  // A: 64 columns, D: 64 columns

// Hash-grid scatter-add of one record's encoding gradient (d0, d1) at level L,
// dtable[L][corner] += w_corner * d.  Every lane of the warp calls it (valid =
// false for a lane without a record).  A warp's records are consecutive
// samples of one or two rays, so at the coarse levels runs of neighbouring
// lanes share a cell: levels 0..kAggLevels-1 sum each run's corner gradients
// with shuffles and add them with one atomic per run.  Corners k and k + 1 are
// one aligned entry pair {i, i ^ 1} half the time (a dense level's even index;
// a hashed level's even x, the x prime being 1): one 16-byte atomic then.
constexpr int kAggLevels = 13;  // levels whose scatter-add is warp-aggregated (N <= 776)
static_assert(level_res(kAggLevels - 1) < 1024, "cell key packs 10 bits per coordinate");

__device__ __forceinline__ void add_pair(float2* __restrict__ gt, uint32_t i, uint32_t j, float2 a, float2 b) {
  if ((i ^ j) == 1u) {
    const float4 v = (i & 1u) ? make_float4(b.x, b.y, a.x, a.y) : make_float4(a.x, a.y, b.x, b.y);
    atomicAdd(reinterpret_cast<float4*>(gt + (i & ~1u)), v);
  } else {
    atomicAdd(gt + i, a);
    atomicAdd(gt + j, b);
  }
}

__device__ __forceinline__ void scatter_add_level(int L, int N, float2* __restrict__ gtable, uint32_t T,
                                                  uint32_t dense_mask, const float3& x, float d0, float d1, bool valid,
                                                  uint32_t lane) {
  const LevelCell c = level_cell(x, N);
  uint32_t idx[8];
  corner_indices(c, N, (dense_mask >> L) & 1u, T, idx);
  float w[8];
  corner_weights(c, w);
  float2* gt = gtable + (size_t)L * T;
  uint32_t heads = 0xffffffffu;  // lanes that start a run
  if (L < kAggLevels) {
    // Runs of lanes with the same cell (invalid lanes form runs of their own
    // and add nothing).  N <= 776 here: 10 bits per coordinate.
    const uint32_t key = valid ? (c.ix | (c.iy << 10) | (c.iz << 20)) : (0x80000000u | lane);
    const uint32_t kprev = __shfl_up_sync(0xffffffffu, key, 1);
    heads = __ballot_sync(0xffffffffu, lane == 0 || kprev != key);
  }
  if (heads == 0xffffffffu) {  // no lane shares its cell
    if (valid)
#pragma unroll
      for (int k = 0; k < 8; k += 2)
        add_pair(gt, idx[k], idx[k + 1], make_float2(w[k] * d0, w[k] * d1), make_float2(w[k + 1] * d0, w[k + 1] * d1));
    return;
  }
  // Step o adds the partial sum of lane + o when no run starts in (lane, lane
  // + o]; afterwards each run's first lane holds its total.  Steps beyond the
  // warp's longest run are left out (more[b]: some run has over 2^b lanes).
  uint32_t more = ~heads, take = 0;
  int steps = 0;
#pragma unroll
  for (int o = 1, b = 0; o < 32; o <<= 1, ++b) {
    const uint32_t span = (uint32_t)(((1ull << o) - 1ull) << (lane + 1));  // lanes lane+1 .. lane+o
    if (lane + o < 32u && (heads & span) == 0u) take |= 1u << b;
    if (more != 0u) steps = b + 1;
    more &= more >> o;
  }
  const bool add = valid && ((heads >> lane) & 1u);
  float a[16];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    a[2 * k] = w[k] * d0;
    a[2 * k + 1] = w[k] * d1;
  }
  for (int b = 0; b < steps; ++b) {
    const bool t = (take >> b) & 1u;
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const float p = __shfl_down_sync(0xffffffffu, a[e], 1 << b);
      if (t) a[e] += p;
    }
  }
  if (add)
#pragma unroll
    for (int k = 0; k < 8; k += 2)
      add_pair(gt, idx[k], idx[k + 1], make_float2(a[2 * k], a[2 * k + 1]), make_float2(a[2 * k + 2], a[2 * k + 3]));
}

// The encoding gradients of `count` records from `first` -> the gradient table.
// In a kernel of its own the atomics of 36 warps per SM overlap, where the
// backward's TMEM leaves 16; it is bound by them: 73 sectors a record, 0.92 ms
// per 2^22 records = 330 G sectors/s (inside the MLP kernel it took 44 of 161
// ms at 122 M records, here 27).
constexpr int kScatThreads = 256;
__global__ void __launch_bounds__(kScatThreads)
scatter_kernel(const SampleRec* __restrict__ recs, uint32_t first, uint32_t count, const DevScene sc,
               const float* __restrict__ denc, float2* __restrict__ gtable) {
  const uint32_t s = blockIdx.x * kScatThreads + threadIdx.x;
  const bool valid = s < count;
  float3 x = make_float3(0.0f, 0.0f, 0.0f);
  if (valid) {
    const float4 q = __ldg(reinterpret_cast<const float4*>(recs + first + s));
    x = make_float3(q.x, q.y, q.z);
  }
  // One copy of the level's code: unrolled, the sixteen levels overran the
  // instruction caches.
#pragma unroll 1
  for (int l = 0; l < kLevels; ++l) {
    float2 d = make_float2(0.0f, 0.0f);
    if (valid) d = __ldg(reinterpret_cast<const float2*>(denc + (size_t)(s >> 5) * kEncTileFloats + (l >> 1) * 128 +
                                                         (s & 31u) * 4 + (l & 1) * 2));
    scatter_add_level(l, level_res_table[l], gtable, sc.T, sc.dense_mask, x, d.x, d.y, valid, threadIdx.x & 31u);
  }
}

// Weight images, [N][K] K-major, no swizzle, FP32 bits read as TF32: core
// matrices of 8 rows x 4 elements (16 B rows, 128 B each), K-adjacent at
// 128 B (LBO), 8-row groups K/4 x 128 B apart (SBO).
__host__ __device__ constexpr uint32_t tf32_off(int n, int k, int K) {
  return (uint32_t)((n >> 3) * (K * 32) + (k >> 2) * 128 + (n & 7) * 16 + (k & 3) * 4);
}
struct BtImage {
  uint32_t off, N, K;
};
constexpr int kBtImages = 10;
// dW1, dW2, cW1, cW2, cW3 (rows 3..15 zero), cW3^T (k 3..15 zero), cW2^T,
// cW1 geometry columns transposed ([n][j] = cW1[j][16 + n], row 15 zero),
// dW2^T, dW1^T.
__host__ __device__ constexpr BtImage bt_image(int i) {
  return i == 0   ? BtImage{0, 64, 32}
         : i == 1 ? BtImage{8192, 16, 64}
         : i == 2 ? BtImage{12288, 64, 32}
         : i == 3 ? BtImage{20480, 64, 64}
         : i == 4 ? BtImage{36864, 16, 64}
         : i == 5 ? BtImage{40960, 64, 16}
         : i == 6 ? BtImage{45056, 64, 64}
         : i == 7 ? BtImage{61440, 16, 64}
         : i == 8 ? BtImage{65536, 64, 16}
                  : BtImage{69632, 32, 64};
}
constexpr uint32_t kBtImageBytes = 77824;
static_assert(bt_image(9).off + bt_image(9).N * bt_image(9).K * 4 == kBtImageBytes, "image table");

// Value of element (n, k) of image i from the FP32 weight blob.
__device__ __forceinline__ float bt_value(const float* __restrict__ w, int i, int n, int k) {
  switch (i) {
    case 0: return w[kOffDW1 + n * kEnc + k];
    case 1: return w[kOffDW2 + n * kHid + k];
    case 2: return w[kOffCW1 + n * kCIn + k];
    case 3: return w[kOffCW2 + n * kHid + k];
    case 4: return n < 3 ? w[kOffCW3 + n * kHid + k] : 0.0f;
    case 5: return k < 3 ? w[kOffCW3 + k * kHid + n] : 0.0f;
    case 6: return w[kOffCW2 + k * kHid + n];
    case 7: return n < 15 ? w[kOffCW1 + k * kCIn + 16 + n] : 0.0f;
    case 8: return w[kOffDW2 + k * kHid + n];
    default: return w[kOffDW1 + k * kEnc + n];
  }
}

__global__ void pack_bt_images_kernel(const float* __restrict__ w, uint8_t* __restrict__ img) {
  const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;  // element of the concatenated images
  if (e >= kBtImageBytes / 4) return;
  int i = 0;
  while (i + 1 < kBtImages && e >= bt_image(i + 1).off / 4) ++i;
  const BtImage b = bt_image(i);
  const uint32_t local = e - b.off / 4;
  const int n = (int)(local / b.K), k = (int)(local % b.K);
  *reinterpret_cast<float*>(img + b.off + tf32_off(n, k, (int)b.K)) = bt_value(w, i, n, k);
}

__device__ __forceinline__ uint32_t f2u(float v) { return __float_as_uint(v); }

// Staging of features f..f+7 (f % 8 == 0) of this thread's record as BF16,
// in the canonical MN-major layout of a 16-bit tensor-core operand with
// K = record: a record's 8 features are one 16-byte row, 8 records a 128-byte
// core matrix, record groups of 8 at 128 B, feature groups of 8 at 512 B; an
// F-wide array's 32-record tile is F x 64 contiguous bytes.  A thread's row
// needs nothing from its neighbours and a warp's 32 rows are one contiguous
// 512-byte block.  (The K-major layout, whose rows hold one feature of 8
// records, took an 8x8 transpose by six shuffles per call: 45 of the backward
// phase's 161 ms at 122 M records.)
__device__ __forceinline__ void stage8(float* arr, int F, uint32_t s, int f, float a0, float a1, float a2, float a3,
                                       float a4, float a5, float a6, float a7, bool stage) {
  if (stage) {
    uint8_t* tile = reinterpret_cast<uint8_t*>(arr) + (size_t)(s >> 5) * (size_t)F * 64u;
    *reinterpret_cast<uint4*>(tile + (f >> 3) * 512 + (s & 31u) * 16) =
        make_uint4(bf16x2(a0, a1), bf16x2(a2, a3), bf16x2(a4, a5), bf16x2(a6, a7));
  }
}

__global__ void __launch_bounds__(kBtThreads, 1)
backward_tc_kernel(const SampleRec* __restrict__ recs, uint32_t first, uint32_t count,
                   const uint2* __restrict__ list, const TrainRay* __restrict__ rays, const float* __restrict__ encs,
                   const uint8_t* __restrict__ images, Staging st, float* __restrict__ denc,
                   uint32_t* __restrict__ err) {
  extern __shared__ __align__(128) uint8_t smem_bt[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_bt + kBtImageBytes);  // [group] mma, [kBtGroups] weights
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + kBtGroups + 1);
  const int tid = threadIdx.x, warp = tid >> 5, g = tid >> 7, row = tid & 127;
  if (tid == 0) {
    for (int k = 0; k <= kBtGroups; ++k) tc::mbar_init(bars + k, 1);
    tc::fence_mbar_init();
  }
  if (warp == 0) {
    tc::tmem_alloc(tslot, kBtColsPerGroup * kBtGroups);
    tc::tmem_relinquish();
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = *tslot;
  bool fail = false;
  if (tid == 0) {
    tc::mbar_arrive_expect_tx(bars + kBtGroups, kBtImageBytes);
    tc::bulk_g2s(smem_bt, images, kBtImageBytes, bars + kBtGroups);
    fail = !tc::mbar_wait(bars + kBtGroups, 0);
  }
  fail = __syncthreads_or(fail);
  const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
  const uint32_t a_col = tmem + g * kBtColsPerGroup, d_col = a_col + 64;
  const uint32_t a_row = a_col + lane_off, d_row = d_col + lane_off;
  const uint32_t sB = tc::smem_addr(smem_bt);
  const uint32_t gbar = 1 + g;
  uint64_t* mbar = bars + g;
  uint32_t pm = 0;
  bool ok = true;
  // D[:, :N] = A[:, :K] B_i^T.  Every thread publishes its TMEM writes; the
  // group learns of any failed wait here and stops as a whole.
  auto mma = [&](int i) -> bool {
    tc::tmem_wait_st();
    tc::fence_before();
    if (tc::named_sync_or(gbar, 128, !ok)) return false;
    const BtImage b = bt_image(i);
    if (row == 0) {
      tc::fence_after();
      const uint32_t idesc = tc::idesc_tf32_f32(128, (int)b.N);
      for (uint32_t j = 0; j < b.K / 8; ++j)
        tc::mma_tf32_at(d_col, a_col + 8 * j, tc::sdesc(sB + b.off + 256 * j, 128, b.K * 32), idesc, j > 0 ? 1u : 0u);
      tc::mma_commit(mbar);
    }
    ok = tc::mbar_wait(mbar, pm) && ok;
    pm ^= 1u;
    tc::fence_after();
    return true;
  };

  const uint32_t ntiles = (count + 127u) / 128u;
  const uint32_t staged = (count + 31u) & ~31u;  // rows the weight-gradient GEMMs read
  if (!fail) {
    for (uint32_t tile = blockIdx.x * kBtGroups + g; tile < ntiles; tile += gridDim.x * kBtGroups) {
      const uint32_t s = tile * 128u + (uint32_t)row;
      const bool valid = s < count, stage = s < staged;
      SampleRec q;
      if (valid) {
        q = recs[first + s];
      } else {
        q.place = 0;
        q.dsigma = q.dcr = q.dcg = q.dcb = 0.0f;
      }
      uint32_t u[32];
      float v[32];
      // ---- forward recompute ----
      {
        float enc[kEnc];
        if (valid) {
          load_enc(encs, q.place, enc);
        } else {
#pragma unroll
          for (int k = 0; k < kEnc; ++k) enc[k] = 0.0f;
        }
#pragma unroll
        for (int k = 0; k < kEnc; ++k) u[k] = f2u(enc[k]);
        tc::tmem_st32_nowait(a_row, u);
#pragma unroll
        for (int k = 0; k < kEnc; k += 8) stage8(st.enc, kEnc, s, k, enc[k + 0], enc[k + 1], enc[k + 2], enc[k + 3], enc[k + 4], enc[k + 5], enc[k + 6], enc[k + 7], stage);
      }
      if (!mma(0)) break;
      uint32_t m_h1[2], m_g1[2], m_g2[2];
      // ReLU of D[:, :64] -> staging, mask, next A.
      auto relu64 = [&](float* act, uint32_t (&m)[2]) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          tc::tmem_ld32(d_row + 32 * c, v);
          uint32_t bits = 0;
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            v[j] = valid ? fmaxf(v[j], 0.0f) : 0.0f;
            bits |= v[j] > 0.0f ? 1u << j : 0u;
            u[j] = f2u(v[j]);
          }
          // Opaque: a mask whose bits were known as predicates was kept as the
          // activations themselves, 129 registers spilled per tile, whose
          // write-back was a third of the kernel's DRAM traffic (36.0 ms at
          // 122 M records, 23.9 without).
          asm volatile("" : "+r"(bits));
          m[c] = bits;
          tc::tmem_st32_nowait(a_row + 32 * c, u);
#pragma unroll
          for (int j = 0; j < 32; j += 8) stage8(act, kHid, s, 32 * c + j, v[j + 0], v[j + 1], v[j + 2], v[j + 3], v[j + 4], v[j + 5], v[j + 6], v[j + 7], stage);
        }
      };
      relu64(st.h1, m_h1);
      if (!mma(1)) break;
      float sigma;
      {
        float out[16];
        tc::tmem_ld16(d_row, reinterpret_cast<float(&)[16]>(out));
        sigma = expf(out[0] - 1.0f);
        float cin[kCIn];
        const TrainRay& r = rays[list[q.place].x];
        sh16(make_float3(r.dx, r.dy, r.dz), cin);
#pragma unroll
        for (int k = 0; k < 15; ++k) cin[16 + k] = out[1 + k];
        cin[31] = 0.0f;
#pragma unroll
        for (int k = 0; k < kCIn; ++k) {
          cin[k] = valid ? cin[k] : 0.0f;
          u[k] = f2u(cin[k]);
        }
        tc::tmem_st32_nowait(a_row, u);
#pragma unroll
        for (int k = 0; k < kCIn; k += 8) stage8(st.cin, kCIn, s, k, cin[k + 0], cin[k + 1], cin[k + 2], cin[k + 3], cin[k + 4], cin[k + 5], cin[k + 6], cin[k + 7], stage);
      }
      if (!mma(2)) break;
      relu64(st.g1, m_g1);
      if (!mma(3)) break;
      relu64(st.g2, m_g2);
      if (!mma(4)) break;
      // ---- backward ----
      {
        float lg[16];
        tc::tmem_ld16(d_row, reinterpret_cast<float(&)[16]>(lg));
        const float c0 = sigmoidf(lg[0]), c1 = sigmoidf(lg[1]), c2 = sigmoidf(lg[2]);
        const float dl[3] = {q.dcr * c0 * (1.0f - c0), q.dcg * c1 * (1.0f - c1), q.dcb * c2 * (1.0f - c2)};
        uint32_t w16[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) w16[k] = k < 3 ? f2u(dl[k]) : 0u;
        tc::tmem_st16_nowait(a_row, w16);
        // FP32: the weight-gradient kernel makes its dlog and dg2 operands of it.
        if (stage) reinterpret_cast<float4*>(st.dlog)[s] = make_float4(dl[0], dl[1], dl[2], 0.0f);
      }
      // Masked D[:, :64] -> staging (if any), next A.
      auto mask64 = [&](float* delta, const uint32_t (&m)[2]) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          tc::tmem_ld32(d_row + 32 * c, v);
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            v[j] = ((m[c] >> j) & 1u) ? v[j] : 0.0f;
            u[j] = f2u(v[j]);
          }
          tc::tmem_st32_nowait(a_row + 32 * c, u);
#pragma unroll
          for (int j = 0; j < 32; j += 8) stage8(delta, kHid, s, 32 * c + j, v[j + 0], v[j + 1], v[j + 2], v[j + 3], v[j + 4], v[j + 5], v[j + 6], v[j + 7], stage && delta);
        }
      };
      if (!mma(5)) break;
      mask64(nullptr, m_g2);
      if (!mma(6)) break;
      mask64(st.dg1, m_g1);
      if (!mma(7)) break;
      {
        float geo[16];
        tc::tmem_ld16(d_row, reinterpret_cast<float(&)[16]>(geo));
        uint32_t w16[16];
        float dout[16];
        dout[0] = q.dsigma * sigma;
#pragma unroll
        for (int m = 0; m < 15; ++m) dout[1 + m] = geo[m];
#pragma unroll
        for (int m = 0; m < 16; ++m) w16[m] = f2u(dout[m]);
        tc::tmem_st16_nowait(a_row, w16);
#pragma unroll
        for (int m = 0; m < kDOut; m += 8) stage8(st.dout, kDOut, s, m, dout[m + 0], dout[m + 1], dout[m + 2], dout[m + 3], dout[m + 4], dout[m + 5], dout[m + 6], dout[m + 7], stage);
      }
      if (!mma(8)) break;
      mask64(st.dh1, m_h1);
      if (!mma(9)) break;
      tc::tmem_ld32(d_row, v);  // denc
      // The next tile's first product overwrites D: its sync follows these reads.
      if (valid)
#pragma unroll
        for (int k = 0; k < kEnc; k += 4) *enc_chunk(denc, s, k / 4) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
    }
  }
  if (fail || !ok) atomicExch(err, kErrTimeout);
  tc::fence_before();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after();
    tc::tmem_dealloc(tmem, kBtColsPerGroup * kBtGroups);
  }
}
constexpr int kBtSmem = (int)kBtImageBytes + 8 * (kBtGroups + 1) + 16;

// ---------------- the forward's field evaluation on the tensor cores, 3xTF32 ----------------
// eval_kernel's work as tcgen05 kind::tf32 products at FP32-level accuracy:
// every operand is split into its TF32 rounding (hi) and the FP32 remainder
// (lo), and each layer accumulates A_hi B_hi + A_lo B_hi + A_hi B_lo in FP32.
// The dropped A_lo B_lo term and the remainders' own TF32 truncation are
// below 2^-21 of each product, so the loss keeps the FP32 evaluation's value
// (plain TF32 products would move it by ~1e-3 relative: a refit whose
// rendered colour sits within 1e-2 of the target then sees a few per cent of
// error in its loss and adjoints).  One CTA per SM, four independent groups of
// 4 warps; a group takes 128 listed samples at a time (thread = sample = TMEM
// lane), writes each layer's input as A_hi into TMEM and as A_lo into shared
// memory, one thread issues the three K-chains against the weight images'
// high and low parts in shared memory, and every thread reads its row of D
// back for the elementwise step (ReLU, exp, SH, sigmoid) and the next layer's
// input.  The encodings of a group's next tile are read under the last
// layer's MMAs.  A group's layers are one serial chain, so the groups in
// flight set the rate: with A_lo and the next encoding in TMEM two fit, which
// took 28.0 of the forward phase's 52.2 ms at 122 M samples; four bring the
// phase to 44.1.
constexpr int kEtGroups = 4;
constexpr int kEtThreads = 128 * kEtGroups;
constexpr uint32_t kEtColsPerGroup = 128;  // A_hi: 64 columns, D: 64 columns
constexpr uint32_t kFwdImageBytes = 40960;  // bt_image 0..4: dW1, dW2, cW1, cW2, cW3
static_assert(bt_image(5).off == kFwdImageBytes, "forward images first");
constexpr uint32_t kEtImageBytes = 2 * kFwdImageBytes;  // high parts, then low parts
constexpr uint32_t kEtLoBytes = 128 * kHid * 4;         // a group's A_lo, laid out as a weight image
constexpr uint32_t kEtBars = kEtImageBytes + kEtGroups * kEtLoBytes;
constexpr int kEtSmem = (int)kEtBars + 8 * (kEtGroups + 1) + 16;
static_assert(2 * kEtSmem > 228 * 1024, "one CTA per SM: its TMEM allocation takes all columns");

__device__ __forceinline__ float tf32_hi(float v) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
  return __uint_as_float(r);
}

// The forward images' high and low parts from the FP32 weights.
__global__ void pack_et_images_kernel(const float* __restrict__ w, uint8_t* __restrict__ img) {
  const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= kFwdImageBytes / 4) return;
  int i = 0;
  while (i + 1 < 5 && e >= bt_image(i + 1).off / 4) ++i;
  const BtImage b = bt_image(i);
  const uint32_t local = e - b.off / 4;
  const int n = (int)(local / b.K), k = (int)(local % b.K);
  const float v = bt_value(w, i, n, k), hi = tf32_hi(v);
  const uint32_t o = b.off + tf32_off(n, k, (int)b.K);
  *reinterpret_cast<float*>(img + o) = hi;
  *reinterpret_cast<float*>(img + kFwdImageBytes + o) = v - hi;
}

// One listed sample's inputs.
struct EtSample {
  float t;
  float3 d;
  bool valid;
};

__device__ __forceinline__ EtSample et_sample(const uint2* __restrict__ list, uint32_t j, uint32_t m,
                                              const TrainRay* __restrict__ rays) {
  EtSample q;
  q.valid = j < m;
  q.t = 0.0f;
  q.d = make_float3(0.0f, 0.0f, 1.0f);
  if (q.valid) {
    const uint2 e = list[j];
    const TrainRay& r = rays[e.x];
    q.t = fmaf((float)e.y + 0.5f, kDt, r.ts);
    q.d = make_float3(r.dx, r.dy, r.dz);
  }
  return q;
}

__global__ void __launch_bounds__(kEtThreads, 1)
eval_tc_kernel(const uint2* __restrict__ list, uint32_t m, const TrainRay* __restrict__ rays,
               const float* __restrict__ encs, const uint8_t* __restrict__ images, ScratchSample* __restrict__ scratch,
               uint32_t* __restrict__ err) {
  extern __shared__ __align__(128) uint8_t smem_et[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_et + kEtBars);  // [group] mma, [kEtGroups] images
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + kEtGroups + 1);
  const int tid = threadIdx.x, warp = tid >> 5, g = tid >> 7, row = tid & 127;
  if (tid == 0) {
    for (int k = 0; k <= kEtGroups; ++k) tc::mbar_init(bars + k, 1);
    tc::fence_mbar_init();
  }
  if (warp == 0) {
    tc::tmem_alloc(tslot, kEtColsPerGroup * kEtGroups);
    tc::tmem_relinquish();
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = *tslot;
  bool fail = false;
  if (tid == 0) {
    tc::mbar_arrive_expect_tx(bars + kEtGroups, kEtImageBytes);
    tc::bulk_g2s(smem_et, images, kEtImageBytes, bars + kEtGroups);
    fail = !tc::mbar_wait(bars + kEtGroups, 0);
  }
  fail = __syncthreads_or(fail);
  const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
  const uint32_t hi_col = tmem + g * kEtColsPerGroup, d_col = hi_col + 64;
  const uint32_t hi_row = hi_col + lane_off, d_row = d_col + lane_off;
  uint8_t* const lo = smem_et + kEtImageBytes + g * kEtLoBytes;
  const uint32_t sB = tc::smem_addr(smem_et), s_lo = tc::smem_addr(lo);
  const uint32_t gbar = 1 + g;
  uint64_t* mbar = bars + g;
  uint32_t pm = 0;
  bool ok = true;
  // Columns 32 c .. 32 c + 31 of a K-wide layer input -> A_hi, A_lo (no wait:
  // the next issue waits).
  auto put32 = [&](const float (&x)[32], int c, int K) {
    uint32_t uh[32];
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
      float l[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float h = tf32_hi(x[j + e]);
        uh[j + e] = __float_as_uint(h);
        l[e] = x[j + e] - h;
      }
      *reinterpret_cast<float4*>(lo + tf32_off(row, 32 * c + j, K)) = make_float4(l[0], l[1], l[2], l[3]);
    }
    tc::tmem_st32_nowait(hi_row + 32 * c, uh);
  };
  // D[:, :N] = A B_i^T at 3xTF32: every thread publishes its writes of A, one
  // thread issues; the group learns of any failed wait here and stops as a
  // whole.
  auto issue = [&](int i) -> bool {
    tc::tmem_wait_st();
    tc::fence_async_smem();
    tc::fence_before();
    if (tc::named_sync_or(gbar, 128, !ok)) return false;
    const BtImage b = bt_image(i);
    if (row == 0) {
      tc::fence_after();
      const uint32_t idesc = tc::idesc_tf32_f32(128, (int)b.N);
      const uint32_t steps = b.K / 8;
      for (uint32_t j = 0; j < steps; ++j)
        tc::mma_tf32_at(d_col, hi_col + 8 * j, tc::sdesc(sB + b.off + 256 * j, 128, b.K * 32), idesc, j > 0 ? 1u : 0u);
      for (uint32_t j = 0; j < steps; ++j)
        tc::mma_tf32(d_col, tc::sdesc(s_lo + 256 * j, 128, b.K * 32), tc::sdesc(sB + b.off + 256 * j, 128, b.K * 32),
                     idesc, 1u);
      for (uint32_t j = 0; j < steps; ++j)
        tc::mma_tf32_at(d_col, hi_col + 8 * j, tc::sdesc(sB + kFwdImageBytes + b.off + 256 * j, 128, b.K * 32),
                        idesc, 1u);
      tc::mma_commit(mbar);
    }
    return true;
  };
  auto wait = [&]() {
    ok = tc::mbar_wait(mbar, pm) && ok;
    pm ^= 1u;
    tc::fence_after();
  };
  // ReLU of D[:, :64] -> the next layer's input.
  auto relu64 = [&]() {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      float v[32];
      tc::tmem_ld32(d_row + 32 * c, v);
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.0f);
      put32(v, c, kHid);
    }
  };
  auto load = [&](uint32_t j, bool valid, float (&enc)[kEnc]) {
    if (valid) {
      load_enc(encs, j, enc);
    } else {
#pragma unroll
      for (int k = 0; k < kEnc; ++k) enc[k] = 0.0f;
    }
  };

  const uint32_t ntiles = (m + 127u) / 128u;
  const uint32_t stride = gridDim.x * kEtGroups;
  uint32_t tile = blockIdx.x * kEtGroups + g;
  if (!fail && tile < ntiles) {
    uint32_t j = tile * 128u + (uint32_t)row;
    EtSample cur = et_sample(list, j, m, rays);
    float enc[kEnc];
    load(j, cur.valid, enc);
    for (; tile < ntiles; tile += stride, j += stride * 128u) {
      const uint32_t jn = j + stride * 128u;
      put32(enc, 0, kEnc);
      if (!issue(0)) break;  // h1 = relu(enc dW1^T)
      const EtSample nxt = et_sample(list, jn, tile + stride < ntiles ? m : 0u, rays);
      wait();
      relu64();
      if (!issue(1)) break;  // out = h1 dW2^T
      float x[32];
      {
        float sh[16];
        sh16(cur.d, sh);
#pragma unroll
        for (int q = 0; q < 16; ++q) x[q] = sh[q];
      }
      wait();
      float sigma;
      {
        float out[16];
        tc::tmem_ld16(d_row, out);
        sigma = expf(out[0] - 1.0f);
#pragma unroll
        for (int q = 0; q < 15; ++q) x[16 + q] = out[1 + q];
        x[31] = 0.0f;
      }
      put32(x, 0, kCIn);
      if (!issue(2)) break;  // g1 = relu(cin cW1^T)
      wait();
      relu64();
      if (!issue(3)) break;  // g2 = relu(g1 cW2^T)
      wait();
      relu64();
      if (!issue(4)) break;  // logit = g2 cW3^T
      load(jn, nxt.valid, enc);
      wait();
      float lg[16];
      tc::tmem_ld16(d_row, lg);
      // The next tile's first product overwrites D: its sync follows these reads.
      if (cur.valid) {
        const float alpha = -expm1f(-sigma * kDt);
        scratch[j] =
            ScratchSample{cur.t, alpha, 0.0f, sigmoidf(lg[0]), sigmoidf(lg[1]), sigmoidf(lg[2]), 0.0f, 0.0f};
      }
      cur = nxt;
    }
  }
  if (fail || !ok) atomicExch(err, kErrTimeout);
  tc::fence_before();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after();
    tc::tmem_dealloc(tmem, kEtColsPerGroup * kEtGroups);
  }
}

__global__ void adam_kernel(float* __restrict__ p, float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                            size_t n, float lr, float b1, float b2, float eps, float bc1, float bc2) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    g[i] = 0.0f;
  }
}

// ---------------- FP64 loss (finite differences) ----------------

struct ParamsF64 {
  const float* table;  // FP32 table, read as double
  const float* w;      // FP32 weight blob
  int which;           // perturbed array: 0 table, 1 weights
  uint64_t index;
  double delta;
};

__device__ __forceinline__ double tab(const ParamsF64& P, uint64_t i) {
  return (double)P.table[i] + ((P.which == 0 && i == P.index) ? P.delta : 0.0);
}
__device__ __forceinline__ double wt(const ParamsF64& P, int i) {
  return (double)P.w[i] + ((P.which == 1 && (uint64_t)i == P.index) ? P.delta : 0.0);
}

// Field query in FP64: same cells and hash indices as encode_fp32 (the cell
// is chosen from the FP32 position), FP64 weights and MLPs.
__device__ void query_f64(const ParamsF64& P, const DevScene& sc, const float3 xf, const float3 d, double& sigma,
                          double rgb[3]) {
  double enc[kEnc];
  const double x[3] = {xf.x, xf.y, xf.z};
  for (int l = 0; l < kLevels; ++l) {
    const int N = level_res(l);
    const LevelCell c = level_cell(xf, N);
    uint32_t idx[8];
    corner_indices(c, N, (sc.dense_mask >> l) & 1u, sc.T, idx);
    const double f[3] = {x[0] * N - (double)c.ix, x[1] * N - (double)c.iy, x[2] * N - (double)c.iz};
    double a0 = 0, a1 = 0;
    for (int k = 0; k < 8; ++k) {
      const double w = ((k & 1) ? f[0] : 1 - f[0]) * ((k & 2) ? f[1] : 1 - f[1]) * ((k & 4) ? f[2] : 1 - f[2]);
      const uint64_t e = ((uint64_t)l * sc.T + idx[k]) * 2;
      a0 += w * tab(P, e);
      a1 += w * tab(P, e + 1);
    }
    enc[2 * l] = a0;
    enc[2 * l + 1] = a1;
  }
  double h1[kHid], out[kDOut];
  for (int j = 0; j < kHid; ++j) {
    double a = 0;
    for (int k = 0; k < kEnc; ++k) a += wt(P, kOffDW1 + j * kEnc + k) * enc[k];
    h1[j] = a > 0 ? a : 0;
  }
  for (int m = 0; m < kDOut; ++m) {
    double a = 0;
    for (int j = 0; j < kHid; ++j) a += wt(P, kOffDW2 + m * kHid + j) * h1[j];
    out[m] = a;
  }
  sigma = exp(out[0] - 1);
  float sh[16];
  sh16(d, sh);  // the direction basis as rendered (FP32): it holds no parameter
  double cin[kCIn];
  for (int k = 0; k < 16; ++k) cin[k] = sh[k];
  for (int k = 0; k < 15; ++k) cin[16 + k] = out[1 + k];
  cin[31] = 0;
  double g1[kHid];
  for (int j = 0; j < kHid; ++j) {
    double a = 0;
    for (int k = 0; k < kCIn; ++k) a += wt(P, kOffCW1 + j * kCIn + k) * cin[k];
    g1[j] = a > 0 ? a : 0;
  }
  double lg[3] = {0, 0, 0};
  for (int j = 0; j < kHid; ++j) {
    double a = 0;
    for (int k = 0; k < kHid; ++k) a += wt(P, kOffCW2 + j * kHid + k) * g1[k];
    a = a > 0 ? a : 0;
    for (int c = 0; c < 3; ++c) lg[c] += wt(P, kOffCW3 + c * kHid + j) * a;
  }
  for (int c = 0; c < 3; ++c) rgb[c] = 1 / (1 + exp(-lg[c]));
}

// The FP32 forward's sample set (same t, positions and occupancy decisions),
// everything downstream in FP64.
__global__ void loss_f64_kernel(const TrainRay* __restrict__ rays, int n, const DevScene sc, ParamsF64 P,
                                double* __restrict__ loss_sum, double depth_w, double inv_n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const TrainRay r = rays[i];
  double C[3] = {0, 0, 0}, D = 0, T = 1;
  const float3 o = make_float3(r.ox, r.oy, r.oz), d = make_float3(r.dx, r.dy, r.dz);
  for (int s = 0; s < r.n; ++s) {
    const float t = fmaf((float)s + 0.5f, kDt, r.ts);
    const float3 x = sample_pos(o, d, t);
    if (!occupied(sc.occ, x)) continue;
    double sigma, c[3];
    query_f64(P, sc, x, d, sigma, c);
    const double alpha = -expm1(-sigma * (double)kDt);
    const double w = T * alpha;
    for (int a = 0; a < 3; ++a) C[a] += w * c[a];
    D += w * (double)t;
    T -= w;
    if (T < (double)kTStop) break;
  }
  const double e0 = C[0] - r.tr, e1 = C[1] - r.tg, e2 = C[2] - r.tb, ed = D - r.td;
  atomicAdd(loss_sum, (e0 * e0 + e1 * e1 + e2 * e2 + depth_w * ed * ed) * inv_n);
}

// The same loss for m perturbations at once (blockIdx.y = perturbation):
// a central-difference check of many parameters in one launch instead of one
// launch per evaluation (each evaluation alone fills one or two SMs).
struct PerturbF64 {
  int which;
  uint64_t index;
  double delta;
};

__global__ void loss_f64_batch_kernel(const TrainRay* __restrict__ rays, int n, const DevScene sc, const float* table,
                                      const float* w, const PerturbF64* __restrict__ pert,
                                      double* __restrict__ loss_sums, double depth_w, double inv_n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const PerturbF64 q = pert[blockIdx.y];
  ParamsF64 P;
  P.table = table;
  P.w = w;
  P.which = q.which;
  P.index = q.index;
  P.delta = q.delta;
  const TrainRay r = rays[i];
  double C[3] = {0, 0, 0}, D = 0, T = 1;
  const float3 o = make_float3(r.ox, r.oy, r.oz), d = make_float3(r.dx, r.dy, r.dz);
  for (int s = 0; s < r.n; ++s) {
    const float t = fmaf((float)s + 0.5f, kDt, r.ts);
    const float3 x = sample_pos(o, d, t);
    if (!occupied(sc.occ, x)) continue;
    double sigma, c[3];
    query_f64(P, sc, x, d, sigma, c);
    const double alpha = -expm1(-sigma * (double)kDt);
    const double wgt = T * alpha;
    for (int a = 0; a < 3; ++a) C[a] += wgt * c[a];
    D += wgt * (double)t;
    T -= wgt;
    if (T < (double)kTStop) break;
  }
  const double e0 = C[0] - r.tr, e1 = C[1] - r.tg, e2 = C[2] - r.tb, ed = D - r.td;
  atomicAdd(loss_sums + blockIdx.y, (e0 * e0 + e1 * e1 + e2 * e2 + depth_w * ed * ed) * inv_n);
}

}  // namespace

struct nes_trainer {
  nes_ctx* ctx = nullptr;
  nes_train_config cfg{};
  cudaStream_t st = nullptr;
  TrainView* d_views = nullptr;
  int nviews = 0;
  const float* trgb = nullptr;
  const float* tdep = nullptr;
  uint32_t max_rays = 0;
  int2* d_pairs = nullptr;
  TrainRay* d_rays = nullptr;
  // Per listed sample (list_capacity of each): list entry, encoding, state (in
  // d_stage) and record of the backward.
  uint32_t list_capacity = 0;
  uint2* d_list = nullptr;
  float* d_enc = nullptr;
  ScratchSample* d_scratch = nullptr;
  SampleRec* d_recs = nullptr;
  uint32_t* d_ctr = nullptr;  // [0] record cursor, [1] error word
  RayOut* d_rout = nullptr;
  uint32_t* d_block_count = nullptr;  // samples per block of kRayBlock rays
  uint32_t* d_block_first = nullptr;  // and before each block (one more entry: all)
  uint32_t* h_block_first = nullptr;  // pinned copy
  double* d_loss = nullptr;
  float2* d_gtable = nullptr;
  float* d_gw = nullptr;
  float *d_mt = nullptr, *d_vt = nullptr, *d_mw = nullptr, *d_vw = nullptr;
  void* d_stage = nullptr;  // a backward chunk's staging; before it, the part's d_scratch
  float* d_denc = nullptr;  // encoding gradients of a backward chunk, tiled as d_enc
  uint8_t* d_bimg = nullptr;  // TF32 weight images of backward_tc_kernel
  uint8_t* d_eimg = nullptr;  // high/low TF32 forward images of eval_tc_kernel
  uint32_t chunk = 0;  // records of a backward chunk
  uint64_t steps = 0;
  uint64_t last_samples = 0;
  // Phase events on the trainer's stream: 0 start of a part's forward, 1 its
  // end, 2 end of the part's backward and weight gradients (read before the
  // next part records them), 3 Adam start, 4 Adam end.
  cudaEvent_t ev[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
  float phase_ms[3] = {0.0f, 0.0f, 0.0f};
};

namespace {

#define TR_CUDA(call)                      \
  do {                                     \
    cudaError_t e_ = (call);               \
    if (e_ != cudaSuccess) return NES_EIO; \
  } while (0)


// A staged record's bytes: FP32 in the strict mode; the tensor-core mode has
// BF16 (dlog as four FP32), and dg2 is not staged there.
constexpr size_t stage_bytes(bool exact) { return exact ? kStageFloats * sizeof(float) : (kStageFloats - kHid) * 2; }

// Samples of the list and records of a backward chunk, by the trainer's device
// memory: at most 64 KiB per ray of the batch and kTrainBytes (8 MB less than
// the FP32 staging of 2^21 records, for the small arrays).  A record takes
// stage_bytes and its encoding gradient, a listed sample kSampleBytes; its
// state, read for the last time before the first record is staged, lies in the
// staging.  The list gets 512 samples a ray (a view of the seeded field, occupied
// throughout, lists 465) while the chunk keeps half its largest size, the chunk
// the rest.  Batches of 180,000 rays and more have both at their largest.  With
// the list at 1024 samples a ray and the largest chunk, 65,536 rays took 17.9
// GB in place of 8.2.
constexpr size_t kSampleBytes = sizeof(uint2) + kEnc * sizeof(float) + sizeof(SampleRec);
constexpr size_t kTrainBytes = ((size_t)1 << 21) * kStageFloats * sizeof(float) - ((size_t)8 << 20);
constexpr size_t kListSamples = (size_t)1 << 26;
struct TrainerSizes {
  size_t samples, records, stage_bytes;  // multiples of 32 and of 128
};
TrainerSizes trainer_sizes(size_t rays, bool exact) {
  const size_t stage = stage_bytes(exact), record = stage + kEnc * sizeof(float), most = (size_t)1 << (exact ? 21 : 22);
  const size_t bytes = rays * (64u << 10) + kTrainBytes, block = std::min<size_t>(rays, kRayBlock) * kMaxSteps;
  TrainerSizes z;
  z.samples = std::min({rays * 512, kListSamples, (bytes - most / 2 * record) / kSampleBytes});
  z.samples = std::max(z.samples, block) & ~(size_t)31;  // a block of rays fits
  z.records = std::min({most, rays * kMaxSteps, (bytes - z.samples * kSampleBytes) / record}) & ~(size_t)127;
  z.samples = std::max(std::min(z.samples, z.records * stage / sizeof(ScratchSample)), block) & ~(size_t)31;
  z.stage_bytes = std::max(z.records * stage, z.samples * sizeof(ScratchSample));
  return z;
}

Staging staging(const nes_trainer* t) {
  Staging s{};
  const bool exact = t->cfg.exact_weight_grads != 0;
  float* p = static_cast<float*>(t->d_stage);
  auto take = [&](int F) {  // an F-wide array of the chunk's records, FP32 or BF16
    float* const a = p;
    p += (size_t)t->chunk * F / (exact ? 1 : 2);
    return a;
  };
  s.enc = take(kEnc);
  s.h1 = take(kHid);
  s.cin = take(kCIn);
  s.g1 = take(kHid);
  s.g2 = take(kHid);
  s.dh1 = take(kHid);
  s.dout = take(kDOut);
  s.dg1 = take(kHid);
  if (exact) s.dg2 = take(kHid);
  s.dlog = take(kFDlog);
  return s;
}

template <int IN, int OUT, int LDD, int P, int Q>
cudaError_t launch_dw(const float* act, const float* delta, uint32_t tiles, float* dw, int num_sms, cudaStream_t st) {
  const uint32_t pairs = (tiles + 1) / 2, want = 2u * (uint32_t)num_sms;  // two resident blocks per SM
  dw_kernel<IN, OUT, LDD, P, Q><<<pairs < want ? pairs : want, kDwThreads, 0, st>>>(act, delta, tiles, dw);
  return cudaGetLastError();
}

// Backward of the `total` records in d_recs, accumulated into d_gtable / d_gw.
int backward_records(nes_trainer* t, const TrainRay* rays, uint32_t total) {
  nes_ctx* c = t->ctx;
  const Staging sg = staging(t);
  float* gw = t->d_gw;
  const int sms = c->num_sms;
  for (uint32_t first = 0; first < total; first += t->chunk) {
    const uint32_t cnt = std::min(total - first, t->chunk);
    if (t->cfg.exact_weight_grads) {
      const uint32_t tiles = (cnt + 31) / 32, want = (tiles + kBwdWarps - 1) / kBwdWarps;
      backward_kernel<<<want < (uint32_t)sms ? want : (uint32_t)sms, 32 * kBwdWarps, (int)sizeof(BackwardSmem),
                        t->st>>>(t->d_recs, first, cnt, t->d_list, rays, t->d_enc, c->scene, sg, t->d_denc);
      TR_CUDA(cudaGetLastError());
      TR_CUDA((launch_dw<kEnc, kHid, kHid, 4, 8>(sg.enc, sg.dh1, tiles, gw + kOffDW1, sms, t->st)));
      TR_CUDA((launch_dw<kHid, kDOut, kDOut, 8, 4>(sg.h1, sg.dout, tiles, gw + kOffDW2, sms, t->st)));
      TR_CUDA((launch_dw<kCIn, kHid, kHid, 4, 8>(sg.cin, sg.dg1, tiles, gw + kOffCW1, sms, t->st)));
      TR_CUDA((launch_dw<kHid, kHid, kHid, 8, 4>(sg.g1, sg.dg2, tiles, gw + kOffCW2, sms, t->st)));
      TR_CUDA((launch_dw<kHid, 3, kFDlog, 8, 4>(sg.g2, sg.dlog, tiles, gw + kOffCW3, sms, t->st)));
    } else {
      const uint32_t groups = (cnt + 127u) / 128u;
      const uint32_t want = (groups + kBtGroups - 1) / kBtGroups;
      backward_tc_kernel<<<want < (uint32_t)sms ? want : (uint32_t)sms, kBtThreads, kBtSmem, t->st>>>(
          t->d_recs, first, cnt, t->d_list, rays, t->d_enc, t->d_bimg, sg, t->d_denc, t->d_ctr + 1);
      TR_CUDA(cudaGetLastError());
      const uint32_t tiles = (cnt + 31) / 32;
      const uint32_t grid = tiles < (uint32_t)sms ? tiles : (uint32_t)sms;
      dw_tc_kernel<<<grid, kDwTcThreads, sizeof(DwTcSmem), t->st>>>(sg, c->d_weights + kOffCW3, tiles, gw, t->d_ctr + 1);
      TR_CUDA(cudaGetLastError());
    }
    scatter_kernel<<<(cnt + kScatThreads - 1) / kScatThreads, kScatThreads, 0, t->st>>>(
        t->d_recs, first, cnt, c->scene, t->d_denc, t->d_gtable);
    TR_CUDA(cudaGetLastError());
  }
  return NES_OK;
}

int train_error(uint32_t word) {
  switch (word) {
    case 0: return NES_OK;
    case kErrOverflow: return NES_ENOMEM;
    case kErrTimeout: return NES_ETIMEDOUT;
    default: return NES_EINVAL;
  }
}

int clear_gradients(nes_trainer* t) {
  TR_CUDA(cudaMemsetAsync(t->d_gtable, 0, (size_t)kLevels * t->ctx->scene.T * sizeof(float2), t->st));
  TR_CUDA(cudaMemsetAsync(t->d_gw, 0, kWeightFloats * sizeof(float), t->st));
  TR_CUDA(cudaStreamSynchronize(t->st));
  return NES_OK;
}

int accumulate_parts(nes_trainer* t, int n, double* loss) {
  nes_ctx* c = t->ctx;
  const int blocks = (n + kRayBlock - 1) / kRayBlock;
  t->last_samples = 0;
  t->phase_ms[0] = t->phase_ms[1] = 0.0f;
  TR_CUDA(cudaMemsetAsync(t->d_loss, 0, sizeof(double), t->st));
  TR_CUDA(cudaEventRecord(t->ev[0], t->st));
  count_kernel<<<blocks, kWalkThreads, 0, t->st>>>(t->d_rays, n, c->scene, t->d_rout, t->d_block_count);
  TR_CUDA(cudaGetLastError());
  scan_kernel<<<1, kScanThreads, 0, t->st>>>(t->d_block_count, blocks, t->d_block_first);
  TR_CUDA(cudaGetLastError());
  TR_CUDA(cudaMemcpyAsync(t->h_block_first, t->d_block_first, (size_t)(blocks + 1) * sizeof(uint32_t),
                          cudaMemcpyDeviceToHost, t->st));
  if (!t->cfg.exact_weight_grads) {  // this step's weights as TF32 operand images
    pack_et_images_kernel<<<(kFwdImageBytes / 4 + 255) / 256, 256, 0, t->st>>>(c->d_weights, t->d_eimg);
    TR_CUDA(cudaGetLastError());
    pack_bt_images_kernel<<<(kBtImageBytes / 4 + 255) / 256, 256, 0, t->st>>>(c->d_weights, t->d_bimg);
    TR_CUDA(cudaGetLastError());
  }
  TR_CUDA(cudaStreamSynchronize(t->st));
  const uint32_t* first = t->h_block_first;
  for (int b0 = 0; b0 < blocks;) {
    int b1 = b0 + 1;
    while (b1 < blocks && first[b1 + 1] - first[b0] <= t->list_capacity) ++b1;
    const uint32_t base = first[b0], m = first[b1] - base;
    const int r0 = b0 * kRayBlock, nr = std::min(n, b1 * kRayBlock) - r0, nb = b1 - b0;
    const TrainRay* rays = t->d_rays + r0;
    RayOut* rout = t->d_rout + r0;
    const uint32_t* block_first = t->d_block_first + b0;
    if (b0 > 0) TR_CUDA(cudaEventRecord(t->ev[0], t->st));
    TR_CUDA(cudaMemsetAsync(t->d_ctr, 0, sizeof(uint32_t), t->st));  // the error word is cleared by the caller
    if (m > 0) {
      list_kernel<<<nb, kWalkThreads, 0, t->st>>>(rays, nr, c->scene, rout, block_first, base, t->d_list);
      TR_CUDA(cudaGetLastError());
      encode_kernel<<<(m + kEncThreads - 1) / kEncThreads, kEncThreads, 0, t->st>>>(t->d_list, m, rays, c->scene,
                                                                                  t->d_enc);
      TR_CUDA(cudaGetLastError());
      if (t->cfg.exact_weight_grads)
        eval_kernel<<<c->num_sms, 32 * kEvalWarps, (int)sizeof(EvalSmem), t->st>>>(t->d_list, m, rays, c->scene, t->d_enc,
                                                                  t->d_scratch);
      else
        eval_tc_kernel<<<c->num_sms, kEtThreads, kEtSmem, t->st>>>(t->d_list, m, rays, t->d_enc, t->d_eimg,
                                                                  t->d_scratch, t->d_ctr + 1);
      TR_CUDA(cudaGetLastError());
    }
    composite_kernel<<<nb, kRayBlock, 0, t->st>>>(nr, t->d_scratch, block_first, base, rout);
    TR_CUDA(cudaGetLastError());
    adjoint_kernel<<<nb, kRayBlock, 0, t->st>>>(rays, rout, nr, t->d_scratch, block_first, base, t->d_recs,
                                                t->list_capacity, t->d_ctr, t->d_ctr + 1, t->d_loss,
                                                t->cfg.depth_weight, 1.0f / (float)n);
    TR_CUDA(cudaGetLastError());
    TR_CUDA(cudaEventRecord(t->ev[1], t->st));
    uint32_t h[2] = {0, 0};
    TR_CUDA(cudaMemcpyAsync(h, t->d_ctr, sizeof(h), cudaMemcpyDeviceToHost, t->st));
    TR_CUDA(cudaMemcpyAsync(loss, t->d_loss, sizeof(double), cudaMemcpyDeviceToHost, t->st));
    TR_CUDA(cudaStreamSynchronize(t->st));
    int rc = train_error(h[1]);
    if (rc != NES_OK) return rc;
    t->last_samples += h[0];
    if ((rc = backward_records(t, rays, h[0])) != NES_OK) return rc;
    TR_CUDA(cudaEventRecord(t->ev[2], t->st));
    // A tensor-core wait that ran out reports through the error word.
    TR_CUDA(cudaMemcpyAsync(h, t->d_ctr, sizeof(h), cudaMemcpyDeviceToHost, t->st));
    TR_CUDA(cudaStreamSynchronize(t->st));
    if ((rc = train_error(h[1])) != NES_OK) return rc;
    float ms = 0.0f;
    TR_CUDA(cudaEventElapsedTime(&ms, t->ev[0], t->ev[1]));
    t->phase_ms[0] += ms;
    TR_CUDA(cudaEventElapsedTime(&ms, t->ev[1], t->ev[2]));
    t->phase_ms[1] += ms;
    b0 = b1;
  }
  return NES_OK;
}

// Loss and gradients (accumulated into d_gtable / d_gw) for the n rays in
// d_rays, as many blocks of kRayBlock rays at a time as the sample list holds.
// A batch that fails in one part leaves no gradient of its earlier ones.
int loss_and_grad(nes_trainer* t, int n, double* loss) {
  const int rc = accumulate_parts(t, n, loss);
  if (rc != NES_OK) clear_gradients(t);
  return rc;
}

int upload_rays(nes_trainer* t, const int32_t* rays, int n) {
  if (!rays || n < 1 || (uint32_t)n > t->max_rays || t->nviews == 0) return NES_EINVAL;
  TR_CUDA(cudaMemsetAsync(t->d_ctr + 1, 0, sizeof(uint32_t), t->st));
  TR_CUDA(cudaMemcpyAsync(t->d_pairs, rays, (size_t)n * sizeof(int2), cudaMemcpyHostToDevice, t->st));
  make_rays_kernel<<<(n + 255) / 256, 256, 0, t->st>>>(t->d_pairs, n, t->d_views, t->nviews, t->trgb, t->tdep,
                                                       t->d_rays, t->d_ctr + 1);
  TR_CUDA(cudaGetLastError());
  return NES_OK;
}

int adam(nes_trainer* t) {
  nes_ctx* c = t->ctx;
  t->steps++;
  const float b1 = t->cfg.beta1, b2 = t->cfg.beta2;
  const float bc1 = (float)(1.0 - std::pow((double)b1, (double)t->steps));
  const float bc2 = (float)(1.0 - std::pow((double)b2, (double)t->steps));
  const size_t nt = (size_t)kLevels * c->scene.T * 2;
  TR_CUDA(cudaEventRecord(t->ev[3], t->st));
  adam_kernel<<<4 * c->num_sms, 256, 0, t->st>>>(reinterpret_cast<float*>(c->d_table32),
                                                 reinterpret_cast<float*>(t->d_gtable), t->d_mt, t->d_vt, nt,
                                                 t->cfg.lr, b1, b2, t->cfg.eps, bc1, bc2);
  TR_CUDA(cudaGetLastError());
  adam_kernel<<<(kWeightFloats + 255) / 256, 256, 0, t->st>>>(c->d_weights, t->d_gw, t->d_mw, t->d_vw,
                                                              (size_t)kWeightFloats, t->cfg.lr, b1, b2, t->cfg.eps,
                                                              bc1, bc2);
  TR_CUDA(cudaGetLastError());
  TR_CUDA(cudaEventRecord(t->ev[4], t->st));
  TR_CUDA(cudaStreamSynchronize(t->st));
  TR_CUDA(cudaEventElapsedTime(&t->phase_ms[2], t->ev[3], t->ev[4]));
  return NES_OK;
}

void free_trainer(nes_trainer* t) {
  cudaFree(t->d_views);
  cudaFree(t->d_pairs);
  cudaFree(t->d_rays);
  cudaFree(t->d_list);
  cudaFree(t->d_enc);
  cudaFree(t->d_recs);
  cudaFree(t->d_block_count);
  cudaFree(t->d_block_first);
  if (t->h_block_first) cudaFreeHost(t->h_block_first);
  cudaFree(t->d_rout);
  cudaFree(t->d_ctr);
  cudaFree(t->d_loss);
  cudaFree(t->d_gtable);
  cudaFree(t->d_gw);
  cudaFree(t->d_mt);
  cudaFree(t->d_vt);
  cudaFree(t->d_mw);
  cudaFree(t->d_vw);
  cudaFree(t->d_stage);
  cudaFree(t->d_denc);
  cudaFree(t->d_bimg);
  cudaFree(t->d_eimg);
  for (cudaEvent_t e : t->ev)
    if (e) cudaEventDestroy(e);
  if (t->st) cudaStreamDestroy(t->st);
  delete t;
}

}  // namespace

extern "C" {

void nes_train_config_default(nes_train_config* cfg) {
  std::memset(cfg, 0, sizeof(*cfg));
  cfg->batch_rays = 1u << 18;
  cfg->lr = 1e-2f;
  cfg->beta1 = 0.9f;
  cfg->beta2 = 0.99f;
  cfg->eps = 1e-15f;
  cfg->depth_weight = 0.1f;
  cfg->exact_weight_grads = 0;
}

int nes_trainer_create(nes_ctx* ctx, const nes_train_config* cfg, nes_trainer** out) {
  if (!ctx || !cfg || !out) return NES_EINVAL;
  *out = nullptr;
  if (ctx->cfg.precision != NES_PREC_FP32) return NES_EINVAL;
  if (cfg->batch_rays == 0 || cfg->batch_rays > (1u << 20) || !(cfg->lr > 0.0f) || !(cfg->beta1 >= 0.0f) ||
      !(cfg->beta1 < 1.0f) || !(cfg->beta2 >= 0.0f) || !(cfg->beta2 < 1.0f) || !(cfg->eps >= 0.0f) ||
      !(cfg->depth_weight >= 0.0f))
    return NES_EINVAL;
  if (cudaSetDevice(ctx->cfg.device) != cudaSuccess) return NES_ENODEV;
  nes_trainer* t = new (std::nothrow) nes_trainer;
  if (!t) return NES_ENOMEM;
  t->ctx = ctx;
  t->cfg = *cfg;
  t->max_rays = cfg->batch_rays;
  auto fail = [&](int code) {
    free_trainer(t);
    return code;
  };
  if (cudaStreamCreateWithFlags(&t->st, cudaStreamNonBlocking) != cudaSuccess) return fail(NES_EIO);
  for (cudaEvent_t& e : t->ev)
    if (cudaEventCreate(&e) != cudaSuccess) return fail(NES_EIO);
  const size_t nt = (size_t)kLevels * ctx->scene.T * 2;
  const size_t blocks = (t->max_rays + kRayBlock - 1) / kRayBlock;
  const bool exact = cfg->exact_weight_grads != 0;
  const TrainerSizes sizes = trainer_sizes(t->max_rays, exact);
  const size_t max_samples = sizes.samples;
  t->list_capacity = (uint32_t)sizes.samples;
  t->chunk = (uint32_t)sizes.records;
  if (cudaMalloc(&t->d_pairs, (size_t)t->max_rays * sizeof(int2)) != cudaSuccess ||
      cudaMalloc(&t->d_rays, (size_t)t->max_rays * sizeof(TrainRay)) != cudaSuccess ||
      cudaMalloc(&t->d_list, max_samples * sizeof(uint2)) != cudaSuccess ||
      cudaMalloc(&t->d_enc, max_samples * kEnc * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&t->d_block_count, blocks * sizeof(uint32_t)) != cudaSuccess ||
      cudaMalloc(&t->d_block_first, (blocks + 1) * sizeof(uint32_t)) != cudaSuccess ||
      cudaMallocHost(&t->h_block_first, (blocks + 1) * sizeof(uint32_t)) != cudaSuccess ||
      cudaMalloc(&t->d_recs, max_samples * sizeof(SampleRec)) != cudaSuccess ||
      cudaMalloc(&t->d_rout, (size_t)t->max_rays * sizeof(RayOut)) != cudaSuccess ||
      cudaMalloc(&t->d_ctr, 4 * sizeof(uint32_t)) != cudaSuccess ||
      cudaMalloc(&t->d_loss, sizeof(double)) != cudaSuccess ||
      cudaMalloc(&t->d_gtable, nt * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&t->d_gw, kWeightFloats * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&t->d_mt, nt * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&t->d_vt, nt * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&t->d_mw, kWeightFloats * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&t->d_vw, kWeightFloats * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&t->d_stage, sizes.stage_bytes) != cudaSuccess ||
      cudaMalloc(&t->d_denc, (size_t)t->chunk * kEnc * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&t->d_bimg, kBtImageBytes) != cudaSuccess ||
      cudaMalloc(&t->d_eimg, kEtImageBytes) != cudaSuccess)
    return fail(NES_ENOMEM);
  t->d_scratch = static_cast<ScratchSample*>(t->d_stage);
  if (cudaMemset(t->d_gtable, 0, nt * sizeof(float)) != cudaSuccess ||
      cudaMemset(t->d_gw, 0, kWeightFloats * sizeof(float)) != cudaSuccess ||
      cudaMemset(t->d_mt, 0, nt * sizeof(float)) != cudaSuccess ||
      cudaMemset(t->d_vt, 0, nt * sizeof(float)) != cudaSuccess ||
      cudaMemset(t->d_mw, 0, kWeightFloats * sizeof(float)) != cudaSuccess ||
      cudaMemset(t->d_vw, 0, kWeightFloats * sizeof(float)) != cudaSuccess ||
      cudaMemset(t->d_ctr, 0, 4 * sizeof(uint32_t)) != cudaSuccess)
    return fail(NES_EIO);
  if (cudaFuncSetAttribute(eval_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(EvalSmem)) != cudaSuccess ||
      cudaFuncSetAttribute(backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BackwardSmem)) != cudaSuccess ||
      cudaFuncSetAttribute(dw_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DwTcSmem)) !=
          cudaSuccess ||
      cudaFuncSetAttribute(backward_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBtSmem) != cudaSuccess ||
      cudaFuncSetAttribute(eval_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kEtSmem) != cudaSuccess)
    return fail(NES_EIO);
  {
    // backward_tc_kernel allocates all 512 TMEM columns: one CTA per SM,
    // which its register footprint (512 threads x > 64) guarantees.
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, backward_tc_kernel) != cudaSuccess || fa.numRegs <= 64) return fail(NES_EIO);
  }
  *out = t;
  return NES_OK;
}

void nes_trainer_destroy(nes_trainer* t) {
  if (!t) return;
  cudaSetDevice(t->ctx->cfg.device);
  cudaStreamSynchronize(t->st);
  free_trainer(t);
}

int nes_trainer_set_targets(nes_trainer* t, const nes_view* views, int nviews, const float* rgb_dev,
                            const float* depth_dev) {
  if (!t || !views || nviews < 1 || nviews > 1024 || !rgb_dev || !depth_dev) return NES_EINVAL;
  std::lock_guard<std::mutex> lk(t->ctx->mu);  // no render of the context meanwhile
  TR_CUDA(cudaSetDevice(t->ctx->cfg.device));
  std::vector<TrainView> hv(nviews);
  uint64_t off = 0;
  for (int i = 0; i < nviews; ++i) {
    const uint64_t px = (uint64_t)views[i].width * views[i].height;
    if (!view_ok(views[i])) return NES_EINVAL;  // the renderer's own view check
    std::memcpy(hv[i].M, views[i].matrix, sizeof(hv[i].M));
    hv[i].W = (int)views[i].width;
    hv[i].H = (int)views[i].height;
    hv[i].focal = views[i].focal_px;
    hv[i].pad = 0;
    hv[i].offset = off;
    off += px;
  }
  TrainView* dv = nullptr;
  TR_CUDA(cudaMalloc(&dv, nviews * sizeof(TrainView)));
  if (cudaMemcpy(dv, hv.data(), nviews * sizeof(TrainView), cudaMemcpyHostToDevice) != cudaSuccess) {
    cudaFree(dv);
    return NES_EIO;
  }
  cudaFree(t->d_views);
  t->d_views = dv;
  t->nviews = nviews;
  t->trgb = rgb_dev;
  t->tdep = depth_dev;
  return NES_OK;
}

int nes_trainer_step(nes_trainer* t, uint64_t seed, double* loss) {
  if (!t || !loss || t->nviews == 0) return NES_EINVAL;
  std::lock_guard<std::mutex> lk(t->ctx->mu);  // no render of the context meanwhile
  TR_CUDA(cudaSetDevice(t->ctx->cfg.device));
  const int n = (int)t->cfg.batch_rays;
  TR_CUDA(cudaMemsetAsync(t->d_ctr + 1, 0, sizeof(uint32_t), t->st));
  sample_pairs_kernel<<<(n + 255) / 256, 256, 0, t->st>>>(seed, n, t->d_views, t->nviews, t->d_pairs);
  TR_CUDA(cudaGetLastError());
  make_rays_kernel<<<(n + 255) / 256, 256, 0, t->st>>>(t->d_pairs, n, t->d_views, t->nviews, t->trgb, t->tdep,
                                                       t->d_rays, t->d_ctr + 1);
  TR_CUDA(cudaGetLastError());
  const int rc = loss_and_grad(t, n, loss);
  if (rc != NES_OK) return rc;
  return adam(t);
}

int nes_trainer_step_rays(nes_trainer* t, const int32_t* rays, int n, double* loss) {
  if (!t || !loss) return NES_EINVAL;
  std::lock_guard<std::mutex> lk(t->ctx->mu);  // no render of the context meanwhile
  TR_CUDA(cudaSetDevice(t->ctx->cfg.device));
  int rc = upload_rays(t, rays, n);
  if (rc != NES_OK) return rc;
  if ((rc = loss_and_grad(t, n, loss)) != NES_OK) return rc;
  return adam(t);
}

int nes_trainer_grad(nes_trainer* t, const int32_t* rays, int n, double* loss, float* grad_table,
                     float* grad_weights) {
  if (!t || !loss) return NES_EINVAL;
  std::lock_guard<std::mutex> lk(t->ctx->mu);  // no render of the context meanwhile
  TR_CUDA(cudaSetDevice(t->ctx->cfg.device));
  int rc = upload_rays(t, rays, n);
  if (rc == NES_OK) rc = loss_and_grad(t, n, loss);
  const size_t nt = (size_t)kLevels * t->ctx->scene.T * 2;
  if (rc == NES_OK && grad_table &&
      cudaMemcpyAsync(grad_table, t->d_gtable, nt * sizeof(float), cudaMemcpyDeviceToHost, t->st) != cudaSuccess)
    rc = NES_EIO;
  if (rc == NES_OK && grad_weights &&
      cudaMemcpyAsync(grad_weights, t->d_gw, kWeightFloats * sizeof(float), cudaMemcpyDeviceToHost, t->st) !=
          cudaSuccess)
    rc = NES_EIO;
  const int cleared = clear_gradients(t);
  return rc != NES_OK ? rc : cleared;
}

int nes_trainer_loss_fp64(nes_trainer* t, const int32_t* rays, int n, int which, uint64_t index, double delta,
                          double* loss) {
  if (!t || !loss || (which != 0 && which != 1)) return NES_EINVAL;
  const uint64_t limit = which == 0 ? (uint64_t)kLevels * t->ctx->scene.T * 2 : (uint64_t)kWeightFloats;
  if (index >= limit) return NES_EINVAL;
  std::lock_guard<std::mutex> lk(t->ctx->mu);  // no render of the context meanwhile
  TR_CUDA(cudaSetDevice(t->ctx->cfg.device));
  int rc = upload_rays(t, rays, n);
  if (rc != NES_OK) return rc;
  ParamsF64 P;
  P.table = reinterpret_cast<const float*>(t->ctx->d_table32);
  P.w = t->ctx->d_weights;
  P.which = which;
  P.index = index;
  P.delta = delta;
  TR_CUDA(cudaMemsetAsync(t->d_loss, 0, sizeof(double), t->st));
  loss_f64_kernel<<<(n + 63) / 64, 64, 0, t->st>>>(t->d_rays, n, t->ctx->scene, P, t->d_loss,
                                                   (double)t->cfg.depth_weight, 1.0 / (double)n);
  TR_CUDA(cudaGetLastError());
  uint32_t err = 0;
  TR_CUDA(cudaMemcpyAsync(&err, t->d_ctr + 1, sizeof(err), cudaMemcpyDeviceToHost, t->st));
  TR_CUDA(cudaMemcpyAsync(loss, t->d_loss, sizeof(double), cudaMemcpyDeviceToHost, t->st));
  TR_CUDA(cudaStreamSynchronize(t->st));
  return err ? NES_EINVAL : NES_OK;
}

int nes_trainer_loss_fp64_batch(nes_trainer* t, const int32_t* rays, int n, int m, const int32_t* which,
                                const uint64_t* index, const double* delta, double* losses) {
  if (!t || !which || !index || !delta || !losses || m < 1 || m > 65535) return NES_EINVAL;
  const uint64_t limits[2] = {(uint64_t)kLevels * t->ctx->scene.T * 2, (uint64_t)kWeightFloats};
  std::vector<PerturbF64> host((size_t)m);
  for (int j = 0; j < m; ++j) {
    if (which[j] != 0 && which[j] != 1) return NES_EINVAL;
    if (index[j] >= limits[which[j]]) return NES_EINVAL;
    host[j] = PerturbF64{which[j], index[j], delta[j]};
  }
  std::lock_guard<std::mutex> lk(t->ctx->mu);  // no render of the context meanwhile
  TR_CUDA(cudaSetDevice(t->ctx->cfg.device));
  int rc = upload_rays(t, rays, n);
  if (rc != NES_OK) return rc;
  PerturbF64* d_pert = nullptr;
  double* d_loss = nullptr;
  if (cudaMalloc(&d_pert, sizeof(PerturbF64) * (size_t)m) != cudaSuccess) return NES_ENOMEM;
  if (cudaMalloc(&d_loss, sizeof(double) * (size_t)m) != cudaSuccess) {
    cudaFree(d_pert);
    return NES_ENOMEM;
  }
  cudaError_t e = cudaMemcpyAsync(d_pert, host.data(), sizeof(PerturbF64) * (size_t)m, cudaMemcpyHostToDevice, t->st);
  if (e == cudaSuccess) e = cudaMemsetAsync(d_loss, 0, sizeof(double) * (size_t)m, t->st);
  if (e == cudaSuccess) {
    loss_f64_batch_kernel<<<dim3((n + 63) / 64, m), 64, 0, t->st>>>(
        t->d_rays, n, t->ctx->scene, reinterpret_cast<const float*>(t->ctx->d_table32), t->ctx->d_weights, d_pert,
        d_loss, (double)t->cfg.depth_weight, 1.0 / (double)n);
    e = cudaGetLastError();
  }
  uint32_t err = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&err, t->d_ctr + 1, sizeof(err), cudaMemcpyDeviceToHost, t->st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(losses, d_loss, sizeof(double) * (size_t)m, cudaMemcpyDeviceToHost, t->st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(t->st);
  cudaFree(d_pert);
  cudaFree(d_loss);
  if (e != cudaSuccess) return NES_EIO;
  return err ? NES_EINVAL : NES_OK;
}

uint64_t nes_trainer_last_samples(const nes_trainer* t) { return t ? t->last_samples : 0; }

int nes_trainer_last_timings(const nes_trainer* t, float* forward_ms, float* backward_ms, float* adam_ms) {
  if (!t || !forward_ms || !backward_ms || !adam_ms) return NES_EINVAL;
  if (t->steps == 0) return NES_EAGAIN;
  *forward_ms = t->phase_ms[0];
  *backward_ms = t->phase_ms[1];
  *adam_ms = t->phase_ms[2];
  return NES_OK;
}

}  // extern "C"
