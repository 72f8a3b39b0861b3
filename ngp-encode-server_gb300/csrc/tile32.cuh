// tile32.cuh -- the FP32 density and colour MLPs of 32 samples by one warp,
// on the CUDA cores (the plain FP32 march, the trainer's strict mode).
//
// Evaluated one sample per thread, every weight costs a shared-memory read
// per four multiply-adds and the L1 / shared-memory pipe, not the FMA pipe,
// sets the time (85 % against 39 % busy).  Here the warp multiplies its 32
// samples' activations, kept in shared memory, by the weights as a matrix
// product: a lane owns 8 samples x 8 outputs in registers, so four 16-byte
// reads feed 64 multiply-adds.  Every output still accumulates over its inputs
// in order from zero with one FMA each, so the results are those of the
// one-sample form bit for bit.
#pragma once
#include "render_common.cuh"

namespace nes {

// Weights in shared memory, [input][output].
struct TileWeights32 {
  float dw1[kEnc * kHid];
  float dw2[kHid * kDOut];
  float cw1[kCIn * kHid];
  float cw2[kHid * kHid];
  float cw3[kHid * 4];  // output 3 is padding
};

// Activations of a warp's 32 samples: row = feature, 32 floats.  The two
// 64-byte halves of a row are swapped in every other group of four rows, so
// that the lanes' 16-byte stores of a layer's outputs (rows four apart) do not
// meet in the same banks.
constexpr int kTileFloats = kHid * 32;
__host__ __device__ constexpr int tile_swap(int row) { return ((row >> 2) & 1) << 4; }

__device__ inline void load_tile_weights32(TileWeights32& W, const float* __restrict__ g) {
  for (int i = threadIdx.x; i < kEnc * kHid; i += blockDim.x) W.dw1[i] = g[kOffDW1 + (i % kHid) * kEnc + i / kHid];
  for (int i = threadIdx.x; i < kHid * kDOut; i += blockDim.x) W.dw2[i] = g[kOffDW2 + (i % kDOut) * kHid + i / kDOut];
  for (int i = threadIdx.x; i < kCIn * kHid; i += blockDim.x) W.cw1[i] = g[kOffCW1 + (i % kHid) * kCIn + i / kHid];
  for (int i = threadIdx.x; i < kHid * kHid; i += blockDim.x) W.cw2[i] = g[kOffCW2 + (i % kHid) * kHid + i / kHid];
  for (int i = threadIdx.x; i < kHid * 4; i += blockDim.x) W.cw3[i] = i % 4 < 3 ? g[kOffCW3 + (i % 4) * kHid + i / 4] : 0.0f;
}

// acc.{lo, hi} = w * x.{lo, hi} + acc.{lo, hi}: two FP32 FMAs, each rounded
// as fmaf rounds.
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long w, unsigned long long x) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(w), "l"(x));
}
__device__ __forceinline__ unsigned long long twice(float w) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(w));
  return r;
}
__device__ __forceinline__ float4 four(unsigned long long a, unsigned long long b) {
  float4 v;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(a));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v.z), "=f"(v.w) : "l"(b));
  return v;
}
__device__ __forceinline__ float4 relu4(const float4& v) {
  return make_float4(fmaxf(v.x, 0.0f), fmaxf(v.y, 0.0f), fmaxf(v.z, 0.0f), fmaxf(v.w, 0.0f));
}

// X[0..64) = ep(W^T in[0..K)) for the warp's samples, W [K][64], K a multiple
// of 8 (in may be X); ep(i, row, sample, v) gets this lane's i-th four outputs
// (i < 16): output `row` of samples sample .. sample + 3.  Around each eight
// inputs' products, bg.begin(i) and bg.finish(i), i = bg0 + (input / 8): other
// work whose memory reads they hide.  A lane has samples 4 sg + {0..3, 16..19}
// and outputs 4 og + {0..3, 32..35}, the samples two by two in packed FMAs.  A
// 16-byte shared-memory read costs two passes instead of four when lanes i and
// i ^ 1 (or i ^ 2) want the same address: bit 0 of the lane is og's and bit 1
// is sg's, so both operands' reads do.  Seeded 1080p view: 232 ms one sample per
// thread; 155 ms as a product with sg in bits 0-1 (four passes for the
// activations), 150 ms so, 145 ms with packed FMAs (12 warps, 32 steps per ray).
template <class Bg, class Ep>
__device__ __forceinline__ void tile_layer64(const float* __restrict__ W, int K, const float* in, float* X, int lane,
                                             Bg& bg, int bg0, Ep&& ep) {
  const int sg = 4 * ((lane >> 1) & 3), og = 4 * ((lane & 1) | ((lane >> 2) & 6));
  unsigned long long acc[8][4];  // [output][pair of samples]
#pragma unroll
  for (int o = 0; o < 8; ++o)
#pragma unroll
    for (int s = 0; s < 4; ++s) acc[o][s] = 0ull;
#pragma unroll 1
  for (int k0 = 0; k0 < K; k0 += 8) {
    bg.begin(bg0 + k0 / 8);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float* xr = in + (k0 + k) * 32;
      const float* wr = W + (k0 + k) * kHid + og;
      const ulonglong2 x0 = *reinterpret_cast<const ulonglong2*>(xr + (sg ^ tile_swap(k)));
      const ulonglong2 x1 = *reinterpret_cast<const ulonglong2*>(xr + ((sg + 16) ^ tile_swap(k)));
      const float4 w0 = *reinterpret_cast<const float4*>(wr);
      const float4 w1 = *reinterpret_cast<const float4*>(wr + 32);
      const unsigned long long x[4] = {x0.x, x0.y, x1.x, x1.y};
      const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
      for (int o = 0; o < 8; ++o) {
        const unsigned long long ww = twice(w[o]);
#pragma unroll
        for (int s = 0; s < 4; ++s) fma2(acc[o][s], ww, x[s]);
      }
    }
    __syncwarp();  // in[k0 .. k0 + 8) has been read: finish may write there
    bg.finish(bg0 + k0 / 8);
  }
  __syncwarp();
  const int swap = tile_swap(og);
#pragma unroll
  for (int o = 0; o < 8; ++o) {
    const int row = og + (o & 3) + (o >> 2) * 32;
    float* xr = X + row * 32;
    *reinterpret_cast<float4*>(xr + (sg ^ swap)) = ep(2 * o, row, sg, four(acc[o][0], acc[o][1]));
    *reinterpret_cast<float4*>(xr + ((sg + 16) ^ swap)) = ep(2 * o + 1, row, sg + 16, four(acc[o][2], acc[o][3]));
  }
  __syncwarp();
}

// W^T X[0..K) for the warp's samples, 16 outputs, W [K][kLd]: ep(row, sample,
// v) gets output `row` of samples sample .. sample + 3 after every lane has
// read X.
template <int K, int kLd, class Ep>
__device__ __forceinline__ void tile_layer16(const float* __restrict__ W, const float* X, int lane, Ep&& ep) {
  const int sg = 4 * ((lane >> 1) & 7), og = 4 * ((lane & 1) | ((lane >> 3) & 2));
  float acc[4][4];
#pragma unroll
  for (int o = 0; o < 4; ++o)
#pragma unroll
    for (int s = 0; s < 4; ++s) acc[o][s] = 0.0f;
#pragma unroll 1
  for (int k0 = 0; k0 < K; k0 += 8) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float4 xv = *reinterpret_cast<const float4*>(X + (k0 + k) * 32 + (sg ^ tile_swap(k)));
      const float4 wv = *reinterpret_cast<const float4*>(W + (k0 + k) * kLd + og);
      const float x[4] = {xv.x, xv.y, xv.z, xv.w}, w[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
      for (int o = 0; o < 4; ++o)
#pragma unroll
        for (int s = 0; s < 4; ++s) acc[o][s] = fmaf(w[o], x[s], acc[o][s]);
    }
  }
  __syncwarp();
#pragma unroll
  for (int o = 0; o < 4; ++o) ep(og + o, sg, make_float4(acc[o][0], acc[o][1], acc[o][2], acc[o][3]));
}

// The colour logits of the lane's own sample, X[0..64) = the last hidden
// layer.
__device__ __forceinline__ float3 tile_logits(const float* __restrict__ cw3, const float* X, int lane) {
  float r = 0.0f, g = 0.0f, b = 0.0f;
#pragma unroll 8
  for (int k = 0; k < kHid; ++k) {
    const float a = X[k * 32 + (lane ^ tile_swap(k))];
    const float4 c3 = *reinterpret_cast<const float4*>(cw3 + k * 4);
    r = fmaf(c3.x, a, r);
    g = fmaf(c3.y, a, g);
    b = fmaf(c3.z, a, b);
  }
  __syncwarp();  // X may be written again
  return make_float3(r, g, b);
}

// The density MLP's second layer and the colour input: X[0..64) = the hidden
// layer -> X[0..32) = [SH16(d) | outputs 1..15 | 0]; every lane gets its own
// sample's output 0 and SH basis.
__device__ __forceinline__ float tile_colour_input(const float* __restrict__ dw2, float* X, int lane, const float3& d,
                                                   float (&sh)[16]) {
  // Output 0 passes through row 31, which is then the input's zero.
  tile_layer16<kHid, kDOut>(dw2, X, lane, [&](int m, int sample, const float4& v) {
    const int row = m == 0 ? 31 : 15 + m;
    *reinterpret_cast<float4*>(X + row * 32 + (sample ^ tile_swap(row))) = v;
  });
  sh16(d, sh);
#pragma unroll
  for (int k = 0; k < 16; ++k) X[k * 32 + (lane ^ tile_swap(k))] = sh[k];
  __syncwarp();
  float* const row31 = X + 31 * 32 + (lane ^ tile_swap(31));
  const float logit = *row31;
  *row31 = 0.0f;
  __syncwarp();
  return logit;
}

// No other work under the products.
struct NoOtherWork {
  __device__ __forceinline__ void begin(int) {}
  __device__ __forceinline__ void finish(int) {}
};

// Both MLPs of the warp's samples, whose 32 encoded features are in E; X is
// scratch.  Every lane gets its own sample's density and colour; d is its
// direction.  bg.begin(i) and bg.finish(i) are called for i = 0..15 on the
// way; after finish(i), rows 2 i and 2 i + 1 of E are free.  The three 64-wide
// layers run through one copy of the product: with three, the march waited for
// instructions (0.46 of its stalls per issue), 128.1 ms per 1080p view; 120.4
// so.
template <class Bg>
__device__ __forceinline__ float tile_mlp32(const TileWeights32& W, const float* E, float* X, int lane,
                                            const float3& d, float3* rgb, Bg& bg) {
  float logit = 0.0f;
#pragma unroll 1
  for (int layer = 0; layer < 3; ++layer) {
    tile_layer64(layer == 0 ? W.dw1 : layer == 1 ? W.cw1 : W.cw2, layer < 2 ? 32 : 64, layer == 0 ? E : X, X, lane, bg,
                 4 * layer, [](int, int, int, const float4& v) { return relu4(v); });
    if (layer == 0) {
      float sh[16];
      logit = tile_colour_input(W.dw2, X, lane, d, sh);
    }
  }
  const float3 lg = tile_logits(W.cw3, X, lane);
  *rgb = make_float3(sigmoidf(lg.x), sigmoidf(lg.y), sigmoidf(lg.z));
  return expf(logit - 1.0f);
}

}  // namespace nes
