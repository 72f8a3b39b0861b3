// glue.cu -- frame glue kernels: RGB24/GRAY8 -> YUV420P, depth packing and
// quantisation.  They replace RenderedFrame::convert_frame, which runs
// libswscale on the CPU once per eye and frame
// (include/base/video/rendered_frame.h:24-33,
// src/base/video/type_managers.cc:143-153), writing the YUV420P plane layout
// that AVCodecContextManager::send_frame consumes (src/encode.cpp:136-137).
//
// Conversion: ITU-R BT.601 studio range in fixed point (coefficients in
// nes_spec.h).  Luma per pixel with 16 fractional bits; chroma from the sum
// of each 2x2 block (18 fractional bits = block average), with the last row
// and column replicated when a dimension is odd.  All integer, so the result
// is bit-exact against the CPU restatement.  Every kernel is HBM-bound.
#include <algorithm>
#include <cstring>

#include "kernels.h"

namespace nes {

namespace {

constexpr int kGlueThreads = 256;
constexpr int kSms = 152;

__device__ __forceinline__ uint8_t clamp8(int32_t v) { return (uint8_t)min(max(v, 0), 255); }

__device__ __forceinline__ uint8_t luma(int r, int g, int b) {
  return clamp8((kYR * r + kYG * g + kYB * b + (16 << 16) + (1 << 15)) >> 16);
}

// One 2x2 block: 4 luma samples and one Cb/Cr pair.
__device__ __forceinline__ void rgb_block_scalar(const uint8_t* __restrict__ rgb, int w, int h, int rgb_ls,
                                                 uint8_t* __restrict__ Y, uint8_t* __restrict__ U,
                                                 uint8_t* __restrict__ V, int ls0, int ls1, int ls2, int cx,
                                                 int cy) {
  int sr = 0, sg = 0, sb = 0;
#pragma unroll
  for (int dy = 0; dy < 2; ++dy) {
    const int yy = 2 * cy + dy;
    const uint8_t* row = rgb + (size_t)min(yy, h - 1) * rgb_ls;
#pragma unroll
    for (int dx = 0; dx < 2; ++dx) {
      const int xx = 2 * cx + dx;
      const int rx = min(xx, w - 1);
      const int r = row[3 * rx], g = row[3 * rx + 1], b = row[3 * rx + 2];
      sr += r;
      sg += g;
      sb += b;
      if (yy < h && xx < w) Y[(size_t)yy * ls0 + xx] = luma(r, g, b);
    }
  }
  U[(size_t)cy * ls1 + cx] = clamp8((kUR * sr + kUG * sg + kUB * sb + (128 << 18) + (1 << 17)) >> 18);
  V[(size_t)cy * ls2 + cx] = clamp8((kVR * sr + kVG * sg + kVB * sb + (128 << 18) + (1 << 17)) >> 18);
}

__device__ __forceinline__ void gray_block_scalar(const uint8_t* __restrict__ g, int w, int h, int g_ls,
                                                  uint8_t* __restrict__ Y, uint8_t* __restrict__ U,
                                                  uint8_t* __restrict__ V, int ls0, int ls1, int ls2, int cx,
                                                  int cy) {
  constexpr int32_t ys = kYR + kYG + kYB;
#pragma unroll
  for (int dy = 0; dy < 2; ++dy) {
    const int yy = 2 * cy + dy;
    if (yy >= h) break;
#pragma unroll
    for (int dx = 0; dx < 2; ++dx) {
      const int xx = 2 * cx + dx;
      if (xx < w) Y[(size_t)yy * ls0 + xx] = clamp8((ys * g[(size_t)yy * g_ls + xx] + (16 << 16) + (1 << 15)) >> 16);
    }
  }
  U[(size_t)cy * ls1 + cx] = 128;
  V[(size_t)cy * ls2 + cx] = 128;
}

template <int kPx>
struct Word;
template <>
struct Word<16> {
  using type = uint4;
};
template <>
struct Word<8> {
  using type = uint2;
};
template <>
struct Word<4> {
  using type = uint32_t;
};
// kBytes bytes at p, which is aligned to them, to and from 32-bit words.
template <int kBytes>
__device__ __forceinline__ void load_word(const uint8_t* __restrict__ p, uint32_t* out) {
  const auto v = __ldg(reinterpret_cast<const typename Word<kBytes>::type*>(p));
  memcpy(out, &v, kBytes);
}
template <int kBytes>
__device__ __forceinline__ void store_word(uint8_t* p, const uint32_t* in) {
  typename Word<kBytes>::type v;
  memcpy(&v, in, kBytes);
  *reinterpret_cast<typename Word<kBytes>::type*>(p) = v;
}

template <int kPx>
__device__ __forceinline__ void rgb24_to_yuv420p_vec(const uint8_t* __restrict__ rgb, int w, int h, int rgb_ls,
                                                     uint8_t* __restrict__ Y, uint8_t* __restrict__ U,
                                                     uint8_t* __restrict__ V, int ls0, int ls1, int ls2,
                                                     int x0, int cy) {
  const int cw = (w + 1) >> 1;
  if (x0 + kPx > w || 2 * cy + 1 >= h) {
    for (int cx = x0 / 2; cx < min(x0 / 2 + kPx / 2, cw); ++cx)
      rgb_block_scalar(rgb, w, h, rgb_ls, Y, U, V, ls0, ls1, ls2, cx, cy);
    return;
  }
  uint32_t px[2][3 * kPx / 4];  // two rows of RGB pixels
#pragma unroll
  for (int dy = 0; dy < 2; ++dy) {
    const uint8_t* row = rgb + (size_t)(2 * cy + dy) * rgb_ls + 3 * x0;
#pragma unroll
    for (int k = 0; k < 3; ++k) load_word<kPx>(row + k * kPx, px[dy] + k * kPx / 4);
  }
  int sr[kPx / 2] = {}, sg[kPx / 2] = {}, sb[kPx / 2] = {};
#pragma unroll
  for (int dy = 0; dy < 2; ++dy) {
    uint32_t yw[kPx / 4] = {};
#pragma unroll
    for (int i = 0; i < kPx; ++i) {
      const int r = (px[dy][(3 * i) >> 2] >> (8 * ((3 * i) & 3))) & 0xff;
      const int g = (px[dy][(3 * i + 1) >> 2] >> (8 * ((3 * i + 1) & 3))) & 0xff;
      const int b = (px[dy][(3 * i + 2) >> 2] >> (8 * ((3 * i + 2) & 3))) & 0xff;
      yw[i >> 2] |= (uint32_t)luma(r, g, b) << (8 * (i & 3));
      sr[i >> 1] += r;
      sg[i >> 1] += g;
      sb[i >> 1] += b;
    }
    store_word<kPx>(Y + (size_t)(2 * cy + dy) * ls0 + x0, yw);
  }
  uint32_t uw[kPx / 8] = {}, vw[kPx / 8] = {};
#pragma unroll
  for (int c = 0; c < kPx / 2; ++c) {
    uw[c >> 2] |= (uint32_t)clamp8((kUR * sr[c] + kUG * sg[c] + kUB * sb[c] + (128 << 18) + (1 << 17)) >> 18)
                  << (8 * (c & 3));
    vw[c >> 2] |= (uint32_t)clamp8((kVR * sr[c] + kVG * sg[c] + kVB * sb[c] + (128 << 18) + (1 << 17)) >> 18)
                  << (8 * (c & 3));
  }
  store_word<kPx / 2>(U + (size_t)cy * ls1 + x0 / 2, uw);
  store_word<kPx / 2>(V + (size_t)cy * ls2 + x0 / 2, vw);
}

template <int kPx>
__device__ __forceinline__ void gray8_to_yuv420p_vec(const uint8_t* __restrict__ g, int w, int h, int g_ls,
                                                     uint8_t* __restrict__ Y, uint8_t* __restrict__ U,
                                                     uint8_t* __restrict__ V, int ls0, int ls1, int ls2,
                                                     int x0, int cy) {
  const int cw = (w + 1) >> 1;
  constexpr int32_t ys = kYR + kYG + kYB;
  if (x0 + kPx > w || 2 * cy + 1 >= h) {
    for (int cx = x0 / 2; cx < min(x0 / 2 + kPx / 2, cw); ++cx)
      gray_block_scalar(g, w, h, g_ls, Y, U, V, ls0, ls1, ls2, cx, cy);
    return;
  }
  uint32_t in[2][kPx / 4];
#pragma unroll
  for (int dy = 0; dy < 2; ++dy) load_word<kPx>(g + (size_t)(2 * cy + dy) * g_ls + x0, in[dy]);
#pragma unroll
  for (int dy = 0; dy < 2; ++dy) {
    uint32_t yw[kPx / 4] = {};
#pragma unroll
    for (int i = 0; i < kPx; ++i) {
      const int gv = (in[dy][i >> 2] >> (8 * (i & 3))) & 0xff;
      yw[i >> 2] |= (uint32_t)clamp8((ys * gv + (16 << 16) + (1 << 15)) >> 16) << (8 * (i & 3));
    }
    store_word<kPx>(Y + (size_t)(2 * cy + dy) * ls0 + x0, yw);
  }
  uint32_t c[kPx / 8];
#pragma unroll
  for (int k = 0; k < kPx / 8; ++k) c[k] = 0x80808080u;
  store_word<kPx / 2>(U + (size_t)cy * ls1 + x0 / 2, c);
  store_word<kPx / 2>(V + (size_t)cy * ls2 + x0 / 2, c);
}

// Frame f = blockIdx.y of one launch, same geometry and linesizes for every
// frame, per-frame plane pointers in the parameter table.  A thread has kPx x
// 2 pixels: kPx = 2 for any alignment; 8 and 16 as words of kPx bytes where
// every base pointer and linesize is a multiple (U and V: of kPx / 2), blocks
// cut by the right or bottom edge sample by sample, so results are identical.
// An image's blocks are numbered through: no row ends in idle warps.  30
// frames of 1280 x 720 through this twice (RGB, GRAY) and the depth packing,
// 359 MB: 67.6 us; 71.7 with rows of 8-pixel blocks and the packing's old form
// (53 at the measured copy bandwidth).
template <class Set, int kPx, bool kGray>
__global__ void __launch_bounds__(kGlueThreads)
to_yuv420p_kernel(const Set fs, int w, int h, int src_ls, int ls0, int ls1, int ls2, int cy0) {
  const uint32_t block = blockIdx.x * blockDim.x + threadIdx.x, per_row = (uint32_t)(w + kPx - 1) / kPx;
  const int f = Set::kFrames == 1 ? 0 : blockIdx.y, cy = cy0 + (int)(block / per_row), x0 = (int)(block % per_row) * kPx;
  if (cy >= (h + 1) >> 1) return;
  if constexpr (kPx == 2) {
    (kGray ? gray_block_scalar : rgb_block_scalar)(fs.src[f], w, h, src_ls, fs.y[f], fs.u[f], fs.v[f], ls0, ls1, ls2,
                                                   x0 / 2, cy);
  } else {
    (kGray ? gray8_to_yuv420p_vec<kPx> : rgb24_to_yuv420p_vec<kPx>)(fs.src[f], w, h, src_ls, fs.y[f], fs.u[f], fs.v[f],
                                                                    ls0, ls1, ls2, x0, cy);
  }
}

// round-half-up of d * 1000 in FP32; NaN/negative -> 0; saturate at 65535.
__device__ __forceinline__ uint16_t pack_mm(float d) {
  const float mm = __fmul_rn(d, 1000.0f);
  if (!(mm >= 0.0f)) return 0;
  if (mm >= 65535.0f) return 65535;
  return (uint16_t)__float2uint_rz(__fadd_rn(mm, 0.5f));
}

__device__ __forceinline__ uint8_t gray_q(float d, float dmax) {
  const float q = __fdiv_rn(d, dmax);
  const float c = q > 0.0f ? (q < 1.0f ? q : 1.0f) : 0.0f;
  return (uint8_t)__float2uint_rz(__fadd_rn(__fmul_rn(c, 255.0f), 0.5f));
}

__device__ __forceinline__ uint8_t unit_q(float x) {
  const float c = x > 0.0f ? (x < 1.0f ? x : 1.0f) : 0.0f;
  return (uint8_t)__float2uint_rz(__fadd_rn(__fmul_rn(c, 255.0f), 0.5f));
}

// Depth packing: frame f = blockIdx.y, n elements per frame.  A thread has
// kPackGroups (four; one for inputs that do not fill the chip) groups of four
// elements, all read before the first is written, a block's width apart: one group per step of a grid-sized stride leaves fewer bytes in
// flight than HBM needs (30 frames of 1280 x 720, 166 MB, launch included: 77
// us so, 70 now).  Groups as one 16-byte load when the input is 16-byte aligned
// and the output aligned to 8 (the host checks), else element by element.
template <class Set, int kPackGroups>
__global__ void __launch_bounds__(kGlueThreads) depth_pack_u16mm_kernel(const Set ds, size_t n, int vec) {
  const int f = Set::kFrames == 1 ? 0 : blockIdx.y;
  const float* __restrict__ d = ds.src[f];
  uint16_t* __restrict__ out = ds.dst[f];
  const size_t base = (size_t)blockIdx.x * (4 * kPackGroups * kGlueThreads);
  if (!vec) {
    float x[4 * kPackGroups];
#pragma unroll
    for (int k = 0; k < 4 * kPackGroups; ++k) {
      const size_t e = base + k * kGlueThreads + threadIdx.x;
      if (e < n) x[k] = __ldg(d + e);
    }
#pragma unroll
    for (int k = 0; k < 4 * kPackGroups; ++k) {
      const size_t e = base + k * kGlueThreads + threadIdx.x;
      if (e < n) out[e] = pack_mm(x[k]);
    }
    return;
  }
  const size_t first = base / 4 + threadIdx.x, n4 = n / 4;
  float4 v[kPackGroups];
#pragma unroll
  for (int k = 0; k < kPackGroups; ++k)
    if (first + k * kGlueThreads < n4) v[k] = __ldg(reinterpret_cast<const float4*>(d) + first + k * kGlueThreads);
#pragma unroll
  for (int k = 0; k < kPackGroups; ++k) {
    const size_t i = first + k * kGlueThreads;
    if (i < n4)
      reinterpret_cast<uint2*>(out)[i] =
          make_uint2((uint32_t)pack_mm(v[k].x) | ((uint32_t)pack_mm(v[k].y) << 16),
                     (uint32_t)pack_mm(v[k].z) | ((uint32_t)pack_mm(v[k].w) << 16));
    else if (i == n4)
      for (size_t e = 4 * n4; e < n; ++e) out[e] = pack_mm(d[e]);
  }
}

// Elementwise kernels: four elements per step with a float4 load when the
// input is 16-byte aligned and the output aligned to its 4-element store
// (the host checks), elements past the last whole group scalar.
__global__ void depth_to_gray8_kernel(const float* __restrict__ d, size_t n, float dmax, uint8_t* __restrict__ out,
                                      int vec) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  size_t i0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  size_t done = 0;
  if (vec) {
    const size_t n4 = n / 4;
    for (size_t i = i0; i < n4; i += stride) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(d) + i);
      reinterpret_cast<uint32_t*>(out)[i] = (uint32_t)gray_q(v.x, dmax) | ((uint32_t)gray_q(v.y, dmax) << 8) |
                                            ((uint32_t)gray_q(v.z, dmax) << 16) | ((uint32_t)gray_q(v.w, dmax) << 24);
    }
    done = n4 * 4;
  }
  for (size_t i = done + i0; i < n; i += stride) out[i] = gray_q(d[i], dmax);
}

__global__ void rgb_to_rgb24_kernel(const float* __restrict__ rgb, size_t n, uint8_t* __restrict__ out, int vec) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  size_t i0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  size_t done = 0;
  if (vec) {
    const size_t n4 = n / 4;
    for (size_t i = i0; i < n4; i += stride) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(rgb) + i);
      reinterpret_cast<uint32_t*>(out)[i] = (uint32_t)unit_q(v.x) | ((uint32_t)unit_q(v.y) << 8) |
                                            ((uint32_t)unit_q(v.z) << 16) | ((uint32_t)unit_q(v.w) << 24);
    }
    done = n4 * 4;
  }
  for (size_t i = done + i0; i < n; i += stride) out[i] = unit_q(rgb[i]);
}

// A RenderedFrame's payload in one launch: RGB24 and GRAY8 of a view (both
// outputs 4-byte aligned) and the render's three status words.  The outputs
// may be pinned host memory: a small frame then needs no copies.
__global__ void __launch_bounds__(kGlueThreads)
frame_bytes_kernel(const float* __restrict__ rgb, const float* __restrict__ depth, size_t px, float dmax,
                   uint8_t* __restrict__ rgb8, uint8_t* __restrict__ gray, const uint32_t* __restrict__ status,
                   uint32_t* __restrict__ status_out) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i < 3) status_out[i] = status[i];
  const size_t n3 = 3 * px, g3 = (n3 + 3) / 4;
  const bool colour = i < g3;
  const size_t e = 4 * (colour ? i : i - g3), n = colour ? n3 : px;
  if (e >= n) return;
  const float* in = (colour ? rgb : depth) + e;
  uint8_t* out = (colour ? rgb8 : gray) + e;
  if (e + 4 <= n) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(in));
    const float x[4] = {v.x, v.y, v.z, v.w};
    uint32_t word = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) word |= (uint32_t)(colour ? unit_q(x[k]) : gray_q(x[k], dmax)) << (8 * k);
    *reinterpret_cast<uint32_t*>(out) = word;
  } else {
    for (size_t k = 0; e + k < n; ++k) out[k] = colour ? unit_q(in[k]) : gray_q(in[k], dmax);
  }
}

// Fused frame output: one thread per 2x2 pixel block of a view of the
// batch.  Each pixel's FP32 colour is quantised to RGB24 (unit_q), its luma
// written, the block's chroma computed from the quantised 2x2 sum (edge
// pixels replicated for odd sizes, as rgb24_to_yuv420p does) and its depth
// packed to uint16 mm: byte for byte the three-kernel sequence, without the
// RGB24 intermediate in memory.
template <class Src>
__global__ void __launch_bounds__(kGlueThreads) frame_out_kernel(const __grid_constant__ Src src) {
  const FrameBatch& fb = src.get();
  const uint32_t total = fb.total_blocks;
  for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < total; b += gridDim.x * blockDim.x) {
    int vi = 0;
    while (vi + 1 < fb.n && b >= fb.f[vi + 1].first_block) ++vi;
    const FrameOut& F = fb.f[vi];
    const uint32_t local = b - F.first_block;
    const uint32_t cw = (uint32_t)(F.w + 1) >> 1;
    const int cx = (int)(local % cw), cy = (int)(local / cw);
    int sr = 0, sg = 0, sb = 0;
#pragma unroll
    for (int dy = 0; dy < 2; ++dy) {
      const int yy = 2 * cy + dy;
      const size_t row = (size_t)min(yy, F.h - 1) * (size_t)F.w;
#pragma unroll
      for (int dx = 0; dx < 2; ++dx) {
        const int xx = 2 * cx + dx;
        const size_t p = row + (size_t)min(xx, F.w - 1);
        const int r = unit_q(__ldg(F.rgb + 3 * p)), g = unit_q(__ldg(F.rgb + 3 * p + 1)),
                  bl = unit_q(__ldg(F.rgb + 3 * p + 2));
        sr += r;
        sg += g;
        sb += bl;
        if (yy < F.h && xx < F.w) {
          F.y[(size_t)yy * F.ls0 + xx] = luma(r, g, bl);
          if (F.depth_mm) F.depth_mm[p] = pack_mm(__ldg(F.depth + p));
        }
      }
    }
    F.u[(size_t)cy * F.ls1 + cx] = clamp8((kUR * sr + kUG * sg + kUB * sb + (128 << 18) + (1 << 17)) >> 18);
    F.v[(size_t)cy * F.ls2 + cx] = clamp8((kVR * sr + kVG * sg + kVB * sb + (128 << 18) + (1 << 17)) >> 18);
    if (cx == (int)cw - 1) {
      // The row padding up to each linesize is zeroed, so no plane carries
      // bytes of an earlier frame (serving reuses its output arena).
      for (int dy = 0; dy < 2; ++dy) {
        const int yy = 2 * cy + dy;
        if (yy < F.h)
          for (int xx = F.w; xx < F.ls0; ++xx) F.y[(size_t)yy * F.ls0 + xx] = 0;
      }
      for (int xx = (int)cw; xx < F.ls1; ++xx) F.u[(size_t)cy * F.ls1 + xx] = 0;
      for (int xx = (int)cw; xx < F.ls2; ++xx) F.v[(size_t)cy * F.ls2 + xx] = 0;
    }
  }
}

unsigned grid_for(size_t n) {
  size_t b = (n + 4 * kGlueThreads - 1) / (4 * kGlueThreads);
  if (b > 152 * 8) b = 152 * 8;  // grid-stride beyond 8 resident blocks per SM
  return (unsigned)(b ? b : 1);
}

bool aligned(const void* p, size_t a) { return ((uintptr_t)p % a) == 0; }

}  // namespace

namespace {

// The largest word the frames' planes allow: 16, 8 or 2 pixels per thread.
int yuv_word(const uint8_t* src, int src_ls, const uint8_t* y, const uint8_t* u, const uint8_t* v, const int ls[3]) {
  const uintptr_t row = (uintptr_t)src | (uintptr_t)src_ls | (uintptr_t)y | (uintptr_t)ls[0];
  const uintptr_t chroma = (uintptr_t)u | (uintptr_t)v | (uintptr_t)ls[1] | (uintptr_t)ls[2];
  return row % 16 == 0 && chroma % 8 == 0 ? 16 : row % 8 == 0 && chroma % 4 == 0 ? 8 : 2;
}

template <class Set, int kPx, bool kGray>
cudaError_t launch_yuv(const Set& fs, int nframes, int w, int h, int src_ls, const int ls[3],
                       cudaStream_t stream) {
  const int per_row = (w + kPx - 1) / kPx, ch = (h + 1) / 2;
  if (ch > 65535) return cudaErrorInvalidConfiguration;  // the limit of the public calls
  const int band = (int)std::min<size_t>(ch, ((size_t)1 << 31) / per_row);  // rows per launch: 32-bit block numbers
  for (int cy0 = 0; cy0 < ch; cy0 += band) {
    const size_t blocks = (size_t)per_row * std::min(band, ch - cy0);
    const dim3 grid((unsigned)((blocks + kGlueThreads - 1) / kGlueThreads), nframes);
    to_yuv420p_kernel<Set, kPx, kGray><<<grid, kGlueThreads, 0, stream>>>(fs, w, h, src_ls, ls[0], ls[1], ls[2], cy0);
  }
  return cudaGetLastError();
}

template <bool kGray, class Set>
cudaError_t launch_yuv(const Set& fs, int nframes, int w, int h, int src_ls, const int ls[3],
                       cudaStream_t stream) {
  // 16 pixels per thread once they give every SM two blocks; fewer blocks leave
  // a frame to its threads' longer chains (90 launches over 30 frames of 1280 x
  // 720, one frame each: 409 us so, 372 with 8).
  const size_t threads16 = (size_t)((w + 15) / 16) * (size_t)((h + 1) / 2) * (size_t)nframes;
  int px = threads16 >= (size_t)2 * kSms * kGlueThreads ? 16 : 8;
  for (int f = 0; f < nframes; ++f)
    px = std::min(px, yuv_word(fs.src[f], src_ls, fs.y[f], fs.u[f], fs.v[f], ls));
  if (px == 16) return launch_yuv<Set, 16, kGray>(fs, nframes, w, h, src_ls, ls, stream);
  if (px == 8) return launch_yuv<Set, 8, kGray>(fs, nframes, w, h, src_ls, ls, stream);
  return launch_yuv<Set, 2, kGray>(fs, nframes, w, h, src_ls, ls, stream);
}

template <class Set>
cudaError_t launch_pack(const Set& ds, int nframes, size_t n, cudaStream_t stream) {
  bool vec = true;
  for (int f = 0; f < nframes; ++f) vec = vec && aligned(ds.src[f], 16) && aligned(ds.dst[f], 8);
  const bool full = n * (size_t)nframes >= (size_t)2 * kSms * 16 * kGlueThreads;  // as launch_yuv
  const size_t per_block = (full ? 16 : 4) * kGlueThreads;
  const dim3 grid((unsigned)((n + per_block - 1) / per_block), nframes);
  if (full)
    depth_pack_u16mm_kernel<Set, 4><<<grid, kGlueThreads, 0, stream>>>(ds, n, vec);
  else
    depth_pack_u16mm_kernel<Set, 1><<<grid, kGlueThreads, 0, stream>>>(ds, n, vec);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_rgb24_to_yuv420p(const uint8_t* rgb, int w, int h, int rgb_ls, uint8_t* y, uint8_t* u,
                                    uint8_t* v, const int ls[3], cudaStream_t stream) {
  return launch_yuv<false>(Frames<1>{{rgb}, {y}, {u}, {v}}, 1, w, h, rgb_ls, ls, stream);
}

cudaError_t launch_gray8_to_yuv420p(const uint8_t* g, int w, int h, int g_ls, uint8_t* y, uint8_t* u, uint8_t* v,
                                    const int ls[3], cudaStream_t stream) {
  return launch_yuv<true>(Frames<1>{{g}, {y}, {u}, {v}}, 1, w, h, g_ls, ls, stream);
}

cudaError_t launch_depth_pack_u16mm(const float* d, size_t n, uint16_t* out, cudaStream_t stream) {
  return launch_pack(Depths<1>{{d}, {out}}, 1, n, stream);
}

cudaError_t launch_depth_to_gray8(const float* d, size_t n, float dmax, uint8_t* out, cudaStream_t stream) {
  depth_to_gray8_kernel<<<grid_for(n), kGlueThreads, 0, stream>>>(d, n, dmax, out, aligned(d, 16) && aligned(out, 4));
  return cudaGetLastError();
}

cudaError_t launch_rgb_to_rgb24(const float* rgb, size_t n, uint8_t* out, cudaStream_t stream) {
  rgb_to_rgb24_kernel<<<grid_for(n), kGlueThreads, 0, stream>>>(rgb, n, out, aligned(rgb, 16) && aligned(out, 4));
  return cudaGetLastError();
}

cudaError_t launch_frame_bytes(const float* rgb, const float* depth, size_t px, float dmax, uint8_t* rgb8,
                               uint8_t* gray, const uint32_t* status, uint32_t* status_out, cudaStream_t stream) {
  const size_t groups = (3 * px + 3) / 4 + (px + 3) / 4;
  const unsigned blocks = (unsigned)((groups + kGlueThreads - 1) / kGlueThreads);
  frame_bytes_kernel<<<blocks, kGlueThreads, 0, stream>>>(rgb, depth, px, dmax, rgb8, gray, status, status_out);
  return cudaGetLastError();
}

cudaError_t launch_yuv420p_batch(bool gray, const FrameSet& fs, int nframes, int w, int h, int src_ls,
                                 const int ls[3], cudaStream_t stream) {
  if (nframes < 1 || nframes > kMaxBatchFrames) return cudaErrorInvalidValue;
  return gray ? launch_yuv<true>(fs, nframes, w, h, src_ls, ls, stream)
              : launch_yuv<false>(fs, nframes, w, h, src_ls, ls, stream);
}

cudaError_t launch_depth_pack_u16mm_batch(const DepthSet& ds, int nframes, size_t n, cudaStream_t stream) {
  if (nframes < 1 || nframes > kMaxBatchFrames) return cudaErrorInvalidValue;
  return launch_pack(ds, nframes, n, stream);
}

void frame_batch_index(FrameBatch* fb) {
  uint32_t blocks = 0;
  for (int i = 0; i < fb->n; ++i) {
    fb->f[i].first_block = blocks;
    blocks += (uint32_t)((fb->f[i].w + 1) / 2) * (uint32_t)((fb->f[i].h + 1) / 2);
  }
  fb->total_blocks = blocks;
}

cudaError_t launch_frame_out(const FrameBatch& fb, cudaStream_t stream) {
  if (fb.total_blocks == 0) return cudaSuccess;
  frame_out_kernel<<<(fb.total_blocks + kGlueThreads - 1) / kGlueThreads, kGlueThreads, 0, stream>>>(
      InParam<FrameBatch>{fb});
  return cudaGetLastError();
}

cudaError_t launch_frame_out(const FrameBatch* fb_dev, int num_sms, cudaStream_t stream) {
  frame_out_kernel<<<(unsigned)num_sms * 8u, kGlueThreads, 0, stream>>>(InMemory<FrameBatch>{fb_dev});
  return cudaGetLastError();
}

}  // namespace nes
