// ray_slot.cuh -- how a marching warp walks its rays: several steps of each
// ray at a time, in lanes of the warp, occupied steps only.  Used by both
// precisions' marches.
#pragma once
#include "kernels.h"

namespace nes {

// Position of set bit number j (from 0) of m; m has more than j set bits.
__device__ __forceinline__ int nth_set_bit(uint32_t m, int j) {
  int pos = 0;
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) {
    const int c = __popc(m & ((1u << w) - 1u));
    if (j >= c) {
      j -= c;
      m >>= w;
      pos += w;
    }
  }
  return pos;
}

// State of one ray slot (the same in all lanes of the ray).
struct Slot {
  bool live = false;
  float3 o, d;
  float ts = 0.0f;
  int n = 0;
  int wb = 0;        // first step after the window
  uint32_t wm = 0;   // occupied steps of the window [wb - 32, wb) not yet taken
  uint32_t id = 0;

  // The slot's lanes start on compacted ray `ray`.
  __device__ __forceinline__ void start(const ViewBatch& vb, const DevScratch& s, uint32_t ray) {
    const float4 rd = s.ray_dt[ray];
    const RayMeta m = s.ray_meta[ray];
    const DevView& V = vb.v[m.view];
    o = make_float3(V.M[3], V.M[7], V.M[11]);
    d = make_float3(rd.x, rd.y, rd.z);
    ts = rd.w;
    n = m.n;
    id = ray;
    wb = 0;
    wm = 0u;
    live = true;
  }
};

// sample_pos and the occupancy test of it, in fewer instructions: the clamp
// to the unit cube is the FMA's saturation, and a coordinate of at least 0
// needs no lower bound on its cell.
__device__ __forceinline__ float3 sample_pos_sat(const float3& o, const float3& d, float t) {
  return make_float3(__saturatef(fmaf(t, d.x, o.x)), __saturatef(fmaf(t, d.y, o.y)), __saturatef(fmaf(t, d.z, o.z)));
}
__device__ __forceinline__ uint32_t occupied_at(const uint32_t* __restrict__ occ, const float3& x) {
  const int cx = min(__float2int_rd(x.x * kOccRes), kOccRes - 1), cy = min(__float2int_rd(x.y * kOccRes), kOccRes - 1),
            cz = min(__float2int_rd(x.z * kOccRes), kOccRes - 1);
  const uint32_t i = (uint32_t)cx + kOccRes * ((uint32_t)cy + kOccRes * (uint32_t)cz);
  return (__ldg(occ + (i >> 5)) >> (i & 31)) & 1u;
}

// Moves every ray whose window is used up to its next 32-step window with an
// occupied step; a ray without one is no longer live.  The ray's lanes (1 <<
// kShift of them, this one is number j) test the window's steps between them.
// Whole warps call it.
template <int kShift>
__device__ __forceinline__ void next_window(const DevScene& sc, Slot& q, int j) {
  for (;;) {
    const bool need = q.live && q.wm == 0u && q.wb < q.n;
    if (__ballot_sync(0xffffffffu, need) == 0u) break;
    uint32_t bits = 0;
    if (need) {
      const int lim = min(32, q.n - q.wb);
      for (int i = j; i < lim; i += 1 << kShift)
        bits |= occupied_at(sc.occ, sample_pos_sat(q.o, q.d, fmaf((float)(q.wb + i) + 0.5f, kDt, q.ts))) << i;
    }
#pragma unroll
    for (int k = 0; k < kShift; ++k) bits |= __shfl_xor_sync(0xffffffffu, bits, 1 << k);
    if (need) {
      q.wm = bits;
      q.wb += 32;
    }
  }
  if (q.wm == 0u) q.live = false;
}

// Takes the ray's next occupied steps of its window, one per lane in order:
// true, with the sample's t, for a lane that gets one.  Whole warps call it.
template <int kShift>
__device__ __forceinline__ bool take_step(Slot& q, int j, int ray_lane, float* t) {
  constexpr int kLanes = 1 << kShift;
  const bool has = q.live && __popc(q.wm) > j;
  int bit = 31;
  if (has) {  // mostly the window's steps are consecutive from its first one
    const int low = __ffs(q.wm) - 1;
    bit = low + j;
    if ((~(q.wm >> low) & ((2u << j) - 1u)) != 0u) bit = nth_set_bit(q.wm, j);
  }
  *t = has ? fmaf((float)(q.wb - 32 + bit) + 0.5f, kDt, q.ts) : 0.0f;
  q.wm &= ~0u << __shfl_sync(0xffffffffu, bit, ray_lane + kLanes - 1) << 1;
  return has;
}

// Four lanes' four values each -> lane c of the four has value c of all four
// (m[i]: lane i's).
__device__ __forceinline__ void transpose4(float (&m)[4], int lane) {
  const bool o1 = lane & 1, o2 = lane & 2;
  float u = __shfl_xor_sync(0xffffffffu, o1 ? m[0] : m[1], 1);
  if (o1) m[0] = u; else m[1] = u;
  u = __shfl_xor_sync(0xffffffffu, o1 ? m[2] : m[3], 1);
  if (o1) m[2] = u; else m[3] = u;
  u = __shfl_xor_sync(0xffffffffu, o2 ? m[0] : m[2], 2);
  if (o2) m[0] = u; else m[2] = u;
  u = __shfl_xor_sync(0xffffffffu, o2 ? m[1] : m[3], 2);
  if (o2) m[1] = u; else m[3] = u;
}

// Channel c (red, green, blue, expected depth) of a ray's pixel, by lane c of
// the ray's first four.
__device__ __forceinline__ void write_channel(const ViewBatch& vb, const DevScratch& s, uint32_t id, int c, float v) {
  const RayMeta m = s.ray_meta[id];
  const DevView& V = vb.v[m.view];
  if (c < 3) {
    if (V.rgb) V.rgb[(size_t)m.pixel * 3 + c] = v;
  } else if (V.depth) {
    V.depth[m.pixel] = v;
  }
}

// A ray's pixel.
__device__ __forceinline__ void write_ray(const ViewBatch& vb, const DevScratch& s, uint32_t id, float cr, float cg,
                                          float cb, float dep) {
  const RayMeta m = s.ray_meta[id];
  const DevView& V = vb.v[m.view];
  if (V.rgb) {
    V.rgb[(size_t)m.pixel * 3 + 0] = cr;
    V.rgb[(size_t)m.pixel * 3 + 1] = cg;
    V.rgb[(size_t)m.pixel * 3 + 2] = cb;
  }
  if (V.depth) V.depth[m.pixel] = dep;
}

}  // namespace nes
