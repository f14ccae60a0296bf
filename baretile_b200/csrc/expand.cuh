// What the tensor-core matmuls share: a packed weight tile as exact bf16 in registers, and the epilogue's arithmetic.
#pragma once
#include "ptx.cuh"
#include "stream_layout.cuh"

namespace bt {

// One packed tile (streaming layout, shared address `tile`) as bf16 weights times 2^-64. a[h][fs] is what this lane (g = lane / 4,
// t = lane % 4) has of face 2h + fs: channels 16 fs + 2g (registers 0 and 2) and 2g + 1 (1 and 3), the four
// consecutive k from 16h + 4t on (0 and 1 the first pair, 2 and 3 the second). Weights are stored in offset binary: a byte
// (or a masked nibble) zero-extended into a 16-bit lane is the bf16 number code * 2^-133, and one packed fused
// multiply-add with the face row's power of two, minus the offset times it, makes it the exact signed weight
// times 2^(e - 197). A nibble q is worth 16 q: a high nibble stays where it is in its byte (16 * code), a low nibble
// takes 16 times the scale.
constexpr float kExpandedUnscale = 18446744073709551616.f;   // 2^64
struct PackedLane {
  uint4 ev, wv[2];           // the exponents and the values that a lane needs
};
template <int FMT> __device__ __forceinline__ PackedLane packed_lane(uint32_t tile, int lane) {
  PackedLane p;
  p.ev = lds128(tile + (lane & 3) * 16), p.wv[0] = lds128(tile + 64 + lane * 16);
  p.wv[1] = FMT == BT_BFP8 ? lds128(tile + 64 + 512 + lane * 16) : p.wv[0];
  return p;
}
template <int FMT> __device__ __forceinline__ void expand_weights(const PackedLane &p, uint32_t (&a)[2][2][4]) {
  const uint32_t ee[4] = {p.ev.x, p.ev.y, p.ev.z, p.ev.w};
  const uint4(&wv)[2] = p.wv;
#pragma unroll
  for (int h = 0; h < 2; h++) {
#pragma unroll
    for (int fs = 0; fs < 2; fs++) {
      const uint32_t ew = ee[2 * h + fs];
      const uint32_t s01 = scale_pair<0>(ew), s23 = scale_pair<1>(ew);
      uint32_t(&r)[4] = a[h][fs];
      if (FMT == BT_BFP8) {
        const uint32_t w0 = fs ? wv[h].z : wv[h].x, w1 = fs ? wv[h].w : wv[h].y;
        const uint32_t n01 = mul_bf16x2(s01, 0x80808080u), n23 = mul_bf16x2(s23, 0x80808080u);   // -128 * 2^-133 * scale
        r[0] = fma_bf16x2(w0 & 0x00FF00FFu, s01, n01), r[1] = fma_bf16x2(w1 & 0x00FF00FFu, s01, n01);
        r[2] = fma_bf16x2(prmt(w0, 0u, 0x4341u), s23, n23), r[3] = fma_bf16x2(prmt(w1, 0u, 0x4341u), s23, n23);
      } else {
        const uint32_t wb = h ? (fs ? wv[0].w : wv[0].z) : (fs ? wv[0].y : wv[0].x), wo = prmt(wb, 0u, 0x4341u);
        const uint32_t t01 = mul_bf16x2(s01, 0x41804180u), t23 = mul_bf16x2(s23, 0x41804180u);   // 16 * scale: a nibble q is worth 16 q
        const uint32_t n01 = mul_bf16x2(t01, 0x80088008u), n23 = mul_bf16x2(t23, 0x80088008u);   // -8 * 2^-133 * 16 * scale
        r[0] = fma_bf16x2(wb & 0x000F000Fu, t01, n01), r[1] = fma_bf16x2(wb & 0x00F000F0u, s01, n01);
        r[2] = fma_bf16x2(wo & 0x000F000Fu, t23, n23), r[3] = fma_bf16x2(wo & 0x00F000F0u, s23, n23);
      }
    }
  }
}

__device__ __forceinline__ float silu(float v) { return __fdividef(v, 1.0f + __expf(-v)); }
__device__ __forceinline__ uint32_t bf16_half_up(float v) { return (__float_as_uint(v) + 0x8000u) >> 16; }

}  // namespace bt
