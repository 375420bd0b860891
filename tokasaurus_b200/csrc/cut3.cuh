// A float32 number as three bfloat16 numbers, for products on the bfloat16 tensor instructions (sgemm.cu, decay_chunks.cu):
//     x 2^24 = h + m + l, 8 bits each, rounded to nearest.
// The power of two keeps all 24 bits of every number below 2^104, subnormal ones too: the lowest bit that a float32 number can have,
// 2^-149, is 2^-125 here, and the pieces, all of which are multiples of it, are no subnormal numbers.  (Cut as they are, numbers
// below 2^-109 lost bits of their third piece.)  From 2^104 on h is an infinity and a NaN follows: results that are not finite are
// made again by other means.  Sums of products come back by CUT_BACK, in the fused multiply-add that takes them.
#pragma once
#include "common.cuh"

namespace tkb {

constexpr float CUT_SCALE = 16777216.f;                       // 2^24
constexpr float CUT_BACK = 1.f / (CUT_SCALE * CUT_SCALE);     // 2^-48

__device__ __forceinline__ uint32_t cut_pack(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}
// Two numbers' differences at once.
__device__ __forceinline__ void cut_minus(float& a, float& b, uint32_t x, uint32_t y) {
  asm("{\n.reg .b64 p, q;\nmov.b64 p, {%0, %1};\nmov.b64 q, {%2, %3};\nsub.rn.f32x2 p, p, q;\nmov.b64 {%0, %1}, p;\n}"
      : "+f"(a), "+f"(b) : "r"(x), "r"(y));
}
// Two neighbouring numbers.  PAIRED: both differences at once, which wants neighbouring registers (where there are none to spare, spills).
template <bool PAIRED = true>
__device__ __forceinline__ void cut2(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
  asm("{\n.reg .b64 x, s;\nmov.b64 x, {%0, %1};\nmov.b64 s, {%2, %2};\nmul.rn.f32x2 x, x, s;\nmov.b64 {%0, %1}, x;\n}"
      : "+f"(a), "+f"(b) : "f"(CUT_SCALE));  // both at once
  h = cut_pack(a, b);
  if (PAIRED) cut_minus(a, b, h << 16, h & 0xffff0000u);
  else a -= __uint_as_float(h << 16), b -= __uint_as_float(h & 0xffff0000u);
  m = cut_pack(a, b);
  if (PAIRED) cut_minus(a, b, m << 16, m & 0xffff0000u);
  else a -= __uint_as_float(m << 16), b -= __uint_as_float(m & 0xffff0000u);
  l = cut_pack(a, b);
}
// Eight numbers -> three 16-byte pieces.
template <bool PAIRED = true>
__device__ __forceinline__ void cut8(const float4& x, const float4& y, uint4& h, uint4& m, uint4& l) {
  cut2<PAIRED>(x.x, x.y, h.x, m.x, l.x);
  cut2<PAIRED>(x.z, x.w, h.y, m.y, l.y);
  cut2<PAIRED>(y.x, y.y, h.z, m.z, l.z);
  cut2<PAIRED>(y.z, y.w, h.w, m.w, l.w);
}

}  // namespace tkb
