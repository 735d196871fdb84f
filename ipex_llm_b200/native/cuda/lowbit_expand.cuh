// Packed weights to the activation's type, as the dequantizer warps of the tcgen05 products need them: 8 codes of one row
// become 16 bytes of consecutive k.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include <type_traits>

#include "common/utils.cuh"
#include "tcgen05_common.cuh"

namespace {

__device__ __forceinline__ int pair_row(int r) { return (r & 7) * 2 + (r >> 3); }

__device__ __forceinline__ float act_apply(float g, int act) {
  if (act == 1) return g / (1.0f + __expf(-g));
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  return 0.5f * g * (1.0f + tanhf(k0 * (g + k1 * g * g * g)));
}

// ------------------------------------------------------------------------------------------------------------------
// two-lane arithmetic in the activation dtype
// ------------------------------------------------------------------------------------------------------------------
template <typename T> struct V2;
template <> struct V2<__half> {
  using type = __half2;
  static __device__ __forceinline__ type bits(uint32_t u) { return *reinterpret_cast<type*>(&u); }
  static __device__ __forceinline__ uint32_t raw(type v) { return *reinterpret_cast<uint32_t*>(&v); }
  static __device__ __forceinline__ type splat(float f) { return __float2half2_rn(f); }
  static constexpr uint32_t kMagic = 0x64006400u;  // 1024 + q
  static constexpr float kMagicBase = 1024.f;
};
template <> struct V2<__nv_bfloat16> {
  using type = __nv_bfloat162;
  static __device__ __forceinline__ type bits(uint32_t u) { return *reinterpret_cast<type*>(&u); }
  static __device__ __forceinline__ uint32_t raw(type v) { return *reinterpret_cast<uint32_t*>(&v); }
  static __device__ __forceinline__ type splat(float f) { return __float2bfloat162_rn(f); }
  static constexpr uint32_t kMagic = 0x43004300u;  // 128 + q
  static constexpr float kMagicBase = 128.f;
};

// Per-(row, scale group) constants of the dequantizer, already in the two-lane type.
template <typename T>
struct Scale {
  typename V2<T>::type d, m;
};

// 8 codes of one 32-bit word (4-bit families) -> 8 values in k order, packed as 4 x two-lane.
// int4 words hold element k in nibble {0,4,1,5,2,6,3,7}[k]: (w >> 4i) & 0x000F000F is the pair (2i, 2i+1).
template <typename T, int WF>
__device__ __forceinline__ uint4 expand4(uint32_t w, const Scale<T>& sc, const uint32_t* lut2) {
  using V = V2<T>;
  uint32_t r[4];
  if constexpr (WF == WF_LUT4) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t pair = lut2[(w >> (8 * i)) & 0xFFu];  // (lut[lo nibble], lut[hi nibble]) in T
      r[i] = V::raw(__hmul2(V::bits(pair), sc.d));
    }
  } else {
    const typename V::type off = V::splat(V::kMagicBase + (WF == WF_SYM_INT4 ? 8.f : 0.f));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t t = ((w >> (4 * i)) & 0x000F000Fu) | V::kMagic;
      const typename V::type q = __hsub2(V::bits(t), off);  // exact: small integers
      r[i] = V::raw(WF == WF_SYM_INT4 ? __hmul2(q, sc.d) : __hfma2(q, sc.d, sc.m));
    }
  }
  return make_uint4(r[0], r[1], r[2], r[3]);
}

// Exponent re-bias for fp8 -> 16-bit float by bit placement: the fp8 byte goes to the top of the 16-bit lane, the
// 7 magnitude bits are shifted down into the wider exponent field, and the missing 2^delta is folded into the
// scale.  Works for denormals too (both formats are linear there).
template <typename T, int WF> struct Fp8Place;
// `pre` (a power of two, applied to the placed value first) keeps the scale out of fp16's denormal range: e5m2
// codes reach 57344, so their scales are ~1e-6; codes below 2^-12 of full range may flush, which is far under
// the format's own resolution.
template <> struct Fp8Place<__half, WF_FP8_E4M3> {
  static constexpr int sh = 1; static constexpr float mul = 256.f; static constexpr float pre = 1.f;
};
template <> struct Fp8Place<__half, WF_FP8_E5M2> {
  static constexpr int sh = 0; static constexpr float mul = 4096.f; static constexpr float pre = 1.f / 4096.f;
};
template <> struct Fp8Place<__nv_bfloat16, WF_FP8_E4M3> {
  static constexpr int sh = 4; static constexpr float mul = 1.329227995784916e36f /* 2^120 */;
  static constexpr float pre = 1.f;
};
template <> struct Fp8Place<__nv_bfloat16, WF_FP8_E5M2> {
  static constexpr int sh = 3; static constexpr float mul = 5.192296858534828e33f /* 2^112 */;
  static constexpr float pre = 1.f;
};

// 8 bytes (two words) of an 8-bit family -> 8 values.
template <typename T, int WF>
__device__ __forceinline__ uint4 expand8(uint32_t w0, uint32_t w1, const Scale<T>& sc) {
  using V = V2<T>;
  uint32_t r[4];
  const uint32_t ws[2] = {w0, w1};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t w = ws[i >> 1];
    if constexpr (WF == WF_INT8) {
      // (1024 + (b ^ 0x80)) - 1152 = signed value, exact in fp16
      const uint32_t t = __byte_perm(w, 0x64646464u, (i & 1) ? 0x4342 : 0x4140) ^ 0x00800080u;
      const __half2 q = __hsub2(V2<__half>::bits(t), __float2half2_rn(1152.f));
      if constexpr (std::is_same<T, __half>::value) {
        r[i] = V::raw(__hmul2(q, sc.d));
      } else {
        const float2 f = __half22float2(q);
        r[i] = V::raw(__hmul2(__floats2bfloat162_rn(f.x, f.y), sc.d));
      }
    } else {
      using P = Fp8Place<T, WF>;
      const uint32_t t = __byte_perm(w, 0u, (i & 1) ? 0x3424 : 0x1404);  // bytes to the top of each 16-bit lane
      uint32_t b = t;
      if constexpr (P::sh != 0) b = (t & 0x80008000u) | ((t >> P::sh) & (0x7F007F00u >> P::sh));
      typename V::type val = V::bits(b);
      if constexpr (P::pre != 1.f) val = __hmul2(val, V::splat(P::pre));
      r[i] = V::raw(__hmul2(val, sc.d));
    }
  }
  return make_uint4(r[0], r[1], r[2], r[3]);
}

}  // namespace
