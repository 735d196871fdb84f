// GPU quantizers (dense weight -> device tile layout) and dequantizers (tile layout / canonical blocks -> dense).
//
// * quantize: what the reference does on the host through `ggml_quantize_tensor`
//   (python/llm/src/ipex_llm/transformers/low_bit_linear.py:104-175) followed by `ggml_q_format_convet_cpu2xpu`
//   (:178-233) happens here in one pass on the GPU: a lane owns one run of 64, finds its scale and writes codes
//   and scales directly in tile order.  Arithmetic mirrors native/host/quant_core.cpp operation
//   by operation (no fused multiply-add) so that CPU- and GPU-quantized weights are bit-identical for the
//   integer formats.
// * dequantize: the reference's `xe_linear.dequant` (QLoRA backward, :534-538) and
//   `xe_linear.dequantize_rows` (quantized embedding rows, embedding.py:220-222).
#include "common/utils.cuh"
#include <cuda_fp8.h>

namespace {

__constant__ float c_nf4[16] = {-1.0f, -0.6961928009986877f, -0.5250730514526367f, -0.39491748809814453f,
                                -0.28444138169288635f, -0.18477343022823334f, -0.09105003625154495f, 0.0f,
                                0.07958029955625534f, 0.16093020141124725f, 0.24611230194568634f,
                                0.33791524171829224f, 0.44070982933044434f, 0.5626170039176941f,
                                0.7229568362236023f, 1.0f};
__constant__ float c_fp4[8] = {0.0f, 0.5f, 1.0f, 1.5f, 2.0f, 3.0f, 4.0f, 6.0f};
__constant__ float c_nf3[8] = {-1.0f, -0.5350227355957031f, -0.2469314038753510f, 0.0f,
                               0.1833375245332718f, 0.3819939494132996f, 0.6229856610298157f, 1.0f};

__device__ __forceinline__ int pair_row(int r) { return (r & 7) * 2 + (r >> 3); }

// Nearest of N ascending values (a power of two), the lower one where two are as near.  Without branches, so that the searches
// of a lane's elements overlap: 256 x 128 weights to nf4 21 us with a loop, 12 us.
template <int N> __device__ __forceinline__ int nearest_sorted(const float* table, float v) {
  int lo = 0;
#pragma unroll
  for (int step = N / 2; step > 0; step >>= 1)
    if (table[lo + step] <= v) lo += step;
  lo = min(lo, N - 2);
  return (v - table[lo] <= table[lo + 1] - v) ? lo : lo + 1;
}

// The same of sixteen values within [-1, 1] that lie more than 1 / 16 apart: a bucket of 1 / 32 holds one of them at most, so the
// bucket names the value below it and the next one to ask for (two look-ups instead of five in a chain; 7008 x 6400 bf16 to
// nf4 82 -> 56 us).
struct Buckets {
  float2 step[65];      // of a bucket: the next value, and the index of the one below it (as bits)
  float2 pair[16];      // values i and i + 1
  __device__ void fill(const float* values) {
    for (int i = threadIdx.x; i < 65; i += blockDim.x) {
      const float edge = (float)(i - 1) / 32.0f - 1.0f;         // a bucket's width below it: the product that picks it is rounded
      int lo = 0;
      for (int j = 1; j < 15; ++j)
        if (values[j] <= edge) lo = j;
      step[i] = make_float2(values[lo + 1], __int_as_float(lo));
    }
    for (int i = threadIdx.x; i < 15; i += blockDim.x) pair[i] = make_float2(values[i], values[i + 1]);
  }
  __device__ __forceinline__ int nearest(float v) const {
    const float2 st = step[min(64, max(0, (int)__fmaf_rn(v, 32.0f, 32.0f)))];
    const int lo = min(__float_as_int(st.y) + (st.x <= v ? 1 : 0), 14);
    const float2 p = pair[lo];
    return (v - p.x <= p.y - v) ? lo : lo + 1;
  }
};

// Kinds of the tiled formats.
enum { Q_SYM4 = 0, Q_ASYM4 = 1, Q_NF4 = 2, Q_FP4 = 3, Q_E4M3 = 4, Q_E5M2 = 5, Q_INT8 = 6 };

// 64 consecutive elements of a row as raw words; `wide`: the bytes that every run's address is a multiple of (32, 16 or less).
template <typename T> struct Run64 {
  static constexpr int kWords = 64 * (int)sizeof(T) / 4;
  uint32_t w[kWords];
  __device__ __forceinline__ void load(const T* p, int wide) {
    if (wide == 32) {
#pragma unroll
      for (int i = 0; i < kWords; i += 8)
        asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(w[i]), "=r"(w[i + 1]), "=r"(w[i + 2]), "=r"(w[i + 3]), "=r"(w[i + 4]), "=r"(w[i + 5]),
                       "=r"(w[i + 6]), "=r"(w[i + 7])
                     : "l"(reinterpret_cast<const uint32_t*>(p) + i));
    } else if (wide == 16) {
#pragma unroll
      for (int i = 0; i < kWords / 4; ++i) {
        const uint4 q = __ldg(reinterpret_cast<const uint4*>(p) + i);
        w[4 * i] = q.x; w[4 * i + 1] = q.y; w[4 * i + 2] = q.z; w[4 * i + 3] = q.w;
      }
    } else if constexpr (sizeof(T) == 4) {
#pragma unroll
      for (int i = 0; i < kWords; ++i) w[i] = __ldg(reinterpret_cast<const uint32_t*>(p) + i);
    } else {
#pragma unroll
      for (int i = 0; i < kWords; ++i)
        w[i] = (uint32_t)__ldg(reinterpret_cast<const uint16_t*>(p) + 2 * i) |
               ((uint32_t)__ldg(reinterpret_cast<const uint16_t*>(p) + 2 * i + 1) << 16);
    }
  }
  __device__ __forceinline__ float at(int i) const {   // i is a constant wherever this is called
    if constexpr (sizeof(T) == 4) {
      return __uint_as_float(w[i]);
    } else {
      const uint16_t h = (uint16_t)(w[i >> 1] >> (16 * (i & 1)));
      return DT<T>::to_f(*reinterpret_cast<const T*>(&h));
    }
  }
  // Smallest and largest element; NaNs are left out, as fminf and fmaxf do (two 16-bit elements at a time).
  __device__ __forceinline__ void extremes(float& lo, float& hi) const {
    if constexpr (sizeof(T) == 4) {
      lo = hi = at(0);
#pragma unroll
      for (int i = 1; i < 64; ++i) {
        lo = fminf(lo, at(i));
        hi = fmaxf(hi, at(i));
      }
    } else {
      using T2 = std::conditional_t<std::is_same<T, __half>::value, __half2, __nv_bfloat162>;
      T2 l = *reinterpret_cast<const T2*>(&w[0]), h = l;
#pragma unroll
      for (int i = 1; i < kWords; ++i) {
        const T2 v = *reinterpret_cast<const T2*>(&w[i]);
        l = __hmin2(l, v);
        h = __hmax2(h, v);
      }
      lo = fminf(DT<T>::to_f(l.x), DT<T>::to_f(l.y));
      hi = fmaxf(DT<T>::to_f(h.x), DT<T>::to_f(h.y));
    }
  }
  // The first element of the largest magnitude, as a serial loop from element 0 on finds it.
  __device__ __forceinline__ float first_largest(float lo, float hi) const {
    const float first = at(0);
    if (first != first) return first;                    // nothing compares above it
    if (hi > -lo) return hi;
    if (hi < -lo) return lo;
    if (hi == 0.f) return first;                         // zeros of either sign
    float top = first;                                   // both signs
#pragma unroll
    for (int i = 1; i < 64; ++i)
      if (fabsf(at(i)) > fabsf(top)) top = at(i);
    return top;
  }
};

// (int)y within [0, 15] for a whole run of eight, nibble by nibble: the number in the last bits of 2^23 + y, rounded down (what
// is not a number becomes zero, as the conversion has it).  put(k): the element whose code is nibble k.
template <typename F> __device__ __forceinline__ uint32_t nibbles(F&& put) {
  uint32_t w = 0;
#pragma unroll
  for (int k = 7; k >= 0; --k) {
    const float y = fminf(fmaxf(put(k), 0.f), 15.5f);
    w = w * 16 + (__float_as_uint(__fadd_rz(y, 8388608.f)) - 0x4B000000u);
  }
  return w;
}

// 32 bytes at an address that is a multiple of 16, or (`whole`) of 32.
__device__ __forceinline__ void store32(uint8_t* to, uint4 a, uint4 b, bool whole) {
  if (whole) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(to), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x),
                 "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
  } else {
    reinterpret_cast<uint4*>(to)[0] = a;
    reinterpret_cast<uint4*>(to)[1] = b;
  }
}

// Dense rows -> device tiles.  A warp makes one tile of 16 rows x 128 k, a lane one run of 64 in it (row lane / 2, half
// lane & 1): the block's scale is found in the lane's own registers (fp8 blocks of 128: two lanes), without shuffles over
// the warp, and a tile's codes leave as whole sectors.  Every byte is read and written once, padding included
// (rows up to 16, k up to 128 are written as zeros).  Bounded by its instructions, some eight for an element, and by the
// requests: a lane's accesses go along its own run of 128 bytes, so a warp's access touches 32 runs, with 32 bytes to each.
// 11008 x 4096 fp16 to sym_int4, 17 us of bytes: 190 us (behind a 123 us copy to fp32 and a zero fill) with a warp per block
// and two elements a lane; 43 us with 16-byte accesses, an element's scale search, conversion and shift one by one, and warps
// that took two or three tiles each; 33 now (the L2 written over before).
template <typename T, int KIND>
__global__ void __launch_bounds__(256) quantize_kernel(const T* __restrict__ src, uint8_t* __restrict__ dst, int64_t rows,
                                                       int64_t cols, int64_t ld, int wide, bool wide_dst) {
  constexpr bool k4 = KIND <= Q_FP4;
  __shared__ float table[16];
  __shared__ Buckets buckets;
  if (KIND == Q_NF4 || KIND == Q_FP4) {
    if (threadIdx.x < 16) table[threadIdx.x] = KIND == Q_NF4 ? c_nf4[threadIdx.x] : c_fp4[threadIdx.x & 7];
    __syncthreads();
    if (KIND == Q_NF4) {
      buckets.fill(table);
      __syncthreads();
    }
  }
  const int lane = threadIdx.x & 31, rr = lane >> 1, half = lane & 1;
  const int64_t Np = ceil_to_i64(rows, 16), Kp = ceil_to_i64(cols, 128);
  const int64_t kt = Kp / 128, tiles = Np / 16 * kt;
  uint8_t* planes = dst + (k4 ? Np * Kp / 2 : Np * Kp);
  uint16_t* sc16 = reinterpret_cast<uint16_t*>(planes);
  for (int64_t tile = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); tile < tiles;
       tile += (int64_t)gridDim.x * (blockDim.x >> 5)) {
    const int64_t r = tile / kt * 16 + rr, k0 = tile % kt * 128 + half * 64;
    const bool valid = r < rows && k0 < cols;
    Run64<T> v;
    if (valid) {
      v.load(src + r * ld + k0, wide);
    } else {
#pragma unroll
      for (int i = 0; i < Run64<T>::kWords; ++i) v.w[i] = 0;
    }
    if constexpr (k4) {
      float d, mn, hi;
      v.extremes(mn, hi);
      if (KIND == Q_ASYM4) {
        d = __fdiv_rn(__fsub_rn(hi, mn), 15.0f);
      } else {
        const float top = v.first_largest(mn, hi);
        if (KIND == Q_SYM4) d = __fdiv_rn(top, -8.0f);
        else if (KIND == Q_NF4) d = fabsf(top);
        else d = __fdiv_rn(fabsf(top), 6.0f);
      }
      const __half dh = __float2half_rn(d);
      const float ds = (KIND == Q_SYM4 || KIND == Q_ASYM4) ? d : __half2float(dh);
      const float id = ds != 0.f ? __fdiv_rn(1.0f, ds) : 0.f;
      uint32_t w[8];
#pragma unroll
      for (int o = 0; o < 8; ++o) {
        if (KIND == Q_SYM4 || KIND == Q_ASYM4) {
          // nibble of element k: {0, 4, 1, 5, 2, 6, 3, 7}
          w[o] = nibbles([&](int n) {
            const float x = v.at(8 * o + 2 * (n & 3) + (n >> 2));
            return KIND == Q_SYM4 ? __fadd_rn(__fmul_rn(x, id), 8.5f) : __fadd_rn(__fmul_rn(__fsub_rn(x, mn), id), 0.5f);
          });
        } else {
          w[o] = 0;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const float sx = __fmul_rn(v.at(8 * o + k), id);
            const int q = KIND == Q_NF4 ? buckets.nearest(sx) : (nearest_sorted<8>(table, fabsf(sx)) | (sx < 0.f ? 8 : 0));
            w[o] |= (uint32_t)q << (4 * k);
          }
        }
        if (!valid) w[o] = 0;
      }
      // slot t of a row holds 8 bytes of each half: the lanes of a row trade so that each has two whole slots
      uint32_t got[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) got[i] = __shfl_xor_sync(0xffffffffu, half ? w[i] : w[4 + i], 1);
      uint8_t* to = dst + tile * 1024 + rr * 64 + half * 32;
      if (half == 0) store32(to, make_uint4(w[0], w[1], got[0], got[1]), make_uint4(w[2], w[3], got[2], got[3]), wide_dst);
      else store32(to, make_uint4(got[0], got[1], w[4], w[5]), make_uint4(got[2], got[3], w[6], w[7]), wide_dst);
      const int64_t si = (tile * 2 + half) * 16 + pair_row(rr);
      sc16[si] = valid ? __half_as_ushort(dh) : (uint16_t)0;
      if (KIND == Q_ASYM4) (sc16 + Np * (Kp / 64))[si] = valid ? __half_as_ushort(__float2half_rn(mn)) : (uint16_t)0;
    } else {
      float lo, hi;
      v.extremes(lo, hi);
      float amax = fmaxf(0.f, fmaxf(-lo, hi));
      if (KIND != Q_INT8) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
      const float d = __fdiv_rn(amax, KIND == Q_INT8 ? 127.0f : KIND == Q_E4M3 ? 448.0f : 57344.0f);
      const float id = d != 0.f ? __fdiv_rn(1.0f, d) : 0.f;
      uint32_t w[16];
#pragma unroll
      for (int o = 0; o < 16; ++o) {
        float sx[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) sx[k] = __fmul_rn(v.at(4 * o + k), id);
        if (KIND == Q_INT8) {
          w[o] = 0;
#pragma unroll
          for (int k = 0; k < 4; ++k)
            w[o] |= (uint32_t)(uint8_t)(int8_t)min(127, max(-128, __float2int_rn(sx[k]))) << (8 * k);
        } else {
          constexpr auto kFp8 = KIND == Q_E4M3 ? __NV_E4M3 : __NV_E5M2;
          w[o] = (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(sx[0], sx[1]), __NV_SATFINITE, kFp8) |
                 (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(sx[2], sx[3]), __NV_SATFINITE, kFp8) << 16;
        }
        if (!valid) w[o] = 0;
      }
      uint8_t* to = dst + (tile * 2 + half) * 1024 + rr * 64;
#pragma unroll
      for (int i = 0; i < 2; ++i)
        store32(to + 32 * i, make_uint4(w[8 * i], w[8 * i + 1], w[8 * i + 2], w[8 * i + 3]),
                make_uint4(w[8 * i + 4], w[8 * i + 5], w[8 * i + 6], w[8 * i + 7]), wide_dst);
      if (KIND == Q_INT8) {
        sc16[(tile * 2 + half) * 16 + pair_row(rr)] = valid ? __half_as_ushort(__float2half_rn(d)) : (uint16_t)0;
      } else if (half == 0) {
        reinterpret_cast<float*>(planes)[tile * 16 + pair_row(rr)] = valid ? d : 0.f;
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------
// tile layout -> dense [rows, cols] (row-major, leading dimension ld).  A warp takes a tile of 16 rows x 128 k, a lane two
// 16-byte slots of one row (four in the 8-bit formats), so that addresses and scales are worked out once per 64 weights:
// 11008 x 4096 sym_int4 to fp16 39 us with a thread per 8 weights, 27 us now.
// ------------------------------------------------------------------------------------------------
// `wide`: the bytes that every run's address is a multiple of, 32, 16 or less.  With 16 bytes a store a warp leaves half of each
// sector it touches to the next one: 11008 x 4096 sym_int4 to fp32 131 us, 48 with whole sectors, to
// fp16 30 and 27.
template <typename T>
__device__ __forceinline__ void store_run16(T* dst, const float (&v)[16], int wide) {
  __align__(32) T o[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) o[k] = DT<T>::from_f(v[k]);
  const uint4* q = reinterpret_cast<const uint4*>(o);
  if (wide == 32) {
#pragma unroll
    for (int i = 0; i < (int)sizeof(T); i += 2)
      asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(reinterpret_cast<uint4*>(dst) + i), "r"(q[i].x),
                   "r"(q[i].y), "r"(q[i].z), "r"(q[i].w), "r"(q[i + 1].x), "r"(q[i + 1].y), "r"(q[i + 1].z), "r"(q[i + 1].w)
                   : "memory");
  } else if (wide == 16) {
#pragma unroll
    for (int i = 0; i < (int)sizeof(T); ++i) reinterpret_cast<uint4*>(dst)[i] = q[i];
  } else {
#pragma unroll
    for (int k = 0; k < 16; ++k) dst[k] = o[k];
  }
}

template <typename T>
__global__ void __launch_bounds__(256) dequant_tiled_kernel(const uint8_t* __restrict__ w, T* __restrict__ out, int64_t rows,
                                                            int64_t cols, int64_t ld, int wf,
                                                            const float* __restrict__ lut, int wide) {
  __shared__ float table[16];
  if (wf == WF_LUT4) {
    if (threadIdx.x < 16) table[threadIdx.x] = lut[threadIdx.x];
    __syncthreads();
  }
  const int lane = threadIdx.x & 31, rr = lane >> 1, half = lane & 1;
  const int64_t Np = ceil_to_i64(rows, 16), Kp = ceil_to_i64(cols, 128);
  const int64_t kt = Kp / 128, tiles = Np / 16 * kt;
  const bool k4 = wf == WF_SYM_INT4 || wf == WF_ASYM_INT4 || wf == WF_LUT4;
  const uint8_t* planes = w + (k4 ? Np * Kp / 2 : Np * Kp);
  const uint16_t* sc16 = reinterpret_cast<const uint16_t*>(planes);
  for (int64_t tile = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); tile < tiles;
       tile += (int64_t)gridDim.x * (blockDim.x >> 5)) {
    const int64_t r = tile / kt * 16 + rr, kb = tile % kt * 128;
    if (r >= rows) continue;
    T* row = out + r * ld + kb;
    if (k4) {
      const uint4* p = reinterpret_cast<const uint4*>(w + tile * 1024 + rr * 64 + half * 32);
      const uint4 q[2] = {__ldg(p), __ldg(p + 1)};
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        if (kb + g * 64 >= cols) break;
        const int64_t si = (tile * 2 + g) * 16 + pair_row(rr);
        const float d = __half2float(__ushort_as_half(sc16[si]));
        const float mn = wf == WF_ASYM_INT4 ? __half2float(__ushort_as_half((sc16 + Np * (Kp / 64))[si])) : 0.f;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const uint32_t word[2] = {g == 0 ? q[t].x : q[t].z, g == 0 ? q[t].y : q[t].w};
          float v[16];
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            const uint32_t x = word[k >> 3];
            const int j = k & 7;
            if (wf == WF_LUT4) v[k] = table[(x >> (4 * j)) & 0xF] * d;
            else {
              const int c = (x >> (4 * ((j >> 1) + 4 * (j & 1)))) & 0xF;
              v[k] = wf == WF_SYM_INT4 ? (float)(c - 8) * d : (float)c * d + mn;
            }
          }
          store_run16(row + g * 64 + (2 * half + t) * 16, v, wide);
        }
      }
    } else {
      if (kb + half * 64 >= cols) continue;
      const uint4* p = reinterpret_cast<const uint4*>(w + (tile * 2 + half) * 1024 + rr * 64);
      float d;
      if (wf == WF_INT8) d = __half2float(__ushort_as_half(sc16[(tile * 2 + half) * 16 + pair_row(rr)]));
      else d = reinterpret_cast<const float*>(planes)[tile * 16 + pair_row(rr)];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const uint4 q = __ldg(p + t);
        const uint32_t word[4] = {q.x, q.y, q.z, q.w};
        float v[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const uint8_t c = (uint8_t)(word[k >> 2] >> (8 * (k & 3)));
          float x;
          if (wf == WF_INT8) x = (float)(int8_t)c;
          else {
            __half_raw h = __nv_cvt_fp8_to_halfraw(c, wf == WF_FP8_E4M3 ? __NV_E4M3 : __NV_E5M2);
            x = __half2float(*reinterpret_cast<__half*>(&h));
          }
          v[k] = x * d;
        }
        store_run16(row + half * 64 + t * 16, v, wide);
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------
// canonical block decoders (one thread per block) for the qtypes without a tile layout, and for embedding rows
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ float ldh(const uint8_t* p) {
  uint16_t h = (uint16_t)p[0] | ((uint16_t)p[1] << 8);
  return __half2float(__ushort_as_half(h));
}
__device__ __forceinline__ float minifloat(int c, int mbits, int bias) {
  int e = c >> mbits, m = c & ((1 << mbits) - 1);
  if (e == 0) return ldexpf((float)m, 1 - bias - mbits);
  return ldexpf((float)((1 << mbits) + m), e - bias - mbits);
}
__device__ __forceinline__ void scale_min_k4(int j, const uint8_t* q, int* d, int* m) {
  if (j < 4) { *d = q[j] & 63; *m = q[j + 4] & 63; }
  else { *d = (q[j + 4] & 0xF) | ((q[j - 4] >> 6) << 4); *m = (q[j + 4] >> 4) | ((q[j] >> 6) << 4); }
}

// qtype ids as in quant/qtypes.py
template <typename T>
__device__ void decode_block(const uint8_t* y, T* x, int qtype) {
  auto put = [&](int i, float v) { x[i] = DT<T>::from_f(v); };
  switch (qtype) {
    case 2: {  // sym_int4
      float d = ldh(y);
      for (int j = 0; j < 32; j++) { put(j, (float)((y[2 + j] & 0xF) - 8) * d); put(j + 32, (float)((y[2 + j] >> 4) - 8) * d); }
    } break;
    case 3: case 34: {  // asym_int4
      float d = ldh(y), m = ldh(y + 2);
      for (int j = 0; j < 32; j++) { put(j, (float)(y[4 + j] & 0xF) * d + m); put(j + 32, (float)(y[4 + j] >> 4) * d + m); }
    } break;
    case 6: {  // sym_int5
      float d = ldh(y);
      uint32_t qh = y[2] | (y[3] << 8) | (y[4] << 16) | ((uint32_t)y[5] << 24);
      for (int j = 0; j < 16; j++) {
        int a = (y[6 + j] & 0xF) | (((qh >> j) & 1) << 4), b = (y[6 + j] >> 4) | (((qh >> (j + 16)) & 1) << 4);
        put(j, (float)(a - 16) * d); put(j + 16, (float)(b - 16) * d);
      }
    } break;
    case 7: {  // asym_int5
      float d = ldh(y), m = ldh(y + 2);
      uint32_t qh = y[4] | (y[5] << 8) | (y[6] << 16) | ((uint32_t)y[7] << 24);
      for (int j = 0; j < 16; j++) {
        int a = (y[8 + j] & 0xF) | (((qh >> j) & 1) << 4), b = (y[8 + j] >> 4) | (((qh >> (j + 16)) & 1) << 4);
        put(j, (float)a * d + m); put(j + 16, (float)b * d + m);
      }
    } break;
    case 8: {  // sym_int8
      float d = ldh(y);
      for (int i = 0; i < 64; i++) put(i, (float)(int8_t)y[2 + i] * d);
    } break;
    case 10: case 16: {  // nf4 / fp4
      float d = ldh(y);
      for (int j = 0; j < 32; j++) {
        int a = y[2 + j] & 0xF, b = y[2 + j] >> 4;
        float va = qtype == 10 ? c_nf4[a] : ((a & 8) ? -c_fp4[a & 7] : c_fp4[a & 7]);
        float vb = qtype == 10 ? c_nf4[b] : ((b & 8) ? -c_fp4[b & 7] : c_fp4[b & 7]);
        put(j, va * d); put(j + 32, vb * d);
      }
    } break;
    case 11: {  // nf3
      float d = ldh(y);
      for (int i = 0; i < 64; i++) {
        int bit = 3 * i;
        uint32_t v = y[2 + (bit >> 3)];
        if ((bit >> 3) + 1 < 24) v |= (uint32_t)y[2 + (bit >> 3) + 1] << 8;
        put(i, c_nf3[(v >> (bit & 7)) & 7] * d);
      }
    } break;
    case 29: case 30: {  // fp6 (e3m2)
      float d = ldh(y);
      for (int g = 0; g < 16; g++) {
        uint32_t pack = y[2 + 3 * g] | (y[2 + 3 * g + 1] << 8) | (y[2 + 3 * g + 2] << 16);
        for (int k = 0; k < 4; k++) {
          uint32_t c = (pack >> (6 * k)) & 63;
          float m = minifloat(c & 31, 2, 3) * d;
          put(4 * g + k, (c & 32) ? -m : m);
        }
      }
    } break;
    case 15: case 19: {  // fp8 e4m3 / e5m2, 128-block with fp32 scale
      float d;
      memcpy(&d, y, 4);
      for (int i = 0; i < 128; i++) {
        int c = y[4 + i] & 0x7f;
        float m = (qtype == 15 ? (c < 127 ? minifloat(c, 3, 7) : 0.f) : (c < 124 ? minifloat(c, 2, 15) : 0.f)) * d;
        put(i, (y[4 + i] & 0x80) ? -m : m);
      }
    } break;
    case 27: {  // q4_k
      float d = ldh(y), dmin = ldh(y + 2);
      const uint8_t* sc = y + 4;
      const uint8_t* q = y + 16;
      int is = 0;
      for (int j = 0; j < 256; j += 64) {
        int s, m;
        scale_min_k4(is, sc, &s, &m);
        float d1 = d * s, m1 = dmin * m;
        scale_min_k4(is + 1, sc, &s, &m);
        float d2 = d * s, m2 = dmin * m;
        for (int l = 0; l < 32; l++) { put(j + l, d1 * (q[l] & 0xF) - m1); put(j + 32 + l, d2 * (q[l] >> 4) - m2); }
        q += 32; is += 2;
      }
    } break;
    case 28: {  // q5_k
      float d = ldh(y), dmin = ldh(y + 2);
      const uint8_t* sc = y + 4;
      const uint8_t* qh = y + 16;
      const uint8_t* ql = y + 48;
      int is = 0;
      uint8_t u1 = 1, u2 = 2;
      for (int j = 0; j < 256; j += 64) {
        int s, m;
        scale_min_k4(is, sc, &s, &m);
        float d1 = d * s, m1 = dmin * m;
        scale_min_k4(is + 1, sc, &s, &m);
        float d2 = d * s, m2 = dmin * m;
        for (int l = 0; l < 32; l++) {
          put(j + l, d1 * ((ql[l] & 0xF) + ((qh[l] & u1) ? 16 : 0)) - m1);
          put(j + 32 + l, d2 * ((ql[l] >> 4) + ((qh[l] & u2) ? 16 : 0)) - m2);
        }
        ql += 32; is += 2; u1 <<= 2; u2 <<= 2;
      }
    } break;
    case 26: {  // q6_k
      const uint8_t* ql = y;
      const uint8_t* qh = y + 128;
      const int8_t* sc = reinterpret_cast<const int8_t*>(y + 192);
      float d = ldh(y + 208);
      int o = 0;
      for (int n = 0; n < 256; n += 128) {
        for (int l = 0; l < 32; l++) {
          int is = l / 16;
          int q1 = (int)((ql[l] & 0xF) | (((qh[l] >> 0) & 3) << 4)) - 32;
          int q2 = (int)((ql[l + 32] & 0xF) | (((qh[l] >> 2) & 3) << 4)) - 32;
          int q3 = (int)((ql[l] >> 4) | (((qh[l] >> 4) & 3) << 4)) - 32;
          int q4 = (int)((ql[l + 32] >> 4) | (((qh[l] >> 6) & 3) << 4)) - 32;
          put(o + l, d * sc[is] * q1); put(o + l + 32, d * sc[is + 2] * q2);
          put(o + l + 64, d * sc[is + 4] * q3); put(o + l + 96, d * sc[is + 6] * q4);
        }
        o += 128; ql += 64; qh += 32; sc += 8;
      }
    } break;
    case 23: {  // q2_k
      const uint8_t* sc = y;
      const uint8_t* q = y + 16;
      float d = ldh(y + 80), dmin = ldh(y + 82);
      int is = 0, o = 0;
      for (int n = 0; n < 256; n += 128) {
        int shift = 0;
        for (int j = 0; j < 4; j++) {
          uint8_t s = sc[is++];
          float dl = d * (s & 0xF), ml = dmin * (s >> 4);
          for (int l = 0; l < 16; l++) put(o++, dl * ((q[l] >> shift) & 3) - ml);
          s = sc[is++];
          dl = d * (s & 0xF); ml = dmin * (s >> 4);
          for (int l = 0; l < 16; l++) put(o++, dl * ((q[l + 16] >> shift) & 3) - ml);
          shift += 2;
        }
        q += 32;
      }
    } break;
    default: break;
  }
}

template <typename T>
__global__ void dequant_blocks_kernel(const uint8_t* __restrict__ src, T* __restrict__ dst, int64_t nblocks, int qk,
                                      int ts, int qtype) {
  for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < nblocks; b += (int64_t)gridDim.x * blockDim.x)
    decode_block<T>(src + b * ts, dst + b * qk, qtype);
}

// rows of a canonical [vocab, dim] table selected by ids -> out [n, dim]
template <typename T>
__global__ void dequant_rows_kernel(const int64_t* __restrict__ ids, const uint8_t* __restrict__ table,
                                    T* __restrict__ out, int64_t n, int dim, int qk, int ts, int qtype) {
  const int bpr = dim / qk;
  const int64_t total = n * bpr;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = i / bpr;
    const int b = (int)(i % bpr);
    decode_block<T>(table + (ids[row] * bpr + b) * ts, out + row * dim + (int64_t)b * qk, qtype);
  }
}

template <typename F>
int by_dtype3(int dtype, F&& f) {
  if (dtype == DT_F16) return (int)f((__half*)nullptr);
  if (dtype == DT_BF16) return (int)f((__nv_bfloat16*)nullptr);
  if (dtype == DT_F32) return (int)f((float*)nullptr);
  return (int)cudaErrorInvalidValue;
}

}  // namespace

// Dense [rows, cols] (leading dimension ld, dtype) -> device tile layout of weight family `wf` (plus `lut_kind`
// for WF_LUT4: 0 = nf4, 1 = fp4).  `dst` holds ipex_device_bytes(rows, cols, qtype) bytes, all of which are written.
IPEX_API int ipex_quantize_to_tiles(const void* src, void* dst, int64_t rows, int64_t cols, int64_t ld, int wf,
                                    int lut_kind, int dtype, void* stream) {
  if (rows < 1 || cols < 1) return (int)cudaSuccess;
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t work = ceil_to_i64(rows, 16) / 16 * (ceil_to_i64(cols, 128) / 128);
  const int blocks = (int)((work + 7) / 8 < 148 * 64 ? (work + 7) / 8 : 148 * 64);    // a tile to a warp: no last round
  return by_dtype3(dtype, [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    const T* p = (const T*)src;
    uint8_t* d = (uint8_t*)dst;
    const uintptr_t at = reinterpret_cast<uintptr_t>(src) | (uintptr_t)(ld * sizeof(T));
    const int wide = (at & 31) == 0 ? 32 : (at & 15) == 0 ? 16 : 1;
    const bool whole = (reinterpret_cast<uintptr_t>(dst) & 31) == 0;
    switch (wf) {
      case WF_SYM_INT4: quantize_kernel<T, Q_SYM4><<<blocks, 256, 0, s>>>(p, d, rows, cols, ld, wide, whole); break;
      case WF_ASYM_INT4: quantize_kernel<T, Q_ASYM4><<<blocks, 256, 0, s>>>(p, d, rows, cols, ld, wide, whole); break;
      case WF_LUT4:
        if (lut_kind == 0) quantize_kernel<T, Q_NF4><<<blocks, 256, 0, s>>>(p, d, rows, cols, ld, wide, whole);
        else quantize_kernel<T, Q_FP4><<<blocks, 256, 0, s>>>(p, d, rows, cols, ld, wide, whole);
        break;
      case WF_FP8_E4M3: quantize_kernel<T, Q_E4M3><<<blocks, 256, 0, s>>>(p, d, rows, cols, ld, wide, whole); break;
      case WF_FP8_E5M2: quantize_kernel<T, Q_E5M2><<<blocks, 256, 0, s>>>(p, d, rows, cols, ld, wide, whole); break;
      case WF_INT8: quantize_kernel<T, Q_INT8><<<blocks, 256, 0, s>>>(p, d, rows, cols, ld, wide, whole); break;
      default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
  });
}

IPEX_API int ipex_dequantize_tiles(const void* w, void* out, int64_t rows, int64_t cols, int64_t ld, int wf,
                                   const float* lut, int dtype, void* stream) {
  if (rows < 1 || cols < 1) return (int)cudaSuccess;
  const int64_t work = ceil_to_i64(rows, 16) / 16 * (ceil_to_i64(cols, 128) / 128);
  const int blocks = (int)((work + 7) / 8 < 148 * 64 ? (work + 7) / 8 : 148 * 64);
  return by_dtype3(dtype, [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    const uintptr_t at = reinterpret_cast<uintptr_t>(out) | (uintptr_t)(ld * sizeof(T));
    const int wide = (at & 31) == 0 ? 32 : (at & 15) == 0 ? 16 : 1;
    dequant_tiled_kernel<T><<<blocks, 256, 0, (cudaStream_t)stream>>>((const uint8_t*)w, (T*)out, rows, cols, ld, wf, lut,
                                                                      wide);
    return cudaGetLastError();
  });
}

IPEX_API int ipex_dequantize_blocks(const void* src, void* dst, int64_t nblocks, int qk, int ts, int qtype, int dtype,
                                    void* stream) {
  int blocks = (int)((nblocks + 127) / 128);
  if (blocks > 148 * 32) blocks = 148 * 32;
  if (blocks < 1) blocks = 1;
  return by_dtype3(dtype, [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    dequant_blocks_kernel<T><<<blocks, 128, 0, (cudaStream_t)stream>>>((const uint8_t*)src, (T*)dst, nblocks, qk, ts,
                                                                       qtype);
    return cudaGetLastError();
  });
}

IPEX_API int ipex_dequantize_rows(const void* ids, const void* table, void* out, int64_t n, int dim, int qk, int ts,
                                  int qtype, int dtype, void* stream) {
  const int64_t work = n * (dim / qk);
  int blocks = (int)((work + 127) / 128);
  if (blocks > 148 * 32) blocks = 148 * 32;
  if (blocks < 1) blocks = 1;
  return by_dtype3(dtype, [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    dequant_rows_kernel<T><<<blocks, 128, 0, (cudaStream_t)stream>>>((const int64_t*)ids, (const uint8_t*)table,
                                                                     (T*)out, n, dim, qk, ts, qtype);
    return cudaGetLastError();
  });
}
