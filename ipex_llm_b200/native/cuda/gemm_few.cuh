// Products of 1 to 64 token rows with packed weights (decode steps of a batch, drafted continuations): those with up to 24 rows
// (16 with minima), and more where two of them make a token, by this kernel, the others by gemm_few_tcgen05.cuh:
//     out[M, N] = x[M, K] . W[N, K]^T  (+ bias) (+ residual)   or   act(gate) * up  for interleaved gate/up rows
//
// What bounds it: with so few rows the weights' codes have to be taken apart as fast as they arrive, some nine instructions
// for eight codes, and each is used for a few columns only.  So a warp keeps everything to itself: it reads the packed codes
// of 32 weight rows from a ring in shared memory, makes them 16-bit operands in the registers of the very lane that the
// matrix instruction wants them in (the packed layout was made for that: a lane's 16 bytes are consecutive k of one row), and
// multiplies them by token fragments that it loads once for its 32 rows.  No expanded weight is written anywhere, and no other
// warp is waited for before the sums are added up.
//
// The codes themselves are multiplied (small integers, fp8 values: exact in 16 bits; a code book's values are rounded to 16
// bits, but not their product with the scale) and the sums of a scale group are scaled in 32 bits.  A minimum takes part as its
// product with the sum of the group's tokens (more than 32 columns: expanded and scaled in 16 bits).
//
// A CTA holds a tile of 128 weight rows over a share of k, two CTAs fit an SM (one loads or adds up while the other
// multiplies), and a cluster of up to eight CTAs shares the k of a tile: the parts meet through distributed shared memory, in
// a fixed order.  The weights' part of the ring's first stages is asked for before the kernel in front has ended; later the warps
// take turns at filling it.
//
// Measured (us per launch between dependent launches, weights from memory; a tcgen05 form that wrote expanded weights to shared
// memory -> this one): int4, 16 rows, 12288 x 4096 19.4 -> 14.6, 22016 x 4096 32.5 -> 22.1, 32000 x 4096 39.7 -> 23.6.  ncu, 32000
// x 4096 at 8 rows: half of the issue slots are used, 340 instructions for 4096 weights of which 150 take codes apart; from 24
// rows on the matrix pipe (one m16n8k16 in 8 clocks) and the sums cost as much again: gemm_few_tcgen05.cuh.
//
// x may hold two rows per token (2m: the value rounded to 16 bits, 2m + 1: what that left over); their products are added in
// 32 bits at the end.
// Every wait is bounded (error code 22).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common/utils.cuh"
#include "lowbit_expand.cuh"
#include "tcgen05_common.cuh"

namespace few {

using namespace tc5;

constexpr int kBM = 128;             // weight rows of a tile
constexpr int kWarps = 8, kThreads = kWarps * 32;
constexpr int kCtasPerSM = 2;
constexpr int kSmemMax = 113 * 1024;   // of a CTA, so that two fit an SM
constexpr int kMaxSplit = 8;

struct Args {
  const uint8_t* w;
  const void* x;
  int64_t ldx;
  int K;
  const float* lut;
  void* out;
  const void* bias;
  const void* residual;
  int64_t ldo, ldr;
  int M, N;            // M: tokens (rows of out)
  int chunks;          // of 128 k
  int rows;            // of x
  int split;           // CTAs that share a tile's k
  int act;
  int pairs;           // two rows of x per token
  int* err;
};

// A warp has 32 weight rows and NT times eight columns of tokens.  Up to 32 columns (WN = 1) two warps share the rows' k; more
// columns are split between two warps, which take the same codes apart (all of them in one warp leave an SM eight warps of
// 255 registers: no faster).
template <int WF, int NT, int WN> struct Cfg {
  static constexpr bool k4 = WF == WF_SYM_INT4 || WF == WF_ASYM_INT4 || WF == WF_LUT4;
  static constexpr bool codes = WF != WF_ASYM_INT4 || WN == 1;         // scales applied to sums
  static constexpr bool minima = WF == WF_ASYM_INT4 && codes;
  static constexpr bool half_scale = k4 || WF == WF_INT8;              // fp16 per 64 k, else fp32 per 128
  static constexpr int kCols = 8 * NT * WN;
  static constexpr int MT = 2;                                         // 16-row tiles of a warp
  static constexpr int WM = kBM / (16 * MT), WK = kWarps / WM / WN;    // warps along the rows and along k
  static constexpr int kCodes = k4 ? 1024 : 2048, kScales = 64;        // bytes of a 16-row tile's 128 k
  static constexpr int kPlanes = WF == WF_ASYM_INT4 ? 2 : 1;           // scales (and minima)
  // a stage: codes [8 row tiles][WK chunks], tokens [2 WK][columns][64 k] with TMA's 128-byte swizzle, scales
  static constexpr int kXAt = 8 * WK * kCodes;
  static constexpr int kPiece = kCols * 128;
  static constexpr int kScaleAt = kXAt + 2 * WK * kPiece;
  static constexpr int kBytes = kScaleAt + kPlanes * 8 * WK * kScales;
  static constexpr int kStageBytes = (kBytes + 1023) / 1024 * 1024;
  static constexpr int kBook = WF == WF_LUT4 ? 256 * 32 * 4 : 0;       // pairs of values by the byte, a copy per lane
  static constexpr int kTail = 256 + kBook;                            // barriers
  static constexpr int kRedPitch = kBM + 4;
  static constexpr int kRedBytes = WK * kCols * kRedPitch * 4;
  static constexpr int kStagesFit = (kSmemMax - 1024 - kTail) / kStageBytes;
  static constexpr int kStages = kStagesFit > 6 ? 6 : kStagesFit;
  static constexpr int kSmem = 1024 + kStages * kStageBytes + kTail;
  static_assert(kStages >= 2 && kRedBytes <= kStages * kStageBytes, "ring");
};

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* tm, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ float ld_rank(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
template <typename T>
__device__ __forceinline__ void mma16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (std::is_same<T, __half>::value)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The codes of 8 consecutive weights of a row as 16-bit values (not CODES: the weights), in pairs of consecutive k.
template <typename T, int WF, bool CODES>
__device__ __forceinline__ uint4 codes4(uint32_t w, const uint32_t* book, const Scale<T>& sc) {
  using V = V2<T>;
  constexpr float zero = WF == WF_SYM_INT4 ? 8.f : 0.f;
  if constexpr (WF == WF_LUT4) {       // `book` is this lane's copy
    uint4 v = make_uint4(book[(w & 0xFF) * 32], book[((w >> 8) & 0xFF) * 32], book[((w >> 16) & 0xFF) * 32], book[(w >> 24) * 32]);
    if constexpr (!CODES) {
      v.x = V::raw(__hmul2(V::bits(v.x), sc.d));
      v.y = V::raw(__hmul2(V::bits(v.y), sc.d));
      v.z = V::raw(__hmul2(V::bits(v.z), sc.d));
      v.w = V::raw(__hmul2(V::bits(v.w), sc.d));
    }
    return v;
  } else if constexpr (!CODES) {
    return expand4<T, WF>(w, sc, nullptr);
  } else if constexpr (std::is_same<T, __half>::value) {
    // 1024 + q, and 1024 + 16 q for the nibbles above: a shift for every other pair only (integers placed in the last bits of a
    // number of known exponent: Kim et al., "Who Says Elephants Can't Run", 2022)
    const uint32_t u = w >> 8;
    const __half2 off = __float2half2_rn(1024.f + zero), sixteenth = __float2half2_rn(0.0625f),
                  off16 = __float2half2_rn(-64.f - zero);
    return make_uint4(V::raw(__hsub2(V::bits((w & 0x000F000Fu) | 0x64006400u), off)),
                      V::raw(__hfma2(V::bits((w & 0x00F000F0u) | 0x64006400u), sixteenth, off16)),
                      V::raw(__hsub2(V::bits((u & 0x000F000Fu) | 0x64006400u), off)),
                      V::raw(__hfma2(V::bits((u & 0x00F000F0u) | 0x64006400u), sixteenth, off16)));
  } else {
    const typename V::type off = V::splat(V::kMagicBase + zero);
    uint32_t r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = V::raw(__hsub2(V::bits(((w >> (4 * i)) & 0x000F000Fu) | V::kMagic), off));
    return make_uint4(r[0], r[1], r[2], r[3]);
  }
}
// fp8: the byte at the top of the 16-bit lane, its magnitude shifted into the wider exponent field: the value times a power of
// two.  In fp16 the scale takes it back; in bf16 (2^-120: the products would leave the range of the sums) the value does.
template <typename T, int WF>
__device__ __forceinline__ uint4 codes8(uint32_t w0, uint32_t w1) {
  using V = V2<T>;
  uint32_t r[4];
  const uint32_t ws[2] = {w0, w1};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t w = ws[i >> 1];
    if constexpr (WF == WF_INT8) {
      const uint32_t t = __byte_perm(w, 0x64646464u, (i & 1) ? 0x4342 : 0x4140) ^ 0x00800080u;
      const __half2 q = __hsub2(V2<__half>::bits(t), __float2half2_rn(1152.f));
      if constexpr (std::is_same<T, __half>::value) {
        r[i] = V::raw(q);
      } else {
        const float2 f = __half22float2(q);
        r[i] = V::raw(__floats2bfloat162_rn(f.x, f.y));
      }
    } else {
      constexpr int sh = Fp8Place<T, WF>::sh;
      const uint32_t t = __byte_perm(w, 0u, (i & 1) ? 0x3424 : 0x1404);
      r[i] = sh == 0 ? t : (t & 0x80008000u) | ((t >> sh) & (0x7F007F00u >> sh));
      if constexpr (std::is_same<T, __nv_bfloat16>::value)
        r[i] = V::raw(__hmul2(V::bits(r[i]), V::splat(Fp8Place<T, WF>::mul)));
    }
  }
  return make_uint4(r[0], r[1], r[2], r[3]);
}

// One chunk of 128 k: acc += scale * (codes . tokens) for this warp's 16-row tiles.  `ct`: its first tile's codes (tiles WK
// chunks apart), `st`: their scales, `xs`: its chunk's tokens.
template <typename T, int WF, int NT, int WN>
__device__ __forceinline__ void chunk_mma(const uint8_t* ct, const uint8_t* st, const uint8_t* xs, const uint32_t* book,
                                          float (&acc)[Cfg<WF, NT, WN>::MT][NT][4]) {
  using C = Cfg<WF, NT, WN>;
  using V = V2<T>;
  constexpr int MT = C::MT;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  uint4 qa[MT], qb[MT];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (!C::k4 || h == 0) {
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const uint8_t* p = ct + m * C::WK * C::kCodes + (C::k4 ? 0 : h * 1024) + g * 64 + t * 16;
        qa[m] = *reinterpret_cast<const uint4*>(p);
        qb[m] = *reinterpret_cast<const uint4*>(p + 512);
      }
    }
    uint4 b[NT][2];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int o = 0; o < 2; ++o) b[n][o] = *reinterpret_cast<const uint4*>(xs + h * C::kPiece + n * 1024 + g * 128 + (((2 * t + o) ^ g) << 4));
    float sx[NT][4];                                // sums of the tokens' k, in the columns that this lane's sums are in
    if constexpr (C::minima) {
      constexpr uint32_t one = std::is_same<T, __half>::value ? 0x3C003C00u : 0x3F803F80u;
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        sx[n][0] = sx[n][1] = sx[n][2] = sx[n][3] = 0.f;
#pragma unroll
        for (int o = 0; o < 2; ++o) {
          mma16<T>(sx[n], one, one, one, one, b[n][o].x, b[n][o].y);
          mma16<T>(sx[n], one, one, one, one, b[n][o].z, b[n][o].w);
        }
      }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      float d0 = 1.f, d1 = 1.f, m0 = 0.f, m1 = 0.f;     // of rows g and g + 8
      Scale<T> s0, s1;
      const uint8_t* sp = st + m * C::WK * C::kScales;
      if constexpr (C::half_scale) {
        const uint32_t raw = *reinterpret_cast<const uint32_t*>(sp + h * 32 + 4 * g);
        const float2 d = __half22float2(*reinterpret_cast<const __half2*>(&raw));
        if constexpr (C::codes) {
          d0 = d.x;
          d1 = d.y;
        }
        if constexpr (WF == WF_ASYM_INT4) {
          const uint32_t rawm = *reinterpret_cast<const uint32_t*>(sp + 8 * C::WK * C::kScales + h * 32 + 4 * g);
          const float2 mn = __half22float2(*reinterpret_cast<const __half2*>(&rawm));
          if constexpr (C::minima) {
            m0 = mn.x;
            m1 = mn.y;
          } else {
            s0.d = V::splat(d.x); s0.m = V::splat(mn.x);
            s1.d = V::splat(d.y); s1.m = V::splat(mn.y);
          }
        }
      } else {
        const float2 d = *reinterpret_cast<const float2*>(sp + 8 * g);
        constexpr float k = std::is_same<T, __half>::value ? Fp8Place<__half, WF>::mul * Fp8Place<__half, WF>::pre : 1.f;
        d0 = d.x * k;
        d1 = d.y * k;
      }
      float s[NT][4];
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) s[n][i] = C::codes ? 0.f : acc[m][n][i];
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        uint4 ra, rb;
        if constexpr (C::k4) {
          // 16 bytes = [group 0: k 16t..16t+7 | 16t+8..16t+15 | group 1: same]
          ra = codes4<T, WF, C::codes>(h == 0 ? (o == 0 ? qa[m].x : qa[m].y) : (o == 0 ? qa[m].z : qa[m].w), book, s0);
          rb = codes4<T, WF, C::codes>(h == 0 ? (o == 0 ? qb[m].x : qb[m].y) : (o == 0 ? qb[m].z : qb[m].w), book, s1);
        } else {
          ra = o == 0 ? codes8<T, WF>(qa[m].x, qa[m].y) : codes8<T, WF>(qa[m].z, qa[m].w);
          rb = o == 0 ? codes8<T, WF>(qb[m].x, qb[m].y) : codes8<T, WF>(qb[m].z, qb[m].w);
        }
        // k of a lane's operands: any four of the 16 per instruction, as long as weights and tokens take the same
#pragma unroll
        for (int n = 0; n < NT; ++n) mma16<T>(s[n], ra.x, rb.x, ra.y, rb.y, b[n][o].x, b[n][o].y);
#pragma unroll
        for (int n = 0; n < NT; ++n) mma16<T>(s[n], ra.z, rb.z, ra.w, rb.w, b[n][o].z, b[n][o].w);
      }
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc[m][n][i] = C::codes ? fmaf(i < 2 ? d0 : d1, s[n][i], acc[m][n][i]) : s[n][i];
          if constexpr (C::minima) acc[m][n][i] = fmaf(i < 2 ? m0 : m1, sx[n][i & 1], acc[m][n][i]);
        }
    }
  }
}

// The code book: a pair of values by the byte, a copy for each lane, so that no two meet in a bank (eight copies: 22016 x 4096 at
// 64 rows 41 -> 51 us).
template <typename T> __device__ __forceinline__ void fill_book(uint32_t* book, const float* lut) {
  for (int i = threadIdx.x; i < 256 * 8; i += kThreads) {
    const int e = i >> 3;
    const T lo = from_float<T>(lut[e & 15]), hi = from_float<T>(lut[e >> 4]);
    const uint32_t v = (uint32_t)(*reinterpret_cast<const uint16_t*>(&lo)) |
                       ((uint32_t)(*reinterpret_cast<const uint16_t*>(&hi)) << 16);
    reinterpret_cast<uint4*>(book)[i] = make_uint4(v, v, v, v);
  }
}

// Sums that are no number, of this CTA's k0 .. k1 of a format with minima, once more from the weights themselves: beside an
// infinite token the codes' part and the minimum's are infinities of any signs, or a zero code's product with it, where the
// weight's own product is an infinity of the weight's sign.  Only rows with such a token (or without a number) come here.
template <typename T, int PARTS, int COLS>
__device__ __noinline__ void add_up_again(const uint8_t* w, const T* x, int64_t ldx, int rows, int N, int chunks, float* red,
                                          int tile, int k0, int k1) {
  constexpr int kPitch = kBM + 4;
  const int row = threadIdx.x % kBM, n = tile * kBM + row;
  if (n >= N) return;
  const int64_t row_tiles = ceil_to_i64(N, 16) / 16;
  const uint8_t* scales = w + row_tiles * chunks * 1024;
  for (int c = threadIdx.x / kBM; c < rows; c += kThreads / kBM) {
    float* sum = red + c * kPitch + row;
    bool number = true;
    for (int p = 0; p < PARTS; ++p) number = number && sum[p * COLS * kPitch] == sum[p * COLS * kPitch];
    if (number) continue;
    float again = 0.f;
    for (int k = k0; k < k1; ++k) {
      const int64_t chunk = (n >> 4) * (int64_t)chunks + (k >> 7);
      const int h = (k >> 6) & 1, e = k & 7;
      const uint32_t word = *reinterpret_cast<const uint32_t*>(w + chunk * 1024 + (n & 15) * 64 + ((k & 63) >> 4) * 16 + h * 8 +
                                                               ((k >> 3) & 1) * 4);
      const __half* d = reinterpret_cast<const __half*>(scales + chunk * 64) + h * 16 + pair_row(n & 15);
      const float m = __half2float(d[row_tiles * chunks * 32]);
      const float code = (float)((word >> (4 * ((e >> 1) + 4 * (e & 1)))) & 15);
      again = fmaf(fmaf(__half2float(*d), code, m), to_float(x[c * ldx + k]), again);
    }
    for (int p = 0; p < PARTS; ++p) sum[p * COLS * kPitch] = p == 0 ? again : 0.f;
  }
}

// The parts of a tile, PARTS of them [COLS][rows] in `red` of every CTA that shares it: a warp adds up 32 rows of one token at a
// time, bias, residual or activation included.
template <typename T, int PARTS, int COLS>
__device__ __forceinline__ void add_parts(const Args& a, const float* red, int rank, int split, int tile, int warp, int lane) {
  constexpr int kPitch = kBM + 4;
  __syncthreads();
  if (split > 1) cluster_sync_all();
  {
    const T* res = reinterpret_cast<const T*>(a.residual);
    const T* bias = reinterpret_cast<const T*>(a.bias);
    T* out = reinterpret_cast<T*>(a.out);
    const uint32_t base = smem_u32(red);
    for (int item = rank * kWarps + warp; item < 4 * a.M; item += split * kWarps) {
      const int u = item & 3, m = item >> 2, n = tile * kBM + u * 32 + lane;
      if (tile * kBM + u * 32 >= a.N) continue;
      const int col = a.pairs ? 2 * m : m;
      const uint32_t off = (uint32_t)((col * kPitch + u * 32 + lane) * 4);
      float f = 0.f, v[kMaxSplit][PARTS], v2[kMaxSplit][PARTS];
#pragma unroll
      for (int q = 0; q < kMaxSplit; ++q) {
        if (q >= split) break;
        const uint32_t from = (split > 1 ? at_rank(base, q) : base) + off;
#pragma unroll
        for (int k = 0; k < PARTS; ++k) {
          v[q][k] = ld_rank(from + k * COLS * kPitch * 4);
          v2[q][k] = a.pairs ? ld_rank(from + (k * COLS + 1) * kPitch * 4) : 0.f;
        }
      }
#pragma unroll
      for (int q = 0; q < kMaxSplit; ++q) {
        if (q >= split) break;
#pragma unroll
        for (int k = 0; k < PARTS; ++k) f += v[q][k] + v2[q][k];
      }
      if (bias != nullptr && n < a.N) f += to_float(bias[n]);
      if (a.act != 0) {
        const float up = __shfl_down_sync(0xffffffffu, f, 16);
        const int no = (tile * kBM + u * 32) / 2 + lane;
        if (lane < 16 && no < a.N / 2) out[(int64_t)m * a.ldo + no] = from_float<T>(act_apply(f, a.act) * up);
      } else if (n < a.N) {
        if (res != nullptr) f += to_float(res[(int64_t)m * a.ldr + n]);
        out[(int64_t)m * a.ldo + n] = from_float<T>(f);
      }
    }
  }
  if (split > 1) cluster_sync_all();                // no CTA leaves while another may still read its part
}

template <typename T, int WF, int NT, int WN>
__global__ void __launch_bounds__(kThreads, kCtasPerSM)
kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_s, const __grid_constant__ CUtensorMap tm_x,
       const Args a) {
  using C = Cfg<WF, NT, WN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(ring + C::kStages * C::kStageBytes);
  uint64_t* empty = full + C::kStages;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(empty + C::kStages);
  uint32_t* book = reinterpret_cast<uint32_t*>(full) + 64;
  float* red = reinterpret_cast<float*>(ring);      // [WK][column][row], once the ring has been read

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int split = a.split, rank = blockIdx.x % split;
  const int tile = blockIdx.x / split;
  const int all = (a.chunks + C::WK - 1) / C::WK;   // stages of a tile; this CTA's: [st0, st0 + nst)
  const int st0 = all * rank / split, nst = all * (rank + 1) / split - st0;
  constexpr int S = C::kStages;

  auto load_weights = [&](int i, int slot) {        // a converged warp
    if (elect_one()) {
      uint8_t* to = ring + slot * C::kStageBytes;
      const int c = (st0 + i) * C::WK;
      mbar_expect_tx(&full[slot], C::kBytes);
      tma_load_3d(to, &tm_w, 0, c * (C::kCodes / 1024), tile * 8, &full[slot]);
      tma_load_3d(to + C::kScaleAt, &tm_s, c * (C::kScales / 8), tile * 8, 0, &full[slot]);
    }
  };
  auto load_tokens = [&](int i, int slot) {
    if (elect_one()) tma_load_3d(ring + slot * C::kStageBytes + C::kXAt, &tm_x, 0, 0, (st0 + i) * C::WK * 2, &full[slot]);
  };
  if (warp == 0) {
    if (elect_one()) {
      for (int s = 0; s < S; ++s) {
        mbar_init(&full[s], 1);
        mbar_init(&empty[s], kWarps);
      }
      *abort_flag = 0;
      fence_barrier_init();
    }
    __syncwarp();
    for (int i = 0; i < S && i < nst; ++i) load_weights(i, i);
  }
  if constexpr (WF == WF_LUT4) fill_book<T>(book, a.lut);
  __syncthreads();
  pdl_launch_dependents();
  // The tokens come from the kernels before this one, out and residual belong to them until here.  Every warp waits for them
  // here: the bounded waits below then count this kernel's own copies only.
  pdl_wait();
  if (warp == 0) {
    for (int i = 0; i < S && i < nst; ++i) load_tokens(i, i);
  }
  {
    // ---------------- multiply ----------------
    const int wm = warp % C::WM, wn = warp / C::WM % WN, wk = warp / (C::WM * WN), g = lane >> 2, t = lane & 3;
    float acc[C::MT][NT][4];
#pragma unroll
    for (int m = 0; m < C::MT; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[m][n][i] = 0.f;
    int slot = 0;
    uint32_t ph = 0;
    bool ok = true;
#pragma unroll 1
    for (int i = 0; i < nst; ++i) {
      // the warps take turns at filling the slot of the stage before, which all of them have read or are about to have
      if ((i & (kWarps - 1)) == warp && i > 0 && i - 1 + S < nst) {
        const int before = slot == 0 ? S - 1 : slot - 1;
        ok = warp_wait(&empty[before], slot == 0 ? ph ^ 1 : ph, abort_flag);
        if (!ok) break;
        load_weights(i - 1 + S, before);
        load_tokens(i - 1 + S, before);
      }
      ok = warp_wait(&full[slot], ph, abort_flag);
      if (!ok) break;
      const uint8_t* st = ring + slot * C::kStageBytes;
      if ((st0 + i) * C::WK + wk < a.chunks)
        chunk_mma<T, WF, NT, WN>(st + (wm * C::MT * C::WK + wk) * C::kCodes, st + C::kScaleAt + (wm * C::MT * C::WK + wk) * C::kScales,
                             st + C::kXAt + wk * 2 * C::kPiece + wn * NT * 1024, book + lane, acc);
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[slot]);
      if (++slot == S) { slot = 0; ph ^= 1; }
    }
    if (!ok) {
      if (lane == 0) report(a.err, 22);
      for (int s = 0; s < S; ++s) mbar_wait_quiet(&full[s], s < slot ? ph ^ 1 : ph, 1 << 12);   // copies in flight
    }
    __syncthreads();                                // the ring has been read, and every copy has landed
    float* mine = red + (size_t)(wk * C::kCols + wn * NT * 8) * C::kRedPitch + wm * C::MT * 16;
#pragma unroll
    for (int m = 0; m < C::MT; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) mine[(n * 8 + 2 * t + (i & 1)) * C::kRedPitch + m * 16 + g + 8 * (i >> 1)] = acc[m][n][i];
    if constexpr (C::minima) {
      float zero = 0.f;
#pragma unroll
      for (int m = 0; m < C::MT; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i) zero = fmaf(acc[m][n][i], 0.f, zero);
      if (__syncthreads_or(zero != 0.f))
        add_up_again<T, C::WK, C::kCols>(a.w, reinterpret_cast<const T*>(a.x), a.ldx, a.rows, a.N, a.chunks, red, tile,
                                         st0 * C::WK * 128, min(a.K, (st0 + nst) * C::WK * 128));
    }
  }
  add_parts<T, C::WK, C::kCols>(a, red, rank, split, tile, warp, lane);
}

// CTAs that share a tile's k: twice as many, up to eight, while all of them still fit the chip at two per SM or nearly so (a
// few of a second round cost less than a chip half full).  Three, five or seven never won: their clusters do not pack into the
// chip's groups of SMs.  int4, 8 rows, us by 1 / 2 / 4 / 8 CTAs: N = 4096 (32 tiles) 11.2 / 7.7 / 7.4 / 6.4, K = 11008 27.5 /
// 17.9 / 14.1 / 11.0; 12288 (96) 16.2 / 12.2 / 12.2 / 17.3; 22016 (172) 19.9 / 18.0 / 19.9 / 31.3; 32000 (250) 19.9 / 23.6 /
// 27.6 / 42.9.
inline int pick_split(int tiles, int stages, int asked) {
  int s = 1;
  if (asked > 0) s = asked;
  else while (s < kMaxSplit && 2 * s * tiles <= 355) s *= 2;
  return s < stages ? s : stages;
}

// Operands as the host has them.
struct Operands {
  const uint8_t* w;
  const void* x;
  int64_t ldx;
  int N, K;
};

inline bool encode_3d(CUtensorMap* tm, CUtensorMapDataType dt, const void* base, const cuuint64_t (&dims)[3],
                      const cuuint64_t (&strides)[2], const cuuint32_t (&box)[3], CUtensorMapSwizzle sw) {
  EncodeTiledFn enc = tensor_map_encoder();
  const cuuint32_t one[3] = {1, 1, 1};
  return enc != nullptr && enc(tm, dt, 3, const_cast<void*>(base), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

constexpr int kBadMap = -1;          // the driver's encoder refused the operands

// Tensor maps and launch of a kernel whose stage is WK chunks.
template <typename T, int CODES, int PLANES, int COLS, int WK, typename K>
int launch_tiles(K kern, SmemLimit& limit, int smem, const Operands& o, const Args& a, cudaStream_t st, bool pdl) {
  cudaError_t e = limit((const void*)kern, smem);
  if (e != cudaSuccess) return (int)e;
  // codes: [16-row tile][1024 bytes of a chunk][128 words]; planes of scales: [plane][16-row tile][chunk's 8 words]; tokens:
  // [64 k][row][k].  Whatever lies outside is read as zero.
  const cuuint64_t rt = ceil_to_i64(o.N, 16) / 16, ch = a.chunks, pieces = ch * (CODES / 1024);
  CUtensorMap tw, ts, tx;
  if (!encode_3d(&tw, CU_TENSOR_MAP_DATA_TYPE_INT64, o.w, {128, pieces, rt}, {1024, pieces * 1024},
                 {128, (cuuint32_t)(WK * CODES / 1024), 8}, CU_TENSOR_MAP_SWIZZLE_NONE) ||
      !encode_3d(&ts, CU_TENSOR_MAP_DATA_TYPE_INT64, o.w + rt * pieces * 1024, {ch * 8, rt, (cuuint64_t)PLANES},
                 {ch * 64, rt * ch * 64}, {WK * 8, 8, PLANES}, CU_TENSOR_MAP_SWIZZLE_NONE) ||
      !encode_3d(&tx, std::is_same<T, __half>::value ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, o.x,
                 {64, (cuuint64_t)a.rows, (cuuint64_t)o.K / 64}, {(cuuint64_t)o.ldx * 2, 128}, {64, COLS, 2 * WK},
                 CU_TENSOR_MAP_SWIZZLE_128B))
    return kBadMap;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((o.N + kBM - 1) / kBM * a.split);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = a.split;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl ? 2 : 1;
  return (int)cudaLaunchKernelEx(&cfg, kern, tw, ts, tx, a);
}

template <typename T, int WF, int NT, int WN>
int launch(const Operands& o, Args a, cudaStream_t st, bool pdl, int asked) {
  using C = Cfg<WF, NT, WN>;
  a.split = pick_split((o.N + kBM - 1) / kBM, (a.chunks + C::WK - 1) / C::WK, asked);
  static SmemLimit limit;
  return launch_tiles<T, C::kCodes, C::kPlanes, C::kCols, C::WK>(kernel<T, WF, NT, WN>, limit, C::kSmem, o, a, st, pdl);
}

// The instances that ipex_gemm_few's rule leaves to this kernel.
template <typename T, int WF>
int by_columns(const Operands& o, const Args& a, cudaStream_t st, bool pdl, int asked) {
  const int cols = (a.rows + 7) / 8;
  if (cols == 1) return launch<T, WF, 1, 1>(o, a, st, pdl, asked);
  if (cols == 2) return launch<T, WF, 2, 1>(o, a, st, pdl, asked);
  if constexpr (WF != WF_ASYM_INT4)
    if (cols == 3) return launch<T, WF, 3, 1>(o, a, st, pdl, asked);
  if constexpr (WF != WF_FP8_E4M3 && WF != WF_FP8_E5M2) {      // pairs
    if (cols == 5 || cols == 6) return launch<T, WF, 3, 2>(o, a, st, pdl, asked);
    if (cols > 6) return launch<T, WF, 4, 2>(o, a, st, pdl, asked);
  }
  return (int)cudaErrorInvalidValue;
}

template <typename T>
int by_family(int wf, const Operands& o, const Args& a, cudaStream_t st, bool pdl, int asked) {
  switch (wf) {
    case WF_SYM_INT4: return by_columns<T, WF_SYM_INT4>(o, a, st, pdl, asked);
    case WF_ASYM_INT4: return by_columns<T, WF_ASYM_INT4>(o, a, st, pdl, asked);
    case WF_LUT4: return by_columns<T, WF_LUT4>(o, a, st, pdl, asked);
    case WF_FP8_E4M3: return by_columns<T, WF_FP8_E4M3>(o, a, st, pdl, asked);
    case WF_FP8_E5M2: return by_columns<T, WF_FP8_E5M2>(o, a, st, pdl, asked);
    case WF_INT8: return by_columns<T, WF_INT8>(o, a, st, pdl, asked);
    default: return (int)cudaErrorInvalidValue;
  }
}

}  // namespace few
