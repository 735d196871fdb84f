// Products of 25 to 64 token rows (17 to 64 of the format with minima) with packed weights on tcgen05, the weights' operand in
// tensor memory:
//     out[M, N] = x[M, K] . W[N, K]^T  (+ bias) (+ residual)   or   act(gate) * up  for interleaved gate/up rows
// (gemm_few.cuh has the contract, the tensor maps, the ring's layout and the adding up of the parts.)
//
// What bounds it: taking the codes apart, as in gemm_few.cuh; but there the matrix pipe (one m16n8k16 in eight clocks) and the
// sums of every scale group cost as much again from 24 columns on.  Here a lane takes one weight row's codes apart, stores them
// to its lane of tensor memory, and tcgen05.mma multiplies 128 rows by all columns at once.  Nothing of the expanded weights goes
// through shared memory.  us per launch between dependent launches, weights from memory, gemm_few.cuh's form | this: int4, 24
// rows, 22016 x 4096 25.8 | 30, 32 rows 33.5 | 29.4, 64 rows 59.7 | 39.1, 32000 x 4096 at 64 rows 70.7 | 34.7; nf4, 40 rows,
// 22016 x 4096 51.7 | 36.4; fp8 48.4 | 38.3.  (A form that wrote expanded weights to shared memory took 42.5, 55.5 and 65.9 for
// int4 at 32 and 64 rows, 67 for nf4 at 64.)  Columns of 64 of the 8-bit floats spill some 50 to 150 bytes a thread beside two
// CTAs' registers, and are the faster all the same: 64 rows, 22016 x 4096, that form and this: e4m3 fp16 64.2 and 48.5, bf16 64.2
// and 49.1, e5m2 62.3 and 48.3, 64.1 and 49.1.
//
// Up to 32 columns (and in the 8-bit float formats) the codes are multiplied and the sums of each scale group scaled and added
// in 32 bits.  More columns of the other formats are expanded and scaled in 16 bits, as in the kernel for many rows, and the sums
// stay in tensor memory.
//
// Minima up to 32 columns stay apart too: their part is their product with the sums of the tokens, which a team makes (eight
// tokens a warp, products with ones) and adds while its products run: the sums of a stage behind its barrier, their product with
// the minima behind the next one's.  Sums by gemm_few.cuh's way (every warp makes all of them) and this, us at 24 | 32 rows of
// fp16: 12288 x 4096 24.8 / 22.3 | 32.3 / 23.1, 4096 x 11008 20.2 / 18.4 | 26.0 / 18.9, 22016 x 4096 36.5 / 35.1 | 47.8 / 36.6
// (bf16 46.9 / 37.5); weights expanded and scaled in 16 bits (in a form before these) took 22.3, 19.2 and 34.6 at 32 rows.  (The minima's
// product at the end, as tf32, instead of stage by stage: 24.1, 20.4 and 38.4.)
//
// A CTA holds 128 weight rows over a share of k; two teams of four warps take its stages of 128 k in turn, and two CTAs fit an SM,
// so that three teams work while one waits.  A team that has waited for its products knows its stage's slot to be free and has it
// filled again: the ring needs no other barrier.  TMEM of a team: 64 columns of weights, up to 64 of sums.
// Every wait is bounded (error code 24); a warp whose wait ran out still attends its team's barriers.
#pragma once
#include "gemm_few.cuh"

namespace few {
namespace tm {

constexpr int kTeams = 2;
constexpr int kTeamCols = 128;       // of TMEM

template <int WF, int N> struct Cfg {
  static constexpr bool k4 = WF == WF_SYM_INT4 || WF == WF_ASYM_INT4 || WF == WF_LUT4;
  static constexpr bool fp8 = WF == WF_FP8_E4M3 || WF == WF_FP8_E5M2;
  static constexpr bool codes = fp8 || N <= 32;
  static constexpr bool minima = WF == WF_ASYM_INT4 && codes;
  static constexpr int groups = codes && !fp8 ? 2 : 1;                 // sums of a stage
  static constexpr int kCodes = k4 ? 1024 : 2048, kScales = 64;        // bytes of a 16-row tile's 128 k
  static constexpr int kPlanes = WF == WF_ASYM_INT4 ? 2 : 1;
  static constexpr int kXAt = 8 * kCodes;
  static constexpr int kPiece = N * 128;
  static constexpr int kScaleAt = kXAt + 2 * kPiece;
  static constexpr int kBytes = kScaleAt + kPlanes * 8 * kScales;
  static constexpr int kStageBytes = (kBytes + 1023) / 1024 * 1024;
  static constexpr int kBook = WF == WF_LUT4 ? 256 * 32 * 4 : 0;
  static constexpr int kSums = minima ? kTeams * 2 * 2 * N * 4 : 0;    // [team][stage in turn][group][token]
  static constexpr int kTail = 256 + kBook + kSums;
  static constexpr int kRedPitch = kBM + 4;
  static constexpr int kRedBytes = kTeams * N * kRedPitch * 4;
  static constexpr int kStagesFit = (kSmemMax - 1024 - kTail) / kStageBytes;
  static constexpr int kStages = kStagesFit > 8 ? 8 : kStagesFit;
  static constexpr int kSmem = 1024 + kStages * kStageBytes + kTail;
  static_assert(kStages > kTeams && kRedBytes <= kStages * kStageBytes && groups * N <= kTeamCols - 64, "ring");
  static_assert(!minima || N == 32, "eight tokens to each of a team's warps");
};

__device__ __forceinline__ void tmem_st_32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
      "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]),
      "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]),
      "r"(v[31])
      : "memory");
}
// 32 lanes x 16 columns, without the wait
__device__ __forceinline__ void tmem_ld_16(uint32_t taddr, float* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]),
        "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
      : "r"(taddr)
      : "memory");
}
template <int N> __device__ __forceinline__ void tmem_ld_done(float (&v)[N]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
  // the values are only there behind the wait: no use of theirs moves in front of it
#pragma unroll
  for (int j = 0; j < N; ++j) asm volatile("" : "+f"(v[j]));
}
// D[tmem] (+)= A[tmem] . B[smem]; issued by one thread
__device__ __forceinline__ void umma_f16_ts(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "}\n" ::"r"(d),
      "r"(a), "l"(bdesc), "r"(idesc), "r"((uint32_t)accumulate)
      : "memory");
}

// Two sums at once: a0 += d * x0, a1 += d * x1.
__device__ __forceinline__ void fma2(float& a0, float& a1, float d, float x0, float x1) {
  asm("{\n"
      ".reg .b64 a, d, x;\n"
      "mov.b64 a, {%0, %1};\n"
      "mov.b64 d, {%2, %2};\n"
      "mov.b64 x, {%3, %4};\n"
      "fma.rn.f32x2 a, d, x, a;\n"
      "mov.b64 {%0, %1}, a;\n"
      "}\n"
      : "+f"(a0), "+f"(a1)
      : "f"(d), "f"(x0), "f"(x1));
}

template <typename T, int WF, int N>
__global__ void __launch_bounds__(kThreads, kCtasPerSM)
kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_s, const __grid_constant__ CUtensorMap tm_x,
       const Args a) {
  using C = Cfg<WF, N>;
  using V = V2<T>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(ring + C::kStages * C::kStageBytes);
  uint64_t* done = full + 2 * C::kStages;           // [team]: the products of its stage
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + kTeams);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint32_t* book = reinterpret_cast<uint32_t*>(full) + 64;
  float* sums = reinterpret_cast<float*>(book);
  float* red = reinterpret_cast<float*>(ring);      // [team][column][row], once the ring has been read

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int split = a.split, rank = blockIdx.x % split, tile = blockIdx.x / split;
  const int st0 = a.chunks * rank / split, nst = a.chunks * (rank + 1) / split - st0;
  constexpr int S = C::kStages;

  // Two barriers to a slot, for its uses in turn: with an odd number of slots the teams take a slot in turn, and one may wait for
  // its stage while the other's in the same slot is still on its way.  One barrier's parity would tell that wait that it is over.
  auto barrier = [&](int slot, int use) { return &full[(use & 1) * S + slot]; };
  auto load_weights = [&](int i, int slot, int use) {        // a converged warp
    if (elect_one()) {
      uint8_t* to = ring + slot * C::kStageBytes;
      uint64_t* b = barrier(slot, use);
      mbar_expect_tx(b, C::kBytes);
      tma_load_3d(to, &tm_w, 0, (st0 + i) * (C::kCodes / 1024), tile * 8, b);
      tma_load_3d(to + C::kScaleAt, &tm_s, (st0 + i) * (C::kScales / 8), tile * 8, 0, b);
    }
  };
  auto load_tokens = [&](int i, int slot, int use) {
    if (elect_one()) tma_load_3d(ring + slot * C::kStageBytes + C::kXAt, &tm_x, 0, 0, (st0 + i) * 2, barrier(slot, use));
  };
  if (warp == 0) {
    if (elect_one()) {
      for (int s = 0; s < 2 * S; ++s) mbar_init(&full[s], 1);
      for (int t = 0; t < kTeams; ++t) mbar_init(&done[t], 1);
      *abort_flag = 0;
      fence_barrier_init();
    }
    __syncwarp();
    for (int i = 0; i < S && i < nst; ++i) load_weights(i, i, 0);
  }
  if (warp == 1) tmem_alloc(tmem_slot, kTeams * kTeamCols);
  if constexpr (WF == WF_LUT4) fill_book<T>(book, a.lut);
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  pdl_launch_dependents();                          // (with this CTA's columns allocated: a kernel behind may want its own)
  pdl_wait();                                       // the tokens come from the kernels before this one (see gemm_few.cuh)
  if (warp == 0) {
    for (int i = 0; i < S && i < nst; ++i) load_tokens(i, i, 0);
  }

  const int team = warp >> 2, qd = warp & 3;        // TMEM lane quarter this warp may reach
  const bool issuer = qd == team;                   // (of another scheduler in the other team)
  const int r = lane & 15;                          // row of its 16-row tile 2 qd + lane / 16
  const uint32_t tmem = *tmem_slot + team * kTeamCols;
  const uint32_t tA = tmem, tD = tmem + 64, lanes = (uint32_t)(qd * 32) << 16;
  const uint32_t idesc = make_idesc_f16<T>(kBM, N);
  const uint32_t* my_book = book + lane;
  float acc[N];
#pragma unroll
  for (int j = 0; j < N; ++j) acc[j] = 0.f;
  float d[2] = {0.f, 0.f};                          // scales of the sums on their way
  auto fold = [&] {
    constexpr int cols = C::groups * N;
#pragma unroll
    for (int c = 0; c < cols; c += 32) {
      constexpr int step = cols < 32 ? cols : 32;
      float v[step];
#pragma unroll
      for (int j = 0; j < step; j += 16) tmem_ld_16(tD + lanes + c + j, v + j);
      tmem_ld_done(v);
#pragma unroll
      for (int j = 0; j < step; j += 2) {
        if (c + j >= cols) break;
        if constexpr (C::minima) {
          fma2(acc[(c + j) % N], acc[(c + j) % N + 1], d[(c + j) / N], v[j], v[j + 1]);
        } else {
          acc[(c + j) % N] = fmaf(d[(c + j) / N], v[j], acc[(c + j) % N]);
          acc[(c + j) % N + 1] = fmaf(d[(c + j) / N], v[j + 1], acc[(c + j) % N + 1]);
        }
      }
    }
  };
  int turn = 0;                                     // where the stage's sums go
  float dm[2] = {0.f, 0.f};                         // minima of the stage whose sums are there next
  auto add_minima = [&] {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float4* sx = reinterpret_cast<const float4*>(sums + ((team * 2 + (turn ^ 1)) * 2 + h) * N);
#pragma unroll
      for (int j = 0; j < N; j += 4) {
        const float4 x = sx[j / 4];
        fma2(acc[j], acc[j + 1], dm[h], x.x, x.y);
        fma2(acc[j + 2], acc[j + 3], dm[h], x.z, x.w);
      }
    }
  };
  bool ok = true, waiting = false;
  int slot = team, use = 0, last = 0, last_use = 0;
  uint32_t dph = 0;
#pragma unroll 1
  for (int i = team; i < nst; i += kTeams) {
    if (waiting) {
      if (ok) ok = warp_wait(&done[team], dph, abort_flag);
      if (ok) dph ^= 1;
      tcgen05_fence_after();
      if (ok && issuer && i - kTeams + S < nst) {
        load_weights(i - kTeams + S, last, last_use + 1);
        load_tokens(i - kTeams + S, last, last_use + 1);
      }
    }
    if (ok) ok = warp_wait(barrier(slot, use), (use >> 1) & 1, abort_flag);
    const uint8_t* st = ring + slot * C::kStageBytes;
    const uint8_t* ct = st + (2 * qd + (lane >> 4)) * C::kCodes + r * 64;
    const uint8_t* sp = st + C::kScaleAt + (2 * qd + (lane >> 4)) * C::kScales;
    uint4 q[C::k4 ? 4 : 8];
    if (ok) {
#pragma unroll
      for (int j = 0; j < (C::k4 ? 4 : 8); ++j) q[j] = *reinterpret_cast<const uint4*>(ct + (j >> 2) * 1024 + (j & 3) * 16);
    }
    float dn[2] = {1.f, 1.f}, mn[2] = {0.f, 0.f};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if constexpr (!C::fp8) {
        dn[h] = __half2float(reinterpret_cast<const __half*>(sp)[h * 16 + pair_row(r)]);
        if constexpr (WF == WF_ASYM_INT4)
          mn[h] = __half2float(reinterpret_cast<const __half*>(sp + 8 * C::kScales)[h * 16 + pair_row(r)]);
      } else {
        constexpr float k = std::is_same<T, __half>::value ? Fp8Place<__half, WF>::mul * Fp8Place<__half, WF>::pre : 1.f;
        dn[h] = reinterpret_cast<const float*>(sp)[pair_row(r)] * k;
      }
    }
    if (C::codes && waiting && ok) fold();
    if (ok) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        Scale<T> sc;
        sc.d = V::splat(dn[h]);
        sc.m = V::splat(mn[h]);
        uint32_t v[32];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          uint4 lo, hi;
          if constexpr (C::k4) {
            // 16 bytes = [group 0: k 16t..16t+7 | 16t+8..16t+15 | group 1: same]
            const uint32_t w0 = h == 0 ? q[t].x : q[t].z, w1 = h == 0 ? q[t].y : q[t].w;
            lo = codes4<T, WF, C::codes>(w0, my_book, sc);
            hi = codes4<T, WF, C::codes>(w1, my_book, sc);
          } else if constexpr (C::codes) {
            lo = codes8<T, WF>(q[4 * h + t].x, q[4 * h + t].y);
            hi = codes8<T, WF>(q[4 * h + t].z, q[4 * h + t].w);
          } else {
            lo = expand8<T, WF>(q[4 * h + t].x, q[4 * h + t].y, sc);
            hi = expand8<T, WF>(q[4 * h + t].z, q[4 * h + t].w, sc);
          }
          v[8 * t] = lo.x; v[8 * t + 1] = lo.y; v[8 * t + 2] = lo.z; v[8 * t + 3] = lo.w;
          v[8 * t + 4] = hi.x; v[8 * t + 5] = hi.y; v[8 * t + 6] = hi.z; v[8 * t + 7] = hi.w;
        }
        tmem_st_32(tA + lanes + 32 * h, v);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    d[0] = dn[0];
    d[1] = dn[1];
    uint4 xb[C::minima ? 4 : 1];
    if constexpr (C::minima) {
      const int g = lane >> 2, t = lane & 3;
      if (ok) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          xb[i] = *reinterpret_cast<const uint4*>(st + C::kXAt + (i >> 1) * C::kPiece + qd * 1024 + g * 128 +
                                                  (((2 * t + (i & 1)) ^ g) << 4));
      }
    }
    tcgen05_fence_before();
    asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "n"(kThreads / kTeams) : "memory");
    if (issuer && ok) {
      tcgen05_fence_after();
      if (elect_one()) {
        const uint64_t bd = make_desc_sw128(smem_u32(st + C::kXAt));
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            const bool fresh = C::codes ? (C::groups == 2 || h == 0) && kk == 0 : !waiting && h == 0 && kk == 0;
            umma_f16_ts(tD + (C::groups == 2 ? h * N : 0), tA + 32 * h + 8 * kk, bd + (h * C::kPiece >> 4) + 2 * kk, idesc, !fresh);
          }
        umma_commit(&done[team]);
      }
      __syncwarp();
    }
    if constexpr (C::minima) {
      if (ok) {
        if (waiting) add_minima();
        constexpr uint32_t one = std::is_same<T, __half>::value ? 0x3C003C00u : 0x3F803F80u;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int o = 0; o < 2; ++o) {
            mma16<T>(s, one, one, one, one, xb[2 * h + o].x, xb[2 * h + o].y);
            mma16<T>(s, one, one, one, one, xb[2 * h + o].z, xb[2 * h + o].w);
          }
          float* to = sums + ((team * 2 + turn) * 2 + h) * N + 8 * qd;
          if (lane < 4) reinterpret_cast<float2*>(to)[lane] = make_float2(s[0], s[1]);
        }
      }
      dm[0] = mn[0];
      dm[1] = mn[1];
      turn ^= 1;
    }
    waiting = true;
    if (ok) {                                       // (a wait that ran out: the barriers behind the loop are those of its stage)
      last = slot;
      last_use = use;
      slot += kTeams;
      if (slot >= S) { slot -= S; ++use; }
    }
  }
  if (waiting) {
    if constexpr (C::minima) {
      asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "n"(kThreads / kTeams) : "memory");
      add_minima();
    }
    if (ok) ok = warp_wait(&done[team], dph, abort_flag);
    tcgen05_fence_after();
    if (ok) {
      if constexpr (C::codes) {
        fold();
      } else {
#pragma unroll
        for (int j = 0; j < N; j += 16) tmem_ld_16(tD + lanes + j, acc + j);
        tmem_ld_done(acc);
      }
    }
  }
  if (!ok) {
    if (lane == 0) report(a.err, 24);
    mbar_wait_quiet(&done[team], dph, 1 << 12);     // products and copies in flight
    for (int s = 0; s < S; ++s) {
      const int u = s < slot ? use + 1 : use;
      mbar_wait_quiet(barrier(s, u), (u >> 1) & 1, 1 << 10);
    }
  }
  tcgen05_fence_before();
  __syncthreads();                                  // the ring has been read, and every copy has landed
  float* mine = red + (size_t)team * N * C::kRedPitch + qd * 32 + lane;
#pragma unroll
  for (int j = 0; j < N; ++j) mine[j * C::kRedPitch] = acc[j];
  if constexpr (C::minima) {
    float zero = 0.f;
#pragma unroll
    for (int j = 0; j < N; ++j) zero = fmaf(acc[j], 0.f, zero);
    if (__syncthreads_or(zero != 0.f))
      add_up_again<T, kTeams, N>(a.w, reinterpret_cast<const T*>(a.x), a.ldx, a.rows, a.N, a.chunks, red, tile, st0 * 128,
                                 min(a.K, (st0 + nst) * 128));
  }
  add_parts<T, kTeams, N>(a, red, rank, split, tile, warp, lane);
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(*tmem_slot, kTeams * kTeamCols);
  }
}

template <typename T, int WF, int N>
int launch(const Operands& o, Args a, cudaStream_t st, bool pdl, int asked) {
  using C = Cfg<WF, N>;
  a.split = pick_split((o.N + kBM - 1) / kBM, a.chunks, asked);
  static SmemLimit limit;
  return launch_tiles<T, C::kCodes, C::kPlanes, N, 1>(kernel<T, WF, N>, limit, C::kSmem, o, a, st, pdl);
}

template <typename T, int WF>
int by_width(const Operands& o, const Args& a, cudaStream_t st, bool pdl, int asked) {
  if (a.rows <= 32) return launch<T, WF, 32>(o, a, st, pdl, asked);
  if (a.rows <= 48) return launch<T, WF, 48>(o, a, st, pdl, asked);
  return launch<T, WF, 64>(o, a, st, pdl, asked);
}

}  // namespace tm
}  // namespace few
