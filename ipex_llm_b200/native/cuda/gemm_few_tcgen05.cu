// Products of 5 to 64 token rows with packed weights (decode steps of a batch, drafted continuations) on tcgen05:
//     out[M, N] = x[M, K] . W[N, K]^T  (+ bias) (+ residual)   or   act(gate) * up  for interleaved gate/up rows
//
// What bounds it: the packed weights' way from memory, 4.4 KB per 128 x 64 weights, if enough SMs work and the expanders keep
// up.  The tiles of 128 weight rows are too few for that (32 at N = 4096, 148 SMs), so a cluster of kSplit CTAs shares the k
// of a tile and adds the parts up through distributed shared memory: no workspace, no counters, a fixed order of addition.
//
// Up to 32 columns the expanders write the codes themselves (small integers, fp8 values: exact in 16 bits) and the scales are
// applied to the sums of one scale group in 32 bits: nothing of the weight is rounded (a code book's values are, to 16 bits,
// but not their product with the scale), and scaling few sums is cheaper than scaling every weight.  With 64 columns the
// 4-bit formats and int8 are expanded and scaled in 16 bits instead, as in the kernel for many rows, and accumulate over all
// of the CTA's k (12288 x 4096 int4 at 64 rows: 40.5 us by codes, 31 by weights), unless x comes in pairs; so is the format with
// minima always.
//
// A stage holds 128 k.  What the issuing warp does per stage is the clock of the loop (a wait costs it 250 clocks, an MMA 45, a
// commit 60), so it waits for one barrier only, asks for the next stage's before it issues, and the loader has made sure
// that the accumulator is free.
//
// x may hold two rows per token (2m: the value rounded to 16 bits, 2m + 1: what that left over); their products are added in
// 32 bits at the end.
//
// Roles by warp: 0 loads the tokens of each stage by TMA; 1 allocates TMEM and issues the MMAs (the whole warp runs the
// loop, one lane is elected at the instruction); 2..5 fold each group's accumulator into 32-bit sums in registers, exchange
// and store them; 6..17 are three teams of four that expand stages of 128 k in turn, a lane per weight row.  (Eight folding
// warps, each with half of the columns, measured slower: 12288 x 4096 at 32 rows 25.7 us against 23.3.)
// Every wait is bounded (error codes 20 loader, 21 MMA, 22 fold, 23 expander).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common/utils.cuh"
#include "lowbit_expand.cuh"
#include "tcgen05_common.cuh"

namespace {

using namespace tc5;

constexpr int kSplit = 4;            // CTAs that share a tile's k
constexpr int kBM = 128, kBK = 64;
constexpr int kTeamThreads = 128, kTeams = 3;
constexpr int kExpand0 = 192;
constexpr int kThreads = kExpand0 + kTeams * kTeamThreads;
constexpr int kStages = kTeams;       // a stage of 128 k per team

struct FewArgs {
  const uint8_t* w;
  const float* lut;
  void* out;
  const void* bias;
  const void* residual;
  int64_t ldo, ldr;
  int64_t Np, Kp;
  int M, N;            // M: tokens (rows of out)
  int n_tiles;
  int act;
  int pairs;           // two rows of x per token
  int* err;
};

template <int WF, bool CODES> struct FewFam {
  static constexpr bool four_bit = WF == WF_SYM_INT4 || WF == WF_ASYM_INT4 || WF == WF_LUT4;
  static constexpr bool codes = CODES;                                               // scales applied to sums
  static constexpr bool half_scale = four_bit || WF == WF_INT8;                      // fp16 per 64 k, else fp32 per 128
  static constexpr int groups = CODES && half_scale ? 2 : 1;                         // sums per stage
};

template <int BT, int WF, bool CODES> struct FewCfg {
  static constexpr int kABytes = kBM * kBK * 2;                                      // one swizzle atom: 64 k
  static constexpr int kBBytes = BT * kBK * 2;
  static constexpr int kStageBytes = 2 * (kABytes + kBBytes);
  static constexpr int kBufCols = FewFam<WF, CODES>::groups * BT;
  static constexpr int kBufs = 512 / kBufCols < 8 ? 512 / kBufCols : 8;              // accumulators in flight
  static constexpr int kTmemCols = kBufs * kBufCols;
  static constexpr int kPart = BT * kBM;                                             // floats of one exchange buffer
  static constexpr int kSmemBytes = kStages * kStageBytes + 2 * kPart * 4 + 1024 /*alignment*/ + 512 /*barriers*/ +
                                    1024 /*code book*/;
};

// ---- cluster helpers ------------------------------------------------------------------------------------------------
// Values to another CTA's shared memory, counted in bytes by a barrier there (the wait for it acquires at cluster scope).
__device__ __forceinline__ void st_async2(uint32_t addr, uint32_t bar, float a, float b) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(addr), "f"(a),
               "f"(b), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void st_async4(uint32_t addr, uint32_t bar, float a, float b, float c, float d) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
               "f"(a), "f"(b), "f"(c), "f"(d), "r"(bar)
               : "memory");
}
// 32 lanes x N columns, without the wait
template <int N> __device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, float* v) {
  if constexpr (N == 8) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "r"(taddr)
                 : "memory");
  } else {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]),
          "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
        : "r"(taddr)
        : "memory");
    if constexpr (N == 32) tmem_ld_cols<16>(taddr + 16, v + 16);
  }
}
template <int N> __device__ __forceinline__ void tmem_ld_done(float (&v)[N]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
  // the values are only there behind the wait: no use of theirs moves in front of it
#pragma unroll
  for (int j = 0; j < N; ++j) asm volatile("" : "+f"(v[j]));
}

// The codes of 8 weights as 16-bit values (see expand4 / expand8, without their scale).
template <typename T, int WF>
__device__ __forceinline__ uint4 codes4(uint32_t w, const uint32_t* book) {
  using V = V2<T>;
  if constexpr (WF == WF_LUT4)     // pairs of values by the byte (an entry per nibble, without bank conflicts, measured slower)
    return make_uint4(book[w & 0xFF], book[(w >> 8) & 0xFF], book[(w >> 16) & 0xFF], book[w >> 24]);
  const typename V::type off = V::splat(V::kMagicBase + 8.f);
  uint32_t r[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) r[i] = V::raw(__hsub2(V::bits(((w >> (4 * i)) & 0x000F000Fu) | V::kMagic), off));
  return make_uint4(r[0], r[1], r[2], r[3]);
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
// The factor of a group's sums from its raw scale.
template <typename T, int WF, bool CODES>
__device__ __forceinline__ float group_scale(uint32_t raw) {
  if constexpr (!CODES) return 1.f;
  else if constexpr (FewFam<WF, CODES>::half_scale) return __half2float(__ushort_as_half((uint16_t)raw));
  else if constexpr (std::is_same<T, __nv_bfloat16>::value) return __uint_as_float(raw);
  else return __uint_as_float(raw) * (Fp8Place<T, WF>::mul * Fp8Place<T, WF>::pre);
}


// ---- expanders ------------------------------------------------------------------------------------------------------
template <typename T, int BT, int WF, bool CODES>
__device__ __forceinline__ void few_expand(const FewArgs& a, int u_begin, int u_count, uint8_t* sA, uint64_t* full,
                                           uint64_t* empty, volatile int* abort_flag, const uint32_t* book) {
  using C = FewCfg<BT, WF, CODES>;
  using V = V2<T>;
  constexpr bool k4 = FewFam<WF, CODES>::four_bit;
  // a piece is 64 bytes of this thread's row: the 128 k of a stage in 4-bit codes, half of them in bytes
  constexpr int kPieces = k4 ? 1 : 2;
  const int dt = threadIdx.x - kExpand0;
  const int team = dt / kTeamThreads, r = dt % kTeamThreads, lane = threadIdx.x & 31;
  const int tstep = gridDim.x / kSplit;
  const int64_t k128 = a.Kp / 128;
  const uint8_t* planes = a.w + (k4 ? a.Np * a.Kp / 2 : a.Np * a.Kp);
  const uint16_t* sc16 = reinterpret_cast<const uint16_t*>(planes);
  const int prow = pair_row(r & 15);
  const int first = blockIdx.x / kSplit;
  const int my_tiles = first < a.n_tiles ? (a.n_tiles - first + tstep - 1) / tstep : 0;
  const int total = my_tiles * u_count;

  int lt = first, lu = team, lp = 0;               // where the next load stands: tile, stage of this CTA's share, piece
  bool valid = false;
  const uint8_t* wp = nullptr;                     // its bytes, and its row's first scale
  const uint16_t* sp = nullptr;
  auto seat = [&]() {
    while (lu >= u_count) {
      lu -= u_count;
      lt += tstep;
    }
    const int64_t rg = (int64_t)lt * kBM + r;
    valid = lt < a.n_tiles && rg < a.Np;
    if (valid) {
      const int64_t at = (rg >> 4) * k128 + u_begin + lu;
      wp = a.w + at * (kPieces * 1024) + (r & 15) * 64;
      sp = sc16 + at * 32 + prow;
    }
  };
  // raw bits only: a conversion here would wait for the load
  struct Piece { uint4 q[4]; uint32_t d0, d1, m0, m1; };
  auto load = [&](Piece& n) {
    n.q[0] = n.q[1] = n.q[2] = n.q[3] = make_uint4(0, 0, 0, 0);
    n.d0 = n.d1 = n.m0 = n.m1 = 0;
    if (valid) {
      ldg_nc_32b(wp, n.q[0], n.q[1]);
      ldg_nc_32b(wp + 32, n.q[2], n.q[3]);
      if constexpr (!CODES && k4) {
        n.d0 = ldg_nc_u16(sp);
        n.d1 = ldg_nc_u16(sp + 16);
        if constexpr (WF == WF_ASYM_INT4) {
          const uint16_t* mp = sp + a.Np * (a.Kp / 64);
          n.m0 = ldg_nc_u16(mp);
          n.m1 = ldg_nc_u16(mp + 16);
        }
      } else if constexpr (!CODES) {
        n.d0 = ldg_nc_u16(sp + lp * 16);           // int8: a piece is a scale's 64 k
      }
    }
    if (++lp == kPieces) {
      lp = 0;
      lu += kTeams;
      wp += (kTeams * kPieces - (kPieces - 1)) * 1024;
      sp += kTeams * 32;
      if (lu >= u_count) seat();
    } else {
      wp += 1024;
    }
  };

  if (u_count <= 0) return;
  uint32_t ph = 0;
  bool ok = true;
  Piece next;
  seat();
  load(next);
  uint8_t* row = sA + team * C::kStageBytes + r * 128;
#pragma unroll 1
  for (int u = team; u < total; u += kTeams, ph ^= 1) {
#pragma unroll
    for (int p = 0; p < kPieces; ++p) {
      const Piece cur = next;
      load(next);
      if (p == 0 && ok && !warp_wait(&empty[team], ph ^ 1, abort_flag)) {
        if (lane == 0) report(a.err, 23);
        ok = false;
      }
#pragma unroll
      for (int g = 0; g < (k4 ? 2 : 1); ++g) {
        Scale<T> sc;
        if constexpr (!FewFam<WF, CODES>::codes) {
          sc.d = V::splat(__half2float(__ushort_as_half((uint16_t)(g == 0 ? cur.d0 : cur.d1))));
          if constexpr (WF == WF_ASYM_INT4)
            sc.m = V::splat(__half2float(__ushort_as_half((uint16_t)(g == 0 ? cur.m0 : cur.m1))));
        }
        uint8_t* atom = row + (k4 ? g : p) * C::kABytes;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const uint4 q = cur.q[t];
          uint4 lo, hi;
          if constexpr (k4) {
            // uint4 = [group 0: k 16t..16t+7 | 16t+8..16t+15 | group 1: same]
            if constexpr (FewFam<WF, CODES>::codes) {
              lo = codes4<T, WF>(g == 0 ? q.x : q.z, book);
              hi = codes4<T, WF>(g == 0 ? q.y : q.w, book);
            } else {
              lo = expand4<T, WF>(g == 0 ? q.x : q.z, sc, book);
              hi = expand4<T, WF>(g == 0 ? q.y : q.w, sc, book);
            }
          } else if constexpr (CODES) {
            lo = codes8<T, WF>(q.x, q.y);
            hi = codes8<T, WF>(q.z, q.w);
          } else {
            lo = expand8<T, WF>(q.x, q.y, sc);
            hi = expand8<T, WF>(q.z, q.w, sc);
          }
          if (ok) {
            *reinterpret_cast<uint4*>(atom + (((2 * t) ^ (r & 7)) << 4)) = lo;      // 16-byte chunk = 8 consecutive k
            *reinterpret_cast<uint4*>(atom + (((2 * t + 1) ^ (r & 7)) << 4)) = hi;
          }
        }
      }
    }
    // one proxy fence and one arrival for the team, behind a barrier that orders its stores before them (a warp whose wait
    // ran out still attends)
    asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "n"(kTeamThreads) : "memory");
    if (r == 0 && ok) {
      fence_proxy_async_smem();
      mbar_arrive(&full[team]);
    }
  }
}

template <typename T, int BT, int WF, bool CODES>
__global__ void __cluster_dims__(kSplit, 1, 1) __launch_bounds__(kThreads, 1)
gemm_few_kernel(const __grid_constant__ CUtensorMap tm_x, const FewArgs a) {
  using C = FewCfg<BT, WF, CODES>;
  constexpr bool k4 = FewFam<WF, CODES>::four_bit;
  constexpr bool kCodes = FewFam<WF, CODES>::codes;
  constexpr int kGroups = FewFam<WF, CODES>::groups;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;                                                    // a stage: two weight atoms, two token atoms
  float* part = reinterpret_cast<float*>(smem + kStages * C::kStageBytes);   // [2][from][row][token of this CTA]
  uint64_t* full = reinterpret_cast<uint64_t*>(part + 2 * C::kPart);
  uint64_t* empty = full + kStages;
  uint64_t* d_full = empty + kStages;
  uint64_t* d_empty = d_full + C::kBufs;
  uint64_t* p_full = d_empty + C::kBufs;                                 // the parts of a tile have arrived
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(p_full + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint32_t* book = reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(full) + 512);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t rank = cta_rank();
  const int first = blockIdx.x / kSplit, tstep = gridDim.x / kSplit;
  // this CTA's share of every tile's k, in stages of 128
  const int k128 = (int)(a.Kp / 128);
  const int kt0 = (int)((int64_t)k128 * rank / kSplit), nst = (int)((int64_t)k128 * (rank + 1) / kSplit) - kt0;
  const int tq = (a.pairs ? BT / 2 : BT) / kSplit;                       // tokens that each CTA adds up and stores

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 2);                       // the loader and the team
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < C::kBufs; ++i) {
      mbar_init(&d_full[i], 1);
      mbar_init(&d_empty[i], 4);
    }
    for (int i = 0; i < 2; ++i) mbar_init(&p_full[i], 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if constexpr (WF == WF_LUT4) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {
      const T lo = from_float<T>(a.lut[i & 15]), hi = from_float<T>(a.lut[i >> 4]);
      book[i] = (uint32_t)(*reinterpret_cast<const uint16_t*>(&lo)) |
                ((uint32_t)(*reinterpret_cast<const uint16_t*>(&hi)) << 16);
    }
  }
  if (warp == 1) tmem_alloc(tmem_slot, C::kTmemCols);
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ---------------- loader ----------------
    if (elect_one()) prefetch_tmap(&tm_x);
    // The expanders' loads are one unit ahead, which hides L2's latency but not memory's: the bytes of a tile's share are
    // called into L2 two tiles ahead, a lane for each 16-row tile's codes and another for its scales.
    constexpr int kStageCodes = k4 ? 1024 : 2048, kStageScales = 64;     // of 16 rows
    auto call_in = [&](int t) {
      const int64_t rt = (int64_t)t * (kBM / 16) + (lane & 7);
      if (t >= a.n_tiles || rt * 16 >= a.Np || nst == 0) return;
      const uint8_t* planes = a.w + (k4 ? a.Np * a.Kp / 2 : a.Np * a.Kp);
      const int64_t at = rt * k128 + kt0;
      if (lane < 8) prefetch_l2_bulk(a.w + at * kStageCodes, (uint32_t)nst * kStageCodes);
      else if (lane < 16) prefetch_l2_bulk(planes + at * kStageScales, (uint32_t)nst * kStageScales);
    };
    call_in(first);
    call_in(first + tstep);
    pdl_wait();                                     // the tokens come from the kernel before this one
    int s = 0, buf = 0;
    uint32_t ph = 0, dph = 0;
    bool ok = true;
    for (int t = first; t < a.n_tiles && ok; t += tstep) {
      call_in(t + 2 * tstep);
      for (int i = 0; i < nst; ++i) {
        if (kCodes || i == 0) {
          // the stage's accumulator is free: the MMA issuer need not ask
          ok = warp_wait(&d_empty[buf], dph ^ 1, abort_flag);
          if (++buf == C::kBufs) { buf = 0; dph ^= 1; }
        }
        if (ok) ok = warp_wait(&empty[s], ph ^ 1, abort_flag);
        if (!ok) break;
        if (elect_one()) {
          uint8_t* to = sA + s * C::kStageBytes + 2 * C::kABytes;
          mbar_expect_tx(&full[s], 2 * C::kBBytes);
          tma_load_2d(to, &tm_x, (kt0 + i) * 2 * kBK, 0, &full[s]);
          tma_load_2d(to + C::kBBytes, &tm_x, (kt0 + i) * 2 * kBK + kBK, 0, &full[s]);
        }
        if (++s == kStages) { s = 0; ph ^= 1; }
      }
    }
    if (!ok) {
      if (lane == 0) report(a.err, 20);
      for (int i = 0; i < kStages; ++i) mbar_wait_quiet(&full[i], 0, 1 << 12);   // copies in flight
      __syncwarp();
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    const uint32_t idesc = make_idesc_f16<T>(kBM, BT);
    const uint64_t desc0 = make_desc_sw128(smem_u32(sA));
    int s = 0, buf = 0;
    uint32_t ph = 0;
    bool ok = true, ready = false;
    for (int t = first; t < a.n_tiles && ok; t += tstep) {
      for (int i = 0; i < nst; ++i) {
        if (!ready && !warp_wait(&full[s], ph, abort_flag)) {
          ok = false;
          break;
        }
        const int ns = s + 1 == kStages ? 0 : s + 1;
        const uint32_t nph = s + 1 == kStages ? ph ^ 1 : ph;
        const bool more = mbar_try_wait(&full[ns], nph);
        tcgen05_fence_after();
        const bool end = kCodes || i == nst - 1;
        if (elect_one()) {
          const uint64_t ad = desc0 + (uint64_t)(s * (C::kStageBytes >> 4)), bd = ad + (2 * C::kABytes >> 4);
          const uint32_t d = tmem_base + buf * C::kBufCols;
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int kk = 0; kk < kBK / 16; ++kk) {
              const bool fresh = kCodes ? (kGroups == 2 || h == 0) && kk == 0 : i == 0 && h == 0 && kk == 0;
              umma_f16(d + (kGroups == 2 ? h * BT : 0), ad + h * (C::kABytes >> 4) + 2 * kk, bd + h * (C::kBBytes >> 4) + 2 * kk,
                       idesc, !fresh);
            }
          umma_commit(&empty[s]);
          if (end) umma_commit(&d_full[buf]);
        }
        ready = __all_sync(0xffffffffu, more);
        s = ns;
        ph = nph;
        if (end && ++buf == C::kBufs) buf = 0;
      }
    }
    if (!ok && lane == 0) report(a.err, 21);
    __syncwarp();
  } else if (warp < 6) {
    // ---------------- fold, exchange, store ----------------
    const int qd = warp & 3;                        // TMEM lane quarter this warp may read
    const int row = qd * 32 + lane;
    const uint8_t* planes = a.w + (k4 ? a.Np * a.Kp / 2 : a.Np * a.Kp);
    const uint16_t* sc16 = reinterpret_cast<const uint16_t*>(planes);
    const float* sc32 = reinterpret_cast<const float*>(planes);
    const T* res = reinterpret_cast<const T*>(a.residual);
    const T* bias = reinterpret_cast<const T*>(a.bias);
    T* out = reinterpret_cast<T*>(a.out);
    const int nfold = kCodes ? nst : (nst > 0 ? 1 : 0);
    int buf = 0, it = 0;
    uint32_t dph = 0;
    bool waited = false, ok = true;
    for (int t = first; t < a.n_tiles && ok; t += tstep, ++it) {
      const int n = t * kBM + row;
      const int64_t srow = ((int64_t)(n >> 4) * k128 + kt0) * (16 * kGroups) + pair_row(row & 15);
      const bool valid = n < a.Np;
      struct Raw { uint32_t d[kGroups]; };
      auto scale_at = [&](int i) {                  // raw scales of stage i of this CTA's share
        Raw x;
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
          x.d[g] = 0;
          if (kCodes && valid && i < nfold) {
            if constexpr (FewFam<WF, CODES>::half_scale) x.d[g] = ldg_nc_u16(sc16 + srow + (i * 2 + g) * 16);
            else x.d[g] = ldg_nc_u32(sc32 + srow + i * 16);
          }
        }
        return x;
      };
      float acc[BT];
#pragma unroll
      for (int j = 0; j < BT; ++j) acc[j] = 0.f;
      Raw sr[3];                                    // of the next stages, on their way
#pragma unroll
      for (int i = 0; i < 3; ++i) sr[i] = scale_at(i);
#pragma unroll 1
      for (int i0 = 0; i0 < nfold && ok; i0 += 3) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          if (i0 + i >= nfold) break;
          ok = warp_wait(&d_full[buf], dph, abort_flag);
          if (!ok) break;
          tcgen05_fence_after();
          float d[kGroups];
#pragma unroll
          for (int g = 0; g < kGroups; ++g) d[g] = group_scale<T, WF, CODES>(sr[i].d[g]);
          sr[i] = scale_at(i0 + i + 3);
          const uint32_t from = tmem_base + (uint32_t(qd * 32) << 16) + buf * C::kBufCols;
          // 32 columns are read back at once (both groups' where they are that few): each time is a chain of 250 clocks
          constexpr int kCols = C::kBufCols < 32 ? C::kBufCols : BT == 64 ? 16 : 32;
#pragma unroll
          for (int c = 0; c < C::kBufCols; c += kCols) {
            float v[kCols];
            tmem_ld_cols<kCols>(from + c, v);
            tmem_ld_done(v);
            if (c + kCols == C::kBufCols) {
              tcgen05_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(&d_empty[buf]);
            }
#pragma unroll
            for (int j = 0; j < kCols; ++j) acc[(c + j) % BT] = fmaf(d[(c + j) / BT], v[j], acc[(c + j) % BT]);
          }
          if (++buf == C::kBufs) { buf = 0; dph ^= 1; }
        }
      }
      if (!ok) break;
      if (a.pairs) {
#pragma unroll
        for (int j = 0; j < BT / 2; ++j) acc[j] = acc[2 * j] + acc[2 * j + 1];
      }
      // ---- parts of the tile: rank q adds up and stores tokens [q * tq, (q + 1) * tq) ----
      const int pb = it & 1;
      const uint32_t pph = (it >> 1) & 1;
      // The buffer is free: whoever sent the parts of tile it - 1, all of which this warp has waited for, had read those of tile
      // it - 2 before.
      if (warp == 2 && elect_one()) mbar_expect_tx(&p_full[pb], (uint32_t)(kSplit * kBM * tq * 4));
      const uint32_t mine = smem_u32(part + (size_t)pb * C::kPart + ((size_t)rank * kBM + row) * tq);
#pragma unroll
      for (int q = 0; q < kSplit; ++q) {
        const uint32_t to = at_rank(mine, q), bar = at_rank(smem_u32(&p_full[pb]), q);
        constexpr int full_q = BT / kSplit, half_q = BT / 2 / kSplit;
        if (!a.pairs) {
#pragma unroll
          for (int j = 0; j < full_q; j += 4)
            st_async4(to + j * 4, bar, acc[q * full_q + j], acc[q * full_q + j + 1], acc[q * full_q + j + 2],
                      acc[q * full_q + j + 3]);
        } else if constexpr (half_q >= 4) {
#pragma unroll
          for (int j = 0; j < half_q; j += 4)
            st_async4(to + j * 4, bar, acc[q * half_q + j], acc[q * half_q + j + 1], acc[q * half_q + j + 2],
                      acc[q * half_q + j + 3]);
        } else {
          st_async2(to, bar, acc[q * half_q], acc[q * half_q + 1]);
        }
      }
      if (!waited) {
        pdl_wait();                                 // out and residual belong to the kernels before this one until here
        waited = true;
      }
      ok = warp_wait<true>(&p_full[pb], pph, abort_flag);
      if (!ok) break;
      const int m0 = (int)rank * tq;
      const float* got = part + (size_t)pb * C::kPart + (size_t)row * tq;
      const float bv = (bias != nullptr && n < a.N) ? to_float(bias[n]) : 0.f;
      const int n_out = a.act != 0 ? (t * kBM + qd * 32) / 2 + (lane & 15) : n;
      const bool writer = a.act != 0 ? (lane < 16 && n_out < a.N / 2) : n < a.N;
#pragma unroll 1
      for (int j = 0; j < tq; ++j) {
        const int m = m0 + j;
        if (m >= a.M) break;
        float f = bv;
#pragma unroll
        for (int q = 0; q < kSplit; ++q) f += got[q * kBM * tq + j];
        if (a.act != 0) {
          const float u = __shfl_down_sync(0xffffffffu, f, 16);
          if (writer) out[(int64_t)m * a.ldo + n_out] = from_float<T>(act_apply(f, a.act) * u);
        } else if (writer) {
          if (res != nullptr) f += to_float(res[(int64_t)m * a.ldr + n]);
          out[(int64_t)m * a.ldo + n] = from_float<T>(f);
        }
      }
      __syncwarp();
    }
    if (!ok && lane == 0) report(a.err, 22);
    __syncwarp();
  } else {
    few_expand<T, BT, WF, CODES>(a, kt0, nst, sA, full, empty, abort_flag, book);
  }
  pdl_launch_dependents();
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();                                   // no CTA leaves while another may still write into it
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

template <typename T, int BT, int WF, bool CODES>
cudaError_t launch_few(const CUtensorMap& tx, const FewArgs& a, cudaStream_t st, bool pdl) {
  using C = FewCfg<BT, WF, CODES>;
  auto kern = gemm_few_kernel<T, BT, WF, CODES>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
  if (e != cudaSuccess) return e;
  // clusters that the device holds at once (its processor groups do not all hold a multiple of kSplit SMs)
  static const int room = [&] {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kSplit);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = C::kSmemBytes;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kSplit;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) n = 32;
    return n;
  }();
  // as few clusters as the same number of rounds needs
  const int rounds = (a.n_tiles + room - 1) / room;
  const int clusters = (a.n_tiles + rounds - 1) / rounds;
  return launch_kernel(kern, dim3(clusters * kSplit), dim3(kThreads), C::kSmemBytes, st, pdl, tx, a);
}

template <typename T, int WF>
cudaError_t dispatch_bt(int bt, const CUtensorMap& tx, const FewArgs& a, cudaStream_t st, bool pdl) {
  constexpr bool fp8 = WF == WF_FP8_E4M3 || WF == WF_FP8_E5M2, codes = WF != WF_ASYM_INT4;
  switch (bt) {
    case 16: return launch_few<T, 16, WF, codes>(tx, a, st, pdl);
    case 32: return launch_few<T, 32, WF, codes>(tx, a, st, pdl);
    default: return a.pairs ? launch_few<T, 64, WF, codes>(tx, a, st, pdl) : launch_few<T, 64, WF, fp8>(tx, a, st, pdl);
  }
}

template <typename T>
cudaError_t dispatch_wf(int wf, int bt, const CUtensorMap& tx, const FewArgs& a, cudaStream_t st, bool pdl) {
  switch (wf) {
    case WF_SYM_INT4: return dispatch_bt<T, WF_SYM_INT4>(bt, tx, a, st, pdl);
    case WF_ASYM_INT4: return dispatch_bt<T, WF_ASYM_INT4>(bt, tx, a, st, pdl);
    case WF_LUT4: return dispatch_bt<T, WF_LUT4>(bt, tx, a, st, pdl);
    case WF_FP8_E4M3: return dispatch_bt<T, WF_FP8_E4M3>(bt, tx, a, st, pdl);
    case WF_FP8_E5M2: return dispatch_bt<T, WF_FP8_E5M2>(bt, tx, a, st, pdl);
    case WF_INT8: return dispatch_bt<T, WF_INT8>(bt, tx, a, st, pdl);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

// out[M, N] = x . W^T (+ bias) (+ residual), or act(gate) * up with N / 2 columns, packed `w` of family `wf`, M <= 64 (32 with
// `pairs`: x then has 2 M rows, value and remainder of each token).  x: row stride ldx (a multiple of 8 elements), 16-byte
// aligned; w 32-byte aligned.
IPEX_API int ipex_gemm_few_tcgen05(const void* x, const void* w, void* out, const void* bias, const void* residual,
                                   const float* lut, int M, int N, int K, int64_t ldx, int64_t ldo, int64_t ldr, int wf,
                                   int act, int pairs, int dtype, int pdl, int* err, void* stream) {
  const int rows = pairs ? 2 * M : M;
  if (M < 1 || rows > 64 || N < 1 || K < 1 || (ldx % 8) != 0) return (int)cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(w) & 31)) return (int)cudaErrorInvalidValue;
  if (dtype != DT_F16 && dtype != DT_BF16) return (int)cudaErrorInvalidValue;
  if (act != 0 && (residual != nullptr || (N % 32) != 0)) return (int)cudaErrorInvalidValue;
  if (wf == WF_LUT4 && lut == nullptr) return (int)cudaErrorInvalidValue;
  const int bt = rows <= 16 ? 16 : rows <= 32 ? 32 : 64;
  const CUtensorMapDataType tdt = dtype == DT_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  CUtensorMap tx;
  if (!tc5::encode_2d_sw128(&tx, tdt, x, (uint64_t)K, (uint64_t)rows, (uint64_t)ldx * 2, kBK, bt)) return -1;
  FewArgs a = {};
  a.w = reinterpret_cast<const uint8_t*>(w); a.lut = lut;
  a.out = out; a.bias = bias; a.residual = residual; a.ldo = ldo; a.ldr = ldr;
  a.Np = ceil_to_i64(N, 16); a.Kp = ceil_to_i64(K, 128);
  a.M = M; a.N = N;
  a.n_tiles = (N + kBM - 1) / kBM;
  a.act = act;
  a.pairs = pairs;
  a.err = err;
  cudaStream_t st = (cudaStream_t)stream;
  return (int)(dtype == DT_F16 ? dispatch_wf<__half>(wf, bt, tx, a, st, pdl != 0)
                               : dispatch_wf<__nv_bfloat16>(wf, bt, tx, a, st, pdl != 0));
}
