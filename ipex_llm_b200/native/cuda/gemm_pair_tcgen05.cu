// Products with many token rows on pairs of SMs (tcgen05, cta_group::2):
//     out[M, N] = x[M, K] . W[N, K]^T  (+ bias) (+ residual)   or   act(gate) * up  for interleaved gate/up rows
// with W dense fp16 / bf16 or packed low-bit tiles that are expanded inside the kernel.
//
// What bounds it: the tensor pipe, if the operands arrive.  On one SM a 128 x 256 tile needs 32 KB of tokens per 64 k, 64
// bytes a clock at the full rate, which is all that L2 gives an SM; and the packed weights have to be expanded at 16 values a
// clock.  A pair works on 256 weight rows x BT tokens: each SM expands (or loads) its own 128 rows and fetches half of the
// tokens, the instruction reads both halves, so the token traffic is halved.  Weight rows sit on the MMA's M side
// (D[TMEM lane = weight row][TMEM column = token]).
//
// One persistent CTA per SM, two to a cluster; roles by warp:
//   warp 0       one lane issues the TMA loads of this SM's half of the token tile (and of its weight rows when dense);
//   warp 1       allocates TMEM; in the leading CTA one lane issues tcgen05.mma and commits: a commit releases the stage in
//                both CTAs, the last one of a tile hands the accumulator to both epilogues;
//   warps 2..5   epilogue: tcgen05.ld, bias / residual / activation, store.  Two accumulators alternate in TMEM, so the
//                epilogue of a tile overlaps the main loop of the next;
//   warps 6..17  (packed weights) three teams of four expand units of 128 k in turn (a lane owns a weight row), so that a
//                team has the time of six stages for the loads, arithmetic, stores and proxy fences of two; the next
//                unit's bytes are already on their way to registers when a unit is begun, across tiles too.
// All barriers that the MMA issuer waits for live in the leading CTA; the other CTA's expanders count bytes there (send_token),
// its epilogue arrives there remotely.  Waits for what another CTA of the cluster says acquire at cluster scope.
// Every mbarrier wait is bounded; on expiry a role raises its CTA's abort flag, records a code in the error flag
// (16 loader, 17 MMA issuer, 18 epilogue, 19 dequantizer) and leaves its loop; the CTAs meet before TMEM is released.
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

constexpr int kBM = 128;      // weight rows of one CTA (the pair's tile has twice as many)
constexpr int kBK = 64;       // k per stage: one 128-byte swizzle row
constexpr int kTeamThreads = 128;   // one weight row each
constexpr int kTeams = 3;

struct PairArgs {
  const uint8_t* w;
  const float* lut;
  void* out;
  const void* bias;
  const void* residual;
  int64_t ldo, ldr;
  int64_t Np, Kp;
  int M, N, K;
  int m_tiles, n_tiles;   // token tiles of BT, weight tiles of 256 rows
  int act;
  int* err;
  const int* m_range;     // device: (first row, rows) of x and out that this launch covers, or null for all M
};

template <int WF> struct PairFam {
  static constexpr bool dense = WF == WF_F16 || WF == WF_BF16;
  static constexpr bool four_bit = WF == WF_SYM_INT4 || WF == WF_ASYM_INT4 || WF == WF_LUT4;
  static constexpr int threads = 192 + (dense ? 0 : kTeams * kTeamThreads);
};

template <int BT> struct PairCfg {
  static constexpr int kABytes = kBM * kBK * 2;
  static constexpr int kBBytes = BT / 2 * kBK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kStages = BT >= 256 ? 6 : 8;      // even, and at least four (two units in flight)
  static constexpr int kTmemCols = 2 * BT;
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*alignment*/ + 256 /*barriers*/ + 1024 /*pair table*/;
};

// ---- two-CTA forms ------------------------------------------------------------------------------------------------
// 16 bytes of this CTA's shared memory to the leading CTA, counted by a barrier there.  This is how the other CTA says that a
// stage is filled: an arrival released at cluster scope waits some 1400 clocks for itself (by the thread that filled the stage
// 1024 x 12288 x 4096 int4 77 -> 95 us, by a warp that does nothing else 172), while the copy runs behind the proxy fence by
// itself, and completes with a release at that scope.
constexpr uint32_t kTokenBytes = 16;
__device__ __forceinline__ void send_token(uint32_t to, const void* from, uint32_t leader_bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(to),
               "r"(smem_u32(from)), "r"(kTokenBytes), "r"(leader_bar)
               : "memory");
}
// Tile load into this CTA's shared memory whose bytes are counted by a barrier of the leading CTA.
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* tm, int x, int y, uint32_t leader_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(leader_bar)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* slot_in_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot_in_smem)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                              bool accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"((uint32_t)accumulate)
      : "memory");
}
// One arrival at this barrier of both CTAs when every MMA issued so far has finished.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"((uint16_t)3)
      : "memory");
}
// 32 lanes x 16 columns
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ---- dequantizers: fill the weight operand of every stage for this CTA's tiles ---------------------------------------
template <typename T, int BT, int WF>
__device__ __forceinline__ void expand_role(const PairArgs& a, uint8_t* sA, uint64_t* full, uint64_t* empty,
                                            volatile int* abort_flag, const uint32_t* lut2, uint32_t token) {
  using C = PairCfg<BT>;
  using V = V2<T>;
  constexpr bool k4 = PairFam<WF>::four_bit;
  constexpr int kSub = k4 ? 2 : 1;                 // stages that one unit feeds
  constexpr int kStep = kTeams * kSub;
  static_assert(C::kStages % kSub == 0 && kStep <= C::kStages, "a wait looks at most one phase ahead");
  const int dt = threadIdx.x - 192;
  const int team = dt / kTeamThreads;
  const int r = dt % kTeamThreads;                 // weight row of this CTA's tile
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cta_rank();
  const int ntiles = a.m_tiles * a.n_tiles, tstep = gridDim.x >> 1;
  // one unit = 64 bytes of this thread's row: a 128-wide k tile of 4-bit codes, a 64-wide one of bytes
  const int units = k4 ? (int)(a.Kp / 128) : (int)(a.Kp / 64);
  const uint8_t* planes = a.w + (k4 ? a.Np * a.Kp / 2 : a.Np * a.Kp);
  const uint16_t* sc16 = reinterpret_cast<const uint16_t*>(planes);
  const float* sc32 = reinterpret_cast<const float*>(planes);
  const uint16_t* mins = sc16 + a.Np * (a.Kp / 64);
  const int prow = pair_row(r & 15);
  const uint32_t full0 = at_rank(smem_u32(full), 0);

  // where the next load stands: tile, unit, and the row it belongs to
  int lt = blockIdx.x >> 1, lu = team;
  int64_t rt = 0;
  bool valid = false;
  const uint8_t* wrow = nullptr;
  auto seat = [&]() {
    while (lu >= units) {
      lu -= units;
      lt += tstep;
    }
    if (lt < ntiles) {
      const int64_t rg = ((int64_t)(lt / a.m_tiles) * 2 + rank) * kBM + r;
      valid = rg < a.Np;
      rt = valid ? (rg >> 4) : 0;
      wrow = a.w + rt * units * 1024 + (r & 15) * 64;
    } else {
      valid = false;
    }
  };
  // raw bits only: a conversion here would wait for the load
  struct Unit { uint4 q[4]; uint32_t d0, d1, m0, m1; };
  auto load = [&](Unit& n) {
    n.q[0] = n.q[1] = n.q[2] = n.q[3] = make_uint4(0, 0, 0, 0);
    n.d0 = n.d1 = n.m0 = n.m1 = 0;
    if (!valid) return;
    ldg_nc_32b(wrow + (int64_t)lu * 1024, n.q[0], n.q[1]);
    ldg_nc_32b(wrow + (int64_t)lu * 1024 + 32, n.q[2], n.q[3]);
    if constexpr (k4) {
      const int64_t si = ((rt * units + lu) * 2) * 16 + prow;
      n.d0 = ldg_nc_u16(sc16 + si);
      n.d1 = ldg_nc_u16(sc16 + si + 16);
      if constexpr (WF == WF_ASYM_INT4) {
        n.m0 = ldg_nc_u16(mins + si);
        n.m1 = ldg_nc_u16(mins + si + 16);
      }
    } else if constexpr (WF == WF_INT8) {
      n.d0 = ldg_nc_u16(sc16 + (rt * units + lu) * 16 + prow);
    } else {
      n.d0 = ldg_nc_u32(sc32 + (rt * (a.Kp / 128) + (lu >> 1)) * 16 + prow);
    }
  };
  auto scale = [](uint32_t raw) {
    if constexpr (k4 || WF == WF_INT8) return __half2float(__ushort_as_half((uint16_t)raw));
    else return __uint_as_float(raw) * Fp8Place<T, WF>::mul;
  };

  const int my_tiles = (int)(blockIdx.x >> 1) < ntiles ? (ntiles - (int)(blockIdx.x >> 1) + tstep - 1) / tstep : 0;
  const int total = my_tiles * units;              // units of all this CTA's tiles, in the order of the stages
  int s = team * kSub;
  uint32_t ph = 0;
  while (s >= C::kStages) { s -= C::kStages; ph ^= 1; }
  bool ok = true;
  Unit next;
  seat();
  load(next);
#pragma unroll 1
  for (int u = team; u < total; u += kTeams) {
    const Unit cur = next;
    lu += kTeams;
    seat();
    load(next);
#pragma unroll
    for (int g = 0; g < kSub; ++g) {
      Scale<T> sc;
      sc.d = V::splat(scale(g == 0 ? cur.d0 : cur.d1));
      if constexpr (WF == WF_ASYM_INT4) sc.m = V::splat(scale(g == 0 ? cur.m0 : cur.m1));
      if (ok && !warp_wait<true>(&empty[s + g], ph ^ 1, abort_flag)) {
        if (lane == 0) report(a.err, 19);
        ok = false;
      }
      uint8_t* row = sA + (s + g) * C::kABytes + r * 128;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const uint4 q = cur.q[t];
        uint4 lo, hi;
        if constexpr (k4) {
          // uint4 = [group 0: k 16t..16t+7 | 16t+8..16t+15 | group 1: same]
          lo = expand4<T, WF>(g == 0 ? q.x : q.z, sc, lut2);
          hi = expand4<T, WF>(g == 0 ? q.y : q.w, sc, lut2);
        } else {
          lo = expand8<T, WF>(q.x, q.y, sc);
          hi = expand8<T, WF>(q.z, q.w, sc);
        }
        if (ok) {
          *reinterpret_cast<uint4*>(row + (((2 * t) ^ (r & 7)) << 4)) = lo;      // 16-byte chunk = 8 consecutive k
          *reinterpret_cast<uint4*>(row + (((2 * t + 1) ^ (r & 7)) << 4)) = hi;
        }
      }
      // one proxy fence and one arrival for the team, behind a barrier that orders its stores before them (a warp whose wait
      // ran out still attends)
      asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "n"(kTeamThreads) : "memory");
      if (r == 0 && ok) {
        fence_proxy_async_smem();
        if (rank == 0) mbar_arrive(&full[s + g]);
        else send_token(token, sA + (s + g) * C::kABytes, full0 + (s + g) * 8);
      }
    }
    s += kStep;
    while (s >= C::kStages) {
      s -= C::kStages;
      ph ^= 1;
    }
  }
}

template <typename T, int BT, int WF>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PairFam<WF>::threads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, PairArgs a) {
  using C = PairCfg<BT>;
  constexpr bool kDense = PairFam<WF>::dense;
  int row0 = 0;
  if (!kDense && a.m_range != nullptr) {
    row0 = a.m_range[0];
    a.M = a.m_range[1];
    a.m_tiles = (a.M + BT - 1) / BT;
    a.out = reinterpret_cast<T*>(a.out) + (int64_t)row0 * a.ldo;
  }
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + C::kStages * C::kABytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::kStages * C::kStageBytes);   // used in the leading CTA
  uint64_t* empty = full + C::kStages;
  uint64_t* acc_full = empty + C::kStages;
  uint64_t* acc_empty = acc_full + 2;                                                 // used in the leading CTA
  uint64_t* token = acc_empty + 2;                                                    // written in the leading CTA, never read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(token + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint32_t* lut2 = reinterpret_cast<uint32_t*>(smem + C::kStages * C::kStageBytes + 256);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t rank = cta_rank();
  const int first = blockIdx.x >> 1, tstep = gridDim.x >> 1;
  const int ntiles = a.m_tiles * a.n_tiles;
  const int kblocks = kDense ? (a.K + kBK - 1) / kBK : (int)(a.Kp / kBK);

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(&full[s], kDense ? 1 : 2);                             // the loader, and the leading CTA's team
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 8);                                   // the epilogue warps of both CTAs
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if constexpr (WF == WF_LUT4) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {
      const T lo = from_float<T>(a.lut[i & 15]), hi = from_float<T>(a.lut[i >> 4]);
      lut2[i] = (uint32_t)(*reinterpret_cast<const uint16_t*>(&lo)) |
                ((uint32_t)(*reinterpret_cast<const uint16_t*>(&hi)) << 16);
    }
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, C::kTmemCols);
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();          // barriers and TMEM of both CTAs are ready
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ---------------- loader ----------------
    if (elect_one()) {
      if constexpr (kDense) prefetch_tmap(&tm_w);
      prefetch_tmap(&tm_x);
    }
    const uint32_t full0 = at_rank(smem_u32(full), 0);
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int t = first; t < ntiles && ok; t += tstep) {
      const int nb = t / a.m_tiles, mb = t % a.m_tiles;
      for (int kb = 0; kb < kblocks; ++kb) {
        if (!warp_wait<true>(&empty[s], ph ^ 1, abort_flag)) {
          ok = false;
          break;
        }
        if (elect_one()) {
          // the leader expects the bytes of both CTAs; the other's may land first, the phase still waits for the arrivals
          if (rank == 0) mbar_expect_tx(&full[s], kDense ? 2 * C::kStageBytes : 2 * C::kBBytes + kTokenBytes);
          if constexpr (kDense)
            tma_load_2d_pair(sA + s * C::kABytes, &tm_w, kb * kBK, (nb * 2 + (int)rank) * kBM, full0 + s * 8);
          tma_load_2d_pair(sB + s * C::kBBytes, &tm_x, kb * kBK, row0 + mb * BT + (int)rank * (BT / 2), full0 + s * 8);
        }
        if (++s == C::kStages) { s = 0; ph ^= 1; }
      }
    }
    if (!ok) {
      // leaving early: give the copies already issued a bounded time to land before the CTA exits
      if (lane == 0) report(a.err, 16);
      if (rank == 0)
        for (int i = 0; i < C::kStages; ++i) mbar_wait_quiet(&full[i], 0, 1 << 12);
      else
        __nanosleep(1000000);
      __syncwarp();
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leading CTA) ----------------
    if (rank == 0) {
      const uint32_t idesc = make_idesc_f16<T>(2 * kBM, BT);
      const uint64_t adesc0 = make_desc_sw128(smem_u32(sA)), bdesc0 = make_desc_sw128(smem_u32(sB));
      int s = 0;
      uint32_t ph = 0;
      int it = 0;
      bool ok = true;
      for (int t = first; t < ntiles && ok; t += tstep, ++it) {
        const int acc = it & 1;
        const uint32_t acc_ph = (it >> 1) & 1;
        ok = warp_wait<true>(&acc_empty[acc], acc_ph ^ 1, abort_flag);
        tcgen05_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BT;
        for (int kb = 0; kb < kblocks && ok; ++kb) {
          if (!warp_wait<true>(&full[s], ph, abort_flag)) {
            ok = false;
            break;
          }
          tcgen05_fence_after();
          if (elect_one()) {
            const uint64_t adesc = adesc0 + (uint64_t)(s * (C::kABytes >> 4)), bdesc = bdesc0 + (uint64_t)(s * (C::kBBytes >> 4));
#pragma unroll
            for (int kk = 0; kk < kBK / 16; ++kk)   // +32 bytes along K inside the swizzle row = +2 in (address >> 4)
              umma_f16_pair(d_tmem, adesc + 2 * kk, bdesc + 2 * kk, idesc, (kb | kk) != 0);
            umma_commit_pair(&empty[s]);
            if (kb == kblocks - 1) umma_commit_pair(&acc_full[acc]);
          }
          __syncwarp();
          if (++s == C::kStages) { s = 0; ph ^= 1; }
        }
      }
      if (!ok && lane == 0) report(a.err, 17);
    }
    __syncwarp();
  } else if (warp < 6) {
    // ---------------- epilogue ----------------
    const int qd = warp & 3;  // TMEM lane quarter this warp may read
    T* out = reinterpret_cast<T*>(a.out);
    const T* res = reinterpret_cast<const T*>(a.residual);
    const T* bias = reinterpret_cast<const T*>(a.bias);
    const uint32_t acc_empty0 = at_rank(smem_u32(acc_empty), 0);
    int it = 0;
    for (int t = first; t < ntiles; t += tstep, ++it) {
      const int nb = t / a.m_tiles, mb = t % a.m_tiles;
      const int acc = it & 1;
      const uint32_t acc_ph = (it >> 1) & 1;
      const int nw = (nb * 2 + (int)rank) * kBM + qd * 32;    // first weight row of the warp
      const int n = nw + lane;
      const float bv = (bias != nullptr && n < a.N) ? to_float(bias[n]) : 0.f;
      // activation mode: lanes 0..15 hold gate rows, lanes 16..31 the matching up rows; 16 outputs per warp
      const int n_out = a.act != 0 ? nw / 2 + (lane & 15) : n;
      const bool writer = a.act != 0 ? (lane < 16 && n_out < a.N / 2) : (n < a.N);
      if (!warp_wait<true>(&acc_full[acc], acc_ph, abort_flag)) {
        if (lane == 0) report(a.err, 18);
        break;
      }
      tcgen05_fence_after();
#pragma unroll 1
      for (int c = 0; c < BT / 16; ++c) {
        const int m0 = mb * BT + c * 16;
        if (m0 >= a.M) break;
        uint32_t v[16];
        T rv[16];
        if (res != nullptr) {
          // all of the chunk's residuals are requested before the accumulators are read
#pragma unroll
          for (int j = 0; j < 16; ++j) rv[j] = (writer && m0 + j < a.M) ? res[(int64_t)(m0 + j) * a.ldr + n] : T(0.f);
        }
        tmem_ld_32x16(tmem_base + (uint32_t(qd * 32) << 16) + acc * BT + c * 16, v);
        if (a.act != 0) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float g = __uint_as_float(v[j]) + bv;
            const float u = __shfl_down_sync(0xffffffffu, g, 16);
            const int m = m0 + j;
            if (writer && m < a.M) out[(int64_t)m * a.ldo + n_out] = from_float<T>(act_apply(g, a.act) * u);
          }
        } else if (writer) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int m = m0 + j;
            if (m < a.M) {
              float f = __uint_as_float(v[j]) + bv;
              if (res != nullptr) f += to_float(rv[j]);
              out[(int64_t)m * a.ldo + n] = from_float<T>(f);
            }
          }
        }
      }
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(acc_empty0 + acc * 8);
    }
  } else {
    if constexpr (!kDense) expand_role<T, BT, WF>(a, sA, full, empty, abort_flag, lut2, at_rank(smem_u32(token), 0));
  }
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();          // no CTA leaves, or gives its TMEM back, while the other may still arrive or multiply
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc_pair(tmem_base, C::kTmemCols);
  }
}

template <typename T, int BT, int WF>
cudaError_t launch_pair(const CUtensorMap& tw, const CUtensorMap& tx, const PairArgs& a, int sms, cudaStream_t st) {
  using C = PairCfg<BT>;
  auto kern = gemm_pair_kernel<T, BT, WF>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
  if (e != cudaSuccess) return e;
  const int ntiles = a.m_tiles * a.n_tiles;
  const int pairs = ntiles < sms / 2 ? ntiles : sms / 2;
  kern<<<2 * pairs, PairFam<WF>::threads, C::kSmemBytes, st>>>(tw, tx, a);
  return cudaGetLastError();
}

template <typename T, int WF>
cudaError_t dispatch_bt(int bt, const CUtensorMap& tw, const CUtensorMap& tx, const PairArgs& a, int sms,
                        cudaStream_t st) {
  return bt == 128 ? launch_pair<T, 128, WF>(tw, tx, a, sms, st) : launch_pair<T, 256, WF>(tw, tx, a, sms, st);
}

template <typename T>
cudaError_t dispatch_wf(int wf, int bt, const CUtensorMap& tw, const CUtensorMap& tx, const PairArgs& a, int sms,
                        cudaStream_t st) {
  switch (wf) {
    case WF_SYM_INT4: return dispatch_bt<T, WF_SYM_INT4>(bt, tw, tx, a, sms, st);
    case WF_ASYM_INT4: return dispatch_bt<T, WF_ASYM_INT4>(bt, tw, tx, a, sms, st);
    case WF_LUT4: return dispatch_bt<T, WF_LUT4>(bt, tw, tx, a, sms, st);
    case WF_FP8_E4M3: return dispatch_bt<T, WF_FP8_E4M3>(bt, tw, tx, a, sms, st);
    case WF_FP8_E5M2: return dispatch_bt<T, WF_FP8_E5M2>(bt, tw, tx, a, sms, st);
    case WF_INT8: return dispatch_bt<T, WF_INT8>(bt, tw, tx, a, sms, st);
    case WF_F16:
    case WF_BF16: return dispatch_bt<T, WF_F16>(bt, tw, tx, a, sms, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

// Rows [m_range[0], m_range[0] + m_range[1]) (device memory) of x [M, K] when m_range is given, with a grid for m_upper rows.
static int pair_entry(const void* x, const void* w, void* out, const void* bias, const void* residual, const float* lut,
                      const int* m_range, int m_upper, int M, int N, int K, int64_t ldx, int64_t ldw, int64_t ldo,
                      int64_t ldr, int wf, int act, int dtype, int bt, int* err, void* stream) {
  const bool dense = wf == WF_F16 || wf == WF_BF16;
  if (M < 1 || N < 1 || K < 1 || (ldx % 8) != 0 || (bt != 128 && bt != 256)) return (int)cudaErrorInvalidValue;
  if (reinterpret_cast<uintptr_t>(x) & 15) return (int)cudaErrorInvalidValue;
  if (reinterpret_cast<uintptr_t>(w) & (dense ? 15 : 31)) return (int)cudaErrorInvalidValue;
  if (dense && (ldw % 8) != 0) return (int)cudaErrorInvalidValue;
  if (dtype != DT_F16 && dtype != DT_BF16) return (int)cudaErrorInvalidValue;
  if (act != 0 && (residual != nullptr || (N % 32) != 0)) return (int)cudaErrorInvalidValue;
  if (wf == WF_LUT4 && lut == nullptr) return (int)cudaErrorInvalidValue;
  const CUtensorMapDataType tdt = dtype == DT_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  CUtensorMap tx, tw;
  if (!tc5::encode_2d_sw128(&tx, tdt, x, (uint64_t)K, (uint64_t)M, (uint64_t)ldx * 2, kBK, bt / 2)) return -1;
  tw = tx;
  if (dense && !tc5::encode_2d_sw128(&tw, tdt, w, (uint64_t)K, (uint64_t)N, (uint64_t)ldw * 2, kBK, kBM)) return -1;
  PairArgs a = {};
  a.w = reinterpret_cast<const uint8_t*>(w); a.lut = lut;
  a.out = out; a.bias = bias; a.residual = residual; a.ldo = ldo; a.ldr = ldr;
  a.Np = ceil_to_i64(N, 16); a.Kp = ceil_to_i64(K, 128);
  a.M = m_upper; a.N = N; a.K = K;
  a.m_range = m_range;
  a.m_tiles = (m_upper + bt - 1) / bt;
  a.n_tiles = (N + 2 * kBM - 1) / (2 * kBM);
  a.act = act;
  a.err = err;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaStream_t st = (cudaStream_t)stream;
  return (int)(dtype == DT_F16 ? dispatch_wf<__half>(wf, bt, tw, tx, a, sms, st)
                               : dispatch_wf<__nv_bfloat16>(wf, bt, tw, tx, a, sms, st));
}

// The product of ipex_gemm_lowbit_tcgen05 (packed `w`) or ipex_gemm_tcgen05_act (dense `w`, row stride ldw) on SM pairs.
// `bt`: token tile, 128 or 256.  Arguments as checked there.
IPEX_API int ipex_gemm_pair_tcgen05(const void* x, const void* w, void* out, const void* bias, const void* residual,
                                    const float* lut, int M, int N, int K, int64_t ldx, int64_t ldw, int64_t ldo,
                                    int64_t ldr, int wf, int act, int dtype, int bt, int* err, void* stream) {
  return pair_entry(x, w, out, bias, residual, lut, nullptr, M, M, N, K, ldx, ldw, ldo, ldr, wf, act, dtype, bt, err, stream);
}

// One expert's product of ipex_gemm_lowbit_tcgen05_grouped on SM pairs.
IPEX_API int ipex_gemm_pair_tcgen05_grouped(const void* x, const void* w, void* out, const float* lut, const int* m_range,
                                            int M_total, int m_upper, int N, int K, int64_t ldx, int64_t ldo, int wf, int act,
                                            int dtype, int bt, int* err, void* stream) {
  return pair_entry(x, w, out, nullptr, nullptr, lut, m_range, m_upper, M_total, N, K, ldx, 0, ldo, 0, wf, act, dtype, bt, err,
                    stream);
}
