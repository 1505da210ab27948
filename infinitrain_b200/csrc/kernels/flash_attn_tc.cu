// Flash attention forward and backward on the 5th-generation tensor cores (tcgen05, accumulators
// in TMEM, operands staged by TMA), causal or full, grouped-query heads, head size 64 or 128.
//
// Backward: one CTA owns 128 keys of one KV head and walks over the 128-row query tiles (and the query heads
// of the group) that attend to them.  Per tile, with n = key row, m = query row, d = head column:
//
//   S^T[n,m]  = K[n,:] . Q[m,:]            tcgen05.mma  K (K-major)  x Q (K-major)   -> TMEM cols 0..127
//   dP^T[n,m] = V[n,:] . dO[m,:]           tcgen05.mma  V            x dO            -> TMEM cols 128..255
//   P^T  = exp2(S^T c - lse[m])            8 warps, half a key row per thread; bf16 over the spent S^T in TMEM
//   dV[n,d] += P^T[n,m]  dO[m,d]           tcgen05.mma  P^T (from TMEM) x dO (MN-major) -> TMEM cols 256..
//   dS^T = P^T (dP^T - delta[m])           the same warps; bf16 to shared memory in the swizzled operand layout
//   dQ[m,d]  = dS[m,n]   K[n,d]            tcgen05.mma  dS^T read MN-major x K (MN-major) -> TMEM; four warps of
//                                          their own read it out and add it to the fp32 dQ buffer by TMA
//   dK[n,d] += dS^T[n,m] Q[m,d]            tcgen05.mma  dS^T (K-major) x Q  (MN-major) -> TMEM cols 256+D..
//
// The softmax warps, the tensor core and the dQ read-out each work on a different part of the chain: the MMA
// thread issues dV(i) and S(i+1) when P(i) is there, dP(i+1), dQ(i) and dK(i) when dS(i) is there, so S(i+1) is
// computed under the dS phase of tile i, dP(i+1) under the P phase of tile i+1, and dQ(i) is read out meanwhile.
// MMAs complete in the order of issue, so s_full(i+1) says that dV(i) has read P(i).  With head size 64 dQ has
// TMEM columns of its own; with head size 128 it takes the spent dP's, so dP(i+1) comes after dQ(i) and waits for
// its read-out.
//
// What bounds it: the exponentials (16 per cycle and SM: 1024 cycles a tile) and the five contractions (1280
// cycles a tile at head size 64, 2560 at 128).
// Measured (this kernel alone, causal): 16 x 1024 tokens, 12 heads of 64: 280 us when one warp set walked the whole
// chain of a tile, one CTA per key tile; 147 us now.  1 x 8192, 32 query and 8 KV heads of 128: 3018 -> 1435 us.
// 1 x 2048, 32 / 8 heads of 64: 292 -> 75 us.  A tile takes 3260 cycles at head size 64 and 5000 at 128, where shared
// memory is busy most of the time: 288 KB of operands, 128 KB for dQ's way out and 96 KB of loads and dS a tile at
// 128 bytes a cycle are 4100 cycles.
//
// Every wait is bounded; a wait that gives up records a code in the status word and the CTA drains without
// touching the tensor pipe again.
//
// The reference composes attention from batched cuBLAS matmuls, a mask and a 3-pass softmax and
// lets autograd differentiate them (infini_train/src/nn/modules/transformer/causal_self_attention.cc:86-130).
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <float.h>
#include <math.h>
#include <stdint.h>

#include "../common/ptx.cuh"
#include "kernels.h"

namespace itb {

int make_tmap_bf16_3d(CUtensorMap* map, const void* ptr, uint64_t inner, uint64_t d1, uint64_t d2,
                      uint64_t ld1, uint64_t ld2, uint32_t box_inner, uint32_t box_d1);

int make_tmap_f32_3d(CUtensorMap* map, const void* ptr, uint64_t inner, uint64_t d1, uint64_t d2,
                     uint64_t ld1, uint64_t ld2, uint32_t box_d1);

namespace fatc {

constexpr int kThreads = 512;     // 8 softmax warps, 4 dQ read-out warps, TMA warp, MMA warp, two idle warps
constexpr int kAtom = 128 * 128;   // bytes of one [128 rows][64 x bf16] swizzled block
constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void readout_warps_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

__device__ __forceinline__ uint4 pack8(const float* v) {
  uint4 u;
  __nv_bfloat162* b2 = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int e = 0; e < 4; ++e) b2[e] = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
  return u;
}

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

template <int D>
struct BwdCfg {
  static constexpr int kAtoms = D / 64;
  static constexpr int kTile = kAtoms * kAtom;          // one [128][D] bf16 tile
  static constexpr int kdOStages = D == 64 ? 2 : 1;     // dO(i) is spent at dV(i), early enough for one stage
  static constexpr int kKvStages = D == 64 ? 2 : 1;     // head size 64 has room to load the next item's K and V early
  static constexpr int kOffK = 0;
  static constexpr int kOffV = kTile;                        // stage s of K and V: 2 * kTile * s further
  static constexpr int kOffQ = 2 * kKvStages * kTile;        // two stages: S(i+1) is issued before dK(i)
  static constexpr int kOffdO = kOffQ + 2 * kTile;
  static constexpr int kOffdS = kOffdO + kdOStages * kTile;  // [2 m-chunks][128 n][64 m]
  static constexpr int kOffStage = kOffdS + 2 * kAtom;       // dQ on its way out: two fp32 [128][32] blocks
  static constexpr int kOffStat = kOffStage + 2 * kAtom;     // lse*log2e [2][128], delta [2][128]
  static constexpr int kOffBar = kOffStat + 4 * 128 * 4;
  static constexpr int kSmem = kOffBar + 22 * 8 + 16;
  static_assert(kSmem <= 232448, "shared memory of one SM");
};

// What the roles of a CTA walk over: items of (128 keys, KV head, share of its query tiles, batch), each with the
// (query head of the group, query tile) pairs that meet its keys.
//
// The pairs of one key tile and KV head are dealt out to `nparts` items in turn (a.bwd_parts > 1 when whole ones
// would leave SMs idle: few key tiles, one KV head per rank under tensor parallelism); each then writes its dK / dV
// to a slab of fp32 scratch of its own.  With a causal mask the items of the first keys have the most
// tiles: items are ordered by that and dealt out to the CTAs to and fro, so that each gets about the same.
struct BwdItems {
  int nparts, width, total, n_qblocks, G;
  int causal;
  int k;                                  // round of the dealing
  int nb, hk, part, b, iters, mb_first, per_head;
  __device__ explicit BwdItems(const ItbAttnArgs& a) {
    nparts = a.bwd_parts > 1 ? a.bwd_parts : 1;
    width = a.KV * nparts;
    n_qblocks = (a.T + 127) / 128;
    total = n_qblocks * width * a.B;
    G = a.H / a.KV;
    causal = a.causal;
    B = a.B;
    k = -1;
  }
  // the next item of this CTA that has tiles
  __device__ bool next() {
    for (;;) {
      ++k;
      const int base = k * static_cast<int>(gridDim.x);
      if (base >= total) return false;
      const int i = base + static_cast<int>((k & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
      if (i >= total) continue;
      nb = i / (width * B);
      const int r = i % (width * B);
      b = r / width;
      hk = (r % width) / nparts;
      part = r % nparts;
      mb_first = causal ? nb : 0;
      per_head = n_qblocks - mb_first;
      const int pairs = per_head * G;
      iters = pairs > part ? (pairs - part + nparts - 1) / nparts : 0;
      if (iters > 0) return true;
    }
  }
  __device__ void tile(int it, int& h, int& mb) const {
    const int g = part + it * nparts;
    h = hk * G + g / per_head;
    mb = mb_first + g % per_head;
  }
  int B;
};

// Persistent: one CTA per SM; the next item's loads, S and dP run under the last tiles of the one before.  Tiles
// and items are numbered through (n, c), which gives every barrier its parity.
template <int D>
__global__ void __launch_bounds__(kThreads, 1)
flash_bwd_tc_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                    const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap tdo,
                    const __grid_constant__ CUtensorMap tdq, const ItbAttnArgs a, int* err) {
  using Cfg = BwdCfg<D>;
  constexpr int SO = Cfg::kdOStages;
  extern __shared__ __align__(1024) uint8_t smem[];
  // the swizzled tiles need a 1024-byte boundary; there is no room left to round up at head size 128
  if (smem_u32(smem) & 1023) {
    if (threadIdx.x == 0) atomicCAS(err, 0, 200);
    return;
  }
  float* s_lse = reinterpret_cast<float*>(smem + Cfg::kOffStat);
  float* s_delta = s_lse + 2 * 128;
  constexpr int SK = Cfg::kKvStages;
  uint64_t* kv_full = reinterpret_cast<uint64_t*>(smem + Cfg::kOffBar);
  uint64_t* kv_empty = kv_full + 2;
  uint64_t* q_full = kv_empty + 2;      // Q tile and the statistics of its rows
  uint64_t* q_empty = q_full + 2;
  uint64_t* do_full = q_empty + 2;
  uint64_t* do_empty = do_full + 2;
  uint64_t* s_full = do_empty + 2;
  uint64_t* dp_full = s_full + 1;
  uint64_t* p_full = dp_full + 1;
  uint64_t* ds_full = p_full + 1;
  uint64_t* dq_full = ds_full + 1;
  uint64_t* dq_drained = dq_full + 1;
  uint64_t* acc_full = dq_drained + 1;      // dK and dV of an item
  uint64_t* acc_drained = acc_full + 1;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_drained + 1);
  volatile uint32_t* abort_flag = tmem_holder + 1;

  const int warp = __shfl_sync(~0u, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&kv_full[s], 1);
      mbar_init(&kv_empty[s], 1);
      mbar_init(&q_full[s], 2);
      mbar_init(&q_empty[s], 1);
      mbar_init(&do_full[s], 1);
      mbar_init(&do_empty[s], 1);
    }
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_full, 8);
    mbar_init(ds_full, 8);
    mbar_init(dq_full, 1);
    mbar_init(dq_drained, 4);
    mbar_init(acc_full, 1);
    mbar_init(acc_drained, 8);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 13) {
    tmem_alloc(tmem_holder, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_holder;
  const uint32_t tm_S = tmem_base, tm_dP = tmem_base + 128, tm_dV = tmem_base + 256, tm_dK = tmem_base + 256 + D;
  constexpr bool kAlias = D > 64;     // no TMEM columns left for dQ: it goes over the spent dP^T
  const uint32_t tm_dQ = kAlias ? tm_dP : tmem_base + 256 + 2 * D;
  // with columns to spare dS^T goes to TMEM too, as dK's operand: 32 KB less to read from shared memory a tile
  constexpr bool kTmemdS = !kAlias;
  const uint32_t tm_dS = tmem_base + 256 + 3 * D;
  auto give_up = [&](int code) {
    atomicCAS(err, 0, code);
    *abort_flag = 1;
  };
  auto wait = [&](uint64_t* bar, uint32_t parity) { return mbar_wait_warp(bar, parity & 1, abort_flag); };
  BwdItems item(a);

  // 512 threads of 128 registers at the launch, 128 x (2 x 144 + 168 + 56) after the split
  if (warp >= 12) {
    regs_shrink<56>();
    if (warp == 12) {
      // ---------------------------------------------------------------- TMA producer
      if (lane == 0) {
        tma_prefetch_desc(&tq);
        tma_prefetch_desc(&tk);
        tma_prefetch_desc(&tv);
        tma_prefetch_desc(&tdo);
      }
      bool ok = true;
      uint32_t n = 0;
      for (uint32_t c = 0; ok && item.next(); ++c) {
        const int sk = c % SK;
        ok = wait(&kv_empty[sk], c / SK + 1);
        if (!ok) break;
        if (lane == 0) {
          uint8_t* kv = smem + Cfg::kOffK + sk * 2 * Cfg::kTile;
          mbar_expect_tx(&kv_full[sk], 2 * Cfg::kTile);
#pragma unroll
          for (int at = 0; at < Cfg::kAtoms; ++at) {
            tma_load_3d(kv + at * kAtom, &tk, &kv_full[sk], item.hk * D + at * 64, item.nb * 128, item.b);
            tma_load_3d(kv + Cfg::kTile + at * kAtom, &tv, &kv_full[sk], item.hk * D + at * 64, item.nb * 128, item.b);
          }
        }
        for (int it = 0; it < item.iters; ++it, ++n) {
          const int st = n & 1, so = n % SO;
          int h, mb;
          item.tile(it, h, mb);
          // statistics of four query rows per lane, in flight under the wait; rows beyond the sequence get
          // probability 0 (lse = +inf) and delta 0
          float lse4[4], delta4[4];
          const long long so_row = (static_cast<long long>(item.b) * a.H + h) * a.T;
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const int qrow = mb * 128 + r * 32 + lane;
            lse4[r] = qrow < a.T ? __ldg(a.lse + so_row + qrow) * kLog2e : INFINITY;
            delta4[r] = qrow < a.T ? __ldg(a.delta + so_row + qrow) : 0.f;
          }
          ok = wait(&q_empty[st], (n >> 1) + 1);
          if (!ok) break;
          if (lane == 0) {
            mbar_expect_tx(&q_full[st], Cfg::kTile);
#pragma unroll
            for (int at = 0; at < Cfg::kAtoms; ++at)
              tma_load_3d(smem + Cfg::kOffQ + st * Cfg::kTile + at * kAtom, &tq, &q_full[st], h * D + at * 64, mb * 128,
                          item.b);
          }
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            s_lse[st * 128 + r * 32 + lane] = lse4[r];
            s_delta[st * 128 + r * 32 + lane] = delta4[r];
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&q_full[st]);
          ok = wait(&do_empty[so], n / SO + 1);
          if (!ok) break;
          if (lane == 0) {
            mbar_expect_tx(&do_full[so], Cfg::kTile);
#pragma unroll
            for (int at = 0; at < Cfg::kAtoms; ++at)
              tma_load_3d(smem + Cfg::kOffdO + so * Cfg::kTile + at * kAtom, &tdo, &do_full[so], h * D + at * 64, mb * 128,
                          item.b);
          }
        }
      }
      if (!ok) give_up(201);
    } else if (warp == 13) {
      // ---------------------------------------------------------------- MMA issuer: one thread, elected per instruction
      constexpr uint32_t id_s = make_idesc_bf16_f32(128, 128, false, false);
      constexpr uint32_t id_kv = make_idesc_bf16_f32(128, D, false, true);
      constexpr uint32_t id_q = make_idesc_bf16_f32(128, D, true, true);
      const uint32_t aK = smem_u32(smem + Cfg::kOffK), aV = smem_u32(smem + Cfg::kOffV);
      const uint32_t adS = smem_u32(smem + Cfg::kOffdS);
      // Shared-memory descriptors are built once; a stage or k-step only adds its byte offset (>> 4) to them.
      const uint64_t dK_k0 = make_smem_desc_sw128(aK, 16, 1024), dV_k0 = make_smem_desc_sw128(aV, 16, 1024);
      const uint64_t ddS_k = make_smem_desc_sw128(adS, 16, 1024);
      const uint64_t ddS_m = make_smem_desc_sw128(adS, kAtom, 1024), dK_m0 = make_smem_desc_sw128(aK, kAtom, 1024);
      const uint32_t aQ0 = smem_u32(smem + Cfg::kOffQ), adO0 = smem_u32(smem + Cfg::kOffdO);
      const uint64_t dQ_k0 = make_smem_desc_sw128(aQ0, 16, 1024), ddO_k0 = make_smem_desc_sw128(adO0, 16, 1024);
      const uint64_t dQ_m0 = make_smem_desc_sw128(aQ0, kAtom, 1024), ddO_m0 = make_smem_desc_sw128(adO0, kAtom, 1024);
      constexpr uint64_t kStageStep = Cfg::kTile >> 4, kKvStep = (2 * Cfg::kTile) >> 4;
      auto wait_tc = [&](uint64_t* bar, uint32_t parity) {
        const bool ok = wait(bar, parity);
        tc_fence_after_sync();
        return ok;
      };
      auto issue_s = [&](uint32_t c, uint32_t n) {       // S^T of tile n with item c's keys
        const uint64_t dK_k = dK_k0 + (c % SK) * kKvStep, dQ_k = dQ_k0 + (n & 1) * kStageStep;
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint64_t off = ((kk >> 2) * kAtom + (kk & 3) * 32) >> 4;
          umma_f16_ss_elect(tm_S, dK_k + off, dQ_k + off, id_s, kk > 0);
        }
        umma_commit_elect(s_full);
      };
      auto issue_dp = [&](uint32_t c, uint32_t n) {
        const uint64_t dV_k = dV_k0 + (c % SK) * kKvStep, ddO_k = ddO_k0 + (n % SO) * kStageStep;
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint64_t off = ((kk >> 2) * kAtom + (kk & 3) * 32) >> 4;
          umma_f16_ss_elect(tm_dP, dV_k + off, ddO_k + off, id_s, kk > 0);
        }
        umma_commit_elect(dp_full);
      };
      bool more = item.next(), ok = true;
      uint32_t n = 0;
      if (more) {
        ok = wait_tc(&kv_full[0], 0) && wait_tc(&q_full[0], 0);
        if (ok) {
          issue_s(0, 0);
          ok = wait_tc(&do_full[0], 0);
          if (ok) issue_dp(0, 0);
        }
      }
      for (uint32_t c = 0; more && ok; ++c) {
        const int iters = item.iters;
        more = item.next();
        const uint64_t dK_m = dK_m0 + (c % SK) * kKvStep;
        for (int it = 0; it < iters; ++it, ++n) {
          const bool last = it + 1 == iters, next_tile = !last || more;
          const uint32_t cn = last ? c + 1 : c;           // the next tile's item
          ok = wait_tc(p_full, n);
          if (ok && it == 0 && c > 0) ok = wait_tc(acc_drained, c - 1);
          if (!ok) break;
          const uint64_t ddO_m = ddO_m0 + (n % SO) * kStageStep;
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)         // contraction over the 128 query rows of the tile
            umma_f16_ts_elect(tm_dV, tm_S + (kk >> 2) * 64 + (kk & 3) * 8, ddO_m + ((kk * 2048) >> 4), id_kv,
                              it > 0 || kk > 0);
          umma_commit_elect(&do_empty[n % SO]);
          auto next_s = [&]() {
            bool got = true;
            if (last) got = wait_tc(&kv_full[cn % SK], cn / SK);
            if (got) got = wait_tc(&q_full[(n + 1) & 1], (n + 1) >> 1);
            if (got) issue_s(cn, n + 1);
            return got;
          };
          // a single stage of K and V is refilled only behind this tile's dQ
          const bool early = !last || SK > 1;
          if (next_tile && early) ok = next_s();
          if (ok) ok = wait_tc(ds_full, n);
          auto next_dp = [&]() {
            bool got = wait_tc(&do_full[(n + 1) % SO], (n + 1) / SO);
            if (got && kAlias) got = wait_tc(dq_drained, n);
            if (got) issue_dp(cn, n + 1);
            return got;
          };
          // dP of the next tile first where dQ does not need its columns: the softmax warps wait for it
          if (ok && !kAlias && next_tile) ok = next_dp();
          // its own columns: the previous tile's dQ must have been read out (at head size 128 dP waited for that)
          if (ok && !kAlias && n > 0) ok = wait_tc(dq_drained, n - 1);
          if (!ok) break;
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) {       // contraction over the 128 keys
            const uint64_t moff = (kk * 2048) >> 4;                            // MN-major operand: 16 rows down
            umma_f16_ss_elect(tm_dQ, ddS_m + moff, dK_m + moff, id_q, kk > 0);
          }
          umma_commit_elect(dq_full);
          const uint64_t dQ_m = dQ_m0 + (n & 1) * kStageStep;
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) {       // contraction over the 128 query rows of the tile
            const uint64_t koff = ((kk >> 2) * kAtom + (kk & 3) * 32) >> 4;   // K-major operand
            if constexpr (kTmemdS)
              umma_f16_ts_elect(tm_dK, tm_dS + kk * 8, dQ_m + ((kk * 2048) >> 4), id_kv, it > 0 || kk > 0);
            else
              umma_f16_ss_elect(tm_dK, ddS_k + koff, dQ_m + ((kk * 2048) >> 4), id_kv, it > 0 || kk > 0);
          }
          umma_commit_elect(&q_empty[n & 1]);
          if (last) {
            umma_commit_elect(&kv_empty[c % SK]);
            umma_commit_elect(acc_full);
          }
          if (kAlias && next_tile) {
            if (!early) ok = next_s();
            if (ok) ok = next_dp();
            if (!ok) break;
          }
        }
      }
      if (!ok) give_up(204);
    }
  } else if (warp >= 8) {
    // ------------------------------------------------------------------ dQ read-out: query row = TMEM lane
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const bool issuer = warp == 8 && lane == 0;
    regs_grow<168>();
    bool ok = true;       // a warp that gave up keeps meeting the others at the barriers
    uint32_t n = 0;
    while (item.next()) {
      for (int it = 0; it < item.iters; ++it, ++n) {
        int h, mb;
        item.tile(it, h, mb);
        if (ok) {
          ok = wait(dq_full, n);
          if (!ok) give_up(206);
        }
        tc_fence_after_sync();
        // All columns into registers, so that the tensor core gets them back at once; then 64 columns a round through
        // two fp32 staging blocks of 32 columns (128-byte swizzle), one bulk add-reduction each.
        uint32_t r[D / 32][32];
        if (ok) {
#pragma unroll
          for (int c = 0; c < D / 32; ++c) tmem_ld_32x32(tm_dQ + lane_addr + c * 32, r[c]);
          tmem_ld_wait();
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(dq_drained);
        }
#pragma unroll
        for (int round = 0; round < D / 64; ++round) {
          if (issuer) tma_store_wait_read<0>();     // the blocks have been read
          readout_warps_sync();
          if (ok) {
#pragma unroll
            for (int blk = 0; blk < 2; ++blk) {
              uint8_t* dst = smem + Cfg::kOffStage + blk * kAtom + row * 128;
              const uint32_t(&v)[32] = r[round * 2 + blk];
#pragma unroll
              for (int j = 0; j < 8; ++j)
                *reinterpret_cast<float4*>(dst + ((j ^ (row & 7)) << 4)) =
                    make_float4(__uint_as_float(v[4 * j]) * a.scale, __uint_as_float(v[4 * j + 1]) * a.scale,
                                __uint_as_float(v[4 * j + 2]) * a.scale, __uint_as_float(v[4 * j + 3]) * a.scale);
            }
          }
          fence_proxy_async_smem();
          readout_warps_sync();
          if (issuer && ok) {
            tma_reduce_add_3d(&tdq, smem + Cfg::kOffStage, h * D + round * 64, mb * 128, item.b);
            tma_reduce_add_3d(&tdq, smem + Cfg::kOffStage + kAtom, h * D + round * 64 + 32, mb * 128, item.b);
            tma_store_commit();
          }
        }
      }
    }
    if (issuer) tma_store_wait<0>();
  } else {
    // ------------------------------------------------------------------ softmax: key row = TMEM lane
    regs_grow<144>();
    const int half = warp >> 2;                 // which half of the query columns this warp takes
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const float sl2 = a.scale * kLog2e;
    bool ok = true;
    uint32_t n = 0;
    for (uint32_t c = 0; ok && item.next(); ++c) {
      const int n0 = item.nb * 128, krow = n0 + row;
      const bool key_ok = krow < a.T;
      for (int it = 0; it < item.iters; ++it, ++n) {
        int h, mb;
        item.tile(it, h, mb);
        const int st = n & 1;
        ok = wait(s_full, n);
        if (!ok) break;
        tc_fence_after_sync();
        uint32_t rs[2][32];
        tmem_ld_32x32(tm_S + lane_addr + half * 64, rs[0]);
        tmem_ld_32x32(tm_S + lane_addr + half * 64 + 32, rs[1]);
        ok = wait(&q_full[st], n >> 1);      // the statistics have been written (S waited for the tile itself)
        tmem_ld_wait();
        if (!ok) break;
        // the mask matters on the diagonal tile and for the keys beyond the sequence only
        const bool diag = a.causal && mb == item.nb;
        const bool need_mask = diag || (n0 + 128 > a.T);
        const float* lse = s_lse + st * 128 + half * 64;
        const float* dl = s_delta + st * 128 + half * 64;
        float p[64];
#pragma unroll
        for (int cg = 0; cg < 2; ++cg) {
#pragma unroll
          for (int j4 = 0; j4 < 32; j4 += 4) {
            const float4 l4 = *reinterpret_cast<const float4*>(lse + cg * 32 + j4);
            const float lv[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) p[cg * 32 + j4 + e] = ex2(fmaf(__uint_as_float(rs[cg][j4 + e]), sl2, -lv[e]));
          }
          if (need_mask) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (!key_ok || (diag && row > half * 64 + cg * 32 + j)) p[cg * 32 + j] = 0.f;
          }
          uint32_t w[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) w[j] = pack2(p[cg * 32 + 2 * j], p[cg * 32 + 2 * j + 1]);
          // over the first half of the columns that this warp alone has read
          tmem_st_32x16(tm_S + lane_addr + half * 64 + cg * 16, w);
        }
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full);
        ok = wait(dp_full, n);
        if (!ok) break;
        tc_fence_after_sync();
        tmem_ld_32x32(tm_dP + lane_addr + half * 64, rs[0]);
        tmem_ld_32x32(tm_dP + lane_addr + half * 64 + 32, rs[1]);
        // dS of the tile before has been read; at head size 128 dp_full says so
        if (!kAlias && n > 0) ok = wait(&q_empty[(n - 1) & 1], (n - 1) >> 1);
        tmem_ld_wait();
        if (!ok) break;
#pragma unroll
        for (int cg = 0; cg < 2; ++cg) {
          const uint32_t(&rp)[32] = rs[cg];
          uint8_t* rowS = smem + Cfg::kOffdS + half * kAtom + row * 128;
          uint32_t w[16];
#pragma unroll
          for (int j4 = 0; j4 < 32; j4 += 4) {
            const float4 d4 = *reinterpret_cast<const float4*>(dl + cg * 32 + j4);
            const float* pj = &p[cg * 32 + j4];
            w[j4 / 2] = pack2(pj[0] * (__uint_as_float(rp[j4]) - d4.x), pj[1] * (__uint_as_float(rp[j4 + 1]) - d4.y));
            w[j4 / 2 + 1] =
                pack2(pj[2] * (__uint_as_float(rp[j4 + 2]) - d4.z), pj[3] * (__uint_as_float(rp[j4 + 3]) - d4.w));
          }
#pragma unroll
          for (int c8 = 0; c8 < 4; ++c8)
            *reinterpret_cast<uint4*>(rowS + (((cg * 4 + c8) ^ (row & 7)) << 4)) =
                make_uint4(w[4 * c8], w[4 * c8 + 1], w[4 * c8 + 2], w[4 * c8 + 3]);
          if constexpr (kTmemdS) tmem_st_32x16(tm_dS + lane_addr + half * 32 + cg * 16, w);
        }
        if constexpr (kTmemdS) tmem_st_wait();
        fence_proxy_async_smem();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(ds_full);
      }
      if (ok) ok = wait(acc_full, c);
      if (!ok) break;
      tc_fence_after_sync();
      // dK (scaled) and dV of the item's 128 keys; a warp has 32 rows and half of the columns.  As bf16 they go through
      // the warp's part of the spent dS^T, so that neighbouring lanes write neighbouring 16 bytes: with a row per
      // lane each store touched 32 lines, 5000 cycles an item at head size 64.
      if (item.nparts == 1) {
        constexpr int kLanes = D / 16;           // lanes per row
        uint8_t* mine = smem + Cfg::kOffdS + warp * 4096;
#pragma unroll
        for (int which = 0; which < 2; ++which) {
          const uint32_t tm = (which ? tm_dV : tm_dK) + lane_addr + half * (D / 2);
          const float f = which ? 1.f : a.scale;
#pragma unroll
          for (int cc = 0; cc < D / 64; ++cc) {
            uint32_t r[32];
            tmem_ld_32x32(tm + cc * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float v[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(r[8 * j + e]) * f;
              // 16-byte pieces of a row in an order that keeps the lanes on different banks
              *reinterpret_cast<uint4*>(mine + lane * (D == 64 ? 64 : 128) +
                                        (((cc * 4 + j) ^ (D == 64 ? (lane >> 1) & 3 : lane & 7)) << 4)) = pack8(v);
            }
          }
          if (which == 1) tc_fence_before_sync();
          __syncwarp();
          if (which == 1 && lane == 0) mbar_arrive(acc_drained);
          __nv_bfloat16* base = static_cast<__nv_bfloat16*>(which ? a.dv : a.dk) +
                                item.b * (which ? a.v_batch_stride : a.k_batch_stride) + item.hk * D + half * (D / 2);
          const long long stride = which ? a.v_row_stride : a.k_row_stride;
          const int piece = lane % kLanes;
#pragma unroll
          for (int i = 0; i < kLanes; ++i) {
            const int rr = i * (32 / kLanes) + lane / kLanes, key = n0 + (warp & 3) * 32 + rr;
            const uint4 v = *reinterpret_cast<const uint4*>(
                mine + rr * (D == 64 ? 64 : 128) + ((piece ^ (D == 64 ? (rr >> 1) & 3 : rr & 7)) << 4));
            if (key < a.T) *reinterpret_cast<uint4*>(base + key * stride + piece * 8) = v;
          }
          __syncwarp();
        }
      } else {
        // this share's, into its own slab of the fp32 scratch [parts][2][B, T, KV, D]: the conversion adds the slabs up
        // in order, so that the result does not depend on which share came first
        const long long plane = static_cast<long long>(a.B) * a.T * a.KV * D;
        float* dks = a.dkv_accum + item.part * 2 * plane +
                     ((static_cast<long long>(item.b) * a.T + krow) * a.KV + item.hk) * D + half * (D / 2);
#pragma unroll
        for (int which = 0; which < 2; ++which) {
          const uint32_t tm = (which ? tm_dV : tm_dK) + lane_addr + half * (D / 2);
          const float f = which ? 1.f : a.scale;
#pragma unroll
          for (int cc = 0; cc < D / 64; ++cc) {
            uint32_t r[32];
            tmem_ld_32x32(tm + cc * 32, r);
            tmem_ld_wait();
            if (which == 1 && cc + 1 == D / 64) {
              tc_fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive(acc_drained);
            }
            if (key_ok) {
              float4* dst = reinterpret_cast<float4*>(dks + which * plane + cc * 32);
#pragma unroll
              for (int j = 0; j < 8; ++j)
                dst[j] = make_float4(__uint_as_float(r[4 * j]) * f, __uint_as_float(r[4 * j + 1]) * f,
                                     __uint_as_float(r[4 * j + 2]) * f, __uint_as_float(r[4 * j + 3]) * f);
            }
            __syncwarp();
          }
        }
      }
    }
    if (!ok) give_up(205);
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 13) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

// ------------------------------------------------------------------------------------ forward
// One item is 256 query rows of one head, two tiles of 128, walking together over the 128-key tiles up to the
// diagonal; per tile and step
//   S[m,n] = Q[m,:] . K[n,:]     tcgen05.mma  Q (K-major) x K (K-major)          -> TMEM, 128 columns a tile
//   online softmax: one thread per query row holds its row of S in registers, so nothing crosses threads;
//   P goes as bf16 over the spent S in TMEM
//   O[m,d] += P[m,n] V[n,d]      tcgen05.mma  P (from TMEM) x V (MN-major)       -> TMEM, D columns a tile
// While four warps do the softmax of one tile, the tensor core works on the other.  O stays in TMEM: a warp reads it,
// multiplies it by exp2(m_old - m_new) and writes it back when the maximum of one of its rows has grown, after its P
// of the step.  (Left relative to an older maximum until that is 2^8 behind, O is rescaled once or twice a row, but the
// largest probabilities are then no longer 1 and are rounded to bf16 like the others: 1 to 2 % more error against 64
// bits, for nothing at head size 64 and 476 -> 437 us of the 8192-token case below.)  Persistent, one CTA per SM; the
// next item's loads and first S run under the last steps of the one before.
//
// Two query tiles in turn, warp roles and P as the MMA's operand in TMEM are published techniques of flash attention
// for this architecture (FlashAttention-4).
//
// What bounds it: the exponentials, 16 per cycle and SM: 1024 cycles per 128 x 128 scores (head size 128: the two
// contractions take as long).
// Measured (causal): 16 x 1024 tokens, 12 heads of 64: 109 us with one tile per CTA, P through shared memory and O
// added up in registers; 66 us now.  1 x 8192, 32 / 8 heads of 128: 1243 -> 476 us (1155 TFLOP/s, 0.70 of the
// measured GEMM peak).  1 x 2048, 32 / 8 heads of 64: 80 -> 35 us.
template <int D>
struct FwdCfg {
  static constexpr int kAtoms = D / 64;
  static constexpr int kTile = kAtoms * kAtom;
  static constexpr int kStages = D == 64 ? 4 : 2;         // of K and of V
  static constexpr int kOffQ = 0;                         // two tiles
  static constexpr int kOffK = 2 * kTile;
  static constexpr int kOffV = kOffK + kStages * kTile;
  static constexpr int kOffOut = kOffV + kStages * kTile;   // 4 KB a softmax warp: O on its way out
  static constexpr int kOffBar = kOffOut + 8 * 4096;
  static constexpr int kSmem = kOffBar + (2 + 4 * kStages + 6) * 8 + 16;
  static_assert(kSmem <= 232448, "shared memory of one SM");
};
constexpr int kFwdThreads = 320;     // 2 x 4 softmax warps, TMA warp, MMA warp

struct FwdItems {
  int pairs, HB, H, causal, n_blocks, T;
  int k;
  int m0, h, b;
  int steps[2];                 // key tiles of the two query tiles; 0: the tile lies beyond the sequence
  __device__ explicit FwdItems(const ItbAttnArgs& a) {
    T = a.T;
    H = a.H;
    HB = a.H * a.B;
    causal = a.causal;
    n_blocks = (a.T + 127) / 128;
    pairs = (n_blocks + 1) / 2;
    k = -1;
  }
  // Items of later queries have more steps under a causal mask: longest first, dealt out to the CTAs to and fro.
  __device__ bool next() {
    for (;;) {
      ++k;
      const int base = k * static_cast<int>(gridDim.x);
      if (base >= pairs * HB) return false;
      const int i = base + static_cast<int>((k & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
      if (i >= pairs * HB) continue;
      const int pair = pairs - 1 - i / HB, hb = i % HB;
      h = hb % H;
      b = hb / H;
      m0 = pair * 256;
      steps[0] = causal ? min(n_blocks, 2 * pair + 1) : n_blocks;
      steps[1] = m0 + 128 >= T ? 0 : causal ? min(n_blocks, 2 * pair + 2) : n_blocks;
      return true;
    }
  }
};

template <int D>
__global__ void __launch_bounds__(kFwdThreads, 1)
flash_fwd_tc_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                    const __grid_constant__ CUtensorMap tv, const ItbAttnArgs a, int* err) {
  using Cfg = FwdCfg<D>;
  constexpr int S = Cfg::kStages;
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023) {          // the swizzled tiles need a 1024-byte boundary
    if (threadIdx.x == 0) atomicCAS(err, 0, 210);
    return;
  }
  uint64_t* q_full = reinterpret_cast<uint64_t*>(smem + Cfg::kOffBar);
  uint64_t* q_empty = q_full + 1;
  uint64_t* k_full = q_empty + 1;
  uint64_t* k_empty = k_full + S;
  uint64_t* v_full = k_empty + S;
  uint64_t* v_empty = v_full + S;
  uint64_t* s_full = v_empty + S;       // one of each per query tile from here on
  uint64_t* p_full = s_full + 2;
  uint64_t* o_full = p_full + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(o_full + 2);
  volatile uint32_t* abort_flag = tmem_holder + 1;

  const int warp = __shfl_sync(~0u, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    for (int s = 0; s < S; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    for (int t = 0; t < 2; ++t) {
      mbar_init(&s_full[t], 1);
      mbar_init(&p_full[t], 4);
      mbar_init(&o_full[t], 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 9) {
    tmem_alloc(tmem_holder, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_holder;
  const uint32_t tm_S = tmem_base, tm_O = tmem_base + 256;     // tile t: S at + 128 t, O at + D t
  auto give_up = [&](int code) {
    atomicCAS(err, 0, code);
    *abort_flag = 1;
  };
  auto wait = [&](uint64_t* bar, uint32_t parity) { return mbar_wait_warp(bar, parity & 1, abort_flag); };
  FwdItems item(a);

  if (warp == 8) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tma_prefetch_desc(&tq);
      tma_prefetch_desc(&tk);
      tma_prefetch_desc(&tv);
    }
    bool ok = true;
    uint32_t n = 0;                     // key tiles so far
    for (uint32_t c = 0; ok && item.next(); ++c) {
      const int hk = item.h / (a.H / a.KV);
      ok = wait(q_empty, c + 1);
      if (!ok) break;
      if (lane == 0) {
        mbar_expect_tx(q_full, 2 * Cfg::kTile);
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
          for (int at = 0; at < Cfg::kAtoms; ++at)
            tma_load_3d(smem + Cfg::kOffQ + t * Cfg::kTile + at * kAtom, &tq, q_full, item.h * D + at * 64,
                        item.m0 + t * 128, item.b);
      }
      const int steps = max(item.steps[0], item.steps[1]);
      for (int j = 0; j < steps; ++j, ++n) {
        const int st = n % S;
        ok = wait(&k_empty[st], n / S + 1);
        if (!ok) break;
        if (lane == 0) {
          mbar_expect_tx(&k_full[st], Cfg::kTile);
#pragma unroll
          for (int at = 0; at < Cfg::kAtoms; ++at)
            tma_load_3d(smem + Cfg::kOffK + st * Cfg::kTile + at * kAtom, &tk, &k_full[st], hk * D + at * 64, j * 128, item.b);
        }
        ok = wait(&v_empty[st], n / S + 1);
        if (!ok) break;
        if (lane == 0) {
          mbar_expect_tx(&v_full[st], Cfg::kTile);
#pragma unroll
          for (int at = 0; at < Cfg::kAtoms; ++at)
            tma_load_3d(smem + Cfg::kOffV + st * Cfg::kTile + at * kAtom, &tv, &v_full[st], hk * D + at * 64, j * 128, item.b);
        }
      }
    }
    if (!ok) give_up(211);
  } else if (warp == 9) {
    // ------------------------------------------------------------------ MMA issuer: one thread, elected per instruction
    constexpr uint32_t id_s = make_idesc_bf16_f32(128, 128, false, false);
    constexpr uint32_t id_o = make_idesc_bf16_f32(128, D, false, true);
    constexpr uint64_t kStep = Cfg::kTile >> 4;
    const uint64_t dQ0 = make_smem_desc_sw128(smem_u32(smem + Cfg::kOffQ), 16, 1024);
    const uint64_t dK0 = make_smem_desc_sw128(smem_u32(smem + Cfg::kOffK), 16, 1024);
    const uint64_t dV0 = make_smem_desc_sw128(smem_u32(smem + Cfg::kOffV), kAtom, 1024);
    auto wait_tc = [&](uint64_t* bar, uint32_t parity) {
      const bool ok = wait(bar, parity);
      tc_fence_after_sync();
      return ok;
    };
    auto issue_s = [&](int t, uint32_t n) {      // S of query tile t with the key tile numbered n
      const uint64_t dQ = dQ0 + t * kStep, dK = dK0 + (n % S) * kStep;
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        const uint64_t off = ((kk >> 2) * kAtom + (kk & 3) * 32) >> 4;
        umma_f16_ss_elect(tm_S + t * 128, dQ + off, dK + off, id_s, kk > 0);
      }
      umma_commit_elect(&s_full[t]);
    };
    bool ok = true;
    uint32_t n0 = 0;                    // number of the item's first key tile
    uint32_t np[2] = {0, 0};            // P tiles so far
    for (uint32_t c = 0; ok && item.next(); ++c) {
      const int steps = max(item.steps[0], item.steps[1]);
      ok = wait_tc(q_full, c) && wait_tc(&k_full[n0 % S], n0 / S);
      if (!ok) break;
      // S of the item before has been read: its last P tiles were waited for
#pragma unroll
      for (int t = 0; t < 2; ++t)
        if (item.steps[t] > 0) issue_s(t, n0);
      umma_commit_elect(&k_empty[n0 % S]);
      if (steps == 1) umma_commit_elect(q_empty);
      for (int j = 0; j < steps && ok; ++j) {
        const uint32_t n = n0 + j;
        const bool more_keys = j + 1 < steps;
        ok = wait_tc(&v_full[n % S], n / S);
        if (ok && more_keys) ok = wait_tc(&k_full[(n + 1) % S], (n + 1) / S);
        const uint64_t dV = dV0 + (n % S) * kStep;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (!ok || j >= item.steps[t]) continue;
          ok = wait_tc(&p_full[t], np[t]);
          if (!ok) continue;
          ++np[t];
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)       // contraction over the 128 keys of the tile
            umma_f16_ts_elect(tm_O + t * D, tm_S + t * 128 + kk * 8, dV + ((kk * 2048) >> 4), id_o, j > 0 || kk > 0);
          // S goes over this P: MMAs complete in the order of issue
          if (j + 1 < item.steps[t])
            issue_s(t, n + 1);
          else
            umma_commit_elect(&o_full[t]);
        }
        if (!ok) break;
        umma_commit_elect(&v_empty[n % S]);
        if (more_keys) umma_commit_elect(&k_empty[(n + 1) % S]);
        if (j + 2 == steps) umma_commit_elect(q_empty);
      }
      n0 += steps;
    }
    if (!ok) give_up(213);
  } else {
    // ------------------------------------------------------------------ softmax: query row = TMEM lane
    const int t = warp >> 2;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t tS = tm_S + t * 128 + lane_addr, tO = tm_O + t * D + lane_addr;
    // a masked key's score is the infinity whose probability is 0; no score times a scale of 0 is that
    const float sl2 = a.scale == 0.f ? FLT_MIN : a.scale * kLog2e;
    const float hidden = sl2 > 0.f ? -INFINITY : INFINITY;
    bool ok = true;
    uint32_t n = 0, items = 0;
    while (ok && item.next()) {
      const int steps = t ? item.steps[1] : item.steps[0], mb = item.m0 / 128 + t;
      if (steps == 0) continue;
      float m_run = -INFINITY, l_run = 0.f;      // running maximum (scaled, log2 domain) and sum
      for (int j = 0; j < steps; ++j, ++n) {
        ok = wait(&s_full[t], n);
        if (!ok) break;
        tc_fence_after_sync();
        uint32_t s[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_32x32(tS + c * 32, s[c]);
        tmem_ld_wait();
        // only the diagonal tile and a ragged last tile need the mask
        const bool diag = a.causal && j == mb;
        if (diag || (j + 1) * 128 > a.T) {
          const int n_lim = min(diag ? row + 1 : 128, a.T - j * 128);   // keys [0, n_lim) visible
#pragma unroll
          for (int i = 0; i < 128; ++i)
            if (i >= n_lim) s[i >> 5][i & 31] = __float_as_uint(hidden);
        }
        float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < 128; ++i) m4[i & 3] = fmaxf(m4[i & 3], __uint_as_float(s[i >> 5][i & 31]));
        // sl2 > 0: scaling commutes with the maximum (below 0 the lowest score, or none, serves as well).  A row without a
        // maximum takes 0 as its base, so that exp2 yields 0, not NaN.
        const float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * sl2;
        const float m_new = fmaxf(m_run, mx);
        const float base = m_new == -INFINITY ? 0.f : m_new;
        const float corr = ex2(m_run - base);
        const bool rescale = j > 0 && __any_sync(~0u, m_new > m_run);
        m_run = m_new;
        float sum = 0.f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t w[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float p0 = ex2(fmaf(__uint_as_float(s[c][2 * i]), sl2, -base));
            const float p1 = ex2(fmaf(__uint_as_float(s[c][2 * i + 1]), sl2, -base));
            sum += p0;
            sum += p1;
            w[i] = pack2(p0, p1);
          }
          tmem_st_32x16(tS + c * 16, w);
        }
        l_run = l_run * corr + sum;
        // s_full says that the PV of the step before has completed; S is spent, its registers take O on its way through
        if (rescale) {
          uint32_t o[D / 32][32];
#pragma unroll
          for (int c = 0; c < D / 32; ++c) tmem_ld_32x32(tO + c * 32, o[c]);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < D / 16; ++c) {
            uint32_t w[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) w[i] = __float_as_uint(__uint_as_float(o[c >> 1][(c & 1) * 16 + i]) * corr);
            tmem_st_32x16(tO + c * 16, w);
          }
        }
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[t]);
      }
      if (ok) ok = wait(&o_full[t], items);
      if (!ok) break;
      ++items;
      tc_fence_after_sync();
      const int qrow = mb * 128 + row;
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      // 64 columns of the warp's 32 rows at a time through shared memory, so that eight lanes write the 128 bytes
      // of a row together
      uint8_t* mine = smem + Cfg::kOffOut + warp * 4096;
#pragma unroll
      for (int c = 0; c < D / 64; ++c) {
        uint32_t r[2][32];
        tmem_ld_32x32(tO + c * 64, r[0]);
        tmem_ld_32x32(tO + c * 64 + 32, r[1]);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float v[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(r[i >> 2][(i & 3) * 8 + e]) * inv;
          *reinterpret_cast<uint4*>(mine + lane * 128 + ((i ^ (lane & 7)) << 4)) = pack8(v);
        }
        __syncwarp();
        __nv_bfloat16* op = static_cast<__nv_bfloat16*>(a.o) + item.b * a.o_batch_stride + item.h * D + c * 64;
        const int first = mb * 128 + (warp & 3) * 32;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int rr = i * 4 + (lane >> 3);
          const uint4 v = *reinterpret_cast<const uint4*>(mine + rr * 128 + (((lane & 7) ^ (rr & 7)) << 4));
          if (first + rr < a.T) *reinterpret_cast<uint4*>(op + (first + rr) * a.o_row_stride + (lane & 7) * 8) = v;
        }
        __syncwarp();
      }
      if (qrow < a.T)
        a.lse[(static_cast<long long>(item.b) * a.H + item.h) * a.T + qrow] =
            l_run > 0.f ? (m_run == -INFINITY ? 0.f : m_run) * 0.6931471805599453f + logf(l_run) : -FLT_MAX;
      __syncwarp();
    }
    if (!ok) give_up(215);
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

// SMs of the current device: the grid of the persistent kernels.
static cudaError_t sm_count(int* sms) {
  int device = 0;
  const cudaError_t e = cudaGetDevice(&device);
  return e != cudaSuccess ? e : cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, device);
}

template <int D>
static int fwd_launch(const ItbAttnArgs* a, int* err, cudaStream_t s) {
  using Cfg = FwdCfg<D>;
  constexpr int smem = Cfg::kSmem;
  static PerDeviceOnce configured;
  if (configured.first()) {
    cudaError_t e = cudaFuncSetAttribute(flash_fwd_tc_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  CUtensorMap tq, tk, tv;
  int rc = make_tmap_bf16_3d(&tq, a->q, static_cast<uint64_t>(a->H) * D, a->T, a->B, a->q_row_stride,
                             a->q_batch_stride, 64, 128);
  if (!rc) rc = make_tmap_bf16_3d(&tk, a->k, static_cast<uint64_t>(a->KV) * D, a->T, a->B, a->k_row_stride,
                                  a->k_batch_stride, 64, 128);
  if (!rc) rc = make_tmap_bf16_3d(&tv, a->v, static_cast<uint64_t>(a->KV) * D, a->T, a->B, a->v_row_stride,
                                  a->v_batch_stride, 64, 128);
  if (rc) return rc;
  int sms = 0;
  const cudaError_t e = sm_count(&sms);
  if (e != cudaSuccess) return static_cast<int>(e);
  const long long items = static_cast<long long>(((a->T + 127) / 128 + 1) / 2) * a->H * a->B;
  if (items > (1LL << 30)) return -5;      // counted in 32 bits
  flash_fwd_tc_kernel<D><<<static_cast<int>(items < sms ? items : sms), kFwdThreads, smem, s>>>(tq, tk, tv, *a, err);
  return static_cast<int>(cudaGetLastError());
}

// The passes around the backward kernel: one thread per 8 elements of a [B, T, H D] row, 32-bit index arithmetic
// while the count allows it.  Both are bound by memory.
//
// delta[b,h,t] = sum_d dO[b,t,h,d] * O[b,t,h,d], D / 8 threads per sum; the same threads clear the fp32 accumulator of
// dQ, which was a memset of its own (16 x 1024 x 12 heads of 64: memset, delta and conversion 9.8 + 14.9 + 19.0 us
// with 64-bit divisions and 4 elements a thread, 15.8 + 10.6 us now).
template <typename Index>
__global__ void attn_delta_tc_kernel(const ItbAttnArgs a, int D, Index total) {
  const Index i = blockIdx.x * static_cast<Index>(blockDim.x) + threadIdx.x;
  const int per_head = D >> 3;                                   // threads per sum: 8 or 16
  const Index per_row = static_cast<Index>(a.H) * per_head;
  const bool mine = i < total;
  const Index r = mine ? i / per_row : 0;
  const int c = mine ? static_cast<int>(i - r * per_row) : 0;
  const int b = static_cast<int>(r / a.T), t = static_cast<int>(r - static_cast<Index>(b) * a.T);
  float acc = 0.f;
  if (mine) {
    const long long off = b * a.o_batch_stride + static_cast<long long>(t) * a.o_row_stride + c * 8;
    const uint4 x = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(a.o) + off);
    const uint4 y = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(a.dout) + off);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4* dq = reinterpret_cast<float4*>(a.dq_accum) + static_cast<long long>(i) * 2;
    dq[0] = zero;
    dq[1] = zero;
    const __nv_bfloat162* xb = reinterpret_cast<const __nv_bfloat162*>(&x);
    const __nv_bfloat162* yb = reinterpret_cast<const __nv_bfloat162*>(&y);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 xf = __bfloat1622float2(xb[e]), yf = __bfloat1622float2(yb[e]);
      acc += xf.x * yf.x + xf.y * yf.y;
    }
  }
  for (int s = per_head >> 1; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
  const int h = c / per_head;
  if (mine && c % per_head == 0) a.delta[(static_cast<long long>(b) * a.H + h) * a.T + t] = acc;
}

// dq (bf16, strided) = the fp32 accumulator; with split key tiles dk and dv = the sums of the shares' slabs
// [parts][2][B, T, KV, D], those that had a tile, in order
template <typename Index>
__global__ void attn_convert_tc_kernel(const ItbAttnArgs a, int D, Index total, Index kv_total) {
  Index i = blockIdx.x * static_cast<Index>(blockDim.x) + threadIdx.x;
  const float* src = a.dq_accum;
  __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(a.dq);
  long long row_stride = a.q_row_stride, batch_stride = a.q_batch_stride;
  Index per_row = static_cast<Index>(a.H) * (D >> 3);
  if (i >= total) {
    i -= total;
    if (i >= kv_total) return;
    const Index plane = kv_total / 2;
    const bool is_v = i >= plane;
    if (is_v) i -= plane;
    src = a.dkv_accum + (is_v ? static_cast<long long>(plane) * 8 : 0);
    dst = static_cast<__nv_bfloat16*>(is_v ? a.dv : a.dk);
    row_stride = is_v ? a.v_row_stride : a.k_row_stride;
    batch_stride = is_v ? a.v_batch_stride : a.k_batch_stride;
    per_row = static_cast<Index>(a.KV) * (D >> 3);
  }
  const Index r = i / per_row;
  const int c = static_cast<int>(i - r * per_row);
  const int b = static_cast<int>(r / a.T), t = static_cast<int>(r - static_cast<Index>(b) * a.T);
  const float4* v = reinterpret_cast<const float4*>(src) + static_cast<long long>(i) * 2;
  float4 lo = v[0], hi = v[1];
  if (src != a.dq_accum) {
    const int n_qblocks = (a.T + 127) / 128;
    const int pairs = (n_qblocks - (a.causal ? t / 128 : 0)) * (a.H / a.KV);
    const long long step = static_cast<long long>(kv_total) * 2;      // float4s of a slab
    for (int p = 1; p < min(a.bwd_parts, pairs); ++p) {
      const float4 l = v[p * step], h = v[p * step + 1];
      lo.x += l.x, lo.y += l.y, lo.z += l.z, lo.w += l.w;
      hi.x += h.x, hi.y += h.y, hi.z += h.z, hi.w += h.w;
    }
  }
  const float x[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
  *reinterpret_cast<uint4*>(dst + b * batch_stride + t * row_stride + c * 8) = pack8(x);
}

template <int D>
static int bwd_launch(const ItbAttnArgs* a_in, int* err, cudaStream_t s) {
  ItbAttnArgs args = *a_in;
  args.bwd_parts = args.dkv_accum ? itb_flash_attn_bwd_parts(args.B, args.T, args.H, args.KV, args.causal) : 1;
  const ItbAttnArgs* a = &args;
  using Cfg = BwdCfg<D>;
  constexpr int smem = Cfg::kSmem;
  static PerDeviceOnce configured;
  if (configured.first()) {
    cudaError_t e = cudaFuncSetAttribute(flash_bwd_tc_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  CUtensorMap tq, tk, tv, tdo, tdq;
  int rc = make_tmap_f32_3d(&tdq, a->dq_accum, static_cast<uint64_t>(a->H) * D, a->T, a->B,
                            static_cast<uint64_t>(a->H) * D, static_cast<uint64_t>(a->T) * a->H * D, 128);
  if (!rc) rc = make_tmap_bf16_3d(&tq, a->q, static_cast<uint64_t>(a->H) * D, a->T, a->B, a->q_row_stride,
                             a->q_batch_stride, 64, 128);
  if (!rc) rc = make_tmap_bf16_3d(&tk, a->k, static_cast<uint64_t>(a->KV) * D, a->T, a->B, a->k_row_stride,
                                  a->k_batch_stride, 64, 128);
  if (!rc) rc = make_tmap_bf16_3d(&tv, a->v, static_cast<uint64_t>(a->KV) * D, a->T, a->B, a->v_row_stride,
                                  a->v_batch_stride, 64, 128);
  if (!rc) rc = make_tmap_bf16_3d(&tdo, a->dout, static_cast<uint64_t>(a->H) * D, a->T, a->B, a->o_row_stride,
                                  a->o_batch_stride, 64, 128);
  if (rc) return rc;
  const int parts = a->bwd_parts > 1 ? a->bwd_parts : 1;
  const long long vecs = static_cast<long long>(a->B) * a->T * a->H * (D / 8);
  const long long kv_vecs = parts > 1 ? 2LL * a->B * a->T * a->KV * (D / 8) : 0;
  const bool small = vecs + kv_vecs < (1LL << 31);
  const unsigned delta_blocks = static_cast<unsigned>((vecs + 255) / 256);
  const unsigned convert_blocks = static_cast<unsigned>((vecs + kv_vecs + 255) / 256);
  if (small)
    attn_delta_tc_kernel<uint32_t><<<delta_blocks, 256, 0, s>>>(*a, D, static_cast<uint32_t>(vecs));
  else
    attn_delta_tc_kernel<uint64_t><<<delta_blocks, 256, 0, s>>>(*a, D, vecs);
  int sms = 0;
  const cudaError_t e = sm_count(&sms);
  if (e != cudaSuccess) return static_cast<int>(e);
  const long long items = static_cast<long long>((a->T + 127) / 128) * a->KV * parts * a->B;
  if (items > (1LL << 30)) return -5;      // items and their tiles are counted in 32 bits
  flash_bwd_tc_kernel<D><<<static_cast<int>(items < sms ? items : sms), kThreads, smem, s>>>(tq, tk, tv, tdo, tdq, *a, err);
  if (small)
    attn_convert_tc_kernel<uint32_t><<<convert_blocks, 256, 0, s>>>(*a, D, static_cast<uint32_t>(vecs),
                                                                    static_cast<uint32_t>(kv_vecs));
  else
    attn_convert_tc_kernel<uint64_t><<<convert_blocks, 256, 0, s>>>(*a, D, vecs, kv_vecs);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace fatc
}  // namespace itb

// CTAs of one (key tile, KV head, batch).  The longest CTA (the first key tile: every query tile of every head of
// the group) bounds the launch from below, so it is split until it is no longer than an even share of all tiles
// and a little: one sequence of 2048 tokens with 8 KV heads of 4 query heads has 128 CTAs of up to 64 tiles, 29 a
// SM.  Each share pays for fp32 scratch (written, read and converted), so no finer than that.
// (1 x 2048 tokens, 32 / 8 heads of 64, the whole call: 159 us unsplit, 105 us in two shares; 89 us with the slabs
// and passes as they are now.)
extern "C" int itb_flash_attn_bwd_parts(int B, int T, int H, int KV, int causal) {
  if (B <= 0 || T <= 0 || KV <= 0) return 1;
  const long long nt = (T + 127) / 128, G = H / KV;
  const long long most = nt * G;                             // tiles of the longest CTA
  const long long tiles = (causal ? nt * (nt + 1) / 2 : nt * nt) * G * KV * B;
  int sms = 0;
  if (itb::fatc::sm_count(&sms) != cudaSuccess || sms <= 0) sms = 148;     // of a B200, where there is no device to ask
  const long long share = tiles / sms + tiles / (sms * 8) + 1;
  int parts = 1;
  while (parts < 16 && parts < most && (most + parts - 1) / parts > share) ++parts;
  return parts;
}

extern "C" int itb_flash_attn_bwd_tc(const ItbAttnArgs* a, int* err, cudaStream_t s) {
  if (a->B <= 0 || a->T <= 0) return 0;
  if (a->H % a->KV) return -3;
  if ((a->q_row_stride | a->k_row_stride | a->v_row_stride | a->o_row_stride | a->q_batch_stride |
       a->k_batch_stride | a->v_batch_stride | a->o_batch_stride) & 7)
    return -2;
  if ((reinterpret_cast<uintptr_t>(a->q) | reinterpret_cast<uintptr_t>(a->k) | reinterpret_cast<uintptr_t>(a->v) |
       reinterpret_cast<uintptr_t>(a->o) | reinterpret_cast<uintptr_t>(a->dq) | reinterpret_cast<uintptr_t>(a->dk) |
       reinterpret_cast<uintptr_t>(a->dv) | reinterpret_cast<uintptr_t>(a->dout)) & 15)
    return -2;
  if (a->D == 64) return itb::fatc::bwd_launch<64>(a, err, s);
  if (a->D == 128) return itb::fatc::bwd_launch<128>(a, err, s);
  return -4;
}

extern "C" int itb_flash_attn_fwd_tc(const ItbAttnArgs* a, int* err, cudaStream_t s) {
  if (a->B <= 0 || a->T <= 0) return 0;
  if (a->H % a->KV) return -3;
  if ((a->q_row_stride | a->k_row_stride | a->v_row_stride | a->o_row_stride | a->q_batch_stride |
       a->k_batch_stride | a->v_batch_stride | a->o_batch_stride) & 7)
    return -2;
  if ((reinterpret_cast<uintptr_t>(a->q) | reinterpret_cast<uintptr_t>(a->k) | reinterpret_cast<uintptr_t>(a->v) |
       reinterpret_cast<uintptr_t>(a->o)) & 15)
    return -2;
  if (a->D == 64) return itb::fatc::fwd_launch<64>(a, err, s);
  if (a->D == 128) return itb::fatc::fwd_launch<128>(a, err, s);
  return -4;
}
