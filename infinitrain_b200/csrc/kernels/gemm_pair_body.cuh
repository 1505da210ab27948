// Device code of the CTA-pair GEMM (tcgen05 cta_group::2), shared by the single-GPU launcher
// (gemm_tcgen05_2cta.cu) and the tensor-parallel launcher (comm/tp_gemm.cu), which compiles the same
// pipeline with the kTp hooks enabled: a prologue that pushes this rank's activation shard into every
// rank's gathered buffer, loads of A gated on the arrival of the shard they read, an epilogue that
// scatters partial output rows to their owner rank, and a closing phase that sums the partials.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include "../common/ptx.cuh"
#include "gemm_epilogue.cuh"
#include "kernels.h"

namespace itb {
namespace pair {

constexpr int BMC = 128;        // rows of A per CTA (pair: 256)
constexpr int BNC = 128;        // columns of B per CTA (pair: 256)
constexpr int BN = 256;
constexpr int BK = 64;
constexpr int kStages = 5;
constexpr int kABytes = BMC * BK * 2;
constexpr int kBBytes = BNC * BK * 2;
constexpr int kStageBytes = kABytes + kBBytes;                 // 32 KB
constexpr int kSlotBytes = 32 * 128;                           // 32 rows x 64 bf16 or 32 fp32, 128-byte swizzle

// Warps 0 and 1 load and issue; the others are the epilogue.
//
// The epilogue of a tile runs under the main loop of the next one (12 k-blocks are 6144 cycles of tensor core) and must
// neither be longer nor come in bursts.  Four warps, one for each quadrant of rows that may be read of TMEM, are enough
// for a bias or a residual.  GELU and its derivative took them longer than the MMAs (16384 x 3072 x 768, without loads
// and MMAs: 90 and 100 us, of 45 for the MMAs), and so does an fp32 residual, so there eight share the tile, two to a
// quadrant.  Eight warps for all would cost the plain output 8 % (16384 x 2304 x 768: 49.8 -> 53.7 us): twice as many
// stores at a time get in the way of the loads.
template <bool kTp, bool kWide>
struct Cfg {
  static constexpr int kEpiWarps = kWide ? 8 : 4;
  static constexpr int kThreads = 64 + 32 * kEpiWarps;
  static constexpr int kWarpCols = BN / (kEpiWarps / 4);
  static constexpr int kSlots = kTp ? 4 : 2;                   // staging slots of a warp
  static constexpr int kWarpStaging = kSlots * kSlotBytes;
  static constexpr int kStagingOffset = kStages * kStageBytes;
  static constexpr int kBiasOffset = kStagingOffset + kEpiWarps * kWarpStaging;
  static constexpr int kBarOffset = kBiasOffset + (kTp ? 0 : kEpiWarps * 256);      // 64 columns of bias per warp
  static constexpr int kOperandBars = kTp ? 4 : 2 * kEpiWarps;
  static constexpr int kSmemTotal = kBarOffset + (2 * kStages + 4 + kOperandBars) * 8 + 16;
  // without static shared memory the dynamic window starts on a 1024-byte boundary (the kernel looks)
  static constexpr int kSmemLaunch = kTp ? kSmemTotal + 1024 : kSmemTotal;
  static_assert(kSmemLaunch <= 232448, "shared memory of one SM");
};
constexpr uint32_t kTmemCols = 512;                            // two 256-column accumulators

// ---- tensor-parallel hooks -------------------------------------------------------------------
// Rows of the full activation are (b, t) pairs, row = b * T + t; under sequence parallelism rank s
// holds t in [s * Tl, (s + 1) * Tl) of every b as local row b * Tl + (t - s * Tl).
enum { kTpPush = 1, kTpGateA = 2, kTpScatter = 4, kTpBroadcast = 8 };
constexpr int kTpMaxRanks = 8;
constexpr unsigned kTpSpinLimit = 1u << 23;     // polls with a short sleep: seconds of skew

struct TpDev {
  int mode;                 // kTpPush | kTpGateA | kTpScatter
  int rank, world;
  int T, Tl, batch;
  // every launch of a context: `started[r]` on each rank holds 1 + the index of the latest launch
  // rank r has begun; a buffer last used `lag` launches ago is free once every rank has begun the
  // launch after that use
  int* started[kTpMaxRanks];
  int* launch_ctr;          // this GPU: number of launches so far
  unsigned* cta_done;       // this GPU: CTAs that have finished (self-resetting)
  int* err;
  // push: local shard [batch * Tl, push_cols] bf16 -> rows of every rank's gathered buffer
  const uint4* push_src;
  int push_row_vecs;        // 16-byte vectors per row
  uint4* gather[kTpMaxRanks];
  uint4* gather_mc;         // multicast address of the gathered buffer, or null
  int* push_arrive[kTpMaxRanks];   // counters [world] on each rank: warps of rank s that have pushed
  int* push_total;          // this GPU: arrivals per source that the pushes so far add up to
  int push_lag;
  // gate: loads of A wait for the shard they read
  const int* gate_arrive;   // this GPU's counters of the gated buffer
  const int* gate_total;
  int gate_includes_this_launch;
  // scatter: partial rows go to slab [rank] of their owner; the owner sums the slabs
  __nv_bfloat16* slab[kTpMaxRanks];     // [world][batch * Tl, N] bf16 on each rank
  int* rs_arrive[kTpMaxRanks];     // counters [world] on each rank: warp-tiles rank s has delivered
  int* rs_total;            // this GPU: arrivals per source that the launches so far add up to
  int rs_lag;
  void* rs_out;             // [batch * Tl, N]
  long long rs_ld_out;
  int rs_out_f32;
  const float* rs_bias;
  const __nv_bfloat16* rs_residual;
  long long rs_ld_res;
  // broadcast (with scatter): the summed rows go to every rank's full [batch * T, N] bf16 buffer
  // instead of rs_out, which turns the reduce-scatter into an all-reduce
  __nv_bfloat16* ar_out[kTpMaxRanks];
  uint4* ar_mc;             // multicast address of that buffer, or null
  int* ar_arrive[kTpMaxRanks];     // counters [world] on each rank: CTAs of rank s that have delivered
  int* ar_total;            // this GPU: arrivals per source that the launches so far add up to
  int ar_lag;
};

__device__ __forceinline__ void tp_st_release_sys(int* p, int v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int tp_ld_acquire_sys(const int* p) {
  int v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void tp_red_release_sys(int* p, int v) {
  asm volatile("red.release.sys.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Waits until *p - target >= 0 (wrap-safe).  False when the limit ran out.
__device__ __forceinline__ bool tp_wait_ge(const int* p, int target) {
  for (unsigned i = 0; i < kTpSpinLimit; ++i) {
    if (tp_ld_acquire_sys(p) - target >= 0) return true;
    if (i > 16) __nanosleep(200);
  }
  return false;
}

template <int kThreads>
__device__ __forceinline__ void epilogue_warps_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");
}

// kWide (staged outputs only): GELU, its derivative or an fp32 residual in the epilogue.  Otherwise everything else.
template <bool A_MN, bool B_MN, bool kTp, bool kWide>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Cfg<kTp, kWide>::kThreads, 1)
gemm_bf16_pair_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                      const __grid_constant__ CUtensorMap tma_c, const __grid_constant__ CUtensorMap tma_c2,
                      const __grid_constant__ CUtensorMap tma_e, const GemmDev p, const TpDev tp) {
  if constexpr (kTp) {
    // an earlier launch gave up on a peer: do not wait for it again (the status word was written
    // before this launch began, so both CTAs of a pair read the same value)
    if (*static_cast<volatile int*>(p.err) != 0) return;
  }
  using L = Cfg<kTp, kWide>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // Rounded up here although it is a no-op without static shared memory: with a base that the compiler knows, the MMA
  // loop comes out slower (2048 x 2048 x 32768: 212 -> 242 us).
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  if constexpr (!kTp) {
    if (smem != smem_raw) {       // nothing is left to round up with; the same answer in every CTA
      if (threadIdx.x == 0) atomicCAS(p.err, 0, 110);
      return;
    }
  }
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::kBarOffset);
  uint64_t* empty_bar = full_bar + kStages;
  uint64_t* tmem_full = empty_bar + kStages;
  uint64_t* tmem_empty = tmem_full + 2;
  uint64_t* operand_bar = tmem_empty + 2;         // of each epilogue warp (and slot): residual / aux tile landed
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(operand_bar + L::kOperandBars);
  volatile uint32_t* abort_flag = tmem_holder + 1;
  volatile uint32_t* stopped_at = tmem_holder + 2;      // the TMA warp's place in the ring

  const int warp = __shfl_sync(~0u, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank();          // 0 = leader
  const bool leader = cta == 0;
  const int pair_id = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);     // leader: its own arrive.expect_tx (bytes of both CTAs)
      mbar_init(&empty_bar[s], 1);    // one commit from the leader's MMA warp
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tmem_full[i], 1);    // one commit
      mbar_init(&tmem_empty[i], 2 * L::kEpiWarps);      // the epilogue warps of both CTAs (used on the leader only)
    }
    for (int i = 0; i < L::kOperandBars; ++i) mbar_init(&operand_bar[i], 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_holder, kTmemCols);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();      // both CTAs' barriers are initialised before any remote signal
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_holder;

  int tp_launch = 0;
  if constexpr (kTp) {
    tp_launch = *tp.launch_ctr;
    if (blockIdx.x == 0 && threadIdx.x < tp.world)
      tp_st_release_sys(tp.started[threadIdx.x] + tp.rank, tp_launch + 1);
  }
  const int total_tiles = p.tiles_m * p.tiles_n * p.split_k;
  const int kb_per_split = (p.k_blocks + p.split_k - 1) / p.split_k;
  constexpr int kGroupM = 8;
  auto decode_tile = [&](int t, int& tm, int& tn, int& kb0, int& kb1) {
    int ks = t % p.split_k;
    int t2 = t / p.split_k;
    int width = kGroupM * p.tiles_n;
    int group = t2 / width;
    int first_m = group * kGroupM;
    int gsz = min(p.tiles_m - first_m, kGroupM);
    int in_group = t2 - group * width;
    tm = first_m + in_group % gsz;
    tn = in_group / gsz;
    if constexpr (kTp) {
      // visit the shards in ring order: a gated GEMM starts with the rows this rank already holds,
      // a scattering GEMM ends with the rows it keeps
      const int nb = tp.Tl / 256, per = tp.batch * nb;
      const int j = tm / per, rem = tm - j * per;
      const int b = rem / nb, blk = rem - b * nb;
      const int sh = (tp.rank + j + ((tp.mode & kTpScatter) ? 1 : 0)) % tp.world;
      tm = (b * tp.T + sh * tp.Tl) / 256 + blk;
    }
    kb0 = ks * kb_per_split;
    kb1 = min(p.k_blocks, kb0 + kb_per_split);
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    if (lane == 0) {
      tma_prefetch_desc(&tma_a);
      tma_prefetch_desc(&tma_b);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      [[maybe_unused]] uint32_t gate_seen = 0;
      // (probe without loads: nothing holds the leader back for the peer's sake, so the peer's producer
      // could miss a barrier phase; it has no part in that run)
      if ((p.flags & kGemmProbeNoLoad) && !leader) ok = false;
      for (int t = pair_id; t < total_tiles && ok; t += num_pairs) {
        int tm, tn, kb0, kb1;
        decode_tile(t, tm, tn, kb0, kb1);
        const int row0 = tm * 256 + cta * BMC;     // this CTA's rows of A
        const int col0 = tn * 256 + cta * BNC;     // this CTA's columns of B
        if constexpr (kTp) {
          if (tp.mode & kTpGateA) {
            const int sh = ((tm * 256) % tp.T) / tp.Tl;
            if (!((gate_seen >> sh) & 1u)) {
              const int target = *tp.gate_total + (tp.gate_includes_this_launch ? static_cast<int>(gridDim.x) * 4 : 0);
              if (!tp_wait_ge(tp.gate_arrive + sh, target)) {
                atomicCAS(p.err, 0, 121);
                *abort_flag = 1;
                ok = false;
                break;
              }
              gate_seen |= 1u << sh;
              // the shard was written with ordinary stores; the loads below go through the async proxy
              asm volatile("fence.proxy.async;" ::: "memory");
            }
          }
        }
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1) || *abort_flag) {
            atomicCAS(p.err, 0, 111);
            *abort_flag = 1;
            ok = false;
            break;
          }
          uint8_t* sa = smem + stage * kStageBytes;
          uint8_t* sb = sa + kABytes;
          // every load of the pair completes on the LEADER's barrier
          const uint32_t bar = mapa_u32(smem_u32(&full_bar[stage]), 0);
          if (p.flags & kGemmProbeNoLoad) {
            if (leader) mbar_arrive(&full_bar[stage]);
            if (++stage == kStages) {
              stage = 0;
              phase ^= 1;
            }
            continue;
          }
          if (leader) mbar_expect_tx(&full_bar[stage], 2 * kStageBytes);
          if constexpr (!A_MN) {
            tma_load_2d_pair(sa, &tma_a, bar, kb * BK, row0);
          } else {
#pragma unroll
            for (int i = 0; i < BMC / 64; ++i)
              tma_load_2d_pair(sa + i * (64 * BK * 2), &tma_a, bar, row0 + i * 64, kb * BK);
          }
          if constexpr (!B_MN) {
            tma_load_2d_pair(sb, &tma_b, bar, kb * BK, col0);
          } else {
#pragma unroll
            for (int i = 0; i < BNC / 64; ++i)
              tma_load_2d_pair(sb + i * (64 * BK * 2), &tma_b, bar, col0 + i * 64, kb * BK);
          }
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      *stopped_at = ring_position(stage, phase);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader CTA only)
    // The warp stays together through the loop: wait for a stage, issue its four MMAs, release it with one
    // commit that arrives on both CTAs' barriers; the issuing thread is elected at each instruction, so that
    // descriptors stay in uniform registers (from a `lane == 0` branch each MMA moved them there first).
    // 16384 x 2304 x 768: 53.3 -> 50.1 us, 16384 x 50304 x 768: 1004 -> 952 us, 2048 x 2048 x 32768: 206 -> 187 us.
    // No tcgen05 fence inside the k-loop (the operands arrive through the async proxy and the barrier wait
    // orders them); the fence after a thread synchronisation is only needed where the epilogue warps hand an
    // accumulator back.
    if (leader) {
      constexpr uint32_t idesc = make_idesc_bf16_f32(256, BN, A_MN, B_MN);
      const bool probe_no_mma = p.flags & kGemmProbeNoMma;
      int stage = 0;
      uint32_t phase = 0;
      uint32_t acc_phase0 = 0, acc_phase1 = 0;
      int local = 0;
      bool ok = true;
      for (int t = pair_id; t < total_tiles && ok; t += num_pairs, ++local) {
        int tm, tn, kb0, kb1;
        decode_tile(t, tm, tn, kb0, kb1);
        const int acc = local & 1;
        if (kb1 <= kb0) continue;
        const uint32_t ap = acc ? acc_phase1 : acc_phase0;
        if (!mbar_wait_warp(&tmem_empty[acc], ap ^ 1, abort_flag)) {
          atomicCAS(p.err, 0, 112);
          *abort_flag = 1;
          break;
        }
        if (acc) acc_phase1 ^= 1; else acc_phase0 ^= 1;
        tc_fence_after_sync();
        const uint32_t tmem_d = tmem_base + acc * BN;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_warp(&full_bar[stage], phase, abort_flag)) {
            atomicCAS(p.err, 0, 113);
            *abort_flag = 1;
            ok = false;
            break;
          }
          const uint32_t sa = smem_u32(smem + stage * kStageBytes);
          const uint32_t sb = sa + kABytes;
          const uint64_t adesc0 = A_MN ? make_smem_desc_sw128(sa, 64 * BK * 2, 1024)
                                       : make_smem_desc_sw128(sa, 16, 1024);
          const uint64_t bdesc0 = B_MN ? make_smem_desc_sw128(sb, 64 * BK * 2, 1024)
                                       : make_smem_desc_sw128(sb, 16, 1024);
          if (!probe_no_mma) {
#pragma unroll
            for (int k = 0; k < BK / 16; ++k) {
              const uint64_t adesc = adesc0 + (A_MN ? (k * 2048) >> 4 : (k * 32) >> 4);
              const uint64_t bdesc = bdesc0 + (B_MN ? (k * 2048) >> 4 : (k * 32) >> 4);
              umma_f16_ss_pair_elect(tmem_d, adesc, bdesc, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
            }
          }
          // free this stage in both CTAs
          umma_commit_pair_mc_elect(smem_u32(&empty_bar[stage]), 3);
          if (kb == kb1 - 1) umma_commit_pair_mc_elect(smem_u32(&tmem_full[acc]), 3);
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if constexpr (kTp) {
    // ------------------------------------------------------------ epilogue of the tensor-parallel GEMM (4 warps per CTA)
    const int q = warp & 3;
    uint32_t acc_phase[2] = {0, 0};
    int local = 0;
    uint8_t* wstage = smem + L::kStagingOffset + q * L::kWarpStaging;
    const bool has_operand = p.flags & (kGemmResidual | kGemmDGelu);
    const bool dual = p.flags & kGemmGeluDual;
    uint32_t operand_phase = 0;
    int group = 0;
    bool tp_ok = true;
    if (tp.mode & (kTpPush | kTpScatter)) {
      // the buffers written below are free once every rank has begun the launch that follows
      // their previous use
      int lag = 1 << 24;
      if (tp.mode & kTpPush) lag = min(lag, tp.push_lag);
      if (tp.mode & kTpScatter) lag = min(lag, tp.rs_lag);
      if (tp.mode & kTpBroadcast) lag = min(lag, tp.ar_lag);
      bool ok = true;
      if (lane < tp.world) ok = tp_wait_ge(tp.started[tp.rank] + lane, tp_launch - lag + 2);
      tp_ok = __all_sync(0xffffffffu, ok);
      if (!tp_ok) {
        if (lane == 0) atomicCAS(p.err, 0, 122);
        *abort_flag = 1;
      }
    }
    if ((tp.mode & kTpPush) && tp_ok) {
      const long long total = static_cast<long long>(tp.batch) * tp.Tl * tp.push_row_vecs;
      const long long stride = static_cast<long long>(gridDim.x) * 128;
      for (long long v = static_cast<long long>(blockIdx.x) * 128 + (warp - 2) * 32 + lane; v < total; v += stride) {
        const long long l = v / tp.push_row_vecs;
        const int cv = static_cast<int>(v - l * tp.push_row_vecs);
        const int b = static_cast<int>(l / tp.Tl), t = static_cast<int>(l - static_cast<long long>(b) * tp.Tl);
        const long long dst = (static_cast<long long>(b) * tp.T + tp.rank * tp.Tl + t) * tp.push_row_vecs + cv;
        const uint4 u = __ldg(tp.push_src + v);
        if (tp.gather_mc) {
          asm volatile("multimem.st.relaxed.sys.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(tp.gather_mc + dst),
                       "f"(__uint_as_float(u.x)), "f"(__uint_as_float(u.y)), "f"(__uint_as_float(u.z)),
                       "f"(__uint_as_float(u.w))
                       : "memory");
        } else {
          for (int d = 0; d < tp.world; ++d) tp.gather[(tp.rank + d) % tp.world][dst] = u;
        }
      }
      __threadfence_system();
      __syncwarp();
      if (lane < tp.world) tp_red_release_sys(tp.push_arrive[lane] + tp.rank, 1);
    }
    for (int t = pair_id; t < total_tiles && tp_ok; t += num_pairs, ++local) {
      int tm, tn, kb0, kb1;
      decode_tile(t, tm, tn, kb0, kb1);
      const int acc = local & 1;
      if (kb1 <= kb0) continue;
      if (!mbar_wait(&tmem_full[acc], acc_phase[acc]) || *abort_flag) {
        if (lane == 0) atomicCAS(p.err, 0, 114);
        *abort_flag = 1;
        break;
      }
      acc_phase[acc] ^= 1;
      tc_fence_after_sync();
      const int row0 = tm * 256 + cta * BMC + q * 32;
      const uint32_t taddr0 = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BN;
      {
        bool ok = true;
#pragma unroll 1
        for (int c = 0; c < BN && ok; c += 64, ++group) {
          const int col0 = tn * BN + c;
          if (col0 >= p.N) break;
          uint8_t* s0 = wstage + (group & 1) * ((L::kSlots / 2) * kSlotBytes);
          uint8_t* s1 = s0 + kSlotBytes;
          // the slots of this set were last read by the store group issued two groups ago
          if (lane == 0) tma_store_wait_read<1>();
          __syncwarp();
          if (has_operand && lane == 0) {
            mbar_expect_tx(&operand_bar[q], kSlotBytes);
            tma_load_2d(s1, &tma_e, &operand_bar[q], col0, row0);
          }
          uint32_t r0[32], r1[32];
          tmem_ld_32x32(taddr0 + c, r0);
          tmem_ld_32x32(taddr0 + c + 32, r1);
          tmem_ld_wait();
          float v0[32], v1[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v0[j] = __uint_as_float(r0[j]), v1[j] = __uint_as_float(r1[j]);
          if (p.flags & kGemmBias) {
            add_bias32(p, col0, v0);
            add_bias32(p, col0 + 32, v1);
          }
          if (has_operand) {
            if (!mbar_wait(&operand_bar[q], operand_phase) || *abort_flag) {
              if (lane == 0) atomicCAS(p.err, 0, 115);
              *abort_flag = 1;
              ok = false;
            }
            operand_phase ^= 1;
            if (p.flags & kGemmDGelu) {
              stage_fold32<true>(s1, lane, 0, v0);
              stage_fold32<true>(s1, lane, 1, v1);
            } else {
              stage_fold32<false>(s1, lane, 0, v0);
              stage_fold32<false>(s1, lane, 1, v1);
            }
          }
          if (dual) {
            stage_put32_gelu(s0, s1, lane, 0, v0);
            stage_put32_gelu(s0, s1, lane, 1, v1);
          } else {
            stage_put32(s0, lane, 0, v0);
            stage_put32(s0, lane, 1, v1);
          }
          fence_proxy_async_smem();
          __syncwarp();
          bool scattered = false;
          if (tp.mode & kTpScatter) {
            // coalesced 16-byte stores of the slot into this rank's slab on the owner of the rows
            scattered = true;
            const int sh = (row0 % tp.T) / tp.Tl;
            const long long lrow0 = static_cast<long long>(row0 / tp.T) * tp.Tl + (row0 % tp.T) - sh * tp.Tl;
            __nv_bfloat16* dst = tp.slab[sh] + (static_cast<long long>(tp.rank) * tp.batch * tp.Tl + lrow0) * p.N;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int idx = i * 32 + lane, r = idx >> 3, pos = idx & 7;
              const int col = col0 + ((pos ^ (r & 7)) << 3);
              if (col < p.N)
                *reinterpret_cast<uint4*>(dst + static_cast<long long>(r) * p.N + col) =
                    *reinterpret_cast<const uint4*>(s0 + r * 128 + pos * 16);
            }
          }
          if (!scattered && lane == 0 && ok && row0 < p.M) {
            tma_store_2d(&tma_c, s0, col0, row0);
            if (dual) tma_store_2d(&tma_c2, s1, col0, row0);
            tma_store_commit();
          }
        }
        if (tp.mode & kTpScatter) {
          __threadfence_system();
          __syncwarp();
          if (lane == 0) tp_red_release_sys(tp.rs_arrive[(row0 % tp.T) / tp.Tl] + tp.rank, 1);
        }
        if (!ok) break;
      }
      // hand the accumulator back to the leader's MMA warp: one arrival per warp
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&tmem_empty[acc]), 0));
    }
    if (lane == 0) tma_store_wait<0>();   // shared memory stays allocated until the stores have left
  } else {
    // ------------------------------------------------------------ epilogue
    // A warp owns 32 rows x kWarpCols columns of a tile and moves 64 (fp32: 32) columns at a time through its two slots.
    // The operand that is folded in (residual, GELU input) is loaded into the slot that the result leaves from; the
    // first two groups' loads are issued before the accumulator is waited for, as is the load of the bias.
    const int ew = warp - 2, q = warp & 3, warp_col = (ew >> 2) * L::kWarpCols;
    uint8_t* slots = smem + L::kStagingOffset + ew * L::kWarpStaging;
    float* bias_s = reinterpret_cast<float*>(smem + L::kBiasOffset + ew * 256);
    uint64_t* landed = operand_bar + 2 * ew;
    const bool f32 = p.staged == 2;
    const bool has_bias = p.flags & kGemmBias;
    const bool fold = p.staged && (p.flags & (kGemmResidual | kGemmDGelu));
    const bool dual = kWide && (p.flags & kGemmGeluDual);
    const bool add = !kWide && (p.flags & (kGemmAtomic | kGemmAccum));
    const int step = f32 ? 32 : 64;
    uint32_t acc_phase = 0, landed_phase = 0, in_flight = 0;      // a bit per accumulator / slot
    int local = 0, group = 0;
    bool ok = true;
    auto load_operand = [&](int slot, int col, int row) {         // lane 0; the slot has been read
      mbar_expect_tx(&landed[slot], kSlotBytes);
      tma_load_2d(slots + slot * kSlotBytes, &tma_e, &landed[slot], col, row);
    };
    // columns lane and lane + 32 of the group at `col`
    auto load_bias = [&](int col) {
      return make_float2(col + lane < p.N ? __ldg(p.bias + col + lane) : 0.f,
                         !f32 && col + 32 + lane < p.N ? __ldg(p.bias + col + 32 + lane) : 0.f);
    };
    // (a warp that gave up keeps meeting the others at the barrier)
    for (int t = pair_id; t < total_tiles; t += num_pairs, ++local) {
      int tm, tn, kb0, kb1;
      decode_tile(t, tm, tn, kb0, kb1);
      const int acc = local & 1;
      if (kb1 <= kb0) continue;
      const int row0 = tm * 256 + cta * BMC + q * 32;
      const int col_begin = tn * BN + warp_col, col_end = min(col_begin + L::kWarpCols, p.N);
      if (fold && ok) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int col = col_begin + i * step, slot = (group + i) & 1;
          if (col < col_end) {
            if (lane == 0) {
              if (i == 0) tma_store_wait_read<0>();
              load_operand(slot, col, row0);
            }
            in_flight |= 1u << slot;
          }
        }
      }
      float2 bias = make_float2(0.f, 0.f);
      if (has_bias && p.staged) bias = load_bias(col_begin);
      // One warp waits for the accumulator, the others for that warp at a hardware barrier: warps that poll shared memory
      // through the main loop slow it down.
      if (ew == 0 && ok && !mbar_wait_warp(&tmem_full[acc], (acc_phase >> acc) & 1, abort_flag)) {
        if (lane == 0) atomicCAS(p.err, 0, 114);
        *abort_flag = 1;
      }
      epilogue_warps_sync<32 * L::kEpiWarps>();
      if (!ok || *abort_flag) {
        ok = false;
        continue;
      }
      acc_phase ^= 1u << acc;
      tc_fence_after_sync();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BN + warp_col;
      // The accumulator goes back to the leader's MMA warp once its last column is in registers: one arrival per warp.
      // Nothing but those reads has to be ordered, and they have completed: with release semantics at cluster scope the
      // arrival waits for the stores before it (2048 x 2048 x 64: 6.9 -> 6.1 us).
      auto drained = [&]() {
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster_relaxed(mapa_u32(smem_u32(&tmem_empty[acc]), 0));
      };
      if (col_begin >= col_end) {
        drained();
      } else if (!kWide && p.staged == 0) {
#pragma unroll 1
        for (int c = 0; c < L::kWarpCols && col_begin + c < col_end; c += 32) {
          uint32_t r[32];
          tmem_ld_32x32(taddr + c, r);
          tmem_ld_wait();
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
          gemm_epilogue_chunk(p, row0 + lane, row0 + lane < p.M, col_begin + c, v);
        }
        drained();
      } else {
#pragma unroll 1
        for (int c = 0; c < L::kWarpCols; c += step, ++group) {
          const int col0 = col_begin + c, slot = group & 1;
          if (col0 >= col_end) break;
          uint8_t* s0 = slots + (dual ? 0 : slot * kSlotBytes);
          if (!fold && lane == 0) {       // what the slot held has left (a folded operand waited for that)
            if (dual) tma_store_wait_read<0>(); else tma_store_wait_read<1>();
          }
          if (has_bias) {
            bias_s[lane] = bias.x;
            bias_s[lane + 32] = bias.y;
          }
          __syncwarp();
          const bool last = col0 + step >= col_end;
          if (has_bias && !last) bias = load_bias(col0 + step);
          auto operand_landed = [&]() {
            if (!mbar_wait_warp(&landed[slot], (landed_phase >> slot) & 1, abort_flag)) {
              if (lane == 0) atomicCAS(p.err, 0, 115);
              *abort_flag = 1;
              return false;
            }
            landed_phase ^= 1u << slot;
            in_flight &= ~(1u << slot);
            return true;
          };
          if (f32) {
            uint32_t r[32];
            tmem_ld_32x32(taddr + c, r);
            tmem_ld_wait();
            if (last) drained();
            float v[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
            if (has_bias) add_staged_bias32(bias_s, v);
            if (fold) {
              if (!(ok = operand_landed())) break;
              stage_fold32_f32(s0, lane, v);
            }
            stage_put32_f32(s0, lane, v);
          } else {
            uint32_t r0[32], r1[32];
            tmem_ld_32x32(taddr + c, r0);
            tmem_ld_32x32(taddr + c + 32, r1);
            tmem_ld_wait();
            if (last) drained();
            float v0[32], v1[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) v0[j] = __uint_as_float(r0[j]), v1[j] = __uint_as_float(r1[j]);
            if (has_bias) {
              add_staged_bias32(bias_s, v0);
              add_staged_bias32(bias_s + 32, v1);
            }
            if (fold) {
              if (!(ok = operand_landed())) break;
              stage_fold32<kWide>(s0, lane, 0, v0);
              stage_fold32<kWide>(s0, lane, 1, v1);
            }
            if (dual) {
              stage_put32_gelu(s0, s0 + kSlotBytes, lane, 0, v0);
              stage_put32_gelu(s0, s0 + kSlotBytes, lane, 1, v1);
            } else {
              stage_put32(s0, lane, 0, v0);
              stage_put32(s0, lane, 1, v1);
            }
          }
          fence_proxy_async_smem();
          __syncwarp();
          const bool more = fold && col0 + 2 * step < col_end;
          if (lane == 0) {
            if (row0 < p.M) {
              if (add)
                tma_reduce_add_2d(&tma_c, s0, col0, row0);
              else
                tma_store_2d(&tma_c, s0, col0, row0);
              if (dual) tma_store_2d(&tma_c2, s0 + kSlotBytes, col0, row0);
            }
            tma_store_commit();       // an empty group too: the waits above count groups
            if (more) {
              tma_store_wait_read<0>();
              load_operand(slot, col0 + 2 * step, row0);
            }
          }
          if (more) in_flight |= 1u << slot;
        }
      }
    }
    // after an abort: loads still in flight land in this CTA's shared memory
    for (int slot = 0; slot < 2; ++slot)
      if ((in_flight >> slot) & 1) mbar_wait(&landed[slot], (landed_phase >> slot) & 1);
    if (lane == 0) tma_store_wait<0>();   // shared memory stays allocated until the stores have left
  }

  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();      // the peer may still signal this CTA's barriers until it gets here
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
  // Beside the other warp's deallocation, where it costs a launch that succeeds nothing (ahead of the cluster's barrier: 0.08 us).
  // Both CTAs' loads of a stage complete on the leader's barrier; the other CTA gives its own a millisecond.
  if (threadIdx.x == 0 && *abort_flag) {
    if (leader) {
      drain_ring<kStages>(full_bar, *stopped_at);
    } else {
      for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
  }
  if constexpr (kTp) {
    if (tp.mode & kTpScatter) {
      // every rank's partial rows for this rank have to be in the slabs before they are summed
      __shared__ int tail_ok;
      if (threadIdx.x == 0) tail_ok = (*abort_flag == 0);
      __syncthreads();
      const int rows = tp.batch * tp.Tl;
      if (threadIdx.x < tp.world) {
        const int per_launch = (rows / 256) * p.tiles_n * 8;
        if (!tp_wait_ge(tp.rs_arrive[tp.rank] + threadIdx.x, *tp.rs_total + per_launch)) {
          atomicCAS(p.err, 0, 123);
          tail_ok = 0;
        }
      }
      __syncthreads();
      if (tail_ok) {
        const int nv = p.N >> 3;
        const long long total = static_cast<long long>(rows) * nv;
        const uint4* slabs = reinterpret_cast<const uint4*>(tp.slab[tp.rank]);
        for (long long v = static_cast<long long>(blockIdx.x) * L::kThreads + threadIdx.x; v < total;
             v += static_cast<long long>(gridDim.x) * L::kThreads) {
          const long long row = v / nv;
          const int c8 = static_cast<int>(v - row * nv);
          float acc[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[e] = 0.f;
          for (int src = 0; src < tp.world; ++src) {
            const uint4 u = __ldcg(slabs + static_cast<long long>(src) * total + v);
            const __nv_bfloat16* b = reinterpret_cast<const __nv_bfloat16*>(&u);
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] += __bfloat162float(b[e]);
          }
          if (tp.rs_bias) {
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] += __ldg(tp.rs_bias + c8 * 8 + e);
          }
          if (tp.rs_residual) {
            const uint4 u = *reinterpret_cast<const uint4*>(tp.rs_residual + row * tp.rs_ld_res + c8 * 8);
            const __nv_bfloat16* b = reinterpret_cast<const __nv_bfloat16*>(&u);
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] += __bfloat162float(b[e]);
          }
          if (tp.mode & kTpBroadcast) {
            // local row -> row of the full activation; every rank receives the 16 bytes
            const long long bb = row / tp.Tl, tt = row - bb * tp.Tl;
            const long long idx = (bb * tp.T + tp.rank * tp.Tl + tt) * nv + c8;     // in 16-byte units
            const uint4 u = pack8_bf16(acc);
            if (tp.ar_mc) {
              asm volatile("multimem.st.relaxed.sys.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(tp.ar_mc + idx),
                           "f"(__uint_as_float(u.x)), "f"(__uint_as_float(u.y)), "f"(__uint_as_float(u.z)),
                           "f"(__uint_as_float(u.w))
                           : "memory");
            } else {
              for (int d = 0; d < tp.world; ++d)
                reinterpret_cast<uint4*>(tp.ar_out[(tp.rank + d) % tp.world])[idx] = u;
            }
          } else if (tp.rs_out_f32) {
            float* o = static_cast<float*>(tp.rs_out) + row * tp.rs_ld_out + c8 * 8;
            *reinterpret_cast<float4*>(o) = make_float4(acc[0], acc[1], acc[2], acc[3]);
            *reinterpret_cast<float4*>(o + 4) = make_float4(acc[4], acc[5], acc[6], acc[7]);
          } else {
            *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(tp.rs_out) + row * tp.rs_ld_out + c8 * 8) =
                pack8_bf16(acc);
          }
        }
      }
    }
    if (tp.mode & kTpBroadcast) {
      // this CTA's share of the summed rows has left: count it on every rank
      __threadfence_system();
      __syncthreads();
      if (threadIdx.x < tp.world) tp_red_release_sys(tp.ar_arrive[threadIdx.x] + tp.rank, 1);
    }
    // the last CTA to get here advances this GPU's counters for the next launch
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      const unsigned prev = atomicAdd(tp.cta_done, 1u);
      if (prev == gridDim.x - 1) {
        *tp.cta_done = 0;
        *tp.launch_ctr = tp_launch + 1;
        if (tp.mode & kTpPush) *tp.push_total += static_cast<int>(gridDim.x) * 4;
        if (tp.mode & kTpScatter) *tp.rs_total += (tp.batch * tp.Tl / 256) * p.tiles_n * 8;
        if (tp.mode & kTpBroadcast) *tp.ar_total += static_cast<int>(gridDim.x);
        __threadfence();
      }
    }
  }
}

}  // namespace pair
}  // namespace itb
