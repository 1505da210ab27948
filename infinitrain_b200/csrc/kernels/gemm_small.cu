// bf16 GEMM for outputs of at most one wave of 128 x 64 tiles.  Same operand layouts and epilogues as the large kernels
// (gemm_tcgen05.cu, gemm_tcgen05_2cta.cu) except for accumulation into the output.
//
// What bounds it is latency: a CTA takes 414 cycles for a k-block of 24 KB (58 bytes a cycle is what reaches an SM from L2)
// and there are few tiles (96 x 768 has 12).  Unless the caller says that the contraction may be split, a CTA walks the whole
// of it in one order, as the large kernels do: a row's bits do not depend on how many rows are computed beside it.
// Where it may be split (kGemmMaySplit: gradients), a cluster of 1, 2, 4 or 8 CTAs computes a tile, each over its share of the
// contraction, and each finishes its share of the tile's rows.  The fp32 partial tiles meet through distributed shared memory:
// a CTA sends each row of its accumulator to the CTA that finishes it, one cluster barrier, and the owner adds the shares in
// order (the result does not depend on who came first, but on how many shares there are).
// Bias, residual and GELU input are loaded into registers before the accumulator is waited for; read afterwards, a row
// per lane, they made an epilogue of 5300 cycles, as long as 13 k-blocks.
//
// The line to the pairs lies where these tiles need a second wave.  us here (one share) / by pairs of 256 x 256, bias and
// residual, operands not in L2, K 768, 3072, 8192: 256 x 768 (24 tiles) 12.3 / 16.4, 20.5 / 27.4, 38.9 / 51.2; 1152 x 1024
// (144) 12.3 / 18.4, 20.5 / 28.7, 41.0 / 53.2; 2368 x 512 (152) 18.4 / 18.4, 34.8 / 28.7, 71.7 / 53.2; 2304 x 1024 (288)
// 19.2 / 18.4, 36.9 / 29.5, 74.5 / 55.3.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <mutex>

#include "../common/ptx.cuh"
#include "gemm_epilogue.cuh"
#include "kernels.h"

namespace itb {

int make_tmap_bf16_2d(CUtensorMap* map, const void* ptr, uint64_t inner, uint64_t outer, uint64_t ld,
                      uint32_t box_inner, uint32_t box_outer);

namespace small {

constexpr int BM = 128, BN = 64, BK = 64;
constexpr int kThreads = 192;                   // TMA warp, MMA warp, four epilogue warps
constexpr int kABytes = BM * BK * 2, kBBytes = BN * BK * 2, kStageBytes = kABytes + kBBytes;
constexpr int kRowBytes = BN * 4;               // of the fp32 tile
template <int kShares>
struct Cfg {
  static constexpr int kStages = kShares == 1 ? 8 : 6;
  static constexpr int kReceiveOffset = kStages * kStageBytes;              // the other CTAs' shares of this one's rows
  static constexpr int kBarOffset = kReceiveOffset + (kShares - 1) * (BM / kShares) * kRowBytes;
  static constexpr int kSmem = kBarOffset + (2 * kStages + 2) * 8 + 16 + 1024;
  static_assert(kSmem <= 232448, "shared memory of one SM");
};

__device__ __forceinline__ void epilogue_warps_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

__device__ __forceinline__ void unpack8(const uint4& u, float (&v)[8]) {
  const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 f = __bfloat1622float2(b[e]);
    v[2 * e] = f.x, v[2 * e + 1] = f.y;
  }
}

template <bool A_MN, bool B_MN, int kShares>
__global__ void __launch_bounds__(kThreads, 1)
gemm_small_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, const GemmDev p) {
  using L = Cfg<kShares>;
  constexpr int kStages = L::kStages;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::kBarOffset);
  uint64_t* empty_bar = full_bar + kStages;
  uint64_t* acc_full = empty_bar + kStages;
  uint64_t* received = acc_full + 1;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(received + 1);
  volatile uint32_t* abort_flag = tmem_holder + 1;
  volatile uint32_t* stopped_at = tmem_holder + 2;      // the TMA warp's place in the ring

  constexpr int kRows = BM / kShares;            // rows of the tile that a CTA finishes
  constexpr int kPasses = kRows / 16;            // 128 threads take 16 rows of 8 x 8 columns at a time
  const int warp = __shfl_sync(~0u, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int rank = kShares > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int tile = static_cast<int>(blockIdx.x) / kShares;
  const int tm = tile % p.tiles_m, tn = tile / p.tiles_m;
  const int kb0 = p.k_blocks * rank / kShares, kb1 = p.k_blocks * (rank + 1) / kShares;      // never empty

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_b);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(received, 1);
    *abort_flag = 0;
    mbar_fence_init();
    if (kShares > 1) mbar_expect_tx(received, (kShares - 1) * kRows * kRowBytes);
  }
  if (warp == 1) {
    tmem_alloc(tmem_holder, BN);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_holder;
  if constexpr (kShares > 1) cluster_arrive();        // waited for before the first copy to another CTA

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1) || *abort_flag) {
          atomicCAS(p.err, 0, 105);
          *abort_flag = 1;
          break;
        }
        uint8_t* sa = smem + stage * kStageBytes;
        uint8_t* sb = sa + kABytes;
        mbar_expect_tx(&full_bar[stage], kStageBytes);
        if constexpr (!A_MN) {
          tma_load_2d(sa, &tma_a, &full_bar[stage], kb * BK, tm * BM);
        } else {
#pragma unroll
          for (int i = 0; i < BM / 64; ++i)
            tma_load_2d(sa + i * (64 * BK * 2), &tma_a, &full_bar[stage], tm * BM + i * 64, kb * BK);
        }
        if constexpr (!B_MN)
          tma_load_2d(sb, &tma_b, &full_bar[stage], kb * BK, tn * BN);
        else
          tma_load_2d(sb, &tma_b, &full_bar[stage], tn * BN, kb * BK);
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1;
        }
      }
      *stopped_at = ring_position(stage, phase);
    }
    __syncwarp();
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc_bf16_f32(BM, BN, A_MN, B_MN);
    int stage = 0;
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!mbar_wait_warp(&full_bar[stage], phase, abort_flag)) {
        atomicCAS(p.err, 0, 106);
        *abort_flag = 1;
        break;
      }
      const uint32_t sa = smem_u32(smem + stage * kStageBytes);
      const uint32_t sb = sa + kABytes;
      const uint64_t adesc0 = A_MN ? make_smem_desc_sw128(sa, 64 * BK * 2, 1024) : make_smem_desc_sw128(sa, 16, 1024);
      const uint64_t bdesc0 = B_MN ? make_smem_desc_sw128(sb, 64 * BK * 2, 1024) : make_smem_desc_sw128(sb, 16, 1024);
#pragma unroll
      for (int k = 0; k < BK / 16; ++k) {
        const uint64_t adesc = adesc0 + (A_MN ? (k * 2048) >> 4 : (k * 32) >> 4);
        const uint64_t bdesc = bdesc0 + (B_MN ? (k * 2048) >> 4 : (k * 32) >> 4);
        umma_f16_ss_elect(tmem_base, adesc, bdesc, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
      }
      umma_commit_elect(&empty_bar[stage]);
      if (kb == kb1 - 1) umma_commit_elect(acc_full);
      if (++stage == kStages) {
        stage = 0;
        phase ^= 1;
      }
    }
  } else {
    // This thread finishes 8 columns (the c8th eight of the tile) of rows row_in, row_in + 16, ... of the CTA's share.
    const int e = static_cast<int>(threadIdx.x) - 64, c8 = e & 7, row_in = e >> 3;
    const int col = tn * BN + c8 * 8, row_begin = tm * BM + rank * kRows + row_in;
    const bool f32 = p.flags & kGemmOutF32, dgelu = p.flags & kGemmDGelu, residual = p.flags & kGemmResidual;
    const bool dual = p.flags & kGemmGeluDual, has_bias = p.flags & kGemmBias;
    auto aligned = [](const void* q, long long ld, int size) {
      return ((reinterpret_cast<uintptr_t>(q) | static_cast<uintptr_t>(ld * size)) & 15) == 0;
    };
    // 16 bytes at a time where all that the epilogue touches allows it; combinations of a residual and GELU's derivative,
    // and of the latter or GELU with an fp32 output, go element by element
    const bool vec = col + 8 <= p.N && aligned(p.C, p.ldc, f32 ? 4 : 2) && !(dgelu && residual) && !(f32 && (dgelu || dual)) &&
                     (!dual || aligned(p.C2, p.ldc, 2)) && (!residual || aligned(p.residual, p.ldr, f32 ? 4 : 2)) &&
                     (!dgelu || aligned(p.aux, p.ld_aux, 2));
    // one CTA a tile and nothing to add: rows leave from registers (1152 x 1024 x 1024: 8.6 -> 8.1 us)
    const bool direct = kShares == 1 && p.flags == 0 && tn * BN + BN <= p.N && aligned(p.C, p.ldc, 2);
    uint4 operand[kPasses], operand_hi[kPasses];      // residual (of fp32 the second four in operand_hi) or GELU input
    float bias[8] = {};
    if (vec) {
      if (has_bias) {
#pragma unroll
        for (int i = 0; i < 8; ++i) bias[i] = __ldg(p.bias + col + i);
      }
      if (dgelu || residual) {
#pragma unroll
        for (int j = 0; j < kPasses; ++j) {
          const long long row = row_begin + j * 16;
          if (row >= p.M) break;
          if (f32) {
            const float* r = static_cast<const float*>(p.residual) + row * p.ldr + col;
            operand[j] = *reinterpret_cast<const uint4*>(r);
            operand_hi[j] = *reinterpret_cast<const uint4*>(r + 4);
          } else {
            operand[j] = *reinterpret_cast<const uint4*>(
                dgelu ? p.aux + row * p.ld_aux + col : static_cast<const __nv_bfloat16*>(p.residual) + row * p.ldr + col);
          }
        }
      }
    }
    if (!mbar_wait_warp(acc_full, 0, abort_flag)) {
      if (lane == 0) atomicCAS(p.err, 0, 107);
      *abort_flag = 1;
    }
    tc_fence_after_sync();
    // Otherwise the accumulator goes through shared memory (over the spent operands), 16-byte pieces in an order within a
    // row's 256 bytes that keeps eight rows on different banks; the rows of another CTA leave from there.
    {
      const int r = (warp & 3) * 32 + lane;
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
      uint32_t v0[32], v1[32];
      tmem_ld_32x32(taddr, v0);
      tmem_ld_32x32(taddr + 32, v1);
      tmem_ld_wait();
      if (direct) {
        const long long row = tm * BM + r;
        if (row < p.M) {
          uint4* out = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.C) + row * p.ldc + tn * BN);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            out[c] = pack8_bf16(reinterpret_cast<const float*>(v0) + 8 * c);
            out[c + 4] = pack8_bf16(reinterpret_cast<const float*>(v1) + 8 * c);
          }
        }
      } else {
        uint8_t* dst = smem + r * kRowBytes;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          *reinterpret_cast<uint4*>(dst + ((c ^ (r & 7)) << 4)) =
              make_uint4(v0[4 * c], v0[4 * c + 1], v0[4 * c + 2], v0[4 * c + 3]);
          *reinterpret_cast<uint4*>(dst + (((c + 8) ^ (r & 7)) << 4)) =
              make_uint4(v1[4 * c], v1[4 * c + 1], v1[4 * c + 2], v1[4 * c + 3]);
        }
      }
    }
    if constexpr (kShares > 1) {
      fence_proxy_async_smem();
      cluster_wait();           // every CTA has started and its barriers are initialised
      epilogue_warps_sync();
      if (warp == 2 && lane < kShares && lane != rank) {
        const int slot = rank < lane ? rank : rank - 1;
        bulk_copy_to_cta(mapa_u32(smem_u32(smem + L::kReceiveOffset + slot * kRows * kRowBytes), lane),
                         smem + lane * kRows * kRowBytes, kRows * kRowBytes, mapa_u32(smem_u32(received), lane));
      }
      __syncwarp();
      if (!mbar_wait_warp(received, 0, abort_flag)) {
        if (lane == 0) atomicCAS(p.err, 0, 108);
        *abort_flag = 1;
      }
    } else {
      epilogue_warps_sync();
    }
    // the shares' sum of row r of the CTA's rows, in the order of the contraction
    auto sum = [&](int r, float (&v)[8]) {
      // lanes 4 to 7 of eight read their odd piece first: eight lanes on different banks
      const int odd = c8 >> 2;
#pragma unroll
      for (int s = 0; s < kShares; ++s) {
        const uint8_t* src = s == rank ? smem + (rank * kRows + r) * kRowBytes
                                       : smem + L::kReceiveOffset + ((s < rank ? s : s - 1) * kRows + r) * kRowBytes;
        const float4 x = *reinterpret_cast<const float4*>(src + (((2 * c8 + odd) ^ (r & 7)) << 4));
        const float4 y = *reinterpret_cast<const float4*>(src + (((2 * c8 + 1 - odd) ^ (r & 7)) << 4));
        const float4 lo = odd ? y : x, hi = odd ? x : y;
        v[0] = s ? v[0] + lo.x : lo.x, v[1] = s ? v[1] + lo.y : lo.y, v[2] = s ? v[2] + lo.z : lo.z, v[3] = s ? v[3] + lo.w : lo.w;
        v[4] = s ? v[4] + hi.x : hi.x, v[5] = s ? v[5] + hi.y : hi.y, v[6] = s ? v[6] + hi.z : hi.z, v[7] = s ? v[7] + hi.w : hi.w;
      }
    };
    if (direct) {
      // done
    } else if (vec) {
#pragma unroll
      for (int j = 0; j < kPasses; ++j) {
        const long long row = row_begin + j * 16;
        if (row >= p.M) break;
        float v[8];
        sum(row_in + j * 16, v);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = has_bias ? v[i] + bias[i] : v[i];
        if (f32) {
          if (residual) {
            const float4 lo = *reinterpret_cast<const float4*>(&operand[j]), hi = *reinterpret_cast<const float4*>(&operand_hi[j]);
            v[0] += lo.x, v[1] += lo.y, v[2] += lo.z, v[3] += lo.w;
            v[4] += hi.x, v[5] += hi.y, v[6] += hi.z, v[7] += hi.w;
          }
          float* out = static_cast<float*>(p.C) + row * p.ldc + col;
          *reinterpret_cast<float4*>(out) = make_float4(v[0], v[1], v[2], v[3]);
          *reinterpret_cast<float4*>(out + 4) = make_float4(v[4], v[5], v[6], v[7]);
        } else {
          if (dgelu || residual) {
            float o[8];
            unpack8(operand[j], o);
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = dgelu ? v[i] * dgelu_tanh(o[i]) : v[i] + o[i];
          }
          const uint4 stored = pack8_bf16(v);
          *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.C) + row * p.ldc + col) = stored;
          if (dual) {             // of the rounded value: all that the backward pass sees
            float h[8];
            unpack8(stored, h);
#pragma unroll
            for (int i = 0; i < 8; ++i) h[i] = gelu_tanh(h[i]);
            *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.C2) + row * p.ldc + col) = pack8_bf16(h);
          }
        }
      }
    } else {
#pragma unroll 1
      for (int j = 0; j < kPasses; ++j) {
        const long long row = row_begin + j * 16;
        if (row >= p.M) break;
        float v[8];
        sum(row_in + j * 16, v);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (col + i >= p.N) continue;
          float x = v[i];
          if (has_bias) x += __ldg(p.bias + col + i);
          if (dgelu) x *= dgelu_tanh(__bfloat162float(p.aux[row * p.ld_aux + col + i]));
          if (residual)
            x += f32 ? static_cast<const float*>(p.residual)[row * p.ldr + col + i]
                     : __bfloat162float(static_cast<const __nv_bfloat16*>(p.residual)[row * p.ldr + col + i]);
          if (f32 && !dual) {
            static_cast<float*>(p.C)[row * p.ldc + col + i] = x;
          } else {
            const __nv_bfloat16 stored = __float2bfloat16(x);
            static_cast<__nv_bfloat16*>(p.C)[row * p.ldc + col + i] = stored;
            if (dual)
              static_cast<__nv_bfloat16*>(p.C2)[row * p.ldc + col + i] = __float2bfloat16(gelu_tanh(__bfloat162float(stored)));
          }
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag) drain_ring<kStages>(full_bar, *stopped_at);
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, BN);
  }
  __syncwarp();
  if constexpr (kShares > 1) {
    // what this CTA sent has been read: whoever arrives has received everything (waits for the first arrival, if the
    // epilogue has not, then for this one)
    if (warp < 2) cluster_wait();
    cluster_sync_all();
  }
}

template <int kShares>
static int count_resident() {
  auto kern = gemm_small_kernel<false, false, kShares>;      // the other layouts take as much
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<kShares>::kSmem) != cudaSuccess) return 0;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = kShares;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.gridDim = dim3(kShares);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = Cfg<kShares>::kSmem;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess) return n;
  cudaGetLastError();       // no answer: such clusters are not used
  return 0;
}

// How many clusters of 2, 4 and 8 CTAs run at the same time on the current device; null when it cannot be told.
static const int* resident_clusters() {
  static int counts[64][3];
  static std::once_flag known[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  std::call_once(known[dev], [dev] {
    counts[dev][0] = count_resident<2>();
    counts[dev][1] = count_resident<4>();
    counts[dev][2] = count_resident<8>();
  });
  return counts[dev];
}

template <bool A_MN, bool B_MN, int kShares>
static int launch_shares(const CUtensorMap& ta, const CUtensorMap& tb, const GemmDev& p, cudaStream_t stream) {
  auto kern = gemm_small_kernel<A_MN, B_MN, kShares>;
  static PerDeviceOnce configured;
  if (configured.first()) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<kShares>::kSmem);
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = kShares;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.gridDim = dim3(p.tiles_m * p.tiles_n * kShares);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = Cfg<kShares>::kSmem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = kShares > 1;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kern, ta, tb, p));
}

template <bool A_MN, bool B_MN>
static int launch(const CUtensorMap& ta, const CUtensorMap& tb, const GemmDev& p, bool may_split, int wanted,
                  cudaStream_t stream) {
  // The most shares for which every cluster runs at once and a share is at least three k-blocks: the exchange costs as
  // much as two or three.  us with 1 / 2 / 4 / 8 shares, operands not in L2: 96 x 768 (12 tiles) at K 256 / 768 / 3072
  // 4.7 / 5.2 / 4.9 / -, 6.8 / 6.2 / 5.4 / 5.3, 15.0 / 10.3 / 7.4 / 6.5; 512 x 768 (48 tiles) at 3072 16.1 / 10.9 / 15.2 / 24.5.
  int shares = 1;
  if (may_split) {
    const int* resident = resident_clusters();
    for (int i = 0; i < 3; ++i) {
      const int s = 2 << i;
      const bool fits = resident && p.tiles_m * p.tiles_n <= resident[i] && p.k_blocks >= 3 * s;
      if (wanted > 0 ? s <= wanted && s <= p.k_blocks : fits) shares = s;
    }
  }
  if (shares == 8) return launch_shares<A_MN, B_MN, 8>(ta, tb, p, stream);
  if (shares == 4) return launch_shares<A_MN, B_MN, 4>(ta, tb, p, stream);
  if (shares == 2) return launch_shares<A_MN, B_MN, 2>(ta, tb, p, stream);
  return launch_shares<A_MN, B_MN, 1>(ta, tb, p, stream);
}

}  // namespace small
}  // namespace itb

extern "C" int itb_gemm_small(const ItbGemmArgs* a, cudaStream_t stream) {
  using namespace itb;
  using namespace itb::small;
  if (a->M <= 0 || a->N <= 0 || a->K <= 0) return 0;
  if ((reinterpret_cast<uintptr_t>(a->A) & 15) || (reinterpret_cast<uintptr_t>(a->B) & 15) || (a->lda % 8) || (a->ldb % 8))
    return -2;
  CUtensorMap ta, tb;
  int rc = a->a_mn_major ? make_tmap_bf16_2d(&ta, a->A, a->M, a->K, a->lda, 64, 64)
                         : make_tmap_bf16_2d(&ta, a->A, a->K, a->M, a->lda, 64, BM);
  if (!rc)
    rc = a->b_mn_major ? make_tmap_bf16_2d(&tb, a->B, a->N, a->K, a->ldb, 64, 64)
                       : make_tmap_bf16_2d(&tb, a->B, a->K, a->N, a->ldb, 64, BN);
  if (rc) return rc;
  GemmDev p = {};
  p.M = a->M;
  p.N = a->N;
  p.K = a->K;
  p.k_blocks = (a->K + BK - 1) / BK;
  p.tiles_m = (a->M + BM - 1) / BM;
  p.tiles_n = (a->N + BN - 1) / BN;
  p.C = a->C;
  p.ldc = a->ldc;
  p.C2 = a->C2;
  p.bias = a->bias;
  p.residual = a->residual;
  p.ldr = a->ldr;
  p.aux = static_cast<const __nv_bfloat16*>(a->aux);
  p.ld_aux = a->ld_aux;
  p.flags = a->flags & ~kGemmMaySplit;
  p.err = a->err;
  const bool amn = a->a_mn_major, bmn = a->b_mn_major, may_split = a->flags & kGemmMaySplit;
  if (!amn && !bmn) return launch<false, false>(ta, tb, p, may_split, a->split_k, stream);
  if (!amn && bmn) return launch<false, true>(ta, tb, p, may_split, a->split_k, stream);
  if (amn && bmn) return launch<true, true>(ta, tb, p, may_split, a->split_k, stream);
  return launch<true, false>(ta, tb, p, may_split, a->split_k, stream);
}
