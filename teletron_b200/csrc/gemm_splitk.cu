// K-GEMM for outputs of few tiles: C = epilogue(alpha * A * B^T) with the K range of every 128 x 128 tile cut over a
// cluster of 2, 4 or 8 CTAs.
//
// Why: a 256-token sampling step multiplies 256 x 8960 by 8960 x 1536.  As 256 x 256 tiles on CTA pairs that is 12 busy
// SMs pulling 27 MB of weights through 140 serial steps; cut in four, 96 SMs share the weights.  Each CTA accumulates
// its part in tensor memory and parks it as fp32 in its (then free) operand ring; the CTAs of the cluster then each add
// up their share of the rows from all parts through distributed shared memory, in rank order, and run the epilogue.  No
// workspace, no atomics: the result does not depend on timing.
//
// Roles (320 threads): warp 0 TMA producer, warp 1 tensor memory + MMA issue, warps 2..9 drain the accumulator, all
// threads add up.  Every mbarrier wait is bounded.  The two cluster barriers are reached by every thread of every CTA:
// no role returns early, and one whose wait ran out goes on to them with the abort flag set.
#include <atomic>

#include "gemm_epilogue.cuh"

using namespace tt;
using namespace tt_gemm;

namespace {

constexpr int SK_BN = 128, SK_STAGES = 6;
constexpr int SK_STAGE_BYTES = A_BYTES + SK_BN * BK * 2;
constexpr int SK_LD = SK_BN + 4;  // floats per parked row: rows start four banks apart
constexpr int SK_SMEM = SK_STAGES * SK_STAGE_BYTES + 256 + 1024;
static_assert(128 * SK_LD * 4 <= SK_STAGES * SK_STAGE_BYTES, "the parked tile fits the ring");

template <int A_MN, int B_MN>
__global__ void __launch_bounds__(320, 1)
gemm_splitk_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmParams p,
                   const int split) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + SK_STAGES * SK_STAGE_BYTES);
  uint64_t* empty = full + SK_STAGES;
  uint64_t* tfull = empty + SK_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();
  const int tile = blockIdx.x / split;
  const int tiles_n = (p.N + SK_BN - 1) / SK_BN;
  const int m0 = (tile / tiles_n) * BM, n0 = (tile % tiles_n) * SK_BN;
  const int num_kb = (p.K + BK - 1) / BK;
  const int kb0 = (int)((long long)num_kb * rank / split), kb1 = (int)((long long)num_kb * (rank + 1) / split);

  chain_release();
  if (threadIdx.x == 0) {
    for (int s = 0; s < SK_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, SK_BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  chain_wait();
  float* park = reinterpret_cast<float*>(smem);

  if (warp == 0) {
    if (lane == 0) {
      for (int kb = kb0; kb < kb1; ++kb) {
        const int it = kb - kb0, s = it % SK_STAGES;
        if (!mbar_wait(&empty[s], ((it / SK_STAGES) & 1) ^ 1, abort_flag, p.status, TT_ST_TIMEOUT_PRODUCER)) break;
        uint8_t* sa = smem + s * SK_STAGE_BYTES;
        uint8_t* sb = sa + A_BYTES;
        mbar_expect_tx(&full[s], SK_STAGE_BYTES);
        const int k0 = kb * BK;
        if (A_MN) {
#pragma unroll
          for (int i = 0; i < BM / 64; ++i) tma_load_2d(sa + i * 8192, &tmA, &full[s], m0 + i * 64, k0);
        } else {
          tma_load_2d(sa, &tmA, &full[s], k0, m0);
        }
        if (B_MN) {
#pragma unroll
          for (int i = 0; i < SK_BN / 64; ++i) tma_load_2d(sb + i * 8192, &tmB, &full[s], n0 + i * 64, k0);
        } else {
          tma_load_2d(sb, &tmB, &full[s], k0, n0);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = umma_idesc(BM, SK_BN, A_MN, B_MN);
      constexpr uint32_t HI = umma_desc_hi(1024);
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        const int it = kb - kb0, s = it % SK_STAGES;
        if (!mbar_wait(&full[s], (it / SK_STAGES) & 1, abort_flag, p.status, TT_ST_TIMEOUT_MMA + 2)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t a_base = smem_u32(smem + s * SK_STAGE_BYTES);
        const uint32_t a_lo = umma_desc_lo(a_base, A_MN ? 8192 : 16);
        const uint32_t b_lo = umma_desc_lo(a_base + A_BYTES, B_MN ? 8192 : 16);
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)
          umma_ss_lo<HI, HI>(tmem_base, a_lo + k * ((A_MN ? 2048 : 32) >> 4), b_lo + k * ((B_MN ? 2048 : 32) >> 4), idesc,
                             (it | k) != 0 ? 1u : 0u);
        tc_commit(&empty[s]);
      }
      if (ok) tc_commit(tfull);
    }
  } else {
    // all MMAs done: the ring is no longer read, every copy into it has landed
    const int q = warp & 3, eg = (warp - 2) >> 2;
    if (mbar_wait_warp(tfull, 0, abort_flag, p.status, TT_ST_TIMEOUT_EPILOGUE)) {
      tc_fence_after();
      float* row = park + (q * 32 + lane) * SK_LD;
      for (int c = eg * 2; c < eg * 2 + 2; ++c) {
        uint32_t r[32];
        tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(c * 32), r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j)
          *reinterpret_cast<uint4*>(row + c * 32 + j * 4) = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // every part is parked
  if (!*abort_flag) {
    const int rows = BM / split, r0 = rank * rows;
    const uint32_t park_addr = smem_u32(park);
    for (int i = threadIdx.x; i < rows * (SK_BN / 8); i += 320) {
      const int lr = r0 + i / (SK_BN / 8), c = (i % (SK_BN / 8)) * 8;
      const int row = m0 + lr, col = n0 + c;
      if (row >= p.M || col >= p.N) continue;
      float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int s = 0; s < split; ++s) {
        const uint32_t a = map_to_cta(park_addr + (uint32_t)(lr * SK_LD + c) * 4, s);
        float f[8];
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]) : "r"(a) : "memory");
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(f[4]), "=f"(f[5]), "=f"(f[6]), "=f"(f[7]) : "r"(a + 16) : "memory");
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] += f[j];
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] *= p.alpha;
      const float* gate_row = p.epi == EPI_GATE_RES && p.gate ? p.gate + (long long)(row / p.rows_per_gate) * p.gate_ld : nullptr;
      epilogue_vec(p, v, row, col, reinterpret_cast<bf16*>(p.C) + (long long)row * p.ldc, gate_row);
    }
  } else {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);  // copies still in flight land before the shared memory goes away
  }
  __syncwarp();
  cluster_sync_all();  // the peers have read this CTA's part
  if (warp == 1) tmem_dealloc(tmem_base, SK_BN);
}

template <int A_MN, int B_MN>
int launch_splitk(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmParams& p, int split, cudaStream_t stream) {
  auto kern = gemm_splitk_kernel<A_MN, B_MN>;
  TT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SK_SMEM));
  const int tiles = ((p.M + BM - 1) / BM) * ((p.N + SK_BN - 1) / SK_BN);
  TT_CUDA(tt_launch(kern, dim3(tiles * split), dim3(320), SK_SMEM, stream, split, tmA, tmB, p, split));
  TT_LAUNCH_CHECK();
  return 0;
}

}  // namespace

int tt_gemm::splitk_clusters(int split) {
  constexpr int DEVS = 16;
  static std::atomic<int> known[DEVS][4];  // a property of the device and the kernel; 0: not asked yet
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= DEVS) return 0;
  std::atomic<int>& slot = known[dev][split == 2 ? 1 : split == 4 ? 2 : 3];
  if ((n = slot.load(std::memory_order_relaxed)) == 0) {
    auto kern = gemm_splitk_kernel<0, 0>;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = split;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.gridDim = dim3(split);
    cfg.blockDim = dim3(320);
    cfg.dynamicSmemBytes = SK_SMEM;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SK_SMEM) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    slot.store(n, std::memory_order_relaxed);
  }
  return n;
}

int tt_gemm_splitk(const CUtensorMap& tmA, const CUtensorMap& tmB, int a_mn, int b_mn, const GemmParams& p, int split,
                   cudaStream_t stream) {
  if (!a_mn && !b_mn) return launch_splitk<0, 0>(tmA, tmB, p, split, stream);
  if (!a_mn && b_mn) return launch_splitk<0, 1>(tmA, tmB, p, split, stream);
  if (a_mn && b_mn) return launch_splitk<1, 1>(tmA, tmB, p, split, stream);
  return launch_splitk<1, 0>(tmA, tmB, p, split, stream);
}
