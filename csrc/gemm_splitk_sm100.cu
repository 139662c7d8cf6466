// bf16 GEMM for few output tiles (a decode batch): D[M,N] = A[M,K] * B[N,K]^T, same contract as gemm_2cta_sm100.cu.
//
// A batch of 256 tokens times a 3584 x 4096 weight shard is 14 tiles of 256 x 256: the persistent kernel runs them on 14 of
// 74 CTA pairs, one k loop of 64 blocks each, bound by what one SM takes in (31 us; the weights alone need 4.4 us from
// HBM).  Here a cluster of 2 S CTAs shares one tile: S pairs take K / S each (tcgen05 cta_group::2, as in
// gemm_2cta_sm100.cu), then every pair sends the other pairs their column slices of its fp32 accumulator through
// distributed shared memory and finishes one slice itself.  The S partial sums of an element are added in fp32 in the
// order of K, whatever order the pairs finish in; no workspace, no atomics.
//
// S = 4 when all tiles fit into clusters of eight at once, else S = 2 when they fit into clusters of four; with more tiles
// than that the persistent kernel already fills half of the GPU.  Shorter sums than 16 k blocks do not pay for the exchange.
// Persistent kernel / this one, device time in us: 14 tiles K = 1024 13.0 / 12.0, 4096 26.6 / 15.8, 8192 44.4 / 20.8 (S = 4);
// 32 tiles K = 512 9.0 / 9.9, 1024 11.5 / 11.2, 4096 25.0 / 19.0, 8192 43.4 / 29.8 (S = 2).
#include <cuda.h>
#include <cuda_runtime.h>

#include "gemm_sm100.cuh"
#include "gemm_sm100.h"
#include "pair_pipeline.cuh"
#include "umma_2cta.cuh"

namespace msccl {
namespace sm100 {

namespace {

__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint4 v) {
  asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ float4 ld_shared_v4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// A slice is CW gate columns and the CW up columns beside them (plain epilogue: the same columns).  A partial sum of a
// slice lies in the receiver's former pipeline stages as [sender][column / 4][row][4]: 32 lanes (rows) store 512
// consecutive bytes.
template <int EPI, int S>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_splitk_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                   __nv_bfloat16* __restrict__ d, int M, int N, int K, int ldd, int* error_words) {
  constexpr int H = PBN / 2, CW = H / S;                       // S = 4: 32 columns of each half, S = 2: 64
  constexpr uint32_t kSliceBytes = 2 * CW * BM * 4;            // one sender's partial of a slice
  static_assert((S - 1) * kSliceBytes <= kAgStages * kPStageBytes, "partials must fit into the pipeline stages");
  extern __shared__ uint8_t smem_raw[];
  __shared__ int s_skip;
  const PairPipe p = carve_pair<kAgStages>(smem_raw);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const uint32_t rank = cluster_ctarank();
  const uint32_t leader_rank = rank & ~1u;
  const int r = static_cast<int>(rank & 1u), split = static_cast<int>(rank / 2);
  const bool leader = r == 0;
  const uint16_t pair_mask = static_cast<uint16_t>(3u << leader_rank);
  const int tiles_m = (M + 2 * BM - 1) / (2 * BM), tiles_n = N / PBN;
  int tm, tn;
  tile_coords(static_cast<int>(cluster_id_x()), tiles_m, tiles_n, 8, tm, tn);
  const int k_blocks = K / BK, kb0 = k_blocks * split / S, kb1 = k_blocks * (split + 1) / S;

  // an earlier launch gave up: the first CTA's reading decides for the cluster
  if (threadIdx.x == 0) s_skip = (error_words != nullptr && *reinterpret_cast<volatile int*>(error_words) != 0) ? 1 : 0;
  init_pair<kAgStages>(p);
  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_a);
    prefetch_tensormap(&map_b);
  }
  if (warp == 1) tmem_alloc_pair(p.tmem_slot, PBN);
  tc_fence_before_sync();
  cluster_sync_all();
  tc_fence_after_sync();
  const uint32_t tmem_base = *p.tmem_slot;
  const bool skip = ld_shared_cluster_u32(map_to_cta(smem_u32(&s_skip), 0)) != 0;
  const int quarter = warp % 4;
  const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
  bool ok = !skip;

  if (warp == 0) {
    if (lane == 0 && ok) {
      int stage = 0;
      uint32_t phase = 0;
      const int a_row = tm * 2 * BM + r * BM, b_row = tn * PBN + r * (PBN / 2);
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&p.empty_bar[stage], phase ^ 1, p.abort_flag)) {
          gemm_fail(error_words, p.abort_flag, GEMM_TIMEOUT_EMPTY, 0, stage);
          ok = false;
          break;
        }
        uint8_t* a_dst = p.stage_base + static_cast<size_t>(stage) * kPStageBytes;
        if (leader) mbar_expect_tx(&p.full_bar[stage], 2 * kPStageBytes);
        const uint32_t leader_full = map_to_cta(smem_u32(&p.full_bar[stage]), leader_rank);
        tma_load_2d_pair(a_dst, &map_a, leader_full, kb * BK, a_row);
        tma_load_2d_pair(a_dst + kPABytes, &map_b, leader_full, kb * BK, b_row);
        if (++stage == kAgStages) { stage = 0; phase ^= 1; }
      }
      if (!ok) drain_pair<kAgStages>(p, leader);
    }
  } else if (warp == 1) {
    if (lane == 0 && leader && ok) {
      constexpr uint32_t idesc = idesc_bf16_f32(2 * BM, PBN);
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1 && ok; ++kb) {
        if (!mbar_wait(&p.full_bar[stage], phase, p.abort_flag)) {
          gemm_fail(error_words, p.abort_flag, GEMM_TIMEOUT_FULL, 1, stage);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const uint32_t a_addr = smem_u32(p.stage_base + static_cast<size_t>(stage) * kPStageBytes);
        const uint64_t adesc = smem_desc_sw128(a_addr), bdesc = smem_desc_sw128(a_addr + kPABytes);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          umma_bf16_pair(tmem_base, adesc + static_cast<uint64_t>(k * 2), bdesc + static_cast<uint64_t>(k * 2), idesc, kb > kb0 || k > 0);
        tc_commit_pair(&p.empty_bar[stage], pair_mask);
        if (++stage == kAgStages) { stage = 0; phase ^= 1; }
      }
      if (ok) tc_commit_pair(&p.acc_full[0], pair_mask);
    }
  } else if (ok) {
    ok = mbar_wait(&p.acc_full[0], 0, p.abort_flag);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok && lane == 0) gemm_fail(error_words, p.abort_flag, GEMM_TIMEOUT_ACC, 2, 0);
    tc_fence_after_sync();
  }
  // every accumulator of the cluster is complete: no load is in flight and no MMA reads shared memory any more, so the
  // pipeline stages can take the partial sums.  All threads come here whatever happened to their role.
  __syncwarp();
  cluster_sync_all();
  const uint32_t parts = smem_u32(p.stage_base);
  const uint32_t my_row = static_cast<uint32_t>(quarter * 32 + lane) * 16;
  if (warp >= 2 && ok) {
    for (int dst = 0; dst < S; ++dst) {
      if (dst == split) continue;
      const uint32_t base = map_to_cta(parts, static_cast<uint32_t>(2 * dst + r)) +
                            static_cast<uint32_t>(split < dst ? split : split - 1) * kSliceBytes + my_row;
#pragma unroll 1
      for (int c = 0; c < 2 * CW; c += 32) {
        const int col = c < CW ? dst * CW + c : H + dst * CW + (c - CW);
        uint32_t v[32];
        tmem_ld32(taddr + col, v);
        tc_wait_ld();
#pragma unroll
        for (int q = 0; q < 8; ++q)
          st_cluster_v4(base + static_cast<uint32_t>(c / 4 + q) * (BM * 16), make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]));
      }
    }
  }
  __syncwarp();
  cluster_sync_all();                                          // the partial sums have arrived
  // a pair that gave up has sent nothing: its error word is raised, and nobody stores a result
  if (warp >= 2 && ok && (error_words == nullptr || *reinterpret_cast<volatile int*>(error_words) == 0)) {
    const int row = tm * 2 * BM + r * BM + quarter * 32 + lane;
    // 32 columns of the slice, the partial sums in the order of K
    const auto sum = [&](int c, float (&acc)[32]) {
      const int col = c < CW ? split * CW + c : H + split * CW + (c - CW);
      uint32_t own[32];
      tmem_ld32(taddr + col, own);
      tc_wait_ld();
#pragma unroll
      for (int s = 0; s < S; ++s) {
        if (s == split) {
#pragma unroll
          for (int e = 0; e < 32; ++e) acc[e] = s == 0 ? __uint_as_float(own[e]) : acc[e] + __uint_as_float(own[e]);
        } else {
          const uint32_t base = parts + static_cast<uint32_t>(s < split ? s : s - 1) * kSliceBytes + my_row;
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const float4 v = ld_shared_v4(base + static_cast<uint32_t>(c / 4 + q) * (BM * 16));
            acc[4 * q + 0] = s == 0 ? v.x : acc[4 * q + 0] + v.x;
            acc[4 * q + 1] = s == 0 ? v.y : acc[4 * q + 1] + v.y;
            acc[4 * q + 2] = s == 0 ? v.z : acc[4 * q + 2] + v.z;
            acc[4 * q + 3] = s == 0 ? v.w : acc[4 * q + 3] + v.w;
          }
        }
      }
    };
    const auto store = [&](const float (&o)[32], int col) {
      if (row >= M) return;
      uint4* out = reinterpret_cast<uint4*>(d + static_cast<size_t>(row) * ldd + col);
#pragma unroll
      for (int v = 0; v < 4; ++v)
        out[v] = make_uint4(pack_bf16(o[8 * v], o[8 * v + 1]), pack_bf16(o[8 * v + 2], o[8 * v + 3]),
                            pack_bf16(o[8 * v + 4], o[8 * v + 5]), pack_bf16(o[8 * v + 6], o[8 * v + 7]));
    };
#pragma unroll 1
    for (int c = 0; c < CW; c += 32) {
      float g[32], u[32];
      sum(c, g);
      sum(CW + c, u);
      if (EPI == 0) {
        store(g, tn * PBN + split * CW + c);
        store(u, tn * PBN + H + split * CW + c);
      } else {
#pragma unroll
        for (int e = 0; e < 32; ++e) g[e] = g[e] / (1.0f + __expf(-g[e])) * u[e];
        store(g, tn * H + split * CW + c);
      }
    }
  }
  tc_fence_before_sync();
  __syncwarp();
  cluster_sync_all();                                          // tensor memory of the pair is no longer read
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, PBN);
  }
}

template <int EPI, int S>
void fill_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int clusters, cudaStream_t stream) {
  cfg.gridDim = dim3(static_cast<unsigned int>(2 * S * clusters), 1, 1);
  cfg.blockDim = dim3(kGemmThreads, 1, 1);
  cfg.dynamicSmemBytes = kAgSmemBytes;
  cfg.stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2 * S;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
}

// Clusters of 2 S CTAs that the device holds at once.
template <int EPI, int S>
int max_clusters() {
  static int cached[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && cached[dev] > 0) return cached[dev];
  auto kernel = gemm_splitk_kernel<EPI, S>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kAgSmemBytes)) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  fill_config<EPI, S>(cfg, attr, sm_count() / (2 * S), nullptr);
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  if (dev >= 0 && dev < 64) cached[dev] = clusters;
  return clusters;
}

template <int EPI, int S>
cudaError_t launch_split(const CUtensorMap& map_a, const CUtensorMap& map_b, __nv_bfloat16* d, int M, int N, int K, int ldd,
                         int* error_words, int tiles, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  fill_config<EPI, S>(cfg, attr, tiles, stream);
  return cudaLaunchKernelEx(&cfg, gemm_splitk_kernel<EPI, S>, map_a, map_b, d, M, N, K, ldd, error_words);
}

}  // namespace

// How many ways K is split for this shape: 4, 2, or 1 (the persistent kernel).
int splitk_ways(int M, int N, int K, int epilogue) {
  const int tiles = ((M + 2 * BM - 1) / (2 * BM)) * (N / PBN), k_blocks = K / BK;
  if (k_blocks < 16) return 1;
  if (tiles <= (epilogue ? max_clusters<1, 4>() : max_clusters<0, 4>())) return 4;
  if (tiles <= (epilogue ? max_clusters<1, 2>() : max_clusters<0, 2>())) return 2;
  return 1;
}

cudaError_t gemm_bf16_splitk(const CUtensorMap& map_a, const CUtensorMap& map_b, void* d, int M, int N, int K, int ldd, int epilogue,
                             int* error_words, int ways, cudaStream_t stream) {
  const int tiles = ((M + 2 * BM - 1) / (2 * BM)) * (N / PBN);
  auto* out = static_cast<__nv_bfloat16*>(d);
  if (ways == 4) return epilogue ? launch_split<1, 4>(map_a, map_b, out, M, N, K, ldd, error_words, tiles, stream)
                                 : launch_split<0, 4>(map_a, map_b, out, M, N, K, ldd, error_words, tiles, stream);
  if (ways == 2) return epilogue ? launch_split<1, 2>(map_a, map_b, out, M, N, K, ldd, error_words, tiles, stream)
                                 : launch_split<0, 2>(map_a, map_b, out, M, N, K, ldd, error_words, tiles, stream);
  return cudaErrorInvalidValue;
}

}  // namespace sm100
}  // namespace msccl
