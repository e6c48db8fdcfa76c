// GEMM whose contraction is split over the thread blocks of a cluster (included by gemm.cu).
//
//   C[M,N] (+)= act( A[M,K] * B[N,K]^T + bias[N] )        operands as in gemm.cu
//
// For few output tiles and a long contraction: 77 tokens through a 14336 x 4096 projection are 32 tiles of 128 columns, and 32
// SMs cannot stream the weights at the rate of the memory.  The S blocks of a cluster take S equal parts of the k blocks of ONE
// 128 x 128 tile; each leaves its fp32 partial tile in its own shared memory (where the operand stages were), and after a cluster
// barrier every block adds 1 / S of the rows of all parts, always in block order, and writes them out.  No scratch in global
// memory, no second launch, no atomics: results repeat themselves bit for bit.
//
// What bounds it is the latency of the loads, then the memory: six stages of 32 KB and one block per SM (77 tokens, 14336 -> 4096 in
// four parts: 43.0 us with three stages and two blocks per SM, 36.9 with six; whole 65.5; 8 us of each are the launch and the events
// around it; the weights alone take 18 at 6.5 TB/s).
// Set-up, cluster barriers and the exchange of the parts are about 6 us: measured on both sides at choose_split.
#pragma once

namespace csb {

constexpr int SK_BN = 128;
constexpr int SK_MAX_SPLIT = 8;  // portable cluster size
constexpr int SK_THREADS = 256;  // warp 0 TMA, warp 1 MMA, warps 4..7 accumulator -> shared memory; all warps add and store

struct SplitKSmem {
  static constexpr int STAGES = 6;
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + SK_BN * BK * 2;
  static constexpr int BAR_OFFSET = STAGES * STAGE_BYTES;  // the partial tile (64 KB) takes the place of the stages
  static constexpr int TOTAL = BAR_OFFSET + (2 * STAGES + 1) * 8 + 16;
  static constexpr int DYN_BYTES = TOTAL + 1024;
  static_assert(BM * SK_BN * 4 <= BAR_OFFSET, "partial tile fits over the stages");
};

// Byte offset of 16-byte piece `c` (of 32) of row r in the partial tile: the pieces of a row are permuted, so that the 32 rows a
// warp writes at one column, and the 32 pieces a warp reads of one row, both fall on different banks.
__device__ __forceinline__ uint32_t sk_offset(int r, int c) { return static_cast<uint32_t>(r * 512 + ((c ^ (r & 31)) << 4)); }

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t map_cluster(uint32_t addr, uint32_t cta_rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta_rank));
  return r;
}

template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__(SK_THREADS, 1)
gemm_splitk_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, const GemmParams p, const int split) {
  using L = SplitKSmem;
  extern __shared__ uint8_t smem_raw[];
  // the same offset in every block of the cluster: dynamic shared memory starts at one address in all blocks of a kernel
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::BAR_OFFSET);
  uint64_t* empty_bar = full_bar + L::STAGES;
  uint64_t* tmem_full = empty_bar + L::STAGES;
  uint32_t* tmem_addr_slot = reinterpret_cast<uint32_t*>(tmem_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_addr_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();
  const int tile = blockIdx.x / split;
  // column tiles slowest: the blocks that run side by side read the same columns of B with all rows of A
  const int m0 = (tile % p.num_m_blocks) * BM, n0 = (tile / p.num_m_blocks) * SK_BN;
  const int kb0 = (int)((long)p.num_k_blocks * rank / split), kb1 = (int)((long)p.num_k_blocks * (rank + 1) / split);
  const int rows = min(BM, p.M - m0);  // rows of the tile that exist

  if (threadIdx.x == 0) {
    for (int s = 0; s < L::STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(tmem_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_b);
  }
  if (warp == 1) {
    tmem_alloc(tmem_addr_slot, SK_BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_addr_slot;

  if (warp == 0) {
    if (lane == 0) {
      for (int kb = kb0, it = 0; kb < kb1; ++kb, ++it) {
        const int s = it % L::STAGES;
        if (!mbar_wait_abort(&empty_bar[s], ((it / L::STAGES) & 1) ^ 1, abort_flag)) {
          atomicExch(p.status, ST_TIMEOUT_EMPTY);
          *abort_flag = 1;
          break;
        }
        uint8_t* sa = smem + s * L::STAGE_BYTES;
        uint8_t* sb = sa + L::A_BYTES;
        const uint32_t bar = smem_u32(&full_bar[s]);
        mbar_expect_tx(&full_bar[s], L::STAGE_BYTES);
        if constexpr (A_MN) {
#pragma unroll
          for (int j = 0; j < BM / 64; ++j) tma_load_2d_to<1>(sa + j * (64 * BK * 2), &tma_a, bar, m0 + j * 64, kb * BK);
        } else {
          tma_load_2d_to<1>(sa, &tma_a, bar, kb * BK, m0);
        }
        if constexpr (B_MN) {
#pragma unroll
          for (int j = 0; j < SK_BN / 64; ++j) tma_load_2d_to<1>(sb + j * (64 * BK * 2), &tma_b, bar, n0 + j * 64, kb * BK);
        } else {
          tma_load_2d_to<1>(sb, &tma_b, bar, kb * BK, n0);
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // the whole warp walks this code in step (see umma_f16_w)
    constexpr uint32_t idesc = make_idesc_bf16(BM, SK_BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
    constexpr int A_STEP = (A_MN ? UMMA_K * 128 : UMMA_K * 2) >> 4, B_STEP = (B_MN ? UMMA_K * 128 : UMMA_K * 2) >> 4;
    const uint32_t sa0 = smem_u32(smem), sb0 = sa0 + L::A_BYTES;
    const uint64_t adesc = A_MN ? make_desc_mnmajor_sw128(sa0, 64 * BK * 2) : make_desc_kmajor_sw128(sa0);
    const uint64_t bdesc = B_MN ? make_desc_mnmajor_sw128(sb0, 64 * BK * 2) : make_desc_kmajor_sw128(sb0);
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!mbar_wait_abort_w(&full_bar[s], ph, abort_flag)) {
        atomicExch(p.status, ST_TIMEOUT_FULL);
        *abort_flag = 1;
        ok = false;
        break;
      }
      tc_fence_after();
      const uint64_t stage = static_cast<uint64_t>((s * L::STAGE_BYTES) >> 4);
      umma_f16_run4_w<A_STEP, B_STEP>(tmem_base, adesc + stage, bdesc + stage, idesc, kb > kb0 ? 1u : 0u);
      umma_commit_w(&empty_bar[s]);
      if (++s == L::STAGES) { s = 0; ph ^= 1u; }
    }
    if (ok) umma_commit_w(tmem_full);
    __syncwarp();
  } else if (warp >= 4) {
    const int quarter = warp & 3, r = quarter * 32 + lane;
    if (mbar_wait_abort_w(tmem_full, 0, abort_flag)) {  // every MMA has retired: the stages are free
      tc_fence_after();
#pragma unroll
      for (int g = 0; g < SK_BN / 32; ++g) {
        uint32_t v[32];
        __syncwarp();
        tmem_ld_32x32(tmem_base + g * 32 + (static_cast<uint32_t>(quarter * 32) << 16), v);
        tmem_ld_wait();
        if (r < rows) {
#pragma unroll
          for (int c = 0; c < 8; ++c)
            *reinterpret_cast<uint4*>(smem + sk_offset(r, g * 8 + c)) = make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
        }
      }
      tc_fence_before();
    } else {
      if (lane == 0) atomicExch(p.status, ST_TIMEOUT_TMEM_FULL);
      *abort_flag = 1;
    }
  }
  __syncwarp();
  cluster_sync_all();  // every block's partial tile is in its shared memory (a block that gave up has set the status word)

  // this block's share of the rows: one warp per row, 16 bytes per lane and part
  {
    const int r0 = rows * rank / split, r1 = rows * (rank + 1) / split;
    const int col = n0 + lane * 4;
    const int n_cols = min(4, p.N - col);
    float bias[4] = {0.f, 0.f, 0.f, 0.f};
    if (p.bias != nullptr) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < n_cols) bias[j] = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.bias)[col + j]);
    }
    const int elem = p.out_fp32 ? 4 : 2;
    const bool vec = n_cols == 4 && ((reinterpret_cast<uintptr_t>(p.C) | ((uintptr_t)p.ldc * elem)) & (4 * elem - 1)) == 0;
    const uint32_t base = smem_u32(smem);
#pragma unroll 2
    for (int r = r0 + warp; r < r1; r += SK_THREADS / 32) {
      const uint32_t off = base + sk_offset(r, lane);
      float4 part[SK_MAX_SPLIT];
#pragma unroll
      for (int s = 0; s < SK_MAX_SPLIT; ++s)
        if (s < split) part[s] = ld_cluster_f4(map_cluster(off, s));
      float f[4] = {part[0].x, part[0].y, part[0].z, part[0].w};
#pragma unroll
      for (int s = 1; s < SK_MAX_SPLIT; ++s)
        if (s < split) {
          f[0] += part[s].x;
          f[1] += part[s].y;
          f[2] += part[s].z;
          f[3] += part[s].w;
        }
#pragma unroll
      for (int j = 0; j < 4; ++j) f[j] = apply_act(f[j] + bias[j], p.act);
      const size_t at = static_cast<size_t>(m0 + r) * p.ldc + col;
      if (p.out_fp32) {
        float* dst = reinterpret_cast<float*>(p.C) + at;
        if (vec) {
          float4 o = make_float4(f[0], f[1], f[2], f[3]);
          if (p.accumulate) {
            const float4 old = *reinterpret_cast<const float4*>(dst);
            o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w;
          }
          *reinterpret_cast<float4*>(dst) = o;
        } else {
          for (int j = 0; j < n_cols; ++j) dst[j] = p.accumulate ? dst[j] + f[j] : f[j];
        }
      } else {
        __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.C) + at;
        if (vec) {
          if (p.accumulate) {
            const uint2 old = *reinterpret_cast<const uint2*>(dst);
            f[0] += __uint_as_float(old.x << 16);
            f[1] += __uint_as_float(old.x & 0xffff0000u);
            f[2] += __uint_as_float(old.y << 16);
            f[3] += __uint_as_float(old.y & 0xffff0000u);
          }
          *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]));
        } else {
          for (int j = 0; j < n_cols; ++j) dst[j] = __float2bfloat16(p.accumulate ? __bfloat162float(dst[j]) + f[j] : f[j]);
        }
      }
    }
  }
  __syncwarp();
  cluster_sync_all();  // nobody leaves while another block reads its part
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, SK_BN);
  }
}

struct SplitKLaunch {
  cudaLaunchAttribute cluster;
  cudaLaunchConfig_t cfg;
  SplitKLaunch(int tiles, int split, cudaStream_t stream) : cfg{} {
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim.x = (unsigned)split;
    cluster.val.clusterDim.y = 1;
    cluster.val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(tiles * split));
    cfg.blockDim = dim3(SK_THREADS);
    cfg.dynamicSmemBytes = SplitKSmem::DYN_BYTES;
    cfg.stream = stream;
    cfg.attrs = &cluster;
    cfg.numAttrs = 1;
  }
};
template <bool A_MN, bool B_MN>
static cudaError_t splitk_prepare() {
  static bool done = false;
  if (done) return cudaSuccess;
  const cudaError_t e =
      cudaFuncSetAttribute(gemm_splitk_kernel<A_MN, B_MN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SplitKSmem::DYN_BYTES);
  done = e == cudaSuccess;
  return e;
}
// Clusters of `split` blocks that the GPU holds at one time when nothing else runs: an SM belongs to one GPC, and what a GPC has left
// over is lost.
static int splitk_clusters(int split) {
  static int n[SK_MAX_SPLIT + 1] = {};  // (a race writes the same number twice; a query that failed is not kept)
  if (n[split] == 0) {
    int c = 0;
    SplitKLaunch l(1, split, nullptr);
    if (splitk_prepare<false, false>() != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&c, (const void*)gemm_splitk_kernel<false, false>, &l.cfg) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    n[split] = c;
  }
  return n[split];
}

template <bool A_MN, bool B_MN>
static int launch_splitk(const void* A, const void* B, const GemmParams& p, int lda, int ldb, int split, cudaStream_t stream) {
  CUtensorMap ta, tb;
  int r = A_MN ? make_tmap_2d_bf16(&ta, A, p.K, p.M, lda, 64, BK) : make_tmap_2d_bf16(&ta, A, p.M, p.K, lda, BK, BM);
  if (r) return r;
  r = B_MN ? make_tmap_2d_bf16(&tb, B, p.K, p.N, ldb, 64, BK) : make_tmap_2d_bf16(&tb, B, p.N, p.K, ldb, BK, SK_BN);
  if (r) return r;
  cudaError_t e = splitk_prepare<A_MN, B_MN>();
  if (e != cudaSuccess) return (int)e;
  SplitKLaunch l(p.num_m_blocks * p.num_n_blocks, split, stream);
  e = cudaLaunchKernelEx(&l.cfg, gemm_splitk_kernel<A_MN, B_MN>, ta, tb, p, split);
  if (e != cudaSuccess) {
    fprintf(stderr, "[cornstarch_b200] cluster launch of the split GEMM failed: %s\n", cudaGetErrorString(e));
    return (int)e;
  }
  return launch_result();
}

}  // namespace csb
