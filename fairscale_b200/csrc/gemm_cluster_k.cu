// bf16 GEMM for products with few output tiles: the K range of one tile is split over the CTAs of a cluster.
//
//   C[M,N] = epilogue( sum_k A(m,k) * B(n,k) )        operands, layouts and epilogues as in gemm_tcgen05.cu
//
// The persistent kernels of gemm_tcgen05.cu give a whole K loop to one CTA or CTA pair.  A product with few 256-wide
// tiles (a short prompt through every matrix, a weight gradient of a small matrix over many tokens) then runs on a
// handful of SMs, each bound by the latency of its own operand stream.  Here a tile is 128 x 64 or 128 x 128 and
// `splits` (1, 2, 4 or 8) CTAs of one cluster take a slice of K each, so that about all SMs load at once:
//
//   warp 0      TMA producer (192 KB of operand stages: for the short slices of this kernel most of the slice in flight)
//   warp 1      TMEM owner and tcgen05.mma issuer
//   warps 2..5  drain the accumulator; with splits > 1 each CTA leaves its fp32 partial tile in its own shared memory
//               (over the operand ring, which is idle by then), and after a cluster barrier every CTA sums 128 / splits
//               rows over the cluster through distributed shared memory, in rank order: no workspace, no atomics, the
//               same bits every time.
//
// Every load is a per-CTA TMA load of this GPU's own memory and every mbarrier wait is bounded.

#include "gemm_tile.cuh"

namespace fsb {

constexpr int CK_THREADS = 192;

template <int BN>
struct CkSmem {
  static constexpr int A_BYTES = BLOCK_M * BLOCK_K * 2;
  static constexpr int B_BYTES = BN * BLOCK_K * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = BN == 64 ? 8 : 6;
  static constexpr int BAR_OFFSET = STAGES * STAGE_BYTES;
  static constexpr int TOTAL = BAR_OFFSET + 256 + 1024;
  static_assert(BN * BLOCK_M * 4 <= STAGES * STAGE_BYTES, "the fp32 partial tile fits over the operand ring");
};

__device__ __forceinline__ float ld_shared_cluster_f32(uint32_t cluster_addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cluster_addr) : "memory");
  return v;
}

// Epilogue of eight consecutive columns of one row.  `vec`: rows of C and aux start on 16-byte boundaries.
__device__ __forceinline__ void epilogue_cols8(float (&v)[8], int row, int col, const GemmParams& p, bool vec) {
  if (row >= p.M || col >= p.N) return;
  const bool full = vec && col + 8 <= p.N;
  const int n = min(8, p.N - col);
  const int epi = p.epilogue;
  if (epi == EPI_BIAS || epi == EPI_BIAS_GELU || epi == EPI_BIAS_RESIDUAL) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i < n) v[i] += __bfloat162float(p.bias[col + i]);
  }
  if (epi == EPI_BIAS_GELU) {
    if (p.aux_out != nullptr) {
      __nv_bfloat16* po = p.aux_out + static_cast<size_t>(row) * p.ld_aux + col;
      Vec16<__nv_bfloat16> o;
#pragma unroll
      for (int i = 0; i < 8; ++i) o.v[i] = __float2bfloat16_rn(v[i]);
      if (full) st16(po, o);
      else {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (i < n) po[i] = o.v[i];
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = gelu_erf(v[i]);
  } else if (epilogue_needs_aux(epi)) {
    const __nv_bfloat16* pa = p.aux + static_cast<size_t>(row) * p.ld_aux + col;
    Vec16<__nv_bfloat16> a;
    if (full) a = ld16(pa);
    else {
#pragma unroll
      for (int i = 0; i < 8; ++i) a.v[i] = i < n ? pa[i] : __float2bfloat16_rn(0.f);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float f = __bfloat162float(a.v[i]);
      v[i] = epi == EPI_DGELU ? v[i] * gelu_erf_grad(f) : v[i] + f;
    }
  }
  if (p.out_f32) {
    float* pc = reinterpret_cast<float*>(p.C) + static_cast<size_t>(row) * p.ldc + col;
    if (full && !p.accumulate_c) {
      *reinterpret_cast<float4*>(pc) = make_float4(v[0], v[1], v[2], v[3]);
      *reinterpret_cast<float4*>(pc + 4) = make_float4(v[4], v[5], v[6], v[7]);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i < n) pc[i] = p.accumulate_c ? pc[i] + v[i] : v[i];
    }
  } else {
    __nv_bfloat16* pc = reinterpret_cast<__nv_bfloat16*>(p.C) + static_cast<size_t>(row) * p.ldc + col;
    Vec16<__nv_bfloat16> o;
#pragma unroll
    for (int i = 0; i < 8; ++i) o.v[i] = __float2bfloat16_rn(v[i]);
    if (full) st16(pc, o);
    else {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i < n) pc[i] = o.v[i];
    }
  }
}

// grid.x = tiles * splits, clusters of `splits` CTAs along x: the CTAs of one tile are one cluster
template <int BN>
__global__ void __launch_bounds__(CK_THREADS, 1)
gemm_cluster_k_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, GemmParams p, int splits) {
  using L = CkSmem<BN>;
  constexpr int NST = L::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::BAR_OFFSET);
  uint64_t* empty_bar = full_bar + NST;
  uint64_t* done_bar = empty_bar + NST;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);  // warp-uniform
  const int lane = threadIdx.x & 31;
  const int rank = splits > 1 ? static_cast<int>(cluster_ctarank()) : 0;

  const int tiles_m = (p.M + BLOCK_M - 1) / BLOCK_M;
  const int tiles_n = (p.N + BN - 1) / BN;
  const int num_kb = (p.K + BLOCK_K - 1) / BLOCK_K;
  const int kb0 = rank * num_kb / splits, kb1 = (rank + 1) * num_kb / splits;  // never empty: splits <= num_kb
  int tm, tn;
  tile_coords(static_cast<int>(blockIdx.x) / splits, tiles_m, tiles_n, tm, tn);
  const int m0 = tm * BLOCK_M, n0 = tn * BN;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < NST; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(done_bar, 1);
    fence_barrier_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, BN);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  const bool reduce = splits > 1;
  float* part = reinterpret_cast<float*>(smem);  // [BN][128] fp32 partial tile, one column after the other
  const uintptr_t ptrs = reinterpret_cast<uintptr_t>(p.C) | reinterpret_cast<uintptr_t>(p.aux) | reinterpret_cast<uintptr_t>(p.aux_out);
  const bool vec = p.ldc % 8 == 0 && p.ld_aux % 8 == 0 && (ptrs & 15u) == 0;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1u, abort_flag, 100)) break;
        uint8_t* sa = smem + stage * L::STAGE_BYTES;
        uint8_t* sb = sa + L::A_BYTES;
        mbar_expect_tx(&full_bar[stage], L::STAGE_BYTES);
        const int k0 = kb * BLOCK_K;
        if (!p.a_mn_major) {
          tma_load_2d(sa, &tmap_a, &full_bar[stage], k0, m0);
        } else {
#pragma unroll
          for (int j = 0; j < BLOCK_M / 64; ++j) tma_load_2d(sa + j * 8192, &tmap_a, &full_bar[stage], m0 + j * 64, k0);
        }
        if (!p.b_mn_major) {
          tma_load_2d(sb, &tmap_b, &full_bar[stage], k0, n0);
        } else {
#pragma unroll
          for (int j = 0; j < BN / 64; ++j) tma_load_2d(sb + j * 8192, &tmap_b, &full_bar[stage], n0 + j * 64, k0);
        }
        if (++stage == NST) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (the whole warp)
    const uint32_t idesc = make_idesc_f16(BLOCK_M, BN, true, p.a_mn_major != 0, p.b_mn_major != 0);
    const uint32_t a_lbo = p.a_mn_major ? 8192u : 16u, b_lbo = p.b_mn_major ? 8192u : 16u;
    const uint32_t a_kstep = p.a_mn_major ? 2048u : 32u, b_kstep = p.b_mn_major ? 2048u : 32u;
    const uint64_t adesc0 = make_smem_desc(smem_u32(smem), a_lbo, 1024u), bdesc0 = make_smem_desc(smem_u32(smem) + L::A_BYTES, b_lbo, 1024u);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!mbar_wait_warp(&full_bar[stage], phase, abort_flag, 101)) { ok = false; break; }
      tc_fence_after_sync();
      const uint64_t ad = desc_offset(adesc0, stage * L::STAGE_BYTES), bd = desc_offset(bdesc0, stage * L::STAGE_BYTES);
#pragma unroll
      for (int k = 0; k < BLOCK_K / UMMA_K; ++k)
        umma_f16_ss_warp(tmem_base, desc_offset(ad, k * a_kstep), desc_offset(bd, k * b_kstep), idesc, (kb != kb0 || k != 0) ? 1u : 0u);
      umma_commit_warp(&empty_bar[stage]);
      if (++stage == NST) { stage = 0; phase ^= 1u; }
    }
    if (ok) umma_commit_warp(done_bar);
  } else {
    // ------------------------------------------------------------------ accumulator -> partial tile, or straight to the epilogue
    const int quad = warp & 3;
    const uint32_t t_base = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    const int row = quad * 32 + lane;
    if (mbar_wait(done_bar, 0, abort_flag, 102)) {
      tc_fence_after_sync();
      if (!reduce && epilogue_can_coalesce(p)) {
        uint4 pre[8];
        if (epilogue_needs_aux(p.epilogue)) epi_slab_prefetch(pre, p.aux, p.ld_aux, m0 + quad * 32, n0, p.M, p.N, lane);
        epilogue_rows_coalesced(t_base, m0 + quad * 32, n0, BN, p, smem + quad * 4096, lane, pre);
      } else {
#pragma unroll 1
        for (int c = 0; c < BN; c += 32) {
          uint32_t r[32];
          tmem_ld_32x32(t_base + static_cast<uint32_t>(c), r);
          tmem_ld_wait();
          if (reduce) {
#pragma unroll
            for (int i = 0; i < 32; ++i) part[(c + i) * BLOCK_M + row] = __uint_as_float(r[i]);
          } else {
#pragma unroll
            for (int g = 0; g < 32; g += 8) {
              float v[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[g + i]);
              epilogue_cols8(v, m0 + row, n0 + c + g, p, vec);
            }
          }
        }
      }
    }
  }

  __syncwarp();
  if (reduce) {
    cluster_sync_all();  // every CTA's partial tile is in place
    if (warp >= 2 && *abort_flag == 0) {
      const int t = static_cast<int>(threadIdx.x) - 64;
      const int rows = BLOCK_M / splits, cols = BN / splits;  // this thread: one row, `cols` (>= 8) consecutive columns
      const int row = rank * rows + t % rows, col0 = (t / rows) * cols;
      for (int c = col0; c < col0 + cols; c += 8) {
        float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        const uint32_t addr = smem_u32(part + c * BLOCK_M + row);
        for (int r = 0; r < splits; r += 2) {  // two CTAs' sixteen loads in flight
          const uint32_t a0 = map_to_cta(addr, static_cast<uint32_t>(r)), a1 = map_to_cta(addr, static_cast<uint32_t>(r + 1));
          float x[8], y[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) x[i] = ld_shared_cluster_f32(a0 + static_cast<uint32_t>(i * BLOCK_M * 4));
#pragma unroll
          for (int i = 0; i < 8; ++i) y[i] = ld_shared_cluster_f32(a1 + static_cast<uint32_t>(i * BLOCK_M * 4));
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = (v[i] + x[i]) + y[i];
        }
        epilogue_cols8(v, m0 + row, n0 + c, p, vec);
      }
    }
    __syncwarp();
    cluster_sync_all();  // no CTA leaves while another one may still read its partial tile
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    if (threadIdx.x == 0 && p.status != nullptr) atomicExch(p.status, FSB_ERR_WAIT_TIMEOUT | (*abort_flag << 8));
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, BN);
  }
}

}  // namespace fsb

namespace fsb_host {

template <int BN>
static int launch_cluster_k(const CUtensorMap& ta, const CUtensorMap& tb, const fsb::GemmParams& p, int splits, int dev, cudaStream_t stream) {
  using L = fsb::CkSmem<BN>;
  static bool attr_set[64] = {false};
  if (!attr_set[dev & 63]) {
    const cudaError_t e = cudaFuncSetAttribute(fsb::gemm_cluster_k_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_set[dev & 63] = true;
  }
  const int tiles = ((p.M + fsb::BLOCK_M - 1) / fsb::BLOCK_M) * ((p.N + BN - 1) / BN);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(tiles * splits));
  cfg.blockDim = dim3(fsb::CK_THREADS);
  cfg.dynamicSmemBytes = L::TOTAL;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(splits);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, fsb::gemm_cluster_k_kernel<BN>, ta, tb, p, splits));
}

// block_n 64 or 128; splits 1, 2, 4 or 8 and at most the number of 64-wide K blocks.  `p` is complete except for what only
// the persistent kernels read; `ta` is the tensor map of A with the box of gemm_tcgen05.cu.
int gemm_cluster_k(const CUtensorMap& ta, const void* B, int ldb, const fsb::GemmParams& p, int block_n, int splits, int dev, cudaStream_t stream) {
  using namespace fsb;
  const int num_kb = (p.K + BLOCK_K - 1) / BLOCK_K;
  if ((block_n != 64 && block_n != 128) || (splits != 1 && splits != 2 && splits != 4 && splits != 8) || splits > num_kb) return -1;
  CUtensorMap tb;
  const bool ok = !p.b_mn_major ? encode_2d_16bit(&tb, B, (uint64_t)p.K, (uint64_t)p.N, (uint64_t)ldb, BLOCK_K, block_n)
                                : encode_2d_16bit(&tb, B, (uint64_t)p.N, (uint64_t)p.K, (uint64_t)ldb, 64, BLOCK_K);
  if (!ok) return -1;
  return block_n == 64 ? launch_cluster_k<64>(ta, tb, p, splits, dev, stream) : launch_cluster_k<128>(ta, tb, p, splits, dev, stream);
}

}  // namespace fsb_host
