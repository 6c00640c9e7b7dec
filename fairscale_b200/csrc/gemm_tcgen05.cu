// bf16 GEMM on the 5th-generation tensor cores (tcgen05) with fused epilogues.
//
//   C[M,N] = epilogue( sum_k A(m,k) * B(n,k) )        fp32 accumulation in TMEM
//
// A and B are bf16 and can each be stored K-major ([rows, K], K contiguous) or MN-major
// ([K, rows], rows contiguous); this covers the three products of a linear layer without any
// transposed copy:
//   forward  Y  = X  W^T : A = X  (K-major),  B = W  (K-major)
//   dgrad    dX = dY W   : A = dY (K-major),  B = W  (MN-major, stored [N_out... see gemm.py)
//   wgrad    dW = dY^T X : A = dY (MN-major), B = X  (MN-major)
//
// Structure: persistent kernel, one CTA per SM, 192 threads, tiles handed out at run time.
//   warp 0      TMA producer: 128-byte-swizzled 64-wide K slabs of A and B into a 4-stage smem ring
//   warp 1      allocates TMEM (2 x BLOCK_N fp32 columns) and issues tcgen05.mma (the whole warp, umma_f16_ss_warp)
//   warps 2..5  epilogue: tcgen05.ld the finished accumulator (each warp its 32-lane quadrant),
//               apply bias / GELU / GELU' / residual, convert and store; overlaps the next tile's
//               main loop because the accumulator is double-buffered in TMEM.
// All loads are per-CTA TMA loads of this GPU's own memory. Every mbarrier wait is bounded.
//
// Replaces the cuBLAS calls behind F.linear in the reference
// (fairscale/nn/model_parallel/layers.py:290,380 and every nn.Linear of its benchmark models).

#include "gemm_tile.cuh"

#include <cstdlib>
#include <mutex>
#include <unordered_map>

namespace fsb {

constexpr int SCHED_DEPTH = 4;  // tile indices in flight between a CTA's (pair's) scheduler and its readers

// Counters of the run-time tile hand-out, two per slot: tiles handed out, CTAs (pairs) that have finished.  All zero while no
// kernel uses them (the last CTA of a launch puts its slot back).  A slot belongs to one stream, so the launches that share
// it are ordered; slot 0 stands for "no counter" (see sched_slot_of).
constexpr int SCHED_SLOTS = 256;
__device__ unsigned int g_sched_counters[2 * SCHED_SLOTS];

// BATCHED (both kernels): the tensor maps are 3-D (K / MN, rows, problem) and a tile index also selects the problem; used
// for the local experts of an MoE layer (equal capacity per expert), where one launch replaces a Python loop of GEMMs.
template <int BLOCK_N, bool BATCHED>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_bf16_tcgen05_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, GemmParams p) {
  using L = SmemLayout<BLOCK_N>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::BAR_OFFSET);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tmem_full_bar = empty_bar + STAGES;
  uint64_t* tmem_empty_bar = tmem_full_bar + 2;
  uint64_t* sched_full = tmem_empty_bar + 2;              // [SCHED_DEPTH] the slot holds a tile index
  uint64_t* sched_empty = sched_full + SCHED_DEPTH;       // [SCHED_DEPTH] every reader has taken it
  volatile int* sched_tile = reinterpret_cast<volatile int*>(sched_empty + SCHED_DEPTH);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(const_cast<int*>(sched_tile) + SCHED_DEPTH);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);  // warp-uniform
  const int lane = threadIdx.x & 31;

  const int tiles_m = (p.M + BLOCK_M - 1) / BLOCK_M;
  const int tiles_n = (p.N + BLOCK_N - 1) / BLOCK_N;
  const int tiles_per_problem = tiles_m * tiles_n;
  const int num_tiles = tiles_per_problem * (BATCHED ? p.batch : 1);
  const int num_kb = (p.K + BLOCK_K - 1) / BLOCK_K;
  auto load_tile = [&](uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
    if (BATCHED) tma_load_3d_warp(dst, map, bar, x, y, z);
    else         tma_load_2d_warp(dst, map, bar, x, y);
  };

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full_bar[a], 1);
      mbar_init(&tmem_empty_bar[a], 4);  // one arrival per epilogue warp
    }
    for (int q = 0; q < SCHED_DEPTH; ++q) {
      mbar_init(&sched_full[q], 1);
      mbar_init(&sched_empty[q], 5);  // the MMA warp and the epilogue warps
    }
    fence_barrier_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 2 * BLOCK_N);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  // Every CTA starts with the tile of its own index; the tiles after those are handed out at run time, as in the CTA-pair
  // kernel below and for the same reason: the producer takes the next index from a counter in global memory and publishes it
  // (or -1 at the end) through a small ring that the other roles read in order.  A launch with one tile per CTA never
  // touches the counter; one without a counter (p.sched_slot 0) strides through the tiles, which is up to 3 % faster on a
  // device that nothing else uses (16384 x 2048 x 2048: 100 against 102 us).
  int q = 0;            // this role's position in the ring
  uint32_t qphase = 0;
  unsigned int* const sched = g_sched_counters + 2 * p.sched_slot;
  const bool counted = num_tiles > static_cast<int>(gridDim.x) && p.sched_slot != 0;
  // Reader side, by all lanes of a warp: the next tile (-1: no more, -2: the wait ran out).
  auto take_tile = [&]() -> int {
    int t = -2;
    if (lane == 0 && mbar_wait(&sched_full[q], qphase, abort_flag)) {
      t = sched_tile[q];
      mbar_arrive(&sched_empty[q]);
    }
    if (++q == SCHED_DEPTH) { q = 0; qphase ^= 1u; }
    return __shfl_sync(0xffffffffu, t, 0);
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (the whole warp, as in the CTA-pair kernel below and for the same reason)
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    auto fetch = [&](int before) -> int {  // `before`: the last index this CTA was given; lane 0 holds the result
      return static_cast<int>(gridDim.x) + (counted ? (lane == 0 ? static_cast<int>(atomicAdd(&sched[0], 1u)) : 0) : before);
    };
    const uint32_t smem0 = smem_u32(smem), full0 = smem_u32(full_bar);
    int nxt = fetch(static_cast<int>(blockIdx.x));  // needed when the first tile's loads are all on their way
    for (int tile = blockIdx.x, next_tile = -1; tile >= 0 && ok; tile = next_tile) {
      const int pb = BATCHED ? tile / tiles_per_problem : 0;
      int tm, tn;
      tile_coords(tile - pb * tiles_per_problem, tiles_m, tiles_n, tm, tn);
      const int m0 = tm * BLOCK_M, n0 = tn * BLOCK_N;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!mbar_wait_warp(&empty_bar[stage], phase ^ 1u, abort_flag)) { ok = false; break; }
        const uint32_t sa = smem0 + stage * L::STAGE_BYTES, sb = sa + L::A_BYTES, bar = full0 + stage * 8;
        mbar_expect_tx_warp(bar, L::STAGE_BYTES);
        const int k0 = kb * BLOCK_K;
        if (!p.a_mn_major) {
          load_tile(sa, &tmap_a, bar, k0, m0, pb);
        } else {
#pragma unroll
          for (int j = 0; j < BLOCK_M / 64; ++j) load_tile(sa + j * 8192, &tmap_a, bar, m0 + j * 64, k0, pb);
        }
        if (!p.b_mn_major) {
          load_tile(sb, &tmap_b, bar, k0, n0, pb);
        } else {
#pragma unroll
          for (int j = 0; j < BLOCK_N / 64; ++j) load_tile(sb + j * 8192, &tmap_b, bar, n0 + j * 64, k0, pb);
        }
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
      if (!ok) break;
      // the other roles are a ring of loads behind and look for the next index after this
      nxt = __shfl_sync(0xffffffffu, nxt, 0);
      next_tile = nxt < num_tiles ? nxt : -1;
      if (!mbar_wait_warp(&sched_empty[q], qphase ^ 1u, abort_flag)) break;
      if (lane == 0) {
        sched_tile[q] = next_tile;
        mbar_arrive(&sched_full[q]);
      }
      __syncwarp();
      if (++q == SCHED_DEPTH) { q = 0; qphase ^= 1u; }
      if (next_tile >= 0) nxt = fetch(next_tile);  // used one tile from now
    }
    if (counted && lane == 0) {
      // The last CTA to get here has seen every CTA's final fetch (each adds to sched[1] after the value of its last fetch
      // came back, so no fence is needed): put the counters back for the next launch.
      if (atomicAdd(&sched[1], 1u) == gridDim.x - 1u) {
        sched[0] = 0u;
        sched[1] = 0u;
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (the whole warp, see umma_f16_ss_warp)
    {
      const uint32_t idesc = make_idesc_f16(BLOCK_M, BLOCK_N, true, p.a_mn_major != 0, p.b_mn_major != 0);
      // K-major: LBO unused, SBO 1024; UMMA_K advance = 32 B inside the swizzle row.
      // MN-major: LBO = 8192 (next 64 MN elements), SBO 1024; UMMA_K advance = 16 k-rows = 2048 B.
      const uint32_t a_lbo = p.a_mn_major ? 8192u : 16u, b_lbo = p.b_mn_major ? 8192u : 16u;
      const uint32_t a_kstep = p.a_mn_major ? 2048u : 32u, b_kstep = p.b_mn_major ? 2048u : 32u;
      const uint64_t adesc0 = make_smem_desc(smem_u32(smem), a_lbo, 1024u), bdesc0 = make_smem_desc(smem_u32(smem) + L::A_BYTES, b_lbo, 1024u);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile >= 0 && ok; tile = take_tile()) {
        if (!mbar_wait_warp(&tmem_empty_bar[acc], acc_phase ^ 1u, abort_flag)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * BLOCK_N);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait_warp(&full_bar[stage], phase, abort_flag)) { ok = false; break; }
          tc_fence_after_sync();
          const uint64_t ad = desc_offset(adesc0, stage * L::STAGE_BYTES), bd = desc_offset(bdesc0, stage * L::STAGE_BYTES);
#pragma unroll
          for (int k = 0; k < BLOCK_K / UMMA_K; ++k)
            umma_f16_ss_warp(d_tmem, desc_offset(ad, k * a_kstep), desc_offset(bd, k * b_kstep), idesc, (kb | k) != 0 ? 1u : 0u);
          umma_commit_warp(&empty_bar[stage]);  // frees the smem slot once these MMAs have read it
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        umma_commit_warp(&tmem_full_bar[acc]);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue warps
    const int quad = warp & 3;  // TMEM lane quadrant this warp may access
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile >= 0 && ok; tile = take_tile()) {
      const int pb = BATCHED ? tile / tiles_per_problem : 0;
      int tm, tn;
      tile_coords(tile - pb * tiles_per_problem, tiles_m, tiles_n, tm, tn);
      const int row = tm * BLOCK_M + quad * 32 + lane;
      const int n0 = tn * BLOCK_N;
      if (!mbar_wait(&tmem_full_bar[acc], acc_phase, abort_flag)) { ok = false; break; }
      tc_fence_after_sync();
      const uint32_t t_base = tmem_base + static_cast<uint32_t>(acc * BLOCK_N) + (static_cast<uint32_t>(quad * 32) << 16);
      const GemmParams pt = BATCHED ? gemm_params_of_batch(p, pb) : p;
      uint4 pre[8];
      if (epilogue_can_coalesce(pt) && epilogue_needs_aux(pt.epilogue)) epi_slab_prefetch(pre, pt.aux, pt.ld_aux, row - lane, n0, pt.M, pt.N, lane);
      if (epilogue_can_coalesce(pt)) epilogue_rows_coalesced(t_base, row - lane, n0, BLOCK_N, pt, smem + L::EPI_OFFSET + quad * 4096, lane, pre);
      else                           epilogue_rows<BLOCK_N>(t_base, row, n0, pt);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tmem_empty_bar[acc]);
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  }

  // ------------------------------------------------------------------ teardown
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    // a wait ran out: report, give in-flight TMA copies time to land, then release TMEM and leave
    if (threadIdx.x == 0 && p.status != nullptr) atomicExch(p.status, FSB_ERR_WAIT_TIMEOUT);
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 2 * BLOCK_N);
  }
}

// ------------------------------------------------------------------------------------------------
// CTA-pair variant: a cluster of two CTAs (two SMs) computes one 256 x 256 tile with
// tcgen05.mma.cta_group::2. Each CTA stages only its 128 rows of A and its 128 columns of B, so the
// shared-memory traffic per MMA drops by a third and 6 stages fit. CTA 0 (the leader) issues the MMAs;
// both CTAs load with their own per-CTA TMA (nothing is broadcast), and both drain their half of the
// accumulator. Barriers: full[] lives in the leader and counts both CTAs' bytes; empty[] and tmem_full[]
// exist in both CTAs and are signalled by one commit to both; tmem_empty[] lives in the leader
// and collects the 8 epilogue warps of the pair.
// ------------------------------------------------------------------------------------------------
constexpr int PAIR_BLOCK_N = 256;
constexpr int PAIR_HALF_N = 128;
constexpr int PAIR_EPI_WARPS = 8;                        // two per TMEM lane quadrant, 128 columns each
constexpr int PAIR_THREADS = 64 + 32 * PAIR_EPI_WARPS;   // producer warp + MMA warp + epilogue warps

// MH: blocks of 128 rows that each CTA of the pair owns.  1: tiles of 256 x 256, two accumulators in TMEM; 2: tiles of
// 512 x 256, whose two row blocks fill TMEM (see the kernel).
template <int MH>
struct PairSmem {
  static constexpr int STAGES = MH == 1 ? 6 : 4;
  static constexpr int A_BYTES = MH * BLOCK_M * BLOCK_K * 2;  // 16 KB per row block
  static constexpr int B_BYTES = PAIR_HALF_N * BLOCK_K * 2;   // 16 KB: this CTA's 128 columns
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int EPI_OFFSET = STAGES * STAGE_BYTES;           // 4 KB of staging per epilogue warp
  static constexpr int BAR_OFFSET = EPI_OFFSET + PAIR_EPI_WARPS * 4096;
  // No slack for re-aligning the base: the kernel has no static shared memory, so its dynamic window starts 1024-byte
  // aligned (checked at run time).  With the 1 KB the hardware reserves per CTA this leaves 2816 bytes of the SM's
  // 228 KB, enough for two of the 128-thread communication CTAs (1 KB reserve + 8 bytes each) to stay resident beside
  // a GEMM CTA; a third would keep the next GEMM CTA off the SM.
  static constexpr int TOTAL = BAR_OFFSET + 256;
  static_assert(8 * (2 * STAGES + 4 + 2 * SCHED_DEPTH + 2) + 4 * (SCHED_DEPTH + 3) <= 256, "barriers, tile indices, TMEM address, abort flag");
};

template <int MH>
__device__ __forceinline__ void pair_tile_coords(const GemmParams& p, int tile, int tiles_m, int tiles_n, int& tm, int& tn) {
  if (MH == 2) {
    tile_coords<8>(tile, tiles_m, tiles_n, tm, tn);
    return;
  }
  if (p.b_ready != nullptr) {  // N-major in sending order of the pieces of B: every M tile of the rows that arrive first
    const int lin = tile / tiles_m;
    tm = tile - lin * tiles_m;
    // first tile that starts inside the first piece sent (rounded up: the tile before it needs the piece sent last)
    const long long tile_bytes = static_cast<long long>(PAIR_BLOCK_N) * p.K * 2;
    const int rot = static_cast<int>((static_cast<long long>(p.b_first_piece) * p.b_piece_bytes + tile_bytes - 1) / tile_bytes);
    tn = (lin + rot) % tiles_n;
  } else if (p.a_ready != nullptr) {  // M-major in arrival order of the row blocks of A, this rank's own block first
    const int lin = tile / tiles_n;
    tn = tile - lin * tiles_n;
    // first tile that starts inside this rank's own block (rounded up: a tile that straddles the block's start also needs
    // rows of the block that arrives last, so it is visited last)
    const int rot = static_cast<int>((static_cast<long long>(p.a_first_shard) * p.a_shard_rows + 2 * BLOCK_M - 1) / (2 * BLOCK_M));
    tm = (lin + rot) % tiles_m;
  } else {
    tile_coords(tile, tiles_m, tiles_n, tm, tn);
  }
}

// Wait until bytes [lo, hi) of the B operand have arrived (see GemmParams::b_ready).  Flags are raised in sending order by
// one stream, so a raised flag vouches for every piece sent before it: `upto` caches the highest sending index seen.
// Returns false when the wait limit ran out.
__device__ __forceinline__ bool wait_b_pieces(const GemmParams& p, long long lo, long long hi, int& upto, volatile int* abort_flag) {
  const int first = static_cast<int>(lo / p.b_piece_bytes), last = static_cast<int>((hi - 1) / p.b_piece_bytes);
  bool waited = false;
  for (int q = first; q <= last; ++q) {
    const int i = (q - p.b_first_piece + p.b_num_pieces) % p.b_num_pieces;  // sending index of piece q
    if (i <= upto) continue;
    const uint64_t t0 = globaltimer_ns();
    unsigned int v;
    while (true) {
      asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p.b_ready + i) : "memory");
      if (static_cast<int>(v - p.b_ready_epoch) >= 0) break;
      if (*abort_flag) return false;
      if (globaltimer_ns() - t0 > p.b_wait_ns) {
        if (*abort_flag == 0) *abort_flag = 10;
        return false;
      }
      __nanosleep(200);
    }
    upto = i;
    waited = true;
  }
  if (waited) asm volatile("fence.proxy.async;" ::: "memory");  // the arrived bytes before this thread's TMA reads of them
  return true;
}

// Wait until rows [r0, r1) of the A operand have arrived (see GemmParams::a_ready).  Flags are raised in index order by
// one stream, so a raised flag vouches for every lower index: `upto` caches the highest index seen.
__device__ __forceinline__ bool wait_a_rows(const GemmParams& p, int r0, int r1, int& upto, volatile int* abort_flag) {
  const int pps = (p.a_shard_rows + p.a_piece_rows - 1) / p.a_piece_rows;
  bool waited = false;
  int r = r0;
  while (r < r1) {
    const int shard = r / p.a_shard_rows, in_shard = r - shard * p.a_shard_rows;
    const int k = (shard - p.a_first_shard + p.a_num_shards) % p.a_num_shards;
    const int j = in_shard / p.a_piece_rows;
    const int idx = k * pps + j;
    if (idx > upto) {
      const uint64_t t0 = globaltimer_ns();
      unsigned int v;
      while (true) {
        asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p.a_ready + idx) : "memory");
        if (static_cast<int>(v - p.a_ready_epoch) >= 0) break;
        if (*abort_flag) return false;
        if (globaltimer_ns() - t0 > p.b_wait_ns) {
          if (*abort_flag == 0) *abort_flag = 11;
          return false;
        }
        __nanosleep(200);
      }
      upto = idx;
      waited = true;
    }
    int next = shard * p.a_shard_rows + (j + 1) * p.a_piece_rows;  // first row of the next piece
    const int shard_end = (shard + 1) * p.a_shard_rows;
    if (next > shard_end) next = shard_end;
    r = next;
  }
  if (waited) asm volatile("fence.proxy.async;" ::: "memory");  // the arrived rows before this thread's TMA reads of them
  return true;
}

// MH 2, tiles of 512 x 256: the operands of a 64-wide K block are 48 KB per CTA for twice the products (64 KB in two 256 x 256
// tiles), and a stage's barriers are paid half as often.  What bounds a long product is the power limit, and the operand stream
// out of L2 is what can be saved there: 8192 x 2048 x 16384 (weight gradient) 486 -> 435 us, 16384 x 50304 x 2048 2696 -> 2518 us,
// 22016 x 4096 x 4096 (weight gradient) 611 -> 555 us (cuBLAS 428, 2594, 550).  The two row blocks fill TMEM, so instead of a second pair of
// accumulators each block is handed back as soon as the epilogue warps hold it in registers, packed to bf16: the last products
// of a tile's second block run while the first block is read, the next tile's first ones while the second is.  Only epilogues
// whose result is final in registers can do that; those that read another operand or write two results stay with MH 1.
template <bool BATCHED, int MH>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1)
gemm_bf16_tcgen05_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, GemmParams p) {
  using L = PairSmem<MH>;
  constexpr int PAIR_STAGES = L::STAGES;
  constexpr int CTA_ROWS = MH * BLOCK_M;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if ((smem_u32(smem_raw) & 1023u) != 0u) {  // same for every thread of the pair: nothing has been set up yet
    if (threadIdx.x == 0 && p.status != nullptr) atomicExch(p.status, FSB_ERR_BAD_ARG);
    return;
  }

  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::BAR_OFFSET);
  uint64_t* empty_bar = full_bar + PAIR_STAGES;
  uint64_t* tmem_full_bar = empty_bar + PAIR_STAGES;
  uint64_t* tmem_empty_bar = tmem_full_bar + 2;
  uint64_t* sched_full = tmem_empty_bar + 2;         // [SCHED_DEPTH] the slot holds a tile index
  uint64_t* sched_empty = sched_full + SCHED_DEPTH;  // [SCHED_DEPTH] every reader in this CTA has taken it
  uint64_t* mail_full = sched_empty + SCHED_DEPTH;   // in the peer: mail_tile holds the next index
  uint64_t* mail_empty = mail_full + 1;              // in the leader: the peer has taken it
  volatile int* sched_tile = reinterpret_cast<volatile int*>(mail_empty + 1);
  volatile int* mail_tile = sched_tile + SCHED_DEPTH;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(const_cast<int*>(mail_tile) + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);  // warp-uniform
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int num_pairs = gridDim.x >> 1;

  const int tiles_m = (p.M + 2 * CTA_ROWS - 1) / (2 * CTA_ROWS);
  const int tiles_n = (p.N + PAIR_BLOCK_N - 1) / PAIR_BLOCK_N;
  const int tiles_per_problem = tiles_m * tiles_n;
  const int num_tiles = tiles_per_problem * (BATCHED ? p.batch : 1);
  const int num_kb = (p.K + BLOCK_K - 1) / BLOCK_K;
  auto load_tile = [&](uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
    if (BATCHED) tma_load_3d_pair_warp(dst, map, bar, x, y, z);
    else         tma_load_2d_pair_warp(dst, map, bar, x, y);
  };
  // Whole lines of C; in a batch every problem's base has to keep the alignment of the first one
  const bool coalesce = MH == 2 || (epilogue_can_coalesce(p) && (!BATCHED || (p.stride_c % 8 == 0 && p.stride_aux % 8 == 0)));
  // Index of this pair's first tile (lane 0 of the leader's producer warp): on its way while the pair sets itself up.
  unsigned int* const sched = g_sched_counters + 2 * p.sched_slot;
  const bool counted = p.sched_slot != 0;
  auto fetch = [&](int before) -> int {  // `before`: the last index this pair was given
    return counted ? static_cast<int>(atomicAdd(&sched[0], 1u)) : before + num_pairs;
  };
  int first = 0;
  if (leader && threadIdx.x == 0) first = fetch(static_cast<int>(blockIdx.x >> 1) - num_pairs);

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < PAIR_STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full_bar[a], 1);
      mbar_init(&tmem_empty_bar[a], 2 * PAIR_EPI_WARPS);  // the epilogue warps of both CTAs of the pair
    }
    for (int q = 0; q < SCHED_DEPTH; ++q) {
      mbar_init(&sched_full[q], 1);
      mbar_init(&sched_empty[q], (leader ? 1 : 0) + PAIR_EPI_WARPS);  // the MMA warp, the epilogue warps
    }
    mbar_init(mail_full, 1);
    mbar_init(mail_empty, 1);
    fence_barrier_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    if (p.b_ready != nullptr) {
      // The first piece of B arrives only after every peer has entered the gather, which can be long after this kernel
      // started (rank skew).  Wait for it here, under the long limit, before any of the pipeline's short waits counts.
      int upto = -1;
      const long long first_byte = static_cast<long long>(p.b_first_piece) * p.b_piece_bytes;
      wait_b_pieces(p, first_byte, first_byte + 1, upto, abort_flag);
    }
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 2 * PAIR_BLOCK_N);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers are initialised before anyone signals them
  tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  // Tiles are handed out at run time: the leader's producer takes the next index from a counter in global memory and sends it
  // (or -1 at the end) to the peer's producer; each of the two publishes it to its own CTA through a small ring that every role
  // reads in order.  An SM that is slowed down or taken by a kernel of another stream (a collective) then simply works off fewer
  // tiles, instead of holding back the ones a static schedule would have given it.  A launch without a counter strides through the tiles.
  // One thread of each CTA takes part in what crosses the pair, and only there is cluster scope needed: the index is a remote
  // store that completes on the peer's barrier, and the peer's producer, which has nothing but loads in flight, hands the word
  // back with a release of cluster scope while its ring of loads is full.  (With every role of both CTAs releasing and acquiring at
  // cluster scope the MMA warp stood still for 2 400 cycles a tile of 20 400, 8192 x 8192 x 2048, and the producers for about as long.)
  // Reader side: wait for slot q of this CTA's ring, take the index, hand the slot back.
  auto take_tile = [&](int q, uint32_t qphase, int site) -> int {
    if (!mbar_wait(&sched_full[q], qphase, abort_flag, site)) return -2;
    const int t = sched_tile[q];
    mbar_arrive(&sched_empty[q]);
    return t;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs, the whole warp)
    // Like the MMAs, the loads are issued from uniform control flow by an elected lane: inside a one-lane branch every
    // operand of a load has to be moved to a uniform register first, and the four loads that a K block of MN-major operands
    // takes cost more than its 512 cycles of tensor time (weight gradient 8192 x 2048 x 16384: 631 -> 543 cycles per block).
    int stage = 0;
    uint32_t phase = 0;
    int q = 0;
    uint32_t qphase = 0;
    bool ok = true;
    auto publish = [&](int t) -> bool {  // to the roles of this CTA
      if (!mbar_wait_warp(&sched_empty[q], qphase ^ 1u, abort_flag, 2)) return false;
      if (lane == 0) {
        sched_tile[q] = t;
        mbar_arrive(&sched_full[q]);
      }
      __syncwarp();
      if (++q == SCHED_DEPTH) { q = 0; qphase ^= 1u; }
      return true;
    };
    uint32_t mail_phase = 0;
    auto send = [&](int t) -> bool {  // leader: to the peer's producer
      if (!mbar_wait_warp<WaitScope::CLUSTER>(mail_empty, mail_phase ^ 1u, abort_flag, 12)) return false;
      if (lane == 0) {
        const uint32_t bar = map_to_cta(smem_u32(mail_full), 1);
        mbar_expect_tx_remote(bar, 4);
        st_async_u32(map_to_cta(smem_u32(const_cast<int*>(mail_tile)), 1), static_cast<uint32_t>(t), bar);
      }
      __syncwarp();
      mail_phase ^= 1u;
      return true;
    };
    auto receive = [&]() -> int {  // peer: what the leader sent, -2 if the wait ran out
      int t = -2;
      if (lane == 0 && mbar_wait<WaitScope::CLUSTER>(mail_full, mail_phase, abort_flag, 3)) {
        t = *mail_tile;
        mbar_arrive_release_cluster(map_to_cta(smem_u32(mail_empty), 0));
      }
      mail_phase ^= 1u;
      return __shfl_sync(0xffffffffu, t, 0);
    };
    // The next index is fetched before the loads of the current tile and handed on behind the first of them, when the ring of
    // loads is full: the atomic's round trip and the way to the peer hide, the readers find theirs without waiting, and neither
    // holds up a tile's first loads.
    // (Not where the epilogue stores a row per thread, fp32 or off the 16-byte pieces, and takes longer than the products: 16384 x
    // 6144 x 2048 fp32 398 us handed on before the loads, 464 behind them; odd rows 341 and 392.  With whole lines it is 502 and 490
    // us at 16384 x 8192 x 2048 with a residual.)
    const int publish_kb = !coalesce ? 0 : num_kb < PAIR_STAGES ? num_kb : PAIR_STAGES;
    int b_upto = -1;  // highest B piece known to have arrived
    int tile;
    if (leader) {
      tile = __shfl_sync(0xffffffffu, first, 0);
      if (tile >= num_tiles) tile = -1;
      ok = publish(tile) && send(tile);
    } else {
      tile = receive();
      ok = tile != -2 && publish(tile);
    }
    const uint32_t smem0 = smem_u32(smem), full_local = smem_u32(full_bar), full0 = map_to_cta(full_local, 0);
    while (ok && tile >= 0) {
      const int pb = BATCHED ? tile / tiles_per_problem : 0;
      int tm, tn;
      pair_tile_coords<MH>(p, tile - pb * tiles_per_problem, tiles_m, tiles_n, tm, tn);
      const int m0 = (tm * 2 + static_cast<int>(rank)) * CTA_ROWS;
      const int n0 = tn * PAIR_BLOCK_N + static_cast<int>(rank) * PAIR_HALF_N;
      // (every lane waits and fences: any of them may be the one that issues the loads)
      if (MH == 1 && p.b_ready != nullptr && n0 < p.N) {
        const long long row_bytes = static_cast<long long>(p.K) * 2;
        const int n1 = n0 + PAIR_HALF_N < p.N ? n0 + PAIR_HALF_N : p.N;
        if (!__all_sync(0xffffffffu, wait_b_pieces(p, n0 * row_bytes, n1 * row_bytes, b_upto, abort_flag))) break;
      }
      if (MH == 1 && p.a_ready != nullptr && m0 < p.M) {
        if (!__all_sync(0xffffffffu, wait_a_rows(p, m0, m0 + BLOCK_M < p.M ? m0 + BLOCK_M : p.M, b_upto, abort_flag))) break;
      }
      auto load_blocks = [&](int kb0, int kb1) -> bool {
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_warp(&empty_bar[stage], phase ^ 1u, abort_flag, 4)) return false;
          const uint32_t sa = smem0 + stage * L::STAGE_BYTES, sb = sa + L::A_BYTES, bar = full0 + stage * 8;
          if (leader) mbar_expect_tx_warp(full_local + stage * 8, 2 * L::STAGE_BYTES);
          const int k0 = kb * BLOCK_K;
          if (!p.a_mn_major) {
#pragma unroll
            for (int h = 0; h < MH; ++h) load_tile(sa + h * 16384, &tmap_a, bar, k0, m0 + h * BLOCK_M, pb);
          } else {
#pragma unroll
            for (int j = 0; j < CTA_ROWS / 64; ++j) load_tile(sa + j * 8192, &tmap_a, bar, m0 + j * 64, k0, pb);
          }
          if (!p.b_mn_major) {
            load_tile(sb, &tmap_b, bar, k0, n0, pb);
          } else {
#pragma unroll
            for (int j = 0; j < PAIR_HALF_N / 64; ++j) load_tile(sb + j * 8192, &tmap_b, bar, n0 + j * 64, k0, pb);
          }
          if (++stage == PAIR_STAGES) { stage = 0; phase ^= 1u; }
        }
        return true;
      };
      int next = -1, nxt = 0;
      if (leader && (lane == 0 || !counted)) nxt = fetch(tile);
      if (!load_blocks(0, publish_kb)) break;
      if (leader) {
        const int nt = __shfl_sync(0xffffffffu, nxt, 0);
        next = nt < num_tiles ? nt : -1;
        if (!publish(next) || !send(next)) break;
      } else {
        next = receive();
        if (next == -2 || !publish(next)) break;
      }
      if (!load_blocks(publish_kb, num_kb)) break;
      tile = next;
    }
    if (leader && counted && lane == 0) {
      // the last pair to get here has seen every pair's final fetch: put the counters back for the next launch
      __threadfence();
      if (atomicAdd(&sched[1], 1u) == static_cast<unsigned int>(num_pairs - 1)) {
        sched[0] = 0u;
        sched[1] = 0u;
        __threadfence();
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (the leader's whole warp, see umma_f16_ss_warp)
    if (leader) {
      const uint32_t idesc = make_idesc_f16(2 * BLOCK_M, PAIR_BLOCK_N, true, p.a_mn_major != 0, p.b_mn_major != 0);
      const uint32_t a_lbo = p.a_mn_major ? 8192u : 16u, b_lbo = p.b_mn_major ? 8192u : 16u;
      const uint32_t a_kstep = p.a_mn_major ? 2048u : 32u, b_kstep = p.b_mn_major ? 2048u : 32u;
      const uint64_t adesc0 = make_smem_desc(smem_u32(smem), a_lbo, 1024u), bdesc0 = make_smem_desc(smem_u32(smem) + L::A_BYTES, b_lbo, 1024u);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      int q = 0;
      uint32_t qphase = 0;
      bool ok = true;
      while (ok) {
        int tile = 0;
        if (lane == 0) tile = take_tile(q, qphase, 5);
        tile = __shfl_sync(0xffffffffu, tile, 0);
        if (++q == SCHED_DEPTH) { q = 0; qphase ^= 1u; }
        if (tile < 0) break;
        if (MH == 1) {
          if (!mbar_wait_warp<WaitScope::CLUSTER_RELAXED>(&tmem_empty_bar[acc], acc_phase ^ 1u, abort_flag, 6)) { ok = false; break; }
          tc_fence_after_sync();
        }
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait_warp(&full_bar[stage], phase, abort_flag, 7)) { ok = false; break; }
          tc_fence_after_sync();
          const uint64_t ad = desc_offset(adesc0, stage * L::STAGE_BYTES), bd = desc_offset(bdesc0, stage * L::STAGE_BYTES);
#pragma unroll
          for (int h = 0; h < MH; ++h) {
            if (MH == 2 && kb == 0) {
              if (!mbar_wait_warp<WaitScope::CLUSTER_RELAXED>(&tmem_empty_bar[h], acc_phase ^ 1u, abort_flag, 6)) { ok = false; break; }
              tc_fence_after_sync();
            }
            const uint32_t d_tmem = tmem_base + static_cast<uint32_t>((MH == 1 ? acc : h) * PAIR_BLOCK_N);
#pragma unroll
            for (int k = 0; k < BLOCK_K / UMMA_K; ++k)
              umma_f16_ss_pair_warp(d_tmem, desc_offset(ad, h * 16384 + k * a_kstep), desc_offset(bd, k * b_kstep), idesc, (kb | k) != 0 ? 1u : 0u);
            if (MH == 2 && kb == num_kb - 1) umma_commit_pair_warp(&tmem_full_bar[h]);
          }
          if (!ok) break;
          umma_commit_pair_warp(&empty_bar[stage]);
          if (++stage == PAIR_STAGES) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        if (MH == 1) {
          umma_commit_pair_warp(&tmem_full_bar[acc]);
          acc ^= 1;
          if (acc == 0) acc_phase ^= 1u;
        } else {
          acc_phase ^= 1u;
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue warps (both CTAs)
    const int quad = warp & 3;            // TMEM lane quadrant this warp may access
    const int half = (warp - 2) >> 2;     // which 128 columns of the 256 this warp drains
    uint8_t* stage = smem + L::EPI_OFFSET + (warp - 2) * 4096;
    int acc = 0;
    uint32_t acc_phase = 0;
    int q = 0;
    uint32_t qphase = 0;
    bool ok = true;
    while (ok) {
      int tile = 0;
      if (lane == 0) tile = take_tile(q, qphase, 8);
      tile = __shfl_sync(0xffffffffu, tile, 0);
      if (++q == SCHED_DEPTH) { q = 0; qphase ^= 1u; }
      if (tile < 0) break;
      const int pb = BATCHED ? tile / tiles_per_problem : 0;
      int tm, tn;
      pair_tile_coords<MH>(p, tile - pb * tiles_per_problem, tiles_m, tiles_n, tm, tn);
      const GemmParams pt = BATCHED ? gemm_params_of_batch(p, pb) : p;
      const int row0 = (tm * 2 + static_cast<int>(rank)) * CTA_ROWS + quad * 32;
      const int n0 = tn * PAIR_BLOCK_N + half * (PAIR_BLOCK_N / 2);
      const uint32_t t_base = tmem_base + static_cast<uint32_t>(half * (PAIR_BLOCK_N / 2)) + (static_cast<uint32_t>(quad * 32) << 16);
      if (MH == 1) {
        uint4 pre[8];
        if (coalesce && epilogue_needs_aux(p.epilogue) && n0 < p.N) epi_slab_prefetch(pre, pt.aux, pt.ld_aux, row0, n0, pt.M, pt.N, lane);
        if (!mbar_wait(&tmem_full_bar[acc], acc_phase, abort_flag, 9)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t t_acc = t_base + static_cast<uint32_t>(acc * PAIR_BLOCK_N);
        if (coalesce) epilogue_rows_coalesced(t_acc, row0, n0, PAIR_BLOCK_N / 2, pt, stage, lane, pre);
        else          epilogue_rows<PAIR_BLOCK_N / 2>(t_acc, row0 + lane, n0, pt);
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_relaxed_cluster(map_to_cta(smem_u32(&tmem_empty_bar[acc]), 0));
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      } else {
        // Both row blocks to registers first, each handed back at once: the next tile's products wait for nothing else.  So the
        // bias waits in the staging buffer already (read from global memory it cost an L2 round trip per 64 columns there).
        uint32_t pk[2][64];
        __nv_bfloat16* const bias = pt.epilogue == EPI_BIAS ? reinterpret_cast<__nv_bfloat16*>(stage) : nullptr;
        if (bias != nullptr) {
#pragma unroll
          for (int i = 0; i < 4; ++i) bias[lane * 4 + i] = n0 + lane * 4 + i < pt.N ? pt.bias[n0 + lane * 4 + i] : __float2bfloat16_rn(0.f);
          __syncwarp();
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (!mbar_wait(&tmem_full_bar[h], acc_phase, abort_flag, 9)) { ok = false; break; }
          tc_fence_after_sync();
#pragma unroll
          for (int c = 0; c < 2; ++c) epi_pack64(t_base + static_cast<uint32_t>(h * PAIR_BLOCK_N + c * 64), bias == nullptr ? nullptr : bias + c * 64, &pk[h][c * 32]);
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive_relaxed_cluster(map_to_cta(smem_u32(&tmem_empty_bar[h]), 0));
        }
        if (!ok) break;
        acc_phase ^= 1u;
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
#pragma unroll
            for (int k = 0; k < 8; ++k)
              *reinterpret_cast<uint4*>(stage + epi_swz(lane, k)) = make_uint4(pk[h][c * 32 + k * 4], pk[h][c * 32 + k * 4 + 1], pk[h][c * 32 + k * 4 + 2], pk[h][c * 32 + k * 4 + 3]);
            __syncwarp();
            epi_slab_store(stage, reinterpret_cast<__nv_bfloat16*>(pt.C), pt.ldc, row0 + h * BLOCK_M, n0 + c * 64, pt.M, pt.N, lane);
            __syncwarp();
          }
        }
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    if (threadIdx.x == 0 && p.status != nullptr) atomicExch(p.status, FSB_ERR_WAIT_TIMEOUT | (*abort_flag << 8));
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  cluster_sync_all();  // neither CTA leaves while its partner may still signal its barriers or read its smem
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, 2 * PAIR_BLOCK_N);
  }
}

}  // namespace fsb

namespace fsb_host {
// gemm_cluster_k.cu
int gemm_cluster_k(const CUtensorMap& ta, const void* B, int ldb, const fsb::GemmParams& p, int block_n, int splits, int dev, cudaStream_t stream);
}  // namespace fsb_host

template <bool BATCHED, int MH>
static int launch_pair(const CUtensorMap& ta, const CUtensorMap& tb, const fsb::GemmParams& p, int num_sms, int di, cudaStream_t stream) {
  using namespace fsb;
  static bool attr_set[64] = {false};  // the attribute is per device
  if (!attr_set[di]) {
    cudaFuncSetAttribute(gemm_bf16_tcgen05_pair_kernel<BATCHED, MH>, cudaFuncAttributeMaxDynamicSharedMemorySize, PairSmem<MH>::TOTAL);
    attr_set[di] = true;
  }
  const long long tiles = static_cast<long long>(p.batch) * ((p.M + 2 * MH * BLOCK_M - 1) / (2 * MH * BLOCK_M)) * ((p.N + PAIR_BLOCK_N - 1) / PAIR_BLOCK_N);
  const int pairs = tiles < num_sms / 2 ? static_cast<int>(tiles) : num_sms / 2;
  gemm_bf16_tcgen05_pair_kernel<BATCHED, MH><<<2 * pairs, PAIR_THREADS, PairSmem<MH>::TOTAL, stream>>>(ta, tb, p);
  return static_cast<int>(cudaGetLastError());
}

// Slot of the tile counters for a launch on `stream`: every stream keeps one of its own for the life of the process, so two
// launches that use the same counters are ordered by their stream, however far the host runs ahead.  Streams are told apart
// by their id, which is never given out twice (a handle is, while the old stream's work may still be running).  0, no
// counter, for the streams that come after SCHED_SLOTS - 1 others and for a launch under capture: a graph is replayed on
// any stream, beside eager launches.  Such a launch strides through its tiles.
static int sched_slot_of(int di, cudaStream_t stream) {
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess) {  // the default stream while another one is captured
    cudaGetLastError();
    return 0;
  }
  if (capture != cudaStreamCaptureStatusNone) return 0;
  unsigned long long id = 0;
  if (cudaStreamGetId(stream, &id) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  static std::mutex mu;
  static std::unordered_map<unsigned long long, int> slots[64];
  std::lock_guard<std::mutex> lock(mu);
  const auto it = slots[di].find(id);
  if (it != slots[di].end()) return it->second;
  const int slot = static_cast<int>(slots[di].size()) + 1;
  if (slot >= fsb::SCHED_SLOTS) return 0;
  slots[di].emplace(id, slot);
  return slot;
}

// The slot that a product launched on `stream` of the current device would use (0: none).
FSB_API int fsb_gemm_sched_slot(cudaStream_t stream) {
  int dev = 0;
  cudaGetDevice(&dev);
  return sched_slot_of(dev & 63, stream);
}

static bool pair_enabled() {  // FSB_GEMM_PAIR=0 disables the CTA-pair kernel
  static const bool on = [] {
    const char* e = getenv("FSB_GEMM_PAIR");
    return e == nullptr || e[0] != '0';
  }();
  return on;
}

// Kernel for a product that is not streamed and has no CTA cap; plan_product has what decides when.  Measured on B200 (us; 64-wide K
// blocks = kb), small products back to back:
//
//   M, N, K              pair   one CTA 128x256   cluster split-K, block_n / splits
//   77, 1024, 4096         -         24.6          64/1 20.5   64/2 15.0   64/4 11.7   128/4 12.8   128/8 12.3
//   128, 1024, 8192        -         43.0          64/1 34.9   64/2 22.5   64/4 15.1   128/4 16.5   128/8 14.3
//   768, 768, 3576       30.5        28.6          64/1 18.5   64/2 14.9   128/1 20.5  128/2 18.2   128/4 22.6
//   1024, 1024, 8192     50.4        43.0          64/1 36.5   64/2 43.1   128/1 38.4  128/2 26.8   128/4 32.8
//   2048, 1024, 1024     19.0        12.3          64/1 16.3   128/1 10.2  128/2 20.5
//   2048, 2048, 2048     24.7        17.3          128/1 25.9
//   3072, 1024, 8192     58.8        52.9          128/1 73.3
//
// One wave of independent CTAs takes about 6 us + K blocks x 0.23 / 0.24 / 0.29 us (tiles 64 / 128 / 256 wide): one CTA's
// operand stream is bound by latency, not by the tensor cores, so shorter slices win until the SMs run out.  A cluster
// costs about 2 us more for its barriers, 4 us at eight CTAs, and clusters of four or eight do not fit the SMs to the last
// one (144 CTAs in clusters of four run in two waves), hence the limits on their number.  (The slopes in the code are those
// of a slower MMA issue, all by the same quarter; with them the rule takes the fastest column of every row above, or one
// within 5 %.)
//
// From 90 tiles on, where choose_persistent below does not come in (fp32 results, rows in no 16-byte pieces, K below 256), it is one
// CTA per tile or a pair per 256 x 256 tile (us, one CTA / pair, in loops of 0.2 s; * operands MN-major):
//
//   M, N, K                    fp32          bf16, N - 1       M, N, K                  fp32          bf16, N - 1
//   952, 12048, 704         32.7 / 35.9      24.3 / 28.3       16384, 6144, 2048      430 / 428       379 / 382
//   8192, 4096, 1024        90.6 / 100       79.1 / 79.3       16384, 8192, 2048      572 / 549       505 / 496
//   5968, 2048, 2048        56.4 / 59.2      53.8 / 56.8       4096, 12288, 4096      391 / 365       367 / 342
//   16384, 2048, 2048        146 / 149        137 / 136        8192, 2048, 16384 *    503 / 505       496 / 500
//   8192, 8192, 2048         288 / 284        254 / 255        2048, 6144, 16384 *    376 / 375       370 / 366
//   16384, 16384, 768        629 / 657        480 / 476        50304, 2048, 16384 *  2924 / 3065     2898 / 2994
//   16384, 16384, 1400      1136 / 1025      1032 / 864        2992, 1976, 13208 *    237 / 183       230 / 179
//   13640, 13184, 616        489 / 477        382 / 358        1936, 5872, 4360       152 / 125       139 / 113
//
// A pair costs some 6 us more per launch and rounds up to larger tiles, but moves a third less operand data.  That counts once
// a product is long enough to run at the power limit, and much sooner where the operands' rows do not start on 128-byte lines
// (a leading dimension that is no multiple of 64): every 128-byte row of a tile is then two lines.  Up to K about 1400 the
// output is what takes the time.  pair_pays puts that into two lines: us per K block and wave of tiles, by the number of operands
// off the lines, and the pair's extra cost.  Over 33 products (M and N 328 .. 50304, K 256 .. 16384) the rule takes 0.7 % longer with
// fp32 results than the faster kernel would on average, 1.1 % with ragged bf16 ones; at worst 11 and 19 %, both at 16384 x 16384 x
// 1400, where the line in K lies.  (It was fitted to slower kernels of both kinds; a single line in operations costs 4.7 %, always the
// pair 8 %, never 7 %.)
struct GemmPlan {
  enum Kind { PAIR, ONE_CTA, CLUSTER_K, WIDE_PAIR } kind;
  int block_n, splits;
};
// Does the pair kernel pay for `problems` products of M x N x K with leading dimensions lda, ldb?
static bool pair_pays(long long problems, int M, int N, int K, int lda, int ldb, int num_sms) {
  const long long tiles = problems * ((M + fsb::BLOCK_M - 1) / fsb::BLOCK_M) * ((N + 255) / 256);
  const long long pair_tiles = problems * ((M + 2 * fsb::BLOCK_M - 1) / (2 * fsb::BLOCK_M)) * ((N + fsb::PAIR_BLOCK_N - 1) / fsb::PAIR_BLOCK_N);
  if (M < 256 || N < 256 || K <= 1400 || tiles < 90) return false;
  static const float one_us[3] = {0.45f, 0.50f, 0.57f}, pair_us[3] = {0.435f, 0.44f, 0.49f};
  const int off_line = (lda % 64 != 0) + (ldb % 64 != 0), num_kb = (K + fsb::BLOCK_K - 1) / fsb::BLOCK_K, pairs = num_sms / 2;
  const float one = one_us[off_line] * num_kb * ((tiles + num_sms - 1) / num_sms);
  const float pair = 8.f + pair_us[off_line] * num_kb * ((pair_tiles + pairs - 1) / pairs);
  return pair < one;
}
// Which of the three persistent kernels for `problems` products with bf16 rows in 16-byte pieces (row_pieces), in estimated us: a
// launch, and per wave of tiles its start and its K blocks, or its epilogue where that takes longer; the share that goes with the
// tiles per SM instead of whole waves is what the card's power limit gives back when a wave is partly empty.
// Plain and bias products: fitted to 90 of them (M and N 256 .. 16384, K 256 .. 32000, one or 4 to 16 stacked, all operand layouts,
// a third with rows off the 128-byte lines).  Over 40 others the choice costs 0.3 % on average and 9 % at worst (2208 x 2640 x 2240,
// wide 32.7, one CTA 30.0); pair_pays' choice between the other two costs 7 %.  Measured (us, wide / pair / one CTA, a quarter of a second each):
//   16384 x 6144 x 2048 323 / 352 / 345       8192 x 2048 x 16384 (wgrad) 435 / 476 / 482     50304 x 2048 x 16384 (wgrad) 2552 / 2837 / 2798
//   4096 x 12288 x 4096 322 / 323 / 345       8192 x 3072 x 1024 50.8 / 55.2 / 52.0           16384 x 50304 x 2048 2527 / 2784 / 2853
//   8 x 2048 x 1024 x 4096 123 / 127 / 133    2792 x 3968 x 256 16.5 / 16.4 / 14.3            16384 x 16384 x 1400 641 / 791 / 895
// The other epilogues take time of their own, and the pair drains a tile with eight warps per CTA instead of four.  Fitted for each
// to 68 products (M 1024 .. 16384, N 256 .. 8192, K 256 .. 12288, half of them off the lines), the mean of bursts of 3 ms and of
// stretches of 0.2 s at the power limit: the choice costs 0.1 % on average and 2.8 % at worst.  (With the residual's constants of a
// plain product but for its start it cost 1 % and 7.3 %.)  Measured (us at the power limit, pair / one CTA):
//   GELU           16384 x 8192 x 2048 482 / 462    16384 x 2048 x 2048 127 / 119    8192 x 2048 x 512 32.4 / 36.8    14724 x 1144 x 2680 106 / 129
//   GELU'          16384 x 8192 x 2048 512 / 523    16384 x 2048 x 2048 134 / 135    8192 x 2048 x 512 45.6 / 48.9    14724 x 1144 x 2680 115 / 136
//   bias+residual  16384 x 8192 x 2048 505 / 482    16384 x 2048 x 2048 133 / 123    8192 x 2048 x 512 35.2 / 39.6    14724 x 1144 x 2680 111 / 134
//   residual       16384 x 8192 x 2048 501 / 479    16384 x 2048 x 2048 131 / 122    8192 x 2048 x 512 31.2 / 34.3    14724 x 1144 x 2680 110 / 133
static bool row_pieces(const fsb::GemmParams& p) {
  const uintptr_t ptrs = reinterpret_cast<uintptr_t>(p.C) | reinterpret_cast<uintptr_t>(p.aux) | reinterpret_cast<uintptr_t>(p.aux_out);
  return !p.out_f32 && p.N % 8 == 0 && p.ldc % 8 == 0 && p.ld_aux % 8 == 0 && p.stride_c % 8 == 0 && p.stride_aux % 8 == 0 && (ptrs & 15u) == 0;
}
// ... of those, what the 512 x 256 tiles take: no operand besides a bias, one result
static bool wide_takes(const fsb::GemmParams& p) {
  return p.M >= 512 && p.N >= 256 && (p.epilogue == fsb::EPI_NONE || p.epilogue == fsb::EPI_BIAS) && row_pieces(p) && p.b_ready == nullptr && p.a_ready == nullptr;
}
static GemmPlan::Kind choose_persistent(const fsb::GemmParams& p, int lda, int ldb, int num_sms) {
  const long long tiles_n = (p.N + 255) / 256;
  auto tiles = [&](int rows) -> long long { return p.batch * ((p.M + rows - 1) / rows) * tiles_n; };
  const int off_line = (lda % 64 != 0) + (ldb % 64 != 0);
  const float num_kb = static_cast<float>((p.K + fsb::BLOCK_K - 1) / fsb::BLOCK_K);
  auto cost = [&](long long n, int units, float launch, float start, float per_wave, float per_share, float epilogue) -> float {
    const float waves = static_cast<float>((n + units - 1) / units), share = static_cast<float>(n) / units;
    const float main_loops = waves * (start + num_kb * per_wave) + num_kb * share * per_share;
    return launch + (main_loops > waves * epilogue ? main_loops : waves * epilogue);
  };
  struct Wave { float start, per_wave, per_off_line, per_share, epilogue; };
  // by EPI_*: none, bias, bias + GELU, bias + residual, GELU', residual
  static const Wave pair_wave[] = {{2.2f, 0.262f, 0.017f, 0.16f, 0.f},   {2.2f, 0.262f, 0.017f, 0.16f, 0.f},   {1.06f, 0.243f, 0.021f, 0.194f, 6.952f},
                                   {2.108f, 0.209f, 0.029f, 0.217f, 7.733f}, {3.58f, 0.194f, 0.025f, 0.228f, 10.249f}, {2.181f, 0.171f, 0.029f, 0.256f, 6.407f}};
  static const Wave one_wave[] = {{1.1f, 0.229f, 0.064f, 0.25f, 0.f},    {1.1f, 0.229f, 0.064f, 0.25f, 0.f},    {0.693f, 0.376f, 0.059f, 0.066f, 8.515f},
                                  {2.111f, 0.349f, 0.068f, 0.074f, 9.57f},  {3.949f, 0.299f, 0.059f, 0.129f, 11.766f}, {2.247f, 0.281f, 0.068f, 0.144f, 7.904f}};
  auto wave_cost = [&](int rows, int units, float launch, const Wave& w) -> float {
    return cost(tiles(rows), units, launch, w.start, w.per_wave + w.per_off_line * off_line, w.per_share, w.epilogue);
  };
  const int epi = p.epilogue >= fsb::EPI_NONE && p.epilogue <= fsb::EPI_RESIDUAL ? p.epilogue : fsb::EPI_NONE;
  const float pair = wave_cost(256, num_sms / 2, 7.2f, pair_wave[epi]), one = wave_cost(128, num_sms, 5.0f, one_wave[epi]);
  if (wide_takes(p)) {
    const float wide = cost(tiles(512), num_sms / 2, 7.2f, 2.0f, 0.52f, 0.25f, 0.f);
    if (wide <= pair && wide <= one) return GemmPlan::WIDE_PAIR;
  }
  return pair < one ? GemmPlan::PAIR : GemmPlan::ONE_CTA;
}
static GemmPlan choose_gemm_plan(int M, int N, int K, int lda, int ldb, int num_sms, bool pair_allowed) {
  const long long tiles_m = (M + fsb::BLOCK_M - 1) / fsb::BLOCK_M;
  const int num_kb = (K + fsb::BLOCK_K - 1) / fsb::BLOCK_K;
  const int one_n = N <= 128 ? 128 : 256;  // tile width of the one-CTA kernel
  auto tiles = [&](int bn) -> long long { return tiles_m * ((N + bn - 1) / bn); };
  GemmPlan best = {GemmPlan::ONE_CTA, one_n, 1};
  if (pair_allowed && pair_pays(1, M, N, K, lda, ldb, num_sms)) best.kind = GemmPlan::PAIR;
  if (best.kind == GemmPlan::PAIR || tiles(one_n) > num_sms) return best;
  float cost = 6.5f + (one_n == 128 ? 0.32f : 0.39f) * num_kb;
  for (int bn = 64; bn <= 128; bn *= 2) {
    for (int c = 1; c <= 8 && c <= num_kb; c *= 2) {
      const long long ctas = tiles(bn) * c;
      const int limit = c <= 2 ? num_sms : c == 4 ? 128 : 64;
      if (ctas > limit) break;
      const float base = c == 1 ? 6.2f : c == 8 ? 10.f : 8.3f;
      const float t = base + (bn == 64 ? 0.28f : 0.32f) * ((num_kb + c - 1) / c);
      if (t < cost) {
        cost = t;
        best = {GemmPlan::CLUSTER_K, bn, c};
      }
    }
  }
  return best;
}

// The kernel of a product, or of `p.batch` stacked ones, that is neither streamed nor capped: what fsb_gemm_bf16 and
// fsb_gemm_bf16_batched launch and fsb_gemm_kernel_of reports.
static GemmPlan plan_product(const fsb::GemmParams& p, bool stacked, int lda, int ldb, int num_sms) {
  const bool pairs = pair_enabled();
  const int block_n = p.N <= 128 ? 128 : 256;
  const long long tiles = static_cast<long long>(p.batch) * ((p.M + fsb::BLOCK_M - 1) / fsb::BLOCK_M) * ((p.N + block_n - 1) / block_n);
  // more tiles than one wave of single CTAs (below, the wide tiles leave most SMs without one) and K as far as it was measured
  if (pairs && tiles > num_sms && p.M >= 256 && p.N >= 256 && p.K >= 256 && row_pieces(p))
    return {choose_persistent(p, lda, ldb, num_sms), block_n, 1};
  if (!stacked) return choose_gemm_plan(p.M, p.N, p.K, lda, ldb, num_sms, pairs);
  return {pairs && pair_pays(p.batch, p.M, p.N, p.K, lda, ldb, num_sms) ? GemmPlan::PAIR : GemmPlan::ONE_CTA, block_n, 1};
}

// What plan_product makes of a product (or of `problems` stacked ones) on a device with `num_sms` SMs, all pointers 16-byte aligned:
// 0 CTA pairs, 1 one CTA per tile, 2 split-K over clusters (a single product only), 3 CTA pairs with tiles of 512 rows.
FSB_API int fsb_gemm_kernel_of(int problems, int M, int N, int K, int lda, int ldb, int ldc, int ld_aux, int epilogue, int out_f32, int num_sms) {
  fsb::GemmParams p{};
  p.M = M; p.N = N; p.K = K;
  p.ldc = ldc; p.ld_aux = ld_aux > 0 ? ld_aux : ldc;
  p.epilogue = epilogue; p.out_f32 = out_f32; p.batch = problems;
  return static_cast<int>(plan_product(p, problems > 1, lda, ldb, num_sms).kind);
}
// The same where choose_persistent does not come in (fp32 or unaligned results, K below 256, one wave or less).
FSB_API int fsb_gemm_plan_of(long long problems, int M, int N, int K, int lda, int ldb, int num_sms) {
  if (problems > 1) return pair_enabled() && pair_pays(problems, M, N, K, lda, ldb, num_sms) ? 0 : 1;
  return static_cast<int>(choose_gemm_plan(M, N, K, lda, ldb, num_sms, pair_enabled()).kind);
}

// C ABI ------------------------------------------------------------------------------------------
// lda / ldb: elements between consecutive rows of the *stored* matrix ([rows,K] when K-major,
// [K,rows] when MN-major). All leading dimensions must be multiples of 8; pointers 16-byte aligned.
// Returns 0 on success, a cudaError_t value, or -1 for an argument / tensor-map problem.
static int gemm_bf16_impl(const void* A, const void* B, void* C, const void* bias, const void* aux, void* aux_out,
                          int M, int N, int K, int lda, int ldb, int ldc, int ld_aux, int a_mn_major, int b_mn_major,
                          int epilogue, int out_f32, int accumulate_c, int max_ctas, int* status, cudaStream_t stream,
                          const unsigned int* b_ready, unsigned int b_ready_epoch, long long b_piece_bytes, unsigned long long b_wait_ns,
                          const unsigned int* a_ready = nullptr, int a_shard_rows = 0, int a_piece_rows = 0, int a_first_shard = 0,
                          int a_num_shards = 0, int b_first_piece = 0, int ck_block_n = 0, int ck_splits = 0, int forced = 0);

FSB_API int fsb_gemm_bf16(const void* A, const void* B, void* C, const void* bias, const void* aux, void* aux_out,
                          int M, int N, int K, int lda, int ldb, int ldc, int ld_aux, int a_mn_major, int b_mn_major,
                          int epilogue, int out_f32, int accumulate_c, int max_ctas, int* status, cudaStream_t stream) {
  return gemm_bf16_impl(A, B, C, bias, aux, aux_out, M, N, K, lda, ldb, ldc, ld_aux, a_mn_major, b_mn_major, epilogue, out_f32,
                        accumulate_c, max_ctas, status, stream, nullptr, 0u, 0, 0ull);
}

// The same product by the cluster split-K kernel (gemm_cluster_k.cu) whatever its shape: block_n 64 or 128, splits 1, 2, 4
// or 8 and no more than the number of 64-wide K blocks (-1 otherwise).  fsb_gemm_bf16 chooses these by itself.
FSB_API int fsb_gemm_bf16_cluster_k(const void* A, const void* B, void* C, const void* bias, const void* aux, void* aux_out,
                                    int M, int N, int K, int lda, int ldb, int ldc, int ld_aux, int a_mn_major, int b_mn_major,
                                    int epilogue, int out_f32, int accumulate_c, int block_n, int splits, int* status, cudaStream_t stream) {
  if (splits < 1) return -1;
  return gemm_bf16_impl(A, B, C, bias, aux, aux_out, M, N, K, lda, ldb, ldc, ld_aux, a_mn_major, b_mn_major, epilogue, out_f32,
                        accumulate_c, 0, status, stream, nullptr, 0u, 0, 0ull, nullptr, 0, 0, 0, 0, 0, block_n, splits);
}

// The same product by one of the persistent kernels whatever its size: plan 1 one CTA per tile, 2 CTA pairs (M and N at
// least 256, -1 otherwise), 3 CTA pairs with tiles of 512 rows (what wide_takes, -1 otherwise).  fsb_gemm_bf16 chooses these by itself.
FSB_API int fsb_gemm_bf16_plan(const void* A, const void* B, void* C, const void* bias, const void* aux, void* aux_out,
                               int M, int N, int K, int lda, int ldb, int ldc, int ld_aux, int a_mn_major, int b_mn_major,
                               int epilogue, int out_f32, int accumulate_c, int plan, int* status, cudaStream_t stream) {
  if (plan != 1 && !((plan == 2 || plan == 3) && M >= 256 && N >= 256)) return -1;
  return gemm_bf16_impl(A, B, C, bias, aux, aux_out, M, N, K, lda, ldb, ldc, ld_aux, a_mn_major, b_mn_major, epilogue, out_f32,
                        accumulate_c, 0, status, stream, nullptr, 0u, 0, 0ull, nullptr, 0, 0, 0, 0, 0, 0, 0, plan);
}

// C[M, N] = epilogue(A[M, K] * B^T + bias) with B ([N, K], rows contiguous: ldb == K) arriving while the kernel runs:
// ready[i] >= ready_epoch means bytes [i * piece_bytes, (i + 1) * piece_bytes) of B are in place (see GemmParams::b_ready).
// Pieces are sent cyclically from `first_piece` on and flags are indexed in sending order.
// Needs the CTA-pair kernel (M, N >= 256); returns -1 otherwise.  wait_ms bounds every wait for a piece.
FSB_API int fsb_gemm_bf16_streamed_b(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, int lda, int ldc,
                                     int epilogue, const unsigned int* ready, unsigned int ready_epoch, long long piece_bytes,
                                     int first_piece, long long wait_ms, int* status, cudaStream_t stream) {
  if (M < 256 || N < 256 || ready == nullptr || piece_bytes <= 0) return -1;
  if (epilogue != fsb::EPI_NONE && epilogue != fsb::EPI_BIAS) return -1;
  if (first_piece < 0) return -1;
  return gemm_bf16_impl(A, B, C, bias, nullptr, nullptr, M, N, K, lda, K, ldc, ldc, 0, 0, epilogue, 0, 0, 0, status, stream, ready,
                        ready_epoch, piece_bytes, static_cast<unsigned long long>(wait_ms > 0 ? wait_ms : 30000) * 1000000ull, nullptr, 0, 0,
                        0, 0, first_piece);
}

// C[M, N] = epilogue(A * B^T + bias) with A ([M, K], rows contiguous) arriving while the kernel runs, row block by row block
// (see GemmParams::a_ready): the all-gather of a sequence-parallel activation consumed by the product it feeds.
// B is [N, K] (ldb) or, with b_mn_major, [K, N].  Needs the CTA-pair kernel (M, N >= 256); returns -1 otherwise.
FSB_API int fsb_gemm_bf16_streamed_a(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, int ldb, int ldc,
                                     int b_mn_major, int epilogue, const unsigned int* ready, unsigned int ready_epoch, int shard_rows,
                                     int piece_rows, int first_shard, int num_shards, long long wait_ms, int* status, cudaStream_t stream) {
  if (M < 256 || N < 256 || ready == nullptr || shard_rows <= 0 || piece_rows <= 0 || num_shards <= 0 || shard_rows * num_shards != M) return -1;
  if (first_shard < 0 || first_shard >= num_shards) return -1;
  if (epilogue != fsb::EPI_NONE && epilogue != fsb::EPI_BIAS && epilogue != fsb::EPI_BIAS_GELU) return -1;
  return gemm_bf16_impl(A, B, C, bias, nullptr, nullptr, M, N, K, K, ldb, ldc, ldc, 0, b_mn_major, epilogue, 0, 0, 0, status, stream, nullptr,
                        ready_epoch, 0, static_cast<unsigned long long>(wait_ms > 0 ? wait_ms : 30000) * 1000000ull, ready, shard_rows,
                        piece_rows, first_shard, num_shards);
}

static int gemm_bf16_impl(const void* A, const void* B, void* C, const void* bias, const void* aux, void* aux_out,
                          int M, int N, int K, int lda, int ldb, int ldc, int ld_aux, int a_mn_major, int b_mn_major,
                          int epilogue, int out_f32, int accumulate_c, int max_ctas, int* status, cudaStream_t stream,
                          const unsigned int* b_ready, unsigned int b_ready_epoch, long long b_piece_bytes, unsigned long long b_wait_ns,
                          const unsigned int* a_ready, int a_shard_rows, int a_piece_rows, int a_first_shard, int a_num_shards,
                          int b_first_piece, int ck_block_n, int ck_splits, int forced) {
  using namespace fsb;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((lda % 8) || (ldb % 8) || (reinterpret_cast<uintptr_t>(A) % 16) || (reinterpret_cast<uintptr_t>(B) % 16)) return -1;
  if (accumulate_c && !out_f32) return -1;

  const int block_n = (N <= 128) ? 128 : 256;
  CUtensorMap ta, tb;
  bool ok = true;
  if (!a_mn_major) ok &= fsb_host::encode_2d_16bit(&ta, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda, BLOCK_K, BLOCK_M);
  else             ok &= fsb_host::encode_2d_16bit(&ta, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, 64, BLOCK_K);
  if (!b_mn_major) ok &= fsb_host::encode_2d_16bit(&tb, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb, BLOCK_K, block_n);
  else             ok &= fsb_host::encode_2d_16bit(&tb, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, 64, BLOCK_K);
  if (!ok) return -1;

  GemmParams p;
  p.C = C;
  p.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  p.aux = reinterpret_cast<const __nv_bfloat16*>(aux);
  p.aux_out = reinterpret_cast<__nv_bfloat16*>(aux_out);
  p.M = M; p.N = N; p.K = K;
  p.ldc = ldc; p.ld_aux = ld_aux > 0 ? ld_aux : ldc;
  p.a_mn_major = a_mn_major; p.b_mn_major = b_mn_major;
  p.epilogue = epilogue; p.out_f32 = out_f32; p.accumulate_c = accumulate_c;
  p.status = status;
  p.batch = 1; p.stride_c = p.stride_aux = p.stride_bias = 0;
  p.sched_slot = 0;
  p.b_ready = b_ready; p.b_ready_epoch = b_ready_epoch; p.b_piece_bytes = b_piece_bytes; p.b_wait_ns = b_wait_ns;
  p.b_num_pieces = b_piece_bytes > 0 ? static_cast<int>((static_cast<long long>(N) * K * 2 + b_piece_bytes - 1) / b_piece_bytes) : 1;
  p.b_first_piece = b_ready != nullptr ? b_first_piece % p.b_num_pieces : 0;
  p.a_ready = a_ready; p.a_ready_epoch = b_ready_epoch; p.a_shard_rows = a_shard_rows; p.a_piece_rows = a_piece_rows;
  p.a_first_shard = a_first_shard; p.a_num_shards = a_num_shards;

  int dev = 0;
  cudaGetDevice(&dev);
  static int num_sms_cache[64] = {0};
  static bool attr_set[64][2] = {{false}};
  const int di = dev & 63;
  if (num_sms_cache[di] == 0) cudaDeviceGetAttribute(&num_sms_cache[di], cudaDevAttrMultiProcessorCount, dev);
  const int num_sms = num_sms_cache[di];
  const int tiles = ((M + BLOCK_M - 1) / BLOCK_M) * ((N + block_n - 1) / block_n);
  int grid = tiles < num_sms ? tiles : num_sms;
  if (max_ctas > 0 && grid > max_ctas) grid = max_ctas;

  if (ck_splits > 0) return fsb_host::gemm_cluster_k(ta, B, ldb, p, ck_block_n, ck_splits, dev, stream);

  if ((b_ready != nullptr || a_ready != nullptr) && !(pair_enabled() && M >= 256 && N >= 256 && max_ctas == 0)) return -1;
  const bool streamed = b_ready != nullptr || a_ready != nullptr;  // only the pair kernel waits for arriving operands
  GemmPlan plan = {GemmPlan::ONE_CTA, block_n, 1};
  if (streamed) plan.kind = GemmPlan::PAIR;
  else if (forced == 3 && !wide_takes(p)) return -1;
  else if (forced != 0) plan.kind = forced == 3 ? GemmPlan::WIDE_PAIR : forced == 2 ? GemmPlan::PAIR : GemmPlan::ONE_CTA;
  else if (max_ctas == 0) plan = plan_product(p, false, lda, ldb, num_sms);
  if (plan.kind == GemmPlan::CLUSTER_K) return fsb_host::gemm_cluster_k(ta, B, ldb, p, plan.block_n, plan.splits, dev, stream);
  // Run-time tile hand-out for products large enough to share the device with a collective; small ones stride.
  if (max_ctas == 0 && M >= 256 && N >= 256 && (plan.kind == GemmPlan::PAIR || plan.kind == GemmPlan::WIDE_PAIR || tiles > num_sms)) {
    p.sched_slot = sched_slot_of(di, stream);
  }
  if (plan.kind == GemmPlan::PAIR || plan.kind == GemmPlan::WIDE_PAIR) {
    // the B map's box is this CTA's 128 columns (K-major) / 64 (MN-major, unchanged)
    if (!b_mn_major && !fsb_host::encode_2d_16bit(&tb, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb, BLOCK_K, PAIR_HALF_N)) return -1;
    return plan.kind == GemmPlan::PAIR ? launch_pair<false, 1>(ta, tb, p, num_sms, di, stream) : launch_pair<false, 2>(ta, tb, p, num_sms, di, stream);
  }
  if (block_n == 256) {
    if (!attr_set[di][0]) {
      cudaFuncSetAttribute(gemm_bf16_tcgen05_kernel<256, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SmemLayout<256>::TOTAL);
      attr_set[di][0] = true;
    }
    gemm_bf16_tcgen05_kernel<256, false><<<grid, GEMM_THREADS, SmemLayout<256>::TOTAL, stream>>>(ta, tb, p);
  } else {
    if (!attr_set[di][1]) {
      cudaFuncSetAttribute(gemm_bf16_tcgen05_kernel<128, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SmemLayout<128>::TOTAL);
      attr_set[di][1] = true;
    }
    gemm_bf16_tcgen05_kernel<128, false><<<grid, GEMM_THREADS, SmemLayout<128>::TOTAL, stream>>>(ta, tb, p);
  }
  return static_cast<int>(cudaGetLastError());
}

// `batch` independent products of one shape in a single launch (the local experts of an MoE layer):
//   C[b] = epilogue( A[b] * B[b]^T ),  b = 0 .. batch-1
// stride_*: elements between consecutive problems (stride_bias may be 0 for a shared bias).  Layout flags, leading
// dimensions and epilogues as for fsb_gemm_bf16.  Rows of a problem never leak into the next one: the tensor maps are
// three-dimensional, so a tile that overhangs M or N reads zeros.
static int gemm_bf16_batched_impl(const void* A, const void* B, void* C, const void* bias, const void* aux, void* aux_out, int batch,
                                  int M, int N, int K, int lda, int ldb, int ldc, int ld_aux, long long stride_a, long long stride_b,
                                  long long stride_c, long long stride_aux, long long stride_bias, int a_mn_major, int b_mn_major,
                                  int epilogue, int out_f32, int accumulate_c, int* status, cudaStream_t stream, int forced) {
  using namespace fsb;
  if (batch <= 0 || M <= 0 || N <= 0 || K <= 0) return 0;
  if ((lda % 8) || (ldb % 8) || (stride_a % 8) || (stride_b % 8) || (reinterpret_cast<uintptr_t>(A) % 16) || (reinterpret_cast<uintptr_t>(B) % 16)) return -1;
  if (accumulate_c && !out_f32) return -1;
  const int block_n = (N <= 128) ? 128 : 256;
  CUtensorMap ta, tb;
  bool ok = true;
  if (!a_mn_major) ok &= fsb_host::encode_3d_16bit(&ta, A, (uint64_t)K, (uint64_t)M, (uint64_t)batch, (uint64_t)lda, (uint64_t)stride_a, BLOCK_K, BLOCK_M, 1);
  else             ok &= fsb_host::encode_3d_16bit(&ta, A, (uint64_t)M, (uint64_t)K, (uint64_t)batch, (uint64_t)lda, (uint64_t)stride_a, 64, BLOCK_K, 1);
  if (!b_mn_major) ok &= fsb_host::encode_3d_16bit(&tb, B, (uint64_t)K, (uint64_t)N, (uint64_t)batch, (uint64_t)ldb, (uint64_t)stride_b, BLOCK_K, block_n, 1);
  else             ok &= fsb_host::encode_3d_16bit(&tb, B, (uint64_t)N, (uint64_t)K, (uint64_t)batch, (uint64_t)ldb, (uint64_t)stride_b, 64, BLOCK_K, 1);
  if (!ok) return -1;
  GemmParams p;
  p.C = C;
  p.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  p.aux = reinterpret_cast<const __nv_bfloat16*>(aux);
  p.aux_out = reinterpret_cast<__nv_bfloat16*>(aux_out);
  p.M = M; p.N = N; p.K = K;
  p.ldc = ldc; p.ld_aux = ld_aux > 0 ? ld_aux : ldc;
  p.a_mn_major = a_mn_major; p.b_mn_major = b_mn_major;
  p.epilogue = epilogue; p.out_f32 = out_f32; p.accumulate_c = accumulate_c;
  p.status = status;
  p.sched_slot = 0;
  p.b_ready = nullptr; p.b_ready_epoch = 0; p.b_piece_bytes = 0; p.b_wait_ns = 0; p.b_first_piece = 0; p.b_num_pieces = 1;
  p.a_ready = nullptr; p.a_ready_epoch = 0; p.a_shard_rows = p.a_piece_rows = p.a_first_shard = p.a_num_shards = 0;
  p.batch = batch; p.stride_c = stride_c; p.stride_aux = stride_aux > 0 ? stride_aux : stride_c; p.stride_bias = stride_bias;
  int dev = 0, num_sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev);
  const long long tiles = static_cast<long long>(batch) * ((M + BLOCK_M - 1) / BLOCK_M) * ((N + block_n - 1) / block_n);
  const int grid = tiles < num_sms ? static_cast<int>(tiles) : num_sms;
  if (forced == 3 && !wide_takes(p)) return -1;
  GemmPlan::Kind kind = forced == 3 ? GemmPlan::WIDE_PAIR : forced == 2 ? GemmPlan::PAIR : GemmPlan::ONE_CTA;
  if (forced == 0) kind = plan_product(p, true, lda, ldb, num_sms).kind;
  if (kind != GemmPlan::ONE_CTA) {
    if (!b_mn_major && !fsb_host::encode_3d_16bit(&tb, B, (uint64_t)K, (uint64_t)N, (uint64_t)batch, (uint64_t)ldb, (uint64_t)stride_b, BLOCK_K, PAIR_HALF_N, 1)) return -1;
    p.sched_slot = sched_slot_of(dev & 63, stream);
    return kind == GemmPlan::WIDE_PAIR ? launch_pair<true, 2>(ta, tb, p, num_sms, dev & 63, stream) : launch_pair<true, 1>(ta, tb, p, num_sms, dev & 63, stream);
  }
  static bool attr_set_dev[64][2] = {{false}};  // the attribute is per device
  bool* attr_set = attr_set_dev[dev & 63];
  if (block_n == 256) {
    if (!attr_set[0]) {
      cudaFuncSetAttribute(gemm_bf16_tcgen05_kernel<256, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SmemLayout<256>::TOTAL);
      attr_set[0] = true;
    }
    gemm_bf16_tcgen05_kernel<256, true><<<grid, GEMM_THREADS, SmemLayout<256>::TOTAL, stream>>>(ta, tb, p);
  } else {
    if (!attr_set[1]) {
      cudaFuncSetAttribute(gemm_bf16_tcgen05_kernel<128, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SmemLayout<128>::TOTAL);
      attr_set[1] = true;
    }
    gemm_bf16_tcgen05_kernel<128, true><<<grid, GEMM_THREADS, SmemLayout<128>::TOTAL, stream>>>(ta, tb, p);
  }
  return static_cast<int>(cudaGetLastError());
}

FSB_API int fsb_gemm_bf16_batched(const void* A, const void* B, void* C, const void* bias, const void* aux, void* aux_out, int batch,
                                  int M, int N, int K, int lda, int ldb, int ldc, int ld_aux, long long stride_a, long long stride_b,
                                  long long stride_c, long long stride_aux, long long stride_bias, int a_mn_major, int b_mn_major,
                                  int epilogue, int out_f32, int accumulate_c, int* status, cudaStream_t stream) {
  return gemm_bf16_batched_impl(A, B, C, bias, aux, aux_out, batch, M, N, K, lda, ldb, ldc, ld_aux, stride_a, stride_b, stride_c, stride_aux, stride_bias, a_mn_major, b_mn_major,
                           epilogue, out_f32, accumulate_c, status, stream, 0);
}

// The same products by one of the persistent kernels whatever their size: plan 1, 2 or 3 as for fsb_gemm_bf16_plan.
// fsb_gemm_bf16_batched chooses by itself.
FSB_API int fsb_gemm_bf16_batched_plan(const void* A, const void* B, void* C, const void* bias, const void* aux, void* aux_out, int batch,
                                  int M, int N, int K, int lda, int ldb, int ldc, int ld_aux, long long stride_a, long long stride_b,
                                  long long stride_c, long long stride_aux, long long stride_bias, int a_mn_major, int b_mn_major,
                                  int epilogue, int out_f32, int accumulate_c, int plan, int* status, cudaStream_t stream) {
  if (plan != 1 && !((plan == 2 || plan == 3) && M >= 256 && N >= 256)) return -1;
  return gemm_bf16_batched_impl(A, B, C, bias, aux, aux_out, batch, M, N, K, lda, ldb, ldc, ld_aux, stride_a, stride_b, stride_c, stride_aux, stride_bias, a_mn_major, b_mn_major,
                           epilogue, out_f32, accumulate_c, status, stream, plan);
}
