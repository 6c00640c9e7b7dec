// Causal flash attention (forward + backward) on tcgen05 / TMEM for packed QKV.
//
//   qkv : bf16 [B, S, 3, H, D]   (the output of the fused QKV projection, untouched)
//   o   : bf16 [B, S, H, D]      lse : fp32 [B, H, S]   (natural-log sum-exp of the scaled scores)
//
// All tiles are fetched straight from the packed tensor with per-CTA TMA loads (no permute / contiguous /
// cat glue kernels) and every product runs on the tensor cores with fp32 accumulators in TMEM:
//
//   forward (attention_fwd_pingpong.cu)        S = Q K^T -> online softmax -> O += P V
//   backward dQ (items of 128 query rows)      S = Q K^T, dP = dO V^T -> dS -> dQ += dS K
//   backward dK/dV (items of 128 key rows)     S^T = K Q^T, dP^T = V dO^T -> P^T, dS^T -> dV += P^T dO, dK += dS^T Q
//
// This file holds the backward.  Thread roles per CTA (608 threads): warp 0 TMA producer, warp 1 issuer of the score products
// (+TMEM allocation), warps 2..17 four groups of four "softmax" warps, one thread per accumulator row (TMEM lane == row), which
// do the exponentials in registers and hand the bf16 results back to the tensor cores through TMEM, warp 18 issuer of the
// accumulating products.  An issuing warp is held until the tensor pipe takes its products, and a wait that does not block
// costs it 100 - 200 cycles all the same; one warp for all products left the pipe idle behind its waits (B2 S8192 H16 D64: of
// 1 290 cycles a step of 64 queries or keys, 650 of products, while the probabilities of the step lay ready for 1 500).
// The score products of an item are issued behind the accumulating ones of the item before (acc_issued): ahead of the last of
// those, whose result the compute warps wait for, they held up items of few steps (HB sequences of all heads, us without / with: S16
// HB1760 D128 85.9 / 83.2, S77 HB640 D64 46.0 / 45.1, S268 HB640 D128 223.6 / 221.1; long ones alike).  What an issuer more still
// costs the shortest sequences is 2 to 4 % (78.6, 43.3 and 221.1 us with one).
// A K-major tile [rows, 64] and an MN-major tile of the same bytes differ only in the MMA descriptor, so each
// streamed tile is loaded once and used both as a "transposed" and a "plain" operand.
// Any sequence length: the tensor maps are three-dimensional (columns, positions, batch), so a tile that overhangs the
// sequence reads zeros; its keys lie above every real query's diagonal, its queries have lse = +inf (probability 0), and
// rows past the end are not stored.
// Every mbarrier wait is bounded (see sm100.cuh).
//
// Replaces nn.MultiheadAttention / bmm+softmax in the reference's models
// (benchmarks/models/transformer_lm.py:107,150-152,169-183).

#include "sm100.cuh"

namespace fsb {

constexpr int ATT_THREADS = 608;  // TMA warp, MMA warp, 16 compute warps (four per TMEM lane quadrant), second MMA warp
constexpr int ATT_ACC_WARP = 18;  // the second MMA warp: accumulating products
constexpr int ATT_BM = 128;  // rows owned by a CTA (TMEM lanes)
constexpr float LOG2E = 1.4426950408889634f;

struct AttnParams {
  int B, S, H, D;
  int S_pad;          // S rounded up to whole tiles of 128: row length of delta
  float scale;        // softmax scale (1/sqrt(D))
  // [2, B, H, S_pad]: scale * rowsum(dO * O), then the base-2 lse, both written by attn_delta_kernel.  Rows past the end
  // hold 0 and +inf, so their probabilities 2^(0 - inf) and dS are exactly zero.
  const float* delta;
  __nv_bfloat16* dqkv;  // [B*S, 3*H*D]
  int* status;
};

__device__ __forceinline__ float ex2_approx(float x) {  // 2^x on the MUFU pipe, one instruction
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Work item of this CTA in round r.  Items are ordered longest first; the rounds run through the CTAs forwards and
// backwards in turn, so that the CTA with the longest item of one round gets the shortest of the next.
__device__ __forceinline__ int snake_item(int r) {
  const int g = static_cast<int>(gridDim.x), b = static_cast<int>(blockIdx.x);
  return (r & 1) ? (r + 1) * g - 1 - b : r * g + b;
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}

// Operand descriptors of tiles made of [rows x 64] slabs of `slab_bytes`, and the byte offsets of their k-steps: K-major 16
// elements (32 bytes inside the swizzle row); MN-major (the same bytes as [k_rows x 64] slabs) 16 k_rows = 2048 bytes.
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t base) { return make_smem_desc(base, 16u, 1024u); }
__device__ __forceinline__ uint64_t desc_mnmajor(uint32_t base, uint32_t slab_bytes) { return make_smem_desc(base, slab_bytes, 1024u); }
__device__ __forceinline__ constexpr uint32_t kstep_kmajor(int ks, uint32_t slab_bytes) {
  return static_cast<uint32_t>(ks >> 2) * slab_bytes + static_cast<uint32_t>(ks & 3) * 32u;
}
__device__ __forceinline__ constexpr uint32_t kstep_mnmajor(int ks) { return static_cast<uint32_t>(ks) * 2048u; }

struct AttnBars {
  uint64_t stat_full;     // stationary tiles landed
  uint64_t stat_empty;    // the item's last products that read the stationary tiles have completed
  uint64_t str_full[6];   // streamed stage landed
  uint64_t str_empty[6];  // streamed stage free again
  uint64_t s_full[3];     // scores and dP of a step are in buffer b
  uint64_t p_full[3];     // the 8 warps of the step have written dS (dQ kernel) / P^T and dS^T (dK/dV kernel) over them
  uint64_t buf_free[3];   // the accumulating products that read buffer b have completed
  uint64_t acc_issued;    // the item's accumulating products are on their way: the next item's score products may follow
  uint64_t acc_done;      // the item's accumulating products have completed
  uint64_t acc_free;      // the 16 compute warps have read the item's output accumulators
  uint32_t tmem_slot;
  int abort_flag;
};

static_assert(sizeof(AttnBars) <= 256, "the barrier block of the shared-memory layouts");

__device__ __forceinline__ void attn_init_bars(AttnBars* b) {
  mbar_init(&b->stat_full, 1);
  mbar_init(&b->stat_empty, 1);
  for (int i = 0; i < 6; ++i) {
    mbar_init(&b->str_full[i], 1);
    mbar_init(&b->str_empty[i], 1);
  }
  for (int i = 0; i < 3; ++i) {
    mbar_init(&b->s_full[i], 1);
    mbar_init(&b->p_full[i], 8);
    mbar_init(&b->buf_free[i], 1);
  }
  mbar_init(&b->acc_issued, 1);
  mbar_init(&b->acc_done, 1);
  mbar_init(&b->acc_free, 16);
  b->abort_flag = 0;
  fence_barrier_init();
}

__device__ __forceinline__ void attn_teardown(AttnBars* bars, int warp, uint32_t tmem_base, uint32_t ncols, int* status) {
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (bars->abort_flag) {
    if (threadIdx.x == 0 && status != nullptr) atomicExch(status, FSB_ERR_WAIT_TIMEOUT | (bars->abort_flag << 8));
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, ncols);
  }
}

// dS for 16 columns (starting at key column `col0` of the 128-key tile) of one row:
// P = 2^(s * sl2 - lse2), dS = P * (dP * scale - delta * scale)
template <bool DIAG>
__device__ __forceinline__ void dq_cols16(const uint32_t (&rs)[16], const uint32_t (&rp)[16], int col0, int row, float sl2,
                                          float lse2, float scale, float delta_s, uint32_t (&pk)[8]) {
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    float p0 = ex2_approx(fmaf(__uint_as_float(rs[i]), sl2, -lse2));
    float p1 = ex2_approx(fmaf(__uint_as_float(rs[i + 1]), sl2, -lse2));
    if (DIAG) {
      if (col0 + i > row) p0 = 0.f;
      if (col0 + i + 1 > row) p1 = 0.f;
    }
    pk[i >> 1] = pack_bf16(p0 * fmaf(__uint_as_float(rp[i]), scale, -delta_s), p1 * fmaf(__uint_as_float(rp[i + 1]), scale, -delta_s));
  }
}

// =================================================================================================
// Backward, dQ: one CTA per 128 query rows; streams K and V tiles and consumes them in steps of 64 keys.
//
// Two sets of eight warps take alternate steps (set b the steps u with u & 1 == b; two threads per query row with 32 keys
// each): while one set is in its exponentials the other one waits for TMEM loads, stores or the
// tensor pipe.  What bounds the kernel is the length of that chain, not a pipe (exponentials 34 %, tensor pipe 25 % busy on
// the busiest SM with one thread per row and set), hence the short slices per thread and the many warps.
// Backward of B2 S8192 H16 D64: 1870 us with eight warps that all worked on the same step and passed dS through shared
// memory, 1447 us with the two sets (B8 S2048 H16 D128 750 -> 690 us).
// dS overwrites scores that the same thread has read (32 keys become the first 16 of their 32 columns) and feeds dS K as
// the TMEM A operand, so it does not pass through shared memory.  Step u uses buffer u mod n; one warp issues S and dP of
// step u + n as soon as dQ(u), issued by another warp, has read the buffer (buf_free).  Head size 64
// leaves TMEM for three buffers: a set that has finished step u then finds the scores of step u + 2 ready, where with two
// it waits for dQ(u) and those products (backward of B2 S8192 H16 D64 1447 -> 1315 us).
// =================================================================================================
template <int D>
struct DqSmem {
  static constexpr int TILE = ATT_BM * D * 2;
  static constexpr int Q_OFF = 0;
  static constexpr int DO_OFF = TILE;
  static constexpr int STAGES = D == 64 ? 4 : 2;  // K / V tiles in flight
  static constexpr int K_OFF = 2 * TILE;
  static constexpr int V_OFF = (2 + STAGES) * TILE;
  static constexpr int BAR_OFF = (2 + 2 * STAGES) * TILE;
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;
};

template <int D>
__global__ void __launch_bounds__(ATT_THREADS, 1)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tm_qkv, const __grid_constant__ CUtensorMap tm_do, AttnParams p) {
  using L = DqSmem<D>;
  constexpr int SLABS = D / 64;
  constexpr uint32_t SLAB = ATT_BM * 128;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  AttnBars* bars = reinterpret_cast<AttnBars*>(smem + L::BAR_OFF);
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;  // warp-uniform
  // Persistent: one CTA per SM walks the work items (one 128-row query tile of one head), long rows first, dealt
  // by snake_item; TMEM, barriers and the K / V ring live for the whole kernel (running counters give the phases).
  const int n_qt = p.S_pad / ATT_BM;
  const int HB = p.H * p.B;
  const int n_items = n_qt * HB;
  const int HD = p.H * D;
  constexpr uint32_t TMEM_COLS = 512;  // buffer b: S [128 b, +64) dP [128 b + 64, +64); then dQ
  constexpr int NBUF = D == 64 ? 3 : 2;
  constexpr uint32_t DQ_COL = NBUF * 128;

  if (threadIdx.x == 0) {
    attn_init_bars(bars);
    tma_prefetch_desc(&tm_qkv);
    tma_prefetch_desc(&tm_do);
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, bars->tmem_slot, 0);

  if (warp == 0) {
    if (lane == 0) {
      uint32_t jt = 0, it = 0;  // key tiles / items so far
      bool ok = true;
      for (int item; ok && (item = snake_item(static_cast<int>(it))) < n_items; ++it) {
        const int qt = n_qt - 1 - item / HB;
        const int hb = item % HB;
        const int h = hb % p.H, b = hb / p.H;
        const int n_kv = qt + 1;
        const int row0 = qt * ATT_BM;
        if (!mbar_wait(&bars->stat_empty, (it & 1u) ^ 1u, abort_flag, 33)) { ok = false; break; }
        mbar_expect_tx(&bars->stat_full, 2 * L::TILE);
#pragma unroll
        for (int c = 0; c < SLABS; ++c) {
          tma_load_3d(smem + L::Q_OFF + c * SLAB, &tm_qkv, &bars->stat_full, h * D + c * 64, row0, b);
          tma_load_3d(smem + L::DO_OFF + c * SLAB, &tm_do, &bars->stat_full, h * D + c * 64, row0, b);
        }
        for (int j = 0; j < n_kv; ++j, ++jt) {
          const int st = jt % L::STAGES;
          if (!mbar_wait(&bars->str_empty[st], ((jt / L::STAGES) & 1u) ^ 1u, abort_flag, 34)) { ok = false; break; }
          const int krow = j * ATT_BM;
          mbar_expect_tx(&bars->str_full[st], 2 * L::TILE);
#pragma unroll
          for (int c = 0; c < SLABS; ++c) {
            tma_load_3d(smem + L::K_OFF + st * L::TILE + c * SLAB, &tm_qkv, &bars->str_full[st], HD + h * D + c * 64, krow, b);
            tma_load_3d(smem + L::V_OFF + st * L::TILE + c * SLAB, &tm_qkv, &bars->str_full[st], 2 * HD + h * D + c * 64, krow, b);
          }
        }
      }
    }
  } else if (warp == 1) {
    // Issuer of S and dP: the whole warp, see umma_f16_ss_warp.  Step u = key tile u / 2, keys [64 (u & 1), +64) of it; stages
    // and buffers go round over the steps of all items.
    const uint32_t idesc_s = make_idesc_f16(ATT_BM, 64, true, false, false);
    const uint64_t dq = desc_kmajor(smem_u32(smem + L::Q_OFF)), ddo = desc_kmajor(smem_u32(smem + L::DO_OFF));
    const uint64_t dk0 = desc_kmajor(smem_u32(smem + L::K_OFF)), dv0 = desc_kmajor(smem_u32(smem + L::V_OFF));
    uint32_t st = 0, st_phase = 0, buf = 0, buf_phase = 0, it = 0;
    bool ok = true;
    for (int item; ok && (item = snake_item(static_cast<int>(it))) < n_items; ++it) {
      const int qt = n_qt - 1 - item / HB;
      const int n_steps = 2 * (qt + 1);
      if (it > 0 && !mbar_wait_warp(&bars->acc_issued, (it - 1u) & 1u, abort_flag, 43)) { ok = false; break; }
      if (!mbar_wait_warp(&bars->stat_full, it & 1u, abort_flag, 37)) { ok = false; break; }
      for (int u = 0; u < n_steps; ++u) {
        if ((u & 1) == 0 && !mbar_wait_warp(&bars->str_full[st], st_phase, abort_flag, 35)) { ok = false; break; }
        if (!mbar_wait_warp(&bars->buf_free[buf], buf_phase ^ 1u, abort_flag, 36)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t off = st * L::TILE + (u & 1) * 8192u;  // rows 64 (u & 1) .. of every slab
        const uint64_t dk = desc_offset(dk0, off), dv = desc_offset(dv0, off);
        const uint32_t t_s = tmem_base + buf * 128;
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
          umma_f16_ss_warp(t_s, desc_offset(dq, kstep_kmajor(ks, SLAB)), desc_offset(dk, kstep_kmajor(ks, SLAB)), idesc_s, ks != 0);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
          umma_f16_ss_warp(t_s + 64, desc_offset(ddo, kstep_kmajor(ks, SLAB)), desc_offset(dv, kstep_kmajor(ks, SLAB)), idesc_s, ks != 0);
        umma_commit_warp(&bars->s_full[buf]);
        if (u == n_steps - 1) umma_commit_warp(&bars->stat_empty);  // the item's last use of Q and dO
        if (++buf == NBUF) { buf = 0; buf_phase ^= 1u; }
        if ((u & 1) != 0 && ++st == L::STAGES) { st = 0; st_phase ^= 1u; }
      }
    }
  } else if (warp == ATT_ACC_WARP) {
    // Issuer of dQ += dS K: dS from TMEM, K tile read MN-major.  (Its stage is full: S of the step was made of it.)
    const uint32_t idesc_q = make_idesc_f16(ATT_BM, D, true, false, true);
    const uint64_t dkt0 = desc_mnmajor(smem_u32(smem + L::K_OFF), SLAB);
    uint32_t st = 0, buf = 0, buf_phase = 0, it = 0;
    bool ok = true;
    for (int item; ok && (item = snake_item(static_cast<int>(it))) < n_items; ++it) {
      const int qt = n_qt - 1 - item / HB;
      const int n_steps = 2 * (qt + 1);
      // the dQ accumulator still belongs to the previous item until its threads have read it
      if (!mbar_wait_warp(&bars->acc_free, (it & 1u) ^ 1u, abort_flag, 38)) { ok = false; break; }
      for (int u = 0; u < n_steps; ++u) {
        if (!mbar_wait_warp(&bars->p_full[buf], buf_phase, abort_flag, 39)) { ok = false; break; }
        tc_fence_after_sync();
        const uint64_t dkt = desc_offset(dkt0, st * L::TILE + (u & 1) * 4 * 2048u);
        const uint32_t t_s = tmem_base + buf * 128;
#pragma unroll
        for (int ks = 0; ks < 64 / 16; ++ks)
          umma_f16_ts_warp(tmem_base + DQ_COL, t_s + (ks >> 1) * 32 + (ks & 1) * 8, desc_offset(dkt, kstep_mnmajor(ks)), idesc_q, (u | ks) != 0);
        umma_commit_warp(&bars->buf_free[buf]);
        if ((u & 1) != 0) umma_commit_warp(&bars->str_empty[st]);
        if (u == n_steps - 1) {
          umma_commit_warp(&bars->acc_done);
          if (lane == 0) mbar_arrive(&bars->acc_issued);
        }
        if (++buf == NBUF) { buf = 0; buf_phase ^= 1u; }
        if ((u & 1) != 0 && ++st == L::STAGES) st = 0;
      }
    }
  } else {
    const int quad = warp & 3;
    const int grp = (warp - 2) >> 2;          // which D/4 output columns
    const int set = grp >> 1, half = grp & 1;  // which of two consecutive steps, which 32 of its 64 keys
    const int row = quad * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t ts0 = tmem_base + half * 32 + lane_off;  // this thread's scores in buffer 0; its dS overwrites the first 16 columns
    const int col0 = set * 64 + half * 32;                  // first key of this thread inside the 128-key tile
    const float sl2 = p.scale * LOG2E;
    uint32_t ut = set, it = 0;  // this set's next step over all items (every item has an even number), items so far
    bool ok = true;
    for (int item; ok && (item = snake_item(static_cast<int>(it))) < n_items; ++it) {
      const int qt = n_qt - 1 - item / HB;
      const int hb = item % HB;
      const int h = hb % p.H, b = hb / p.H;
      const int pos = qt * ATT_BM + row;  // this thread's query (sequence index)
      const size_t stat_idx = (static_cast<size_t>(b) * p.H + h) * p.S_pad + pos;
      const float lse2 = p.delta[static_cast<size_t>(p.B) * p.H * p.S_pad + stat_idx];  // base-2 lse, written by the delta kernel
      const float delta_s = p.delta[stat_idx];                                       // scale * rowsum(dO * O)
      for (int j = 0; j <= qt; ++j, ut += 2) {
        const uint32_t buf = ut % NBUF, ts = ts0 + buf * 128;
        if (!mbar_wait(&bars->s_full[buf], (ut / NBUF) & 1u, abort_flag, 40)) { ok = false; break; }
        tc_fence_after_sync();
        const bool diag = (j == qt);
        uint32_t rs0[16], rp0[16], rs1[16], rp1[16], pk[8];
        tmem_ld_32x16(ts, rs0);
        tmem_ld_32x16(ts + 64, rp0);
        tmem_ld_32x16(ts + 16, rs1);
        tmem_ld_32x16(ts + 80, rp1);
        tmem_ld_wait();
        if (!diag) dq_cols16<false>(rs0, rp0, col0, row, sl2, lse2, p.scale, delta_s, pk);
        else       dq_cols16<true>(rs0, rp0, col0, row, sl2, lse2, p.scale, delta_s, pk);
        tmem_st_32x8(ts, pk);
        if (!diag) dq_cols16<false>(rs1, rp1, col0 + 16, row, sl2, lse2, p.scale, delta_s, pk);
        else       dq_cols16<true>(rs1, rp1, col0 + 16, row, sl2, lse2, p.scale, delta_s, pk);
        tmem_st_32x8(ts + 8, pk);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->p_full[buf]);
      }
      if (!ok) break;
      if (!mbar_wait(&bars->acc_done, it & 1u, abort_flag, 42)) { ok = false; break; }
      tc_fence_after_sync();
      __nv_bfloat16* drow = p.dqkv + (static_cast<size_t>(b) * p.S + pos) * (3 * HD) + h * D + grp * (D / 4);
#pragma unroll 1
      for (int c = 0; c < D / 4; c += 16) {
        uint32_t r[16];
        tmem_ld_32x16(tmem_base + DQ_COL + lane_off + grp * (D / 4) + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          uint4 v;
          v.x = pack_bf16(__uint_as_float(r[q * 8 + 0]), __uint_as_float(r[q * 8 + 1]));
          v.y = pack_bf16(__uint_as_float(r[q * 8 + 2]), __uint_as_float(r[q * 8 + 3]));
          v.z = pack_bf16(__uint_as_float(r[q * 8 + 4]), __uint_as_float(r[q * 8 + 5]));
          v.w = pack_bf16(__uint_as_float(r[q * 8 + 6]), __uint_as_float(r[q * 8 + 7]));
          if (pos < p.S) *reinterpret_cast<uint4*>(drow + c + q * 8) = v;
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->acc_free);
    }
  }
  attn_teardown(bars, warp, tmem_base, TMEM_COLS, p.status);
}

// P^T and dS^T for one key row against 16 queries (`qa0` = sequence index of the first); the per-query statistics come
// from shared memory in 16-byte broadcast loads.  EDGE: the queries may lie before the key or past the end `S` of the
// sequence; the latter get plain zeros, whatever the products with the zero rows of Q and dO gave (K or V may hold
// infinities).
template <bool EDGE>
__device__ __forceinline__ void dkv_cols16(const uint32_t (&rs)[16], const uint32_t (&rp)[16], const float* lse2, const float* delta_s,
                                           int qa0, int key, int S, float sl2, float scale, uint32_t (&pp)[8], uint32_t (&pd)[8]) {
#pragma unroll
  for (int i = 0; i < 16; i += 4) {
    const float4 l = *reinterpret_cast<const float4*>(lse2 + i);
    const float4 e = *reinterpret_cast<const float4*>(delta_s + i);
    const float lv[4] = {l.x, l.y, l.z, l.w}, ev[4] = {e.x, e.y, e.z, e.w};
    float pr[4], dp[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      pr[k] = ex2_approx(fmaf(__uint_as_float(rs[i + k]), sl2, -lv[k]));
      dp[k] = __uint_as_float(rp[i + k]);
      if (EDGE) {
        const int q = qa0 + i + k;
        if (key > q || q >= S) pr[k] = 0.f;
        if (q >= S) dp[k] = 0.f;
      }
    }
    pp[i >> 1] = pack_bf16(pr[0], pr[1]);
    pp[(i >> 1) + 1] = pack_bf16(pr[2], pr[3]);
    pd[i >> 1] = pack_bf16(pr[0] * fmaf(dp[0], scale, -ev[0]), pr[1] * fmaf(dp[1], scale, -ev[1]));
    pd[(i >> 1) + 1] = pack_bf16(pr[2] * fmaf(dp[2], scale, -ev[2]), pr[3] * fmaf(dp[3], scale, -ev[3]));
  }
}

// =================================================================================================
// Backward, dK / dV: one CTA per 128 key rows; streams 64-row Q / dO sub-tiles with their statistics (copied to shared
// memory with the tiles: read from global memory where they are used, each first touch cost an L2 round trip inside the
// softmax chain).  The same scheme as the dQ kernel: two sets of eight warps take alternate sub-tiles, P^T and dS^T overwrite
// their own scores in TMEM and are the A operands of the accumulating products, head size 64 has three score buffers, and two
// warps issue, one the score products, one the accumulating ones.
// =================================================================================================
constexpr int KV_QSUB = 64;

template <int D>
struct DkvSmem {
  static constexpr int TILE = ATT_BM * D * 2;     // K or V tile
  static constexpr int QTILE = KV_QSUB * D * 2;   // Q or dO sub-tile
  static constexpr int K_OFF = 0;
  static constexpr int V_OFF = TILE;
  static constexpr int STAGES = D == 64 ? 6 : 4;               // Q / dO sub-tiles in flight
  static constexpr int Q_OFF = 2 * TILE;
  static constexpr int DO_OFF = 2 * TILE + STAGES * QTILE;
  static constexpr int STAT_OFF = 2 * TILE + 2 * STAGES * QTILE;  // per stage: 64 base-2 lse, then 64 scaled deltas
  static constexpr int STAT_BYTES = 2 * KV_QSUB * 4;
  static constexpr int BAR_OFF = STAT_OFF + STAGES * STAT_BYTES;
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;
};

template <int D>
__global__ void __launch_bounds__(ATT_THREADS, 1)
attn_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tm_kv, const __grid_constant__ CUtensorMap tm_q,
                    const __grid_constant__ CUtensorMap tm_do, AttnParams p) {
  using L = DkvSmem<D>;
  constexpr int SLABS = D / 64;
  constexpr uint32_t SLAB = ATT_BM * 128;    // [128 x 64] slab of K / V
  constexpr uint32_t QSLAB = KV_QSUB * 128;  // [64 x 64] slab of Q / dO
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  AttnBars* bars = reinterpret_cast<AttnBars*>(smem + L::BAR_OFF);
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;  // warp-uniform
  // Persistent: one CTA per SM walks the work items (one 128-row key tile of one head); small key tiles see the most
  // query sub-tiles and come first.  Every item has an even number of sub-tiles, so a set's sub-tiles are the even or the
  // odd ones of the running index as well.
  const int n_kt = p.S_pad / ATT_BM;
  const int HB = p.H * p.B;
  const int n_items = n_kt * HB;
  const int HD = p.H * D;
  // Score buffers: S^T 64 columns, dP^T the next 64.  Head size 64: three at 0, 128, 256, then dV and dK; head size 128:
  // two at 0 and 384, dV and dK between them.
  constexpr uint32_t TMEM_COLS = 512;
  constexpr int NBUF = D == 64 ? 3 : 2;
  constexpr uint32_t BUF_STEP = D == 64 ? 128 : 384;
  constexpr uint32_t DV_COL = D == 64 ? 384 : 128, DK_COL = D == 64 ? 448 : 256;

  if (threadIdx.x == 0) {
    attn_init_bars(bars);
    tma_prefetch_desc(&tm_kv);
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_do);
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, bars->tmem_slot, 0);

  if (warp == 0) {
    if (lane == 0) {
      uint32_t tt = 0, it = 0;  // sub-tiles / items so far
      bool ok = true;
      for (int item; ok && (item = snake_item(static_cast<int>(it))) < n_items; ++it) {
        const int kt = item / HB;
        const int hb = item % HB;
        const int h = hb % p.H, b = hb / p.H;
        const int krow0 = kt * ATT_BM;
        const int first_sub = kt * (ATT_BM / KV_QSUB);
        const int n_sub = p.S_pad / KV_QSUB - first_sub;
        if (!mbar_wait(&bars->stat_empty, (it & 1u) ^ 1u, abort_flag, 65)) { ok = false; break; }
        mbar_expect_tx(&bars->stat_full, 2 * L::TILE);
#pragma unroll
        for (int c = 0; c < SLABS; ++c) {
          tma_load_3d(smem + L::K_OFF + c * SLAB, &tm_kv, &bars->stat_full, HD + h * D + c * 64, krow0, b);
          tma_load_3d(smem + L::V_OFF + c * SLAB, &tm_kv, &bars->stat_full, 2 * HD + h * D + c * 64, krow0, b);
        }
        for (int t = 0; t < n_sub; ++t, ++tt) {
          const int st = tt % L::STAGES;
          if (!mbar_wait(&bars->str_empty[st], ((tt / L::STAGES) & 1u) ^ 1u, abort_flag, 66)) { ok = false; break; }
          const int qrow = (first_sub + t) * KV_QSUB;
          mbar_expect_tx(&bars->str_full[st], 2 * L::QTILE + L::STAT_BYTES);
          const float* delta_q = p.delta + (static_cast<size_t>(b) * p.H + h) * p.S_pad + qrow;  // 256-byte pieces, 256-byte aligned
          bulk_load_1d(smem + L::STAT_OFF + st * L::STAT_BYTES, delta_q + static_cast<size_t>(p.B) * p.H * p.S_pad, KV_QSUB * 4, &bars->str_full[st]);
          bulk_load_1d(smem + L::STAT_OFF + st * L::STAT_BYTES + KV_QSUB * 4, delta_q, KV_QSUB * 4, &bars->str_full[st]);
#pragma unroll
          for (int c = 0; c < SLABS; ++c) {
            tma_load_3d(smem + L::Q_OFF + st * L::QTILE + c * QSLAB, &tm_q, &bars->str_full[st], h * D + c * 64, qrow, b);
            tma_load_3d(smem + L::DO_OFF + st * L::QTILE + c * QSLAB, &tm_do, &bars->str_full[st], h * D + c * 64, qrow, b);
          }
        }
      }
    }
  } else if (warp == 1) {
    // Issuer of S^T(t) = K Q_t^T and dP^T(t) = V dO_t^T: the whole warp, see umma_f16_ss_warp.  Stages and buffers go round over
    // the sub-tiles of all items.
    const uint32_t idesc_s = make_idesc_f16(ATT_BM, KV_QSUB, true, false, false);
    const uint64_t dk = desc_kmajor(smem_u32(smem + L::K_OFF)), dv = desc_kmajor(smem_u32(smem + L::V_OFF));
    const uint64_t dq0 = desc_kmajor(smem_u32(smem + L::Q_OFF)), ddo0 = desc_kmajor(smem_u32(smem + L::DO_OFF));
    uint32_t st = 0, st_phase = 0, buf = 0, buf_phase = 0, it = 0;
    bool ok = true;
    for (int item; ok && (item = snake_item(static_cast<int>(it))) < n_items; ++it) {
      const int kt = item / HB;
      const int n_sub = p.S_pad / KV_QSUB - kt * (ATT_BM / KV_QSUB);
      if (it > 0 && !mbar_wait_warp(&bars->acc_issued, (it - 1u) & 1u, abort_flag, 75)) { ok = false; break; }
      if (!mbar_wait_warp(&bars->stat_full, it & 1u, abort_flag, 69)) { ok = false; break; }
      for (int t = 0; t < n_sub; ++t) {
        if (!mbar_wait_warp(&bars->str_full[st], st_phase, abort_flag, 67)) { ok = false; break; }
        if (!mbar_wait_warp(&bars->buf_free[buf], buf_phase ^ 1u, abort_flag, 68)) { ok = false; break; }
        tc_fence_after_sync();
        const uint64_t dq = desc_offset(dq0, st * L::QTILE), ddo = desc_offset(ddo0, st * L::QTILE);
        const uint32_t t_s = tmem_base + buf * BUF_STEP;
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
          umma_f16_ss_warp(t_s, desc_offset(dk, kstep_kmajor(ks, SLAB)), desc_offset(dq, kstep_kmajor(ks, QSLAB)), idesc_s, ks != 0);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
          umma_f16_ss_warp(t_s + 64, desc_offset(dv, kstep_kmajor(ks, SLAB)), desc_offset(ddo, kstep_kmajor(ks, QSLAB)), idesc_s, ks != 0);
        umma_commit_warp(&bars->s_full[buf]);
        if (t == n_sub - 1) umma_commit_warp(&bars->stat_empty);  // the item's last use of the K and V tiles
        if (++buf == NBUF) { buf = 0; buf_phase ^= 1u; }
        if (++st == L::STAGES) { st = 0; st_phase ^= 1u; }
      }
    }
  } else if (warp == ATT_ACC_WARP) {
    // Issuer of dV += P^T dO and dK += dS^T Q (A in TMEM, B MN-major)
    const uint32_t idesc_a = make_idesc_f16(ATT_BM, D, true, false, true);
    const uint64_t dqt0 = desc_mnmajor(smem_u32(smem + L::Q_OFF), QSLAB), ddot0 = desc_mnmajor(smem_u32(smem + L::DO_OFF), QSLAB);
    uint32_t st = 0, buf = 0, buf_phase = 0, it = 0;
    bool ok = true;
    for (int item; ok && (item = snake_item(static_cast<int>(it))) < n_items; ++it) {
      const int kt = item / HB;
      const int n_sub = p.S_pad / KV_QSUB - kt * (ATT_BM / KV_QSUB);
      // dK / dV still belong to the previous item until its threads have read them
      if (!mbar_wait_warp(&bars->acc_free, (it & 1u) ^ 1u, abort_flag, 70)) { ok = false; break; }
      for (int t = 0; t < n_sub; ++t) {
        if (!mbar_wait_warp(&bars->p_full[buf], buf_phase, abort_flag, 71)) { ok = false; break; }
        tc_fence_after_sync();
        const uint64_t dqt = desc_offset(dqt0, st * L::QTILE), ddot = desc_offset(ddot0, st * L::QTILE);
        const uint32_t t_s = tmem_base + buf * BUF_STEP;
#pragma unroll
        for (int ks = 0; ks < KV_QSUB / 16; ++ks)
          umma_f16_ts_warp(tmem_base + DV_COL, t_s + (ks >> 1) * 32 + (ks & 1) * 8, desc_offset(ddot, kstep_mnmajor(ks)), idesc_a, (t | ks) != 0);
#pragma unroll
        for (int ks = 0; ks < KV_QSUB / 16; ++ks)
          umma_f16_ts_warp(tmem_base + DK_COL, t_s + 64 + (ks >> 1) * 32 + (ks & 1) * 8, desc_offset(dqt, kstep_mnmajor(ks)), idesc_a, (t | ks) != 0);
        umma_commit_warp(&bars->buf_free[buf]);
        umma_commit_warp(&bars->str_empty[st]);
        if (t == n_sub - 1) {
          umma_commit_warp(&bars->acc_done);
          if (lane == 0) mbar_arrive(&bars->acc_issued);
        }
        if (++buf == NBUF) { buf = 0; buf_phase ^= 1u; }
        if (++st == L::STAGES) st = 0;
      }
    }
  } else {
    const int quad = warp & 3;
    const int grp = (warp - 2) >> 2;
    const int set = grp >> 1, half = grp & 1;  // which of two consecutive sub-tiles, which 32 of its 64 queries (and: dK or dV, which D/2 columns)
    const int row = quad * 32 + lane;          // key row inside the tile
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    // this thread's S^T columns in buffer 0, its dP^T at +64; P^T / dS^T overwrite the first 16 columns of each
    const uint32_t ts0 = tmem_base + half * 32 + lane_off;
    const float sl2 = p.scale * LOG2E;
    uint32_t tt0 = 0, it = 0;  // sub-tiles / items so far
    bool ok = true;
    for (int item; ok && (item = snake_item(static_cast<int>(it))) < n_items; ++it) {
      const int kt = item / HB;
      const int hb = item % HB;
      const int h = hb % p.H, b = hb / p.H;
      const int first_sub = kt * (ATT_BM / KV_QSUB);
      const int n_sub = p.S_pad / KV_QSUB - first_sub;
      const int key = kt * ATT_BM + row;  // this thread's key (sequence index)
      for (int t = set; t < n_sub; t += 2) {
        const uint32_t tt = tt0 + t, buf = tt % NBUF, ts = ts0 + buf * BUF_STEP;
        const int st = static_cast<int>(tt % L::STAGES);
        const int qa0 = (first_sub + t) * KV_QSUB + half * 32;  // first query (sequence index) of this thread
        const bool edge = t < ATT_BM / KV_QSUB || qa0 + 32 > p.S;  // may overlap the diagonal block or the sequence's end
        if (!mbar_wait(&bars->s_full[buf], (tt / NBUF) & 1u, abort_flag, 72)) { ok = false; break; }
        tc_fence_after_sync();
        // the statistics landed with the tile that S^T was made of: this wait does not block, it orders the reads behind the copy
        if (!mbar_wait(&bars->str_full[st], (tt / L::STAGES) & 1u, abort_flag, 73)) { ok = false; break; }
        const float* lse2 = reinterpret_cast<const float*>(smem + L::STAT_OFF + st * L::STAT_BYTES) + half * 32;
        const float* delta_s = lse2 + KV_QSUB;
        uint32_t rs0[16], rp0[16], rs1[16], rp1[16], pp[8], pd[8];
        tmem_ld_32x16(ts, rs0);
        tmem_ld_32x16(ts + 64, rp0);
        tmem_ld_32x16(ts + 16, rs1);
        tmem_ld_32x16(ts + 80, rp1);
        tmem_ld_wait();
        if (!edge) dkv_cols16<false>(rs0, rp0, lse2, delta_s, qa0, key, p.S, sl2, p.scale, pp, pd);
        else       dkv_cols16<true>(rs0, rp0, lse2, delta_s, qa0, key, p.S, sl2, p.scale, pp, pd);
        tmem_st_32x8(ts, pp);
        tmem_st_32x8(ts + 64, pd);
        if (!edge) dkv_cols16<false>(rs1, rp1, lse2 + 16, delta_s + 16, qa0 + 16, key, p.S, sl2, p.scale, pp, pd);
        else       dkv_cols16<true>(rs1, rp1, lse2 + 16, delta_s + 16, qa0 + 16, key, p.S, sl2, p.scale, pp, pd);
        tmem_st_32x8(ts + 8, pp);
        tmem_st_32x8(ts + 72, pd);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->p_full[buf]);
      }
      if (!ok) break;
      if (!mbar_wait(&bars->acc_done, it & 1u, abort_flag, 74)) { ok = false; break; }
      tc_fence_after_sync();
      // set 0: dK, set 1: dV
      const uint32_t tcol = tmem_base + (set == 0 ? DK_COL : DV_COL) + static_cast<uint32_t>(half * (D / 2)) + lane_off;
      __nv_bfloat16* drow = p.dqkv + (static_cast<size_t>(b) * p.S + key) * (3 * HD) + (set == 0 ? HD : 2 * HD) + h * D + half * (D / 2);
#pragma unroll 1
      for (int c = 0; c < D / 2; c += 16) {
        uint32_t r[16];
        tmem_ld_32x16(tcol + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          uint4 v;
          v.x = pack_bf16(__uint_as_float(r[q * 8 + 0]), __uint_as_float(r[q * 8 + 1]));
          v.y = pack_bf16(__uint_as_float(r[q * 8 + 2]), __uint_as_float(r[q * 8 + 3]));
          v.z = pack_bf16(__uint_as_float(r[q * 8 + 4]), __uint_as_float(r[q * 8 + 5]));
          v.w = pack_bf16(__uint_as_float(r[q * 8 + 6]), __uint_as_float(r[q * 8 + 7]));
          if (key < p.S) *reinterpret_cast<uint4*>(drow + c + q * 8) = v;
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->acc_free);
      tt0 += static_cast<uint32_t>(n_sub);
    }
  }
  attn_teardown(bars, warp, tmem_base, TMEM_COLS, p.status);
}

// delta[b, h, s] = scale * sum_d dO[b, s, h, d] * O[b, s, h, d].  A warp takes one token at a time; D / 8 lanes share one head
// (16 bytes per lane and tensor), 256 / D heads per step.  Bound by memory once the indices cost nothing: one division per
// token, in 32 bits (two 64-bit divisions per token and head took longer than the loads: 46 us for 16384 tokens of 16 x 128).
// Also writes the base-2 log-sum-exp right behind it, and fills the rows between S and S_pad (see AttnParams::delta).
__global__ void __launch_bounds__(256) attn_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o,
                                                         const float* __restrict__ lse, float* __restrict__ delta, float scale, int B,
                                                         int S, int S_pad, int H, int D) {
  const int lanes_per = D >> 3;             // 8 or 16
  const int lane = threadIdx.x & 31;
  const int sub = lane / lanes_per, sl = lane - sub * lanes_per;
  const int heads_per_step = 32 / lanes_per;
  const int tokens = B * S;
  const long long total_pad = static_cast<long long>(B) * S_pad * H;
  const int n_warps = static_cast<int>((gridDim.x * blockDim.x) >> 5);
  for (int tok = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5); tok < tokens; tok += n_warps) {
    const int bb = tok / S, ss = tok - bb * S;
    const long long row0 = static_cast<long long>(bb) * H;
    const __nv_bfloat16* po = o + static_cast<long long>(tok) * H * D + sl * 8;
    const __nv_bfloat16* pd = d_o + static_cast<long long>(tok) * H * D + sl * 8;
#pragma unroll 4
    for (int h0 = 0; h0 < H; h0 += heads_per_step) {
      const int h = h0 + sub;
      float acc = 0.f;
      if (h < H) {
        const Vec16<__nv_bfloat16> a = ld16(po + h * D), c = ld16(pd + h * D);
#pragma unroll
        for (int k = 0; k < 8; ++k) acc += __bfloat162float(a.v[k]) * __bfloat162float(c.v[k]);
      }
      for (int off = lanes_per >> 1; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
      if (sl == 0 && h < H) {
        const long long row = row0 + h;
        delta[row * S_pad + ss] = acc * scale;
        delta[total_pad + row * S_pad + ss] = lse[row * S + ss] * LOG2E;
      }
    }
  }
  const int pad = S_pad - S;  // < 128
  const long long n_pad = static_cast<long long>(B) * H * pad;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n_pad; i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long idx = (i / pad) * S_pad + S + i % pad;
    delta[idx] = 0.f;
    delta[total_pad + idx] = INFINITY;
  }
}

}  // namespace fsb

// ------------------------------------------------------------------------------------------------
// C ABI.  Any S >= 1, D in {64, 128}; all tensors contiguous, 16-byte aligned.
// ------------------------------------------------------------------------------------------------
template <typename K>
static int set_smem(K kernel, int bytes) {
  return static_cast<int>(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
}
// Each CTA allocates all 512 TMEM columns, so two CTAs must never share an SM: ask for more than half of the
// SM's shared memory even when the tiles need less (D = 64).
static constexpr int kMinSmem = 120 * 1024;
static inline int one_cta_smem(int bytes) { return bytes < kMinSmem ? kMinSmem : bytes; }

FSB_API int fsb_attn_fwd_pingpong(const void* qkv, void* o, float* lse, int B, int S, int H, int D, float scale, int* status,
                                  cudaStream_t stream);

// Debug aid: copies (and clears) the bit set of wait sites that were blocked when an attention kernel aborted.
FSB_API int fsb_attn_wait_sites(unsigned int* out8) {
  unsigned int zero[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  cudaError_t e = cudaMemcpyFromSymbol(out8, fsb::g_blocked_wait_sites, sizeof(zero));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(fsb::g_blocked_wait_sites, zero, sizeof(zero));
  return static_cast<int>(e);
}

FSB_API int fsb_last_tensor_map_result() { return fsb_host::last_encode_result(); }

// Forward (attention_fwd_pingpong.cu): any S >= 1.
FSB_API int fsb_attn_fwd(const void* qkv, void* o, float* lse, int B, int S, int H, int D, float scale, int* status,
                         cudaStream_t stream) {
  return fsb_attn_fwd_pingpong(qkv, o, lse, B, S, H, D, scale, status, stream);
}

// dqkv receives dQ, dK and dV in the packed layout of qkv.  delta: fp32 workspace [2, B, H, S rounded up to 128].
FSB_API int fsb_attn_bwd(const void* qkv, const void* o, const void* d_o, const float* lse, float* delta, void* dqkv, int B, int S,
                         int H, int D, float scale, int* status, cudaStream_t stream) {
  using namespace fsb;
  if (B < 1 || S < 1 || H < 1 || (D != 64 && D != 128) || static_cast<long long>(B) * S > 0x7fffffffll) return -1;
  const int S_pad = (S + ATT_BM - 1) / ATT_BM * ATT_BM;
  // (columns, positions, batch): a tile that overhangs the sequence reads zeros
  const uint64_t w_qkv = (uint64_t)3 * H * D, w_o = (uint64_t)H * D;
  CUtensorMap tm_qkv128, tm_do128, tm_qkv64, tm_do64;
  if (!fsb_host::encode_3d_16bit(&tm_qkv128, qkv, w_qkv, S, B, w_qkv, w_qkv * S, 64, ATT_BM, 1)) return -2;
  if (!fsb_host::encode_3d_16bit(&tm_do128, d_o, w_o, S, B, w_o, w_o * S, 64, ATT_BM, 1)) return -3;
  if (!fsb_host::encode_3d_16bit(&tm_qkv64, qkv, w_qkv, S, B, w_qkv, w_qkv * S, 64, KV_QSUB, 1)) return -4;
  if (!fsb_host::encode_3d_16bit(&tm_do64, d_o, w_o, S, B, w_o, w_o * S, 64, KV_QSUB, 1)) return -5;
  AttnParams p{};
  p.B = B; p.S = S; p.S_pad = S_pad; p.H = H; p.D = D; p.scale = scale;
  p.delta = delta; p.dqkv = static_cast<__nv_bfloat16*>(dqkv); p.status = status;
  {
    const int threads = 256;
    long long blocks = (static_cast<long long>(B) * S + threads / 32 - 1) / (threads / 32);  // one token per warp at most ...
    if (blocks > 148 * 8) blocks = 148 * 8;                                                  // ... but no more CTAs than fill every SM
    attn_delta_kernel<<<static_cast<unsigned>(blocks), threads, 0, stream>>>(static_cast<const __nv_bfloat16*>(o),
                                                                             static_cast<const __nv_bfloat16*>(d_o), lse, delta, scale, B, S, S_pad, H, D);
  }
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int n_items = (S_pad / ATT_BM) * H * B;
  const dim3 grid(n_items < sms ? n_items : sms);  // persistent: one CTA per SM walks the work items
  if (D == 128) {
    set_smem(attn_bwd_dq_kernel<128>, DqSmem<128>::TOTAL);
    set_smem(attn_bwd_dkv_kernel<128>, DkvSmem<128>::TOTAL);
    attn_bwd_dkv_kernel<128><<<grid, ATT_THREADS, DkvSmem<128>::TOTAL, stream>>>(tm_qkv128, tm_qkv64, tm_do64, p);
    attn_bwd_dq_kernel<128><<<grid, ATT_THREADS, DqSmem<128>::TOTAL, stream>>>(tm_qkv128, tm_do128, p);
  } else {
    set_smem(attn_bwd_dq_kernel<64>, one_cta_smem(DqSmem<64>::TOTAL));
    set_smem(attn_bwd_dkv_kernel<64>, one_cta_smem(DkvSmem<64>::TOTAL));
    attn_bwd_dkv_kernel<64><<<grid, ATT_THREADS, one_cta_smem(DkvSmem<64>::TOTAL), stream>>>(tm_qkv128, tm_qkv64, tm_do64, p);
    attn_bwd_dq_kernel<64><<<grid, ATT_THREADS, one_cta_smem(DqSmem<64>::TOTAL), stream>>>(tm_qkv128, tm_do128, p);
  }
  return static_cast<int>(cudaGetLastError());
}
