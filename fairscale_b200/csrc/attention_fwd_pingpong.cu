// Causal flash-attention forward with two query tiles per CTA in ping-pong and the probabilities kept in TMEM.
//
//   qkv : bf16 [B, S, 3, H, D] (packed, read by TMA)      o : bf16 [B, S, H, D]      lse : fp32 [B, H, S]
//
// One CTA owns 256 query rows as two 128-row tiles A and B.  The tensor cores alternate between the tiles, so the
// softmax of one tile runs while the products of the other are in flight:
//
//   tensor pipe :  S_A(j)  S_B(j) | PV_A(j-1) S_A(j) ... ->  PV_A(j)  S_A(j+1)  PV_B(j)  S_B(j+1)  PV_A(j+1) ...
//   softmax A   :          [ softmax A(j) ............ ]              [ softmax A(j+1) ............ ]
//   softmax B   :                    [ softmax B(j) ............ ]              [ softmax B(j+1) ..... ]
//
// Roles (608 threads): warp 0 TMA producer, warp 1 MMA issuer and TMEM owner, warps 2-9 softmax of tile A, warps 10-17
// softmax of tile B, warp 18 MMA issuer of tile B with head size 64 (below).  Two threads share a query row (TMEM lane), 64 of a
// step's 128 keys each: they read their scores once and keep them in registers, pass each other the row maximum and their sums
// through shared memory, and with four warps per scheduler one warp's loads and waits hide behind the exponentials of others.
// (One thread per row read the scores twice, once for the maximum, and left the exponential unit, which bounds head size 64, idle
// 46 % of the time.  Against that, and with an issuer for each tile: B2 S8192 H16 D64 428 -> 395 us, B8 S1024 H16 D64 53.3 -> 45.1,
// B16 S512 H16 D64 41.7 -> 32.6; head size 128, where the products bound the step, 47.1 -> 45.3 us at B2 S2048 H16.  The output and
// the normaliser are to the bit those of one thread per row: a running sum for each thread would take 383 us at B2 S8192 H16 D64,
// and make the result depend on how a row is divided.)
// TMEM (512 columns): S_A [0,128)  S_B [128,256)  O_A [256,256+D)  O_B [384,384+D).  With head size 128 the bf16 probabilities overwrite
// the first 64 columns of their own score tile (two values per 32-bit column) and feed P V as the TMEM A operand of
// tcgen05.mma, so they never pass through shared memory.  The tensor pipe executes in issue order: S_t(j+1) is issued
// after PV_t(j) and therefore cannot overwrite P_t(j) early.
// Tile A skips the last key tile of the item (it lies wholly above A's diagonal).  Every mbarrier wait is bounded.
//
// Head size 64 leaves 128 TMEM columns free, and the probabilities get them (P_A [384,448)  P_B [448,512), O_B [320,384)).
// Then S_t(j+1) need not wait for PV_t(j): it is issued as soon as the softmax warps have read the scores of step j, before
// their exponentials, and is ready when they come back for it:
//
//   tensor pipe :  S_A(j+1)  S_B(j+1)  PV_A(j)  PV_B(j)  S_A(j+2) ...
//
// (In place, the chain exponentials -> PV -> S -> maximum kept the exponential unit, which bounds this head size, at 57 %.)  Each
// tile has an issuer of its own: one for both held up the products of one tile behind its waits for the other (B16 S512 H16 D64
// 44 -> 33 us together with the two threads a row).  With head size 128, in place and bound by the products, strict turns are the
// faster order (B8 S2048 H16 D128 168 us, 177 with two issuers).
//
// Any sequence length: the tensor map is three-dimensional (columns, positions, batch), so a tile that overhangs the
// sequence reads zeros instead of the next sequence's rows; keys past the end lie above every real query's diagonal and
// are masked with it; rows past the end are computed and not stored.  An item whose second query tile would lie wholly
// past the end runs its first tile alone.  (torch's operator, which such lengths went through before, has the faster
// forward but needs the packed tensor permuted and the gradients concatenated: B4 S1543 H16 D128 forward + backward 553 us there,
// 296 us here.  ops/attention.py says which lengths come here.)
//
// The kernel is persistent: one CTA per SM walks a list of work items (256 query rows of one head), longest rows first,
// dealt forwards and backwards in turn (snake_item; B2 S8192 H16 D64: 508 -> 471 us against plain round-robin).  TMEM,
// barriers and the K / V ring live for the whole kernel, and the next item's query tiles are loaded as soon as the last
// Q K^T products of the current item have completed, i.e. during its final softmax and output write.  (With one CTA per
// item an SM sat idle for 7-10 us between consecutive CTAs - launch, 197 KB of shared memory, TMEM allocation - which was
// a third of the kernel's run time.)
//
// Replaces nn.MultiheadAttention / bmm+softmax in the reference's models
// (benchmarks/models/transformer_lm.py:107,150-152,169-183).

#include "sm100.cuh"

#include <cfloat>

namespace fsb {
namespace pp {

constexpr int THREADS = 608;
constexpr int BM = 128;          // rows of a query tile == TMEM lanes
constexpr int BN = 128;          // keys per step
constexpr float LOG2E = 1.4426950408889634f;
constexpr float LN2 = 0.6931471805599453f;

struct Params {
  int B, S, H, D;
  float scale;
  __nv_bfloat16* o;
  float* lse;
  int* status;
};

struct Bars {
  uint64_t q_full;
  uint64_t k_full[2], k_empty[2];  // empty: a commit of every issuer
  uint64_t v_full[2], v_empty[2];
  uint64_t s_full[2];   // per query tile: scores of the current step are in TMEM
  uint64_t p_full[2];   // per query tile: probabilities written (8 warp arrivals)
  uint64_t o_done[2];   // per query tile: P V of the current step has completed
  uint64_t s_read[2];   // per query tile, head size 64: the softmax warps hold all scores of the step (8 warp arrivals)
  uint64_t q_empty;     // the item's last Q K^T products of either tile have completed: the query tiles may be replaced
  uint64_t o_free[2];   // per query tile: the softmax warps have read the item's output accumulator (8 warp arrivals)
  uint64_t pair[2][4];  // per query tile and lane quadrant: both warps of the rows have left a value for each other (2 warp arrivals)
  uint32_t tmem_slot;
  int abort_flag;
};
static_assert(sizeof(Bars) <= 512, "the values that the threads of a row exchange start behind the barriers (Smem::XCH_OFF)");

template <int D>
struct Smem {
  static constexpr int TILE = BM * D * 2;
  static constexpr int Q_OFF = 0;            // two query tiles
  static constexpr int K_OFF = 2 * TILE;     // two stages
  static constexpr int V_OFF = 4 * TILE;     // two stages
  static constexpr int BAR_OFF = 6 * TILE;
  static constexpr int XCH_OFF = BAR_OFF + 512;  // [2 parities][2 tiles][2 halves][3][BM] values passed between the two threads of a row
  static constexpr int TOTAL = XCH_OFF + 2 * 2 * 2 * 3 * BM * 4 + 1024;
};

__device__ __forceinline__ void st_shared_f32(uint32_t addr, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }
__device__ __forceinline__ float ld_shared_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float ex2_approx(float x) {
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
// Operand descriptors: K-major [rows x 64] slabs of `slab_bytes`, k-step ks covers 16 elements (32 bytes inside the swizzle
// row); MN-major the same bytes read as [k_rows x 64] slabs, k-step ks covers 16 k_rows = 2048 bytes.
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t base) { return make_smem_desc(base, 16u, 1024u); }
__device__ __forceinline__ uint64_t desc_mnmajor(uint32_t base, uint32_t slab_bytes) { return make_smem_desc(base, slab_bytes, 1024u); }
__device__ __forceinline__ constexpr uint32_t kstep_kmajor(int ks, uint32_t slab_bytes) {
  return static_cast<uint32_t>(ks >> 2) * slab_bytes + static_cast<uint32_t>(ks & 3) * 32u;
}
__device__ __forceinline__ constexpr uint32_t kstep_mnmajor(int ks) { return static_cast<uint32_t>(ks) * 2048u; }

// Largest of 32 scores of a row and `m`; DIAG: of those of keys col0 + i <= row only.
template <bool DIAG>
__device__ __forceinline__ float chunk_max(const uint32_t (&r)[32], int col0, int row, float m) {
  float a[4] = {m, m, m, m};
#pragma unroll
  for (int i = 0; i < 32; i += 2) {
    float x = __uint_as_float(r[i]), y = __uint_as_float(r[i + 1]);
    if (DIAG) {
      if (col0 + i > row) x = m;
      if (col0 + i + 1 > row) y = m;
    }
    a[(i >> 1) & 3] = fmaxf(fmaxf(a[(i >> 1) & 3], x), y);
  }
  return fmaxf(fmaxf(a[0], a[1]), fmaxf(a[2], a[3]));
}

// Probabilities of 32 scores, packed to bf16; returns their sum: pairs of keys into four partial sums in turn.  (Packed additions
// would be half as many, but take their operands from neighbouring registers, where the conversion to bf16 wants other
// neighbours: B2 S8192 H16 D64 401 us, 412 with them, B4 S1543 H16 D128 67.7 us, 71.5.)
template <bool DIAG>
__device__ __forceinline__ float chunk_exp(const uint32_t (&r)[32], int col0, int row, uint64_t sl2, uint64_t neg_mb, uint32_t (&pk)[16]) {
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 0; i < 32; i += 2) {
    float x, y;
    unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), sl2, neg_mb), x, y);
    float p0 = ex2_approx(x), p1 = ex2_approx(y);
    if (DIAG) {
      if (col0 + i > row) p0 = 0.f;
      if (col0 + i + 1 > row) p1 = 0.f;
    }
    acc[(i >> 1) & 3] += p0 + p1;
    pk[i >> 1] = pack_bf16(p0, p1);
  }
  return (acc[0] + acc[1]) + (acc[2] + acc[3]);
}

template <int D>
__global__ void __launch_bounds__(THREADS, 1)
attn_fwd_pingpong_kernel(const __grid_constant__ CUtensorMap tm_qkv, Params p) {
  using L = Smem<D>;
  constexpr int SLABS = D / 64;
  constexpr uint32_t SLAB = BM * 128;  // bytes of a [128 x 64] bf16 slab
  constexpr uint32_t TMEM_COLS = 512;
  constexpr bool SEP = D == 64;                    // probabilities in columns of their own
  constexpr uint32_t O_COL = 256, O_STEP = SEP ? 64 : 128;
  constexpr uint32_t P_COL = SEP ? 384 : 0, P_STEP = SEP ? 64 : 128;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Bars* bars = reinterpret_cast<Bars*>(smem + L::BAR_OFF);
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;  // warp-uniform
  // Work items (256 query rows of one head) ordered longest first and dealt to the persistent CTAs by snake_item: every
  // role of the CTA walks the same list.  item -> (q2, h, b): all heads of the longest rows come first.
  const int n_tiles = (p.S + BM - 1) / BM;  // 128-row tiles with at least one real row
  const int n_q2 = (n_tiles + 1) / 2;
  const int HB = p.H * p.B;
  const int n_items = n_q2 * HB;
  const int HD = p.H * D;

  if (threadIdx.x == 0) {
    mbar_init(&bars->q_full, 1);
    constexpr int ISSUERS = SEP ? 2 : 1;
    mbar_init(&bars->q_empty, ISSUERS);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->k_full[i], 1);
      mbar_init(&bars->k_empty[i], ISSUERS);
      mbar_init(&bars->v_full[i], 1);
      mbar_init(&bars->v_empty[i], ISSUERS);
      mbar_init(&bars->s_full[i], 1);
      mbar_init(&bars->p_full[i], 8);
      mbar_init(&bars->o_done[i], 1);
      mbar_init(&bars->o_free[i], 8);
      mbar_init(&bars->s_read[i], 8);
      for (int q = 0; q < 4; ++q) mbar_init(&bars->pair[i][q], 2);
    }
    bars->abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tm_qkv);
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
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      uint32_t kt = 0;  // key tiles loaded so far (selects the K / V stage and its phase)
      uint32_t it = 0;  // items started so far
      bool ok = true;
      for (int item; ok && (item = snake_item(static_cast<int>(it))) < n_items; ++it) {
        const int q2 = n_q2 - 1 - item / HB;
        const int hb = item % HB;
        const int h = hb % p.H, b = hb / p.H;
        const int n_q = 2 * q2 + 1 < n_tiles ? 2 : 1;  // query tiles of the item
        const int n_kv = 2 * q2 + n_q;
        const int row0 = q2 * 2 * BM;
        // the query tiles of the previous item are free once its last Q K^T products have completed
        if (!mbar_wait(&bars->q_empty, (it & 1u) ^ 1u, abort_flag)) { ok = false; break; }
        mbar_expect_tx(&bars->q_full, n_q * L::TILE);
        for (int t = 0; t < n_q; ++t)
#pragma unroll
          for (int c = 0; c < SLABS; ++c)
            tma_load_3d(smem + L::Q_OFF + t * L::TILE + c * SLAB, &tm_qkv, &bars->q_full, h * D + c * 64, row0 + t * BM, b);
        for (int j = 0; j < n_kv; ++j, ++kt) {
          const int st = kt & 1;
          const uint32_t par = ((kt >> 1) & 1u) ^ 1u;
          const int krow = j * BN;
          if (!mbar_wait(&bars->k_empty[st], par, abort_flag)) { ok = false; break; }
          mbar_expect_tx(&bars->k_full[st], L::TILE);
#pragma unroll
          for (int c = 0; c < SLABS; ++c)
            tma_load_3d(smem + L::K_OFF + st * L::TILE + c * SLAB, &tm_qkv, &bars->k_full[st], HD + h * D + c * 64, krow, b);
          if (!mbar_wait(&bars->v_empty[st], par, abort_flag)) { ok = false; break; }
          mbar_expect_tx(&bars->v_full[st], L::TILE);
#pragma unroll
          for (int c = 0; c < SLABS; ++c)
            tma_load_3d(smem + L::V_OFF + st * L::TILE + c * SLAB, &tm_qkv, &bars->v_full[st], 2 * HD + h * D + c * 64, krow, b);
        }
      }
    }
  } else if (warp == 1 || warp == 18) {
    // ------------------------------------------------------------------ MMA issuers (whole warps, see umma_f16_ss_warp)
    const uint32_t idesc_s = make_idesc_f16(BM, BN, true, false, false);  // Q K^T: both K-major
    const uint32_t idesc_o = make_idesc_f16(BM, D, true, false, true);    // P V: P from TMEM, V MN-major
    const uint64_t dq0 = desc_kmajor(smem_u32(smem + L::Q_OFF)), dk0 = desc_kmajor(smem_u32(smem + L::K_OFF));
    const uint64_t dv0 = desc_mnmajor(smem_u32(smem + L::V_OFF), SLAB);
    uint32_t kt0 = 0;           // key tiles of earlier items
    // Counted per query tile this warp issues for (i_of), over all items:
    uint32_t cs[2] = {0, 0};    // steps (phase of p_full)
    uint32_t ss[2] = {0, 0};    // score products (phase of s_read)
    uint32_t its[2] = {0, 0};   // items with that tile (phase of o_free)
    auto i_of = [](int t) { return SEP ? 0 : t; };
    uint32_t it = 0;
    bool ok = true;
    auto issue_s = [&](int t, uint32_t kt) -> bool {
      const int st = kt & 1;
      if (!mbar_wait_warp(&bars->k_full[st], (kt >> 1) & 1u, abort_flag)) return false;
      if (SEP && ss[i_of(t)] > 0 && !mbar_wait_warp(&bars->s_read[t], (ss[i_of(t)] - 1u) & 1u, abort_flag)) return false;
      ++ss[i_of(t)];
      tc_fence_after_sync();
      const uint64_t dq = desc_offset(dq0, t * L::TILE), dk = desc_offset(dk0, st * L::TILE);
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks)
        umma_f16_ss_warp(tmem_base + t * 128, desc_offset(dq, kstep_kmajor(ks, SLAB)), desc_offset(dk, kstep_kmajor(ks, SLAB)), idesc_s, ks != 0);
      umma_commit_warp(&bars->s_full[t]);
      return true;
    };
    auto issue_pv = [&](int t, uint32_t kt, bool first) -> bool {
      // the output accumulator still belongs to the previous item until its softmax warps have read it
      if (first && !mbar_wait_warp(&bars->o_free[t], (its[i_of(t)] & 1u) ^ 1u, abort_flag)) return false;
      if (!mbar_wait_warp(&bars->p_full[t], cs[i_of(t)] & 1u, abort_flag)) return false;
      tc_fence_after_sync();
      const uint64_t dv = desc_offset(dv0, (kt & 1) * L::TILE);
#pragma unroll
      for (int ks = 0; ks < BN / 16; ++ks)
        umma_f16_ts_warp(tmem_base + O_COL + t * O_STEP, tmem_base + P_COL + t * P_STEP + ks * 8, desc_offset(dv, kstep_mnmajor(ks)), idesc_o,
                         (!first || ks != 0) ? 1u : 0u);
      umma_commit_warp(&bars->o_done[t]);
      ++cs[i_of(t)];
      return true;
    };
    auto wait_k = [&](uint32_t kt) -> bool { return mbar_wait_warp(&bars->k_full[kt & 1], (kt >> 1) & 1u, abort_flag); };
    auto wait_v = [&](uint32_t kt) -> bool { return mbar_wait_warp(&bars->v_full[kt & 1], (kt >> 1) & 1u, abort_flag); };
    for (int item; ok && (item = snake_item(static_cast<int>(it))) < n_items; ++it) {
      const int q2 = n_q2 - 1 - item / HB;
      const bool has_b = 2 * q2 + 1 < n_tiles;
      const int n_a = 2 * q2 + 1;               // key tiles seen by tile A; tile B sees one more
      const int n_kv = has_b ? n_a + 1 : n_a;
      if (SEP) {
        // an issuer for each tile: neither is held up behind its waits for the other
        const int t = warp == 1 ? 0 : 1;
        const int n_own = t == 0 ? n_a : (has_b ? n_kv : 0);
        if (!mbar_wait_warp(&bars->q_full, it & 1u, abort_flag)) { ok = false; break; }
        for (int j = -1; j < n_own && ok && n_own > 0; ++j) {
          const uint32_t kt = kt0 + j;
          if (j + 1 < n_own) {  // the next step's scores first: they wait for reads that come before the exponentials of this one
            if (!issue_s(t, kt + 1)) { ok = false; break; }
            umma_commit_warp(&bars->k_empty[(kt + 1) & 1]);
            if (j + 2 == n_own) umma_commit_warp(&bars->q_empty);  // that was the tile's last use of its queries
          }
          if (j >= 0) {
            if (!wait_v(kt) || !issue_pv(t, kt, j == 0)) { ok = false; break; }
            umma_commit_warp(&bars->v_empty[kt & 1]);
          }
        }
        if (ok && n_own == 0) umma_commit_warp(&bars->q_empty);
        its[0] += n_own > 0 ? 1u : 0u;
        // key tiles that only the other query tile sees pass by (once they have landed: until then an earlier phase may be open)
        for (int j = n_own; j < n_kv && ok; ++j) {
          const uint32_t kt = kt0 + j;
          if (!wait_k(kt)) { ok = false; break; }
          umma_commit_warp(&bars->k_empty[kt & 1]);
          if (!wait_v(kt)) { ok = false; break; }
          umma_commit_warp(&bars->v_empty[kt & 1]);
        }
      } else {
        // one issuer: the products of the two tiles in turn
        if (warp != 1) break;
        if (!mbar_wait_warp(&bars->q_full, it & 1u, abort_flag)) { ok = false; break; }
        ok = issue_s(0, kt0);
        if (ok && has_b) ok = issue_s(1, kt0);
        if (ok) umma_commit_warp(&bars->k_empty[kt0 & 1]);
        if (ok && n_kv == 1) umma_commit_warp(&bars->q_empty);
        for (int j = 0; j < n_kv && ok; ++j) {
          const uint32_t kt = kt0 + j;
          if (!wait_v(kt)) { ok = false; break; }
          if (j < n_a) {
            if (!issue_pv(0, kt, j == 0)) { ok = false; break; }
            if (j + 1 < n_a && !issue_s(0, kt + 1)) { ok = false; break; }
          }
          if (has_b && !issue_pv(1, kt, j == 0)) { ok = false; break; }
          umma_commit_warp(&bars->v_empty[kt & 1]);
          if (j + 1 < n_kv) {
            if (has_b && !issue_s(1, kt + 1)) { ok = false; break; }
            umma_commit_warp(&bars->k_empty[(kt + 1) & 1]);
            if (j + 2 == n_kv) umma_commit_warp(&bars->q_empty);  // that was the item's last use of the query tiles
          }
        }
        ++its[0];
        its[1] += has_b ? 1u : 0u;
      }
      kt0 += n_kv;
    }
  } else {
    // ------------------------------------------------------------------ softmax warps: two threads per query row
    const int t = (warp - 2) >> 3;           // query tile
    const int half = ((warp - 2) >> 2) & 1;  // which 64 of a step's 128 keys, which D / 2 output columns
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t ts = tmem_base + t * 128 + half * 64 + lane_off;                  // this thread's scores
    const uint32_t tp = tmem_base + P_COL + t * P_STEP + half * 32 + lane_off;        // its probabilities (in columns [0, 64) of the tile's scores unless SEP)
    const uint32_t to = tmem_base + O_COL + t * O_STEP + half * (D / 2) + lane_off;  // its output columns
    const int col0 = half * 64;
    const uint32_t xch = smem_u32(smem + L::XCH_OFF) + (t * 6 * BM + row) * 4;  // + parity * XCH_PARITY + half * XCH_HALF + value * 4 BM
    constexpr uint32_t XCH_PARITY = 12 * BM * 4, XCH_HALF = 3 * BM * 4;
    uint64_t* const pair_bar = &bars->pair[t][quad];
    uint32_t xs = 0;  // exchanges so far (parity of the buffer, phase of pair_bar)
    // What the two threads of a row pass each other at a step: their maxima, and the sums of their probabilities of the step before
    // (leave_sum, per 32 keys).  Both then add up the row in the order of its keys: the four sums of a step one after the other,
    // then on to the running sum.  (With a running sum for each thread the result would depend on how a row is divided.)  The
    // buffers alternate: a thread writes one again only after the partner has arrived at the exchange in between, i.e. has read it.
    auto leave_sum = [&](int k, float v) { st_shared_f32(xch + (xs & 1u) * XCH_PARITY + half * XCH_HALF + (1 + k) * 4 * BM, v); };  // for the next exchange
    auto exchange = [&](float mx, float& other) -> bool {
      const uint32_t x = xch + (xs & 1u) * XCH_PARITY;
      st_shared_f32(x + half * XCH_HALF, mx);
      __syncwarp();
      if (lane == 0) mbar_arrive(pair_bar);
      if (!mbar_wait(pair_bar, xs & 1u, abort_flag)) return false;
      other = ld_shared_f32(x + (half ^ 1) * XCH_HALF);
      ++xs;
      return true;
    };
    auto sums = [&]() -> float {  // of the row at the step before, after this step's exchange and before the next
      const uint32_t x = xch + ((xs & 1u) ^ 1u) * XCH_PARITY;
      return ((ld_shared_f32(x + 4 * BM) + ld_shared_f32(x + 8 * BM)) + ld_shared_f32(x + XCH_HALF + 4 * BM)) + ld_shared_f32(x + XCH_HALF + 8 * BM);
    };
    const float sl2 = p.scale * LOG2E;
    const uint64_t sl2x2 = pack_f32x2(sl2, sl2);
    // The running maximum starts at the lowest value that stays finite when scaled, not at -inf: a row whose keys so far all
    // score -inf then has probabilities 2^(-inf) = 0, where -inf - -inf would be NaN.
    const float m_low = sl2 > 1.f ? -FLT_MAX / sl2 : -FLT_MAX;
    uint32_t cs = 0;  // steps of this tile so far, over all items (phase of s_full / o_done)
    bool ok = true;
    for (int r = 0, item; ok && (item = snake_item(r)) < n_items; ++r) {
      const int q2 = n_q2 - 1 - item / HB;
      const int hb = item % HB;
      const int h = hb % p.H, b = hb / p.H;
      if (2 * q2 + t >= n_tiles) continue;  // the item has no second query tile
      const int n_it = 2 * q2 + 1 + t;
      const int pos = q2 * 2 * BM + t * BM + row;  // this thread's position in the sequence
      const bool row_ok = pos < p.S;
      float m_run = m_low, mo;
      float l_run = 0.f, alpha_run = 0.f;  // sum of the row up to the step before, scaling of that step
      for (int j = 0; j < n_it && ok; ++j, ++cs) {
        if (!mbar_wait(&bars->s_full[t], cs & 1u, abort_flag)) { ok = false; break; }
        tc_fence_after_sync();
        const bool diag = (j == n_it - 1);
        uint32_t r0[32], r1[32];
        tmem_ld_32x32(ts, r0);
        tmem_ld_32x32(ts + 32, r1);
        tmem_ld_wait();
        if (SEP) {  // all scores of the step are in registers: the next products may overwrite them
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->s_read[t]);
        }
        float mx = -INFINITY;
        if (!diag) { mx = chunk_max<false>(r0, col0, row, mx); mx = chunk_max<false>(r1, col0 + 32, row, mx); }
        else       { mx = chunk_max<true>(r0, col0, row, mx);  mx = chunk_max<true>(r1, col0 + 32, row, mx); }
        // (in place, the exchange also keeps this thread's probabilities behind the partner's reads of the same columns)
        tc_fence_before_sync();
        if (!exchange(mx, mo)) { ok = false; break; }
        tc_fence_after_sync();
        // keep the old maximum while the new one is at most 2^8 above it: no rescaling of O, values stay in range
        float m_new = fmaxf(m_run, fmaxf(mx, mo));
        if (j > 0 && (m_new - m_run) * sl2 <= 8.f) m_new = m_run;
        const float alpha = j == 0 ? 0.f : ex2_approx((m_run - m_new) * sl2);
        const float mb = m_new * sl2;
        const uint64_t neg_mb = pack_f32x2(-mb, -mb);
        uint32_t pk[16];
        const float c0 = !diag ? chunk_exp<false>(r0, col0, row, sl2x2, neg_mb, pk) : chunk_exp<true>(r0, col0, row, sl2x2, neg_mb, pk);
        const bool rescale = j > 0 && __any_sync(0xffffffffu, alpha != 1.f);
        if (j > 0 && (SEP || rescale)) {
          // O_t (and P_t, where it has columns of its own) belongs to P V of step j-1 until that has completed; in place it
          // has, because S_t(j) was issued behind it
          if (!mbar_wait(&bars->o_done[t], (cs - 1u) & 1u, abort_flag)) { ok = false; break; }
          tc_fence_after_sync();
        }
        tmem_st_32x16(tp, pk);
        const float c1 = !diag ? chunk_exp<false>(r1, col0 + 32, row, sl2x2, neg_mb, pk) : chunk_exp<true>(r1, col0 + 32, row, sl2x2, neg_mb, pk);
        tmem_st_32x16(tp + 16, pk);
        if (rescale) {
#pragma unroll 1
          for (int c = 0; c < D / 64; ++c) {
            uint32_t o[32];
            tmem_ld_32x32(to + c * 32, o);
            tmem_ld_wait();
            uint32_t lo[16], hi[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              lo[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
              hi[i] = __float_as_uint(__uint_as_float(o[16 + i]) * alpha);
            }
            tmem_st_32x16(to + c * 32, lo);
            tmem_st_32x16(to + c * 32 + 16, hi);
          }
        }
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->p_full[t]);
        // the sums have time: the products wait for nothing below
        leave_sum(0, c0);
        leave_sum(1, c1);
        if (j > 0) l_run = l_run * alpha_run + sums();
        m_run = m_new;
        alpha_run = alpha;
      }
      if (!ok) break;
      // epilogue of the item: normalise and store this thread's half of the output row, then hand the accumulator back
      if (!exchange(0.f, mo)) { ok = false; break; }
      l_run = l_run * alpha_run + sums();
      if (!mbar_wait(&bars->o_done[t], (cs - 1u) & 1u, abort_flag)) { ok = false; break; }
      tc_fence_after_sync();
      const float inv = 1.f / l_run;
      __nv_bfloat16* orow = p.o + (static_cast<size_t>(b) * p.S + pos) * HD + h * D + half * (D / 2);
#pragma unroll 1
      for (int c = 0; c < D / 64; ++c) {
        uint32_t o[32];
        tmem_ld_32x32(to + c * 32, o);
        tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint4 v;
          v.x = pack_bf16(__uint_as_float(o[q * 8 + 0]) * inv, __uint_as_float(o[q * 8 + 1]) * inv);
          v.y = pack_bf16(__uint_as_float(o[q * 8 + 2]) * inv, __uint_as_float(o[q * 8 + 3]) * inv);
          v.z = pack_bf16(__uint_as_float(o[q * 8 + 4]) * inv, __uint_as_float(o[q * 8 + 5]) * inv);
          v.w = pack_bf16(__uint_as_float(o[q * 8 + 6]) * inv, __uint_as_float(o[q * 8 + 7]) * inv);
          if (row_ok) *reinterpret_cast<uint4*>(orow + c * 32 + q * 8) = v;
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->o_free[t]);
      if (half == 0 && p.lse != nullptr && row_ok)
        p.lse[(static_cast<size_t>(b) * p.H + h) * p.S + pos] = (m_run * sl2 + log2f(l_run)) * LN2;
    }
  }

  // ------------------------------------------------------------------ teardown
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (bars->abort_flag) {
    if (threadIdx.x == 0 && p.status != nullptr) atomicExch(p.status, FSB_ERR_WAIT_TIMEOUT);
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

}  // namespace pp
}  // namespace fsb

// C ABI.  Any S >= 1, D in {64, 128}; returns -1 otherwise.  Tensors are contiguous and 16-byte aligned.
FSB_API int fsb_attn_fwd_pingpong(const void* qkv, void* o, float* lse, int B, int S, int H, int D, float scale, int* status,
                                  cudaStream_t stream) {
  using namespace fsb;
  using namespace fsb::pp;
  if (B < 1 || S < 1 || H < 1 || (D != 64 && D != 128)) return -1;
  CUtensorMap tm;
  if (!fsb_host::encode_3d_16bit(&tm, qkv, (uint64_t)3 * H * D, (uint64_t)S, (uint64_t)B, (uint64_t)3 * H * D, (uint64_t)3 * H * D * S, 64, BM, 1)) return -1;
  Params p{};
  p.B = B; p.S = S; p.H = H; p.D = D; p.scale = scale;
  p.o = static_cast<__nv_bfloat16*>(o); p.lse = lse; p.status = status;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int n_items = ((S + 2 * BM - 1) / (2 * BM)) * H * B;
  const dim3 grid(n_items < sms ? n_items : sms);  // persistent: one CTA per SM walks the work items
  // each CTA allocates all 512 TMEM columns, so two CTAs must never share an SM: ask for more than half of its shared memory
  constexpr int kMinSmem = 120 * 1024;
  if (D == 128) {
    constexpr int smem = Smem<128>::TOTAL;
    cudaFuncSetAttribute(attn_fwd_pingpong_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    attn_fwd_pingpong_kernel<128><<<grid, THREADS, smem, stream>>>(tm, p);
  } else {
    constexpr int smem = Smem<64>::TOTAL < kMinSmem ? kMinSmem : Smem<64>::TOTAL;
    cudaFuncSetAttribute(attn_fwd_pingpong_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    attn_fwd_pingpong_kernel<64><<<grid, THREADS, smem, stream>>>(tm, p);
  }
  return static_cast<int>(cudaGetLastError());
}
