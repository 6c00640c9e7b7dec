// LayerNorm / RMSNorm forward and backward for bf16 activations, fp32 statistics.
//
// Forward: a row is read once with 16-byte loads, kept in registers, reduced (mean / variance) and written once; mean
// and rstd are saved for backward.  Backward: same one-pass structure for dx; dgamma / dbeta are accumulated per CTA into
// fp32 partials [n_strips, H], reduced by a second small kernel (no atomics, so the result is deterministic).
// Rows of up to 4096 columns take a warp each forwards and the row-group kernel backwards, longer ones (up to 8192) one
// CTA per row.
// Replaces nn.LayerNorm in the reference's benchmark models (benchmarks/models/transformer_lm.py:109-110).

#include "common.cuh"

#include <atomic>

namespace fsb {

constexpr int NORM_THREADS = 256;
constexpr int NORM_MAX_VEC = 4;  // block-per-row path: up to 4 x 8 bf16 per thread -> H <= 8192
constexpr int NORM_WARPS = 4;    // warp-per-row forward: rows handled per CTA
constexpr int NORM_ROWS_MAX_H = 4096;  // row-group backward: up to 512 threads of 8 columns

// Eight columns of a row in a lane's registers, as fp32 or as they came.
template <bool F32> struct RowPiece {
  float v[8];
  __device__ __forceinline__ void load(const __nv_bfloat16* p) {
    const Vec16<__nv_bfloat16> t = ld16(p);
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = __bfloat162float(t.v[k]);
  }
  __device__ __forceinline__ float operator[](int k) const { return v[k]; }
};
template <> struct RowPiece<false> {
  Vec16<__nv_bfloat16> v;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { v = ld16(p); }
  __device__ __forceinline__ float operator[](int k) const { return __bfloat162float(v.v[k]); }
};

// ---- warp-per-row forward (H <= 4096): a lane keeps VPL pieces of eight columns of the row in registers, all
// reductions are warp shuffles, no shared memory and no block barriers.
// Bound by memory, and by how many rows are in flight: as bf16 a row takes 64 registers a thread at 2048 columns (95 as fp32)
// and 96 at 4096 (164): 16384 x 2048 31.8 -> 25.9 us (20.5 at the copy rate), 16384 x 4096 71 -> 58.  But each value is then
// converted three times, and where registers are no limit that is what takes the time: 65536 x 328 22.9 us as fp32, 25.8 as
// bf16, 16384 x 1024 11.3 and 12.3, 300 x 3072 6.1 and 7.0.  launch_norm_fwd has the line.
template <bool RMS, int VPL, bool F32>
__global__ void __launch_bounds__(NORM_WARPS * 32) norm_fwd_warp_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ gamma,
                                                                        const __nv_bfloat16* __restrict__ beta, __nv_bfloat16* __restrict__ y,
                                                                        float* __restrict__ mean_out, float* __restrict__ rstd_out,
                                                                        long long rows, int H, float eps) {
  const int lane = threadIdx.x & 31;
  const long long row = static_cast<long long>(blockIdx.x) * NORM_WARPS + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int nvec = H / 8;
  const __nv_bfloat16* xr = x + row * H;
  RowPiece<F32> v[VPL];
  float sum = 0.f;
#pragma unroll
  for (int it = 0; it < VPL; ++it) {
    const int j = lane + it * 32;
    if (j < nvec) v[it].load(xr + j * 8);
  }
#pragma unroll
  for (int it = 0; it < VPL; ++it) {
    const int j = lane + it * 32;
    if (j < nvec) {
#pragma unroll
      for (int k = 0; k < 8; ++k) sum += v[it][k];
    }
  }
  const float mean = RMS ? 0.f : warp_sum(sum) / H;
  float sq = 0.f;
#pragma unroll
  for (int it = 0; it < VPL; ++it) {
    const int j = lane + it * 32;
    if (j < nvec) {
#pragma unroll
      for (int k = 0; k < 8; ++k) { const float d = v[it][k] - mean; sq += d * d; }
    }
  }
  const float rstd = rsqrtf(warp_sum(sq) / H + eps);
  if (lane == 0) {
    if (!RMS && mean_out != nullptr) mean_out[row] = mean;
    if (rstd_out != nullptr) rstd_out[row] = rstd;
  }
  __nv_bfloat16* yr = y + row * H;
#pragma unroll
  for (int it = 0; it < VPL; ++it) {
    const int j = lane + it * 32;
    if (j < nvec) {
      const Vec16<__nv_bfloat16> g = ld16(gamma + j * 8);
      Vec16<__nv_bfloat16> o;
      if (!RMS && beta != nullptr) {
        const Vec16<__nv_bfloat16> b = ld16(beta + j * 8);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          o.v[k] = __float2bfloat16_rn((v[it][k] - mean) * rstd * __bfloat162float(g.v[k]) + __bfloat162float(b.v[k]));
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) o.v[k] = __float2bfloat16_rn((v[it][k] - mean) * rstd * __bfloat162float(g.v[k]));
      }
      st16(yr + j * 8, o);
    }
  }
}

// ---- row-group backward (H <= 4096): a thread owns the same 8 columns of every row it sees, so gamma and the dgamma / dbeta
// sums stay in its registers.  A row takes H / 8 lanes: a power of two inside one warp up to 256 columns, whole warps beyond; a
// CTA of about 256 threads holds as many such groups as fit (one from 1032 columns on), and each walks R rows at a time.
// Persistent: two CTAs of up to 256 threads per SM (128 registers per thread), one of 288 to 512 for wider rows.  Bound by memory,
// and what counts is bytes in flight: the next rows' vectors (x, dy and the residual's) are loaded before the current rows' sums,
// and the narrower a row, the more of them are under way side by side.  One group per CTA whatever the width left a narrow row's
// SM with a fraction of its 512 threads and took 65536 x 512 162 us (now 47 us), 16384 x 1024 51 (29), 16384 x 2048 66 (51),
// 16384 x 4096, its grid in two waves, 138 (102); with a residual 16384 x 2048 75 (58).  A warp per row, with all of a row's sums
// in one warp's registers and room for one row only, took 87, 41 and 67 us, two kernels for 4096 columns 188.  (All with the
// reduction of the partial rows, ten calls in a graph.)  The forward has no sums to keep and is faster with a warp per row: 29
// against 41 us.
struct NormRowsShape {
  int lanes;          // lanes of a warp that share a row
  int warps_per_row;  // 1 unless lanes == 32
  int groups;         // rows that the CTA works on side by side
  int threads;
};
__host__ __device__ inline NormRowsShape norm_rows_shape(int H) {
  NormRowsShape s;
  const int need = H / 8;
  s.lanes = 1;
  while (s.lanes < 32 && s.lanes < need) s.lanes *= 2;
  s.warps_per_row = (need + 31) / 32;
  const int warp_groups = s.warps_per_row >= 8 ? 1 : 8 / s.warps_per_row;
  s.groups = warp_groups * (32 / s.lanes);
  s.threads = warp_groups * s.warps_per_row * 32;
  return s;
}

// Sums of N values over the threads that share a row; `red` (per group of warps) holds 2 * 16 * N floats and is used in turn
// (`turn` alternates), so one barrier per call is enough.
template <int N>
__device__ __forceinline__ void row_sums(float (&v)[N], float* red, int turn, int lanes, int warps_per_row, int warp_group, int warp_in_row) {
  for (int o = lanes >> 1; o > 0; o >>= 1) {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
  }
  if (warps_per_row == 1) return;
  float* buf = red + (turn & 1) * 16 * N;
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int i = 0; i < N; ++i) buf[warp_in_row * N + i] = v[i];
  }
  asm volatile("bar.sync %0, %1;" ::"r"(warp_group + 1), "r"(warps_per_row * 32) : "memory");
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = 0.f;
  for (int w = 0; w < warps_per_row; ++w) {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] += buf[w * N + i];
  }
}

// dx and the dgamma / dbeta partials in one pass over dy and x: dgamma_part / dbeta_part are [gridDim.x, H].  RES: `res` is a
// gradient of x from elsewhere - the residual branch around the norm - that is added before dx is rounded.
template <bool RMS, bool RES, int MAX_THREADS>
__global__ void __launch_bounds__(MAX_THREADS, 512 / MAX_THREADS) norm_bwd_rows_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                                                               const __nv_bfloat16* __restrict__ gamma, const float* __restrict__ mean_in,
                                                               const float* __restrict__ rstd_in, const __nv_bfloat16* __restrict__ res,
                                                               __nv_bfloat16* __restrict__ dx, float* __restrict__ dgamma_part,
                                                               float* __restrict__ dbeta_part, long long rows, int H) {
  constexpr int R = 2, N = 2 * R;
  __shared__ float red[4][2 * 16 * N];  // per group of warps (more than one warp per row: at most four groups)
  __shared__ __align__(16) float sums[MAX_THREADS <= 256 ? 256 * 8 : 4];  // one value per group and column, at the end
  const NormRowsShape sh = norm_rows_shape(H);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int warp_group = warp / sh.warps_per_row, warp_in_row = warp - warp_group * sh.warps_per_row;
  const int group = sh.warps_per_row == 1 ? static_cast<int>(threadIdx.x) / sh.lanes : warp_group;
  const int col = sh.warps_per_row == 1 ? (lane & (sh.lanes - 1)) * 8 : (warp_in_row * 32 + lane) * 8;
  const bool mine = col < H;
  float* my_red = red[sh.warps_per_row == 1 ? 0 : warp_group];
  float dg[8], db[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) dg[k] = db[k] = 0.f;
  struct Rows {
    Vec16<__nv_bfloat16> x[R], d[R], t[RES ? R : 1];
    float m[R], r[R];
  } cur, nxt;
  Vec16<__nv_bfloat16> tg;
  tg.raw = make_uint4(0u, 0u, 0u, 0u);
  if (mine) tg = ld16(gamma + col);
  auto load = [&](Rows& v, long long row0) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      v.x[i].raw = v.d[i].raw = make_uint4(0u, 0u, 0u, 0u);
      if (RES) v.t[i].raw = make_uint4(0u, 0u, 0u, 0u);
      v.m[i] = v.r[i] = 0.f;
      if (row0 + i < rows) {
        if (mine) {
          v.x[i] = ld16(x + (row0 + i) * H + col);
          v.d[i] = ld16(dy + (row0 + i) * H + col);
          if (RES) v.t[i] = ld16(res + (row0 + i) * H + col);
        }
        if (!RMS) v.m[i] = mean_in[row0 + i];
        v.r[i] = rstd_in[row0 + i];
      }
    }
  };
  const long long step = static_cast<long long>(gridDim.x) * sh.groups * R;
  long long base = static_cast<long long>(blockIdx.x) * sh.groups * R;  // the CTA's first row: the same trip count for all its lanes
  long long row0 = base + group * R;
  int turn = 0;
  load(cur, row0);
  for (; base < rows; base += step, row0 += step) {
    load(nxt, row0 + step);
    float s[N];  // sum of w, sum of w * xhat, per row
#pragma unroll
    for (int i = 0; i < R; ++i) {
      s[2 * i] = s[2 * i + 1] = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float xh = (__bfloat162float(cur.x[i].v[k]) - cur.m[i]) * cur.r[i];
        const float w = __bfloat162float(cur.d[i].v[k]) * __bfloat162float(tg.v[k]);
        s[2 * i] += w;
        s[2 * i + 1] = fmaf(w, xh, s[2 * i + 1]);
      }
    }
    row_sums<N>(s, my_red, turn++, sh.lanes, sh.warps_per_row, warp_group, warp_in_row);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      if (row0 + i >= rows || !mine) break;
      const float s1 = RMS ? 0.f : s[2 * i] / H, s2 = s[2 * i + 1] / H;
      Vec16<__nv_bfloat16> o;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float xh = (__bfloat162float(cur.x[i].v[k]) - cur.m[i]) * cur.r[i];
        const float d = __bfloat162float(cur.d[i].v[k]);
        const float w = d * __bfloat162float(tg.v[k]);
        o.v[k] = __float2bfloat16_rn(fmaf(cur.r[i], w - s1 - xh * s2, RES ? __bfloat162float(cur.t[RES ? i : 0].v[k]) : 0.f));
        dg[k] = fmaf(d, xh, dg[k]);
        if (!RMS) db[k] += d;
      }
      st16(dx + (row0 + i) * H + col, o);
    }
    cur = nxt;
  }
  // the CTA's partial row: its groups in order, dgamma first and dbeta second through the same buffer
#pragma unroll
  for (int which = 0; which < (RMS ? 1 : 2); ++which) {
    float* out = which == 0 ? dgamma_part : dbeta_part;
    if (out == nullptr) break;  // uniform
    out += static_cast<long long>(blockIdx.x) * H;
    const float (&v)[8] = which == 0 ? dg : db;
    float* to = sh.groups == 1 ? out + col : sums + group * H + col;
    if (which == 1 && sh.groups > 1) __syncthreads();
    if (mine) {
      *reinterpret_cast<float4*>(to) = make_float4(v[0], v[1], v[2], v[3]);
      *reinterpret_cast<float4*>(to + 4) = make_float4(v[4], v[5], v[6], v[7]);
    }
    if (sh.groups == 1) continue;
    __syncthreads();
    for (int c = threadIdx.x; c < H; c += blockDim.x) {
      float acc = 0.f;
      for (int g = 0; g < sh.groups; ++g) acc += sums[g * H + c];
      out[c] = acc;
    }
  }
}

// Partial column sums of dy * xhat (-> dgamma) and dy (-> dbeta) over a strip of rows.
// grid = (ceil(H / 256), strips), block = (32, 8): a thread owns 8 consecutive columns.
template <bool RMS>
__global__ void __launch_bounds__(256) norm_dparam_partial_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                                                                  const float* __restrict__ mean_in, const float* __restrict__ rstd_in,
                                                                  float* __restrict__ dgamma_part, float* __restrict__ dbeta_part,
                                                                  long long rows, int H) {
  const int col0 = (blockIdx.x * 32 + threadIdx.x) * 8;
  const bool active = col0 < H;
  float dg[8] = {0, 0, 0, 0, 0, 0, 0, 0}, db[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (long long r = blockIdx.y * 8 + threadIdx.y; active && r < rows; r += static_cast<long long>(gridDim.y) * 8) {
    const float mean = RMS ? 0.f : mean_in[r];
    const float rstd = rstd_in[r];
    const Vec16<__nv_bfloat16> tx = ld16(x + r * H + col0);
    const Vec16<__nv_bfloat16> td = ld16(dy + r * H + col0);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float d = __bfloat162float(td.v[k]);
      dg[k] += d * (__bfloat162float(tx.v[k]) - mean) * rstd;
      db[k] += d;
    }
  }
  __shared__ float red[2][8][32][9];
#pragma unroll
  for (int k = 0; k < 8; ++k) { red[0][threadIdx.y][threadIdx.x][k] = dg[k]; red[1][threadIdx.y][threadIdx.x][k] = db[k]; }
  __syncthreads();
  if (threadIdx.y < 2 && active) {
    const int which = threadIdx.y;
    if (which == 1 && (RMS || dbeta_part == nullptr)) return;
    float* out = (which == 0 ? dgamma_part : dbeta_part) + static_cast<long long>(blockIdx.y) * H + col0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      float s = 0.f;
#pragma unroll
      for (int yy = 0; yy < 8; ++yy) s += red[which][yy][threadIdx.x][k];
      out[k] = s;
    }
  }
}

template <bool RMS>
__global__ void __launch_bounds__(NORM_THREADS) norm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ gamma,
                                                                const __nv_bfloat16* __restrict__ beta, __nv_bfloat16* __restrict__ y,
                                                                float* __restrict__ mean_out, float* __restrict__ rstd_out, int H, float eps) {
  __shared__ float scratch[32];
  const long long row = blockIdx.x;
  const __nv_bfloat16* xr = x + row * H;
  __nv_bfloat16* yr = y + row * H;
  const int nvec = H / 8;
  float v[NORM_MAX_VEC][8];
  float sum = 0.f;
#pragma unroll
  for (int it = 0; it < NORM_MAX_VEC; ++it) {
    const int j = threadIdx.x + it * NORM_THREADS;
    if (j < nvec) {
      const Vec16<__nv_bfloat16> t = ld16(xr + j * 8);
#pragma unroll
      for (int k = 0; k < 8; ++k) { v[it][k] = __bfloat162float(t.v[k]); sum += v[it][k]; }
    }
  }
  float mean = 0.f;
  if (!RMS) mean = block_sum(sum, scratch) / H;
  float sq = 0.f;
#pragma unroll
  for (int it = 0; it < NORM_MAX_VEC; ++it) {
    const int j = threadIdx.x + it * NORM_THREADS;
    if (j < nvec) {
#pragma unroll
      for (int k = 0; k < 8; ++k) { const float d = v[it][k] - mean; sq += d * d; }
    }
  }
  const float var = block_sum(sq, scratch) / H;
  const float rstd = rsqrtf(var + eps);
  if (threadIdx.x == 0) {
    if (!RMS && mean_out != nullptr) mean_out[row] = mean;
    if (rstd_out != nullptr) rstd_out[row] = rstd;
  }
#pragma unroll
  for (int it = 0; it < NORM_MAX_VEC; ++it) {
    const int j = threadIdx.x + it * NORM_THREADS;
    if (j < nvec) {
      const Vec16<__nv_bfloat16> g = ld16(gamma + j * 8);
      Vec16<__nv_bfloat16> o;
      if (!RMS && beta != nullptr) {
        const Vec16<__nv_bfloat16> b = ld16(beta + j * 8);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          o.v[k] = __float2bfloat16_rn((v[it][k] - mean) * rstd * __bfloat162float(g.v[k]) + __bfloat162float(b.v[k]));
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) o.v[k] = __float2bfloat16_rn((v[it][k] - mean) * rstd * __bfloat162float(g.v[k]));
      }
      st16(yr + j * 8, o);
    }
  }
}

// Block-per-row dx (H > 4096).
template <bool RMS>
__global__ void __launch_bounds__(NORM_THREADS) norm_bwd_dx_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                                                                   const __nv_bfloat16* __restrict__ gamma, const float* __restrict__ mean_in,
                                                                   const float* __restrict__ rstd_in, const __nv_bfloat16* __restrict__ res,
                                                                   __nv_bfloat16* __restrict__ dx, int H) {
  __shared__ float scratch[32];
  const int nvec = H / 8;
  const long long row = blockIdx.x;
  const float mean = RMS ? 0.f : mean_in[row];
  const float rstd = rstd_in[row];
  float xh[NORM_MAX_VEC][8], wdy[NORM_MAX_VEC][8];
  float s1 = 0.f, s2 = 0.f;
#pragma unroll
  for (int it = 0; it < NORM_MAX_VEC; ++it) {
    const int j = threadIdx.x + it * NORM_THREADS;
    if (j < nvec) {
      const Vec16<__nv_bfloat16> tx = ld16(x + row * H + j * 8);
      const Vec16<__nv_bfloat16> td = ld16(dy + row * H + j * 8);
      const Vec16<__nv_bfloat16> tg = ld16(gamma + j * 8);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        xh[it][k] = (__bfloat162float(tx.v[k]) - mean) * rstd;
        wdy[it][k] = __bfloat162float(td.v[k]) * __bfloat162float(tg.v[k]);
        s1 += wdy[it][k];
        s2 += wdy[it][k] * xh[it][k];
      }
    }
  }
  if (!RMS) s1 = block_sum(s1, scratch) / H; else s1 = 0.f;
  s2 = block_sum(s2, scratch) / H;
#pragma unroll
  for (int it = 0; it < NORM_MAX_VEC; ++it) {
    const int j = threadIdx.x + it * NORM_THREADS;
    if (j < nvec) {
      Vec16<__nv_bfloat16> o, tr;
      tr.raw = make_uint4(0u, 0u, 0u, 0u);
      if (res != nullptr) tr = ld16(res + row * H + j * 8);
#pragma unroll
      for (int k = 0; k < 8; ++k) o.v[k] = __float2bfloat16_rn(fmaf(rstd, wdy[it][k] - s1 - xh[it][k] * s2, __bfloat162float(tr.v[k])));
      st16(dx + row * H + j * 8, o);
    }
  }
}

// out[c] = sum_r part[r, c]  (fp32 partials -> bf16 result).  block = (32 columns, 8 row groups): a thread
// adds rows ty, ty + 8, ... of its column in a fixed order, the eight sums are combined through shared memory.
// blockIdx.y: independent matrices stored one after the other; with `out_second` the second one's result goes there (dgamma
// and dbeta of a norm in one launch), otherwise results are stored one after the other as well.
__global__ void __launch_bounds__(256) column_reduce_kernel(const float* __restrict__ part, int rows, int H, __nv_bfloat16* out, __nv_bfloat16* out_second) {
  __shared__ float red[8][33];
  const int c = blockIdx.x * 32 + threadIdx.x;
  part += static_cast<long long>(blockIdx.y) * rows * H;
  if (out_second != nullptr) out = blockIdx.y == 0 ? out : out_second;
  else out += static_cast<long long>(blockIdx.y) * H;
  float acc = 0.f;
  if (c < H) {
#pragma unroll 4
    for (int r = threadIdx.y; r < rows; r += 8) acc += part[static_cast<long long>(r) * H + c];
  }
  red[threadIdx.y][threadIdx.x] = acc;
  __syncthreads();
  if (threadIdx.y == 0 && c < H) {
    float t = 0.f;
#pragma unroll
    for (int y = 0; y < 8; ++y) t += red[y][threadIdx.x];
    out[c] = __float2bfloat16_rn(t);
  }
}

// Column sums of a bf16 matrix [rows, H] (bias gradient): strip partials then reduce.  blockIdx.z: independent matrices
// stored one after the other (the experts of an MoE layer).
__global__ void __launch_bounds__(256) colsum_partial_kernel(const __nv_bfloat16* __restrict__ x, long long rows, int H, float* __restrict__ part) {
  // block = 32 x 8 threads; a block handles 256 columns (8 per thread along x) for a strip of rows
  const int col0 = (blockIdx.x * 32 + threadIdx.x) * 8;
  const bool active = col0 < H;
  x += static_cast<long long>(blockIdx.z) * rows * H;
  part += static_cast<long long>(blockIdx.z) * gridDim.y * H;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  // bound by memory: four loads in flight per thread (16384 x 8192: one load gave 4 TB/s)
  const long long step = static_cast<long long>(gridDim.y) * 8;
  long long r = blockIdx.y * 8 + threadIdx.y;
  for (; active && r + 3 * step < rows; r += 4 * step) {
    Vec16<__nv_bfloat16> t[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) t[u] = ld16(x + (r + u * step) * H + col0);
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] += __bfloat162float(t[u].v[k]);
  }
  for (; active && r < rows; r += step) {
    const Vec16<__nv_bfloat16> t = ld16(x + r * H + col0);
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] += __bfloat162float(t.v[k]);
  }
  __shared__ float red[8][32][9];
#pragma unroll
  for (int k = 0; k < 8; ++k) red[threadIdx.y][threadIdx.x][k] = acc[k];
  __syncthreads();
  if (threadIdx.y == 0 && active) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      float s = 0.f;
#pragma unroll
      for (int y = 0; y < 8; ++y) s += red[y][threadIdx.x][k];
      part[static_cast<long long>(blockIdx.y) * H + col0 + k] = s;
    }
  }
}

}  // namespace fsb

// Rows of the widest warp-per-row forward that the device holds at a time.
template <bool RMS, bool F32>
static long long norm_rows_in_flight() {
  using namespace fsb;
  static std::atomic<int> cache[64];
  int dev = 0;
  cudaGetDevice(&dev);
  int rows = cache[dev & 63].load(std::memory_order_relaxed);
  if (rows == 0) {
    int ctas = 1, sms = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, norm_fwd_warp_kernel<RMS, 16, F32>, NORM_WARPS * 32, 0);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    rows = ctas * sms * NORM_WARPS;
    if (rows < 1) rows = 1;
    cache[dev & 63].store(rows, std::memory_order_relaxed);
  }
  return rows;
}

// Rows in fp32 up to 1024 columns, where they are all in flight either way; as bf16 beyond, up to 2048 columns at any number of
// rows (fewer than one wave: within 5 % of one another); beyond that by the number of waves, of which fp32 takes more (1776 rows
// each, bf16 2960) but shorter ones (us, fp32 / bf16, 4096 columns: 1200 rows 8.6 / 9.0, 2048 13.3 / 9.4, 3200 13.7 / 15.1).
template <bool RMS>
static void launch_norm_fwd(const __nv_bfloat16* x, const __nv_bfloat16* g, const __nv_bfloat16* b, __nv_bfloat16* y, float* mean,
                            float* rstd, long long rows, int H, float eps, cudaStream_t stream) {
  using namespace fsb;
  const unsigned grid = static_cast<unsigned>((rows + NORM_WARPS - 1) / NORM_WARPS);
  const int vpl = (H / 8 + 31) / 32;
  auto warp_rows = [&](auto kernel) { kernel<<<grid, NORM_WARPS * 32, 0, stream>>>(x, g, b, y, mean, rstd, rows, H, eps); };
  if (vpl <= 2)       warp_rows(norm_fwd_warp_kernel<RMS, 2, true>);
  else if (vpl <= 4)  warp_rows(norm_fwd_warp_kernel<RMS, 4, true>);
  else if (vpl <= 8)  warp_rows(norm_fwd_warp_kernel<RMS, 8, false>);
  else if (vpl <= 16) {
    const long long in_f32 = norm_rows_in_flight<RMS, true>(), in_bf16 = norm_rows_in_flight<RMS, false>();
    if ((rows + in_f32 - 1) / in_f32 <= (rows + in_bf16 - 1) / in_bf16) warp_rows(norm_fwd_warp_kernel<RMS, 16, true>);
    else                                                                warp_rows(norm_fwd_warp_kernel<RMS, 16, false>);
  }
  else norm_fwd_kernel<RMS><<<static_cast<unsigned>(rows), NORM_THREADS, 0, stream>>>(x, g, b, y, mean, rstd, H, eps);
}

// H must be a multiple of 8 and <= 8192. mean/rstd are fp32 [rows]. rms != 0 selects RMSNorm
// (beta and mean ignored).
FSB_API int fsb_norm_fwd(const void* x, const void* gamma, const void* beta, void* y, float* mean, float* rstd,
                         long long rows, int H, float eps, int rms, cudaStream_t stream) {
  using namespace fsb;
  if (rows <= 0) return 0;
  if (H % 8 != 0 || H > 8 * NORM_THREADS * NORM_MAX_VEC) return -1;
  auto* xx = static_cast<const __nv_bfloat16*>(x);
  auto* gg = static_cast<const __nv_bfloat16*>(gamma);
  auto* bb = static_cast<const __nv_bfloat16*>(beta);
  auto* yy = static_cast<__nv_bfloat16*>(y);
  if (rms) launch_norm_fwd<true>(xx, gg, bb, yy, mean, rstd, rows, H, eps, stream);
  else     launch_norm_fwd<false>(xx, gg, bb, yy, mean, rstd, rows, H, eps, stream);
  return static_cast<int>(cudaGetLastError());
}

// Rows of fp32 partials the backward needs room for: the row-group kernel (H <= 4096) writes one row per CTA of its persistent
// grid - two CTAs of up to 256 threads or one larger one per SM, never more than there are groups of rows - the two-kernel path
// at most 48.
static int norm_bwd_rows_ctas(long long rows, int groups, int ctas_per_sm) {
  const long long per_cta = 2ll * groups, want = (rows + per_cta - 1) / per_cta, most = 148ll * ctas_per_sm;
  return static_cast<int>(want < 1 ? 1 : (want > most ? most : want));
}
static int norm_bwd_split_strips(long long rows) {
  const long long want = (rows + 7) / 8;
  return static_cast<int>(want < 1 ? 1 : (want > 48 ? 48 : want));
}

FSB_API int fsb_norm_bwd_num_strips(long long rows) {
  const int a = norm_bwd_rows_ctas(rows, 1, 2), b = norm_bwd_split_strips(rows);
  return a > b ? a : b;
}

// partials: fp32 workspace of 2 * n_strips * H floats (n_strips from fsb_norm_bwd_num_strips).
// dgamma / dbeta are bf16 [H] outputs (dbeta may be null, and is ignored for RMSNorm).  res: bf16 [rows, H] added to dx, or null.
FSB_API int fsb_norm_bwd_res(const void* dy, const void* x, const void* gamma, const float* mean, const float* rstd, const void* res, void* dx,
                             void* dgamma, void* dbeta, float* partials, long long rows, int H, int rms, cudaStream_t stream) {
  using namespace fsb;
  if (H % 8 != 0 || H > 8 * NORM_THREADS * NORM_MAX_VEC) return -1;
  if (rows <= 0) {  // an empty sum is zero, and the outputs may be windows of a gradient that is used as it stands
    cudaError_t e = cudaMemsetAsync(dgamma, 0, static_cast<size_t>(H) * 2, stream);
    if (e == cudaSuccess && !rms && dbeta != nullptr) e = cudaMemsetAsync(dbeta, 0, static_cast<size_t>(H) * 2, stream);
    return static_cast<int>(e);
  }
  const bool fused = H <= NORM_ROWS_MAX_H;
  const NormRowsShape sh = norm_rows_shape(H);
  const int strips = fused ? norm_bwd_rows_ctas(rows, sh.groups, sh.threads <= 256 ? 2 : 1) : norm_bwd_split_strips(rows);
  float* pg = partials;
  float* pb = partials + static_cast<long long>(strips) * H;
  auto* d = static_cast<const __nv_bfloat16*>(dy);
  auto* xx = static_cast<const __nv_bfloat16*>(x);
  auto* gg = static_cast<const __nv_bfloat16*>(gamma);
  auto* rr = static_cast<const __nv_bfloat16*>(res);
  auto* o = static_cast<__nv_bfloat16*>(dx);
  const bool want_beta = !rms && dbeta != nullptr;
  if (fused) {
    auto launch = [&](auto kernel) { kernel<<<strips, sh.threads, 0, stream>>>(d, xx, gg, mean, rstd, rr, o, pg, want_beta ? pb : nullptr, rows, H); };
    if (sh.threads <= 256) {
      if (rms) rr != nullptr ? launch(norm_bwd_rows_kernel<true, true, 256>) : launch(norm_bwd_rows_kernel<true, false, 256>);
      else     rr != nullptr ? launch(norm_bwd_rows_kernel<false, true, 256>) : launch(norm_bwd_rows_kernel<false, false, 256>);
    } else {
      if (rms) rr != nullptr ? launch(norm_bwd_rows_kernel<true, true, 512>) : launch(norm_bwd_rows_kernel<true, false, 512>);
      else     rr != nullptr ? launch(norm_bwd_rows_kernel<false, true, 512>) : launch(norm_bwd_rows_kernel<false, false, 512>);
    }
  } else {
    dim3 block(32, 8), grid((H / 8 + 31) / 32, strips);
    if (rms) {
      norm_bwd_dx_kernel<true><<<static_cast<unsigned>(rows), NORM_THREADS, 0, stream>>>(d, xx, gg, mean, rstd, rr, o, H);
      norm_dparam_partial_kernel<true><<<grid, block, 0, stream>>>(d, xx, mean, rstd, pg, nullptr, rows, H);
    } else {
      norm_bwd_dx_kernel<false><<<static_cast<unsigned>(rows), NORM_THREADS, 0, stream>>>(d, xx, gg, mean, rstd, rr, o, H);
      norm_dparam_partial_kernel<false><<<grid, block, 0, stream>>>(d, xx, mean, rstd, pg, want_beta ? pb : nullptr, rows, H);
    }
  }
  const dim3 threads(32, 8);
  const int blocks = (H + 31) / 32;
  // the beta partials follow the gamma partials
  column_reduce_kernel<<<dim3(blocks, want_beta ? 2 : 1), threads, 0, stream>>>(pg, strips, H, static_cast<__nv_bfloat16*>(dgamma),
                                                                                want_beta ? static_cast<__nv_bfloat16*>(dbeta) : nullptr);
  return static_cast<int>(cudaGetLastError());
}

FSB_API int fsb_colsum_num_strips(long long rows) {
  const long long want = (rows + 63) / 64;
  return static_cast<int>(want < 1 ? 1 : (want > 48 ? 48 : want));
}

// out[b, c] = sum_r x[b, r, c]; x bf16 [batch, rows, H] (H % 8 == 0); partials fp32 [batch, n_strips, H]; out bf16 [batch, H].
FSB_API int fsb_colsum_batched(const void* x, int batch, long long rows, int H, float* partials, void* out, cudaStream_t stream) {
  using namespace fsb;
  if (batch <= 0 || rows <= 0 || H <= 0) return 0;
  if (H % 8 != 0 || batch > 65535) return -1;
  const int strips = fsb_colsum_num_strips(rows);
  const dim3 block(32, 8), grid((H / 8 + 31) / 32, strips, batch);
  colsum_partial_kernel<<<grid, block, 0, stream>>>(static_cast<const __nv_bfloat16*>(x), rows, H, partials);
  column_reduce_kernel<<<dim3((H + 31) / 32, batch), block, 0, stream>>>(partials, strips, H, static_cast<__nv_bfloat16*>(out), nullptr);
  return static_cast<int>(cudaGetLastError());
}

FSB_API int fsb_colsum(const void* x, long long rows, int H, float* partials, void* out, cudaStream_t stream) {
  return fsb_colsum_batched(x, 1, rows, H, partials, out, stream);
}

// ---------------------------------------------------------------------------------------------------------
// Allocation-free column sum (declared in fsb_no_alloc.h; no counterpart in the reference library).
// The strip partials go to a fixed array in device memory instead of a workspace from the caller.
// ---------------------------------------------------------------------------------------------------------
#include <mutex>

#include "fsb_no_alloc.h"

namespace {
constexpr int kStaticStrips = 48;   // upper bound of fsb_colsum_num_strips
constexpr int kMaxDevices = 64;
static __device__ __align__(256) float g_colsum_scratch[kStaticStrips * FSB_COLSUM_STATIC_MAX_H];
float* g_colsum_scratch_ptr[kMaxDevices] = {};
std::mutex g_colsum_scratch_mutex;

// Device address of the scratch array on the current device; resolved once per device.
int colsum_scratch_for_current_device(float** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (dev < 0 || dev >= kMaxDevices) return FSB_NOALLOC_ERR_DEVICE;
  std::lock_guard<std::mutex> lock(g_colsum_scratch_mutex);
  if (g_colsum_scratch_ptr[dev] == nullptr) {
    float* p = nullptr;
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_colsum_scratch);
    if (e != cudaSuccess || p == nullptr) {
      (void)cudaGetLastError();
      return FSB_NOALLOC_ERR_SYMBOL;
    }
    g_colsum_scratch_ptr[dev] = p;
  }
  *out = g_colsum_scratch_ptr[dev];
  return 0;
}
}  // namespace

FSB_API int fsb_colsum_static_max_h(void) { return FSB_COLSUM_STATIC_MAX_H; }

FSB_API const char* fsb_colsum_static_strerror(int code) {
  switch (code) {
    case 0: return "ok";
    case FSB_NOALLOC_ERR_SHAPE: return "fsb_colsum_static: H must be a multiple of 8";
    case FSB_NOALLOC_ERR_TOO_LARGE: return "fsb_colsum_static: H exceeds FSB_COLSUM_STATIC_MAX_H (8192); call fsb_colsum with a caller-provided workspace";
    case FSB_NOALLOC_ERR_DEVICE: return "fsb_colsum_static: device ordinal beyond the 64 devices the library tracks";
    case FSB_NOALLOC_ERR_SYMBOL: return "fsb_colsum_static: could not resolve the built-in workspace on this device";
    default: return code > 0 ? cudaGetErrorString(static_cast<cudaError_t>(code)) : "fsb_colsum_static: unknown error";
  }
}

FSB_API int fsb_colsum_static(const void* x, long long rows, int H, void* out, cudaStream_t stream) {
  using namespace fsb;
  if (rows <= 0 || H <= 0) return 0;
  if (H % 8 != 0) return FSB_NOALLOC_ERR_SHAPE;
  if (H > FSB_COLSUM_STATIC_MAX_H) return FSB_NOALLOC_ERR_TOO_LARGE;
  float* scratch = nullptr;
  const int rc = colsum_scratch_for_current_device(&scratch);
  if (rc != 0) return rc;
  const int strips = fsb_colsum_num_strips(rows);  // <= kStaticStrips
  dim3 block(32, 8), grid((H / 8 + 31) / 32, strips);
  // every (strip, column < H) element read by the reduction below is written here first: no clearing needed
  colsum_partial_kernel<<<grid, block, 0, stream>>>(static_cast<const __nv_bfloat16*>(x), rows, H, scratch);
  const dim3 threads(32, 8);
  const int blocks = (H + 31) / 32;
  column_reduce_kernel<<<blocks, threads, 0, stream>>>(scratch, strips, H, static_cast<__nv_bfloat16*>(out), nullptr);
  return static_cast<int>(cudaGetLastError());
}
