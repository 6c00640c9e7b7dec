// Softmax cross-entropy over bf16 or fp32 logits with fp32 math.
//
// Forward: one CTA per token row, one streaming pass (online max / sum) over the vocabulary with
// 16-byte loads; writes the per-row loss and log-sum-exp.  Backward: one pass that turns the logits
// into d(logits) = (softmax - onehot) * g in place or into a separate buffer.  The [tokens, vocab]
// matrix is therefore read twice and written once in total.
// The vocab-parallel variant returns each rank's (max, sum-exp at that max, target logit) triple so
// the caller can combine them with ONE 3-vector all-reduce instead of the three all-reduces of
// fairscale/nn/model_parallel/cross_entropy.py:35,62-71.
// Both passes are bound by memory.  bf16 logits are 8 bits wide, so the fast exponential's error is far below theirs; fp32
// logits take expf / logf (2 ulp), whose extra instructions still hide behind twice the bytes per element.
// (4096 x 32000 fp32 logits: a chain of fifteen elementwise and reduction kernels took 2.6 ms more than these two.)

#include "common.cuh"

namespace fsb {

constexpr int CE_THREADS = 512;

template <typename T> __device__ __forceinline__ float ce_exp(float x);
template <> __device__ __forceinline__ float ce_exp<__nv_bfloat16>(float x) { return __expf(x); }
template <> __device__ __forceinline__ float ce_exp<float>(float x) { return expf(x); }
template <typename T> __device__ __forceinline__ float ce_log(float x);
template <> __device__ __forceinline__ float ce_log<__nv_bfloat16>(float x) { return __logf(x); }
template <> __device__ __forceinline__ float ce_log<float>(float x) { return logf(x); }

// Exponents are taken relative to the largest value; a maximum that is infinite leaves nothing to be relative to (inf - inf).
__device__ __forceinline__ float ce_ref(float m) { return isinf(m) ? 0.f : m; }

// Online softmax over N values at once: one rescaling per vector instead of a branch per value, which made the bf16 forward
// compute-bound (16384 x 50304: 671 us against 250 us of memory time).  fmaxf passes over NaN, so `m` never holds one and a
// NaN shows in `s` alone.  While every value is -inf or NaN, `m` is -inf and `s` is 0 or NaN; from the first +inf on, `s` is
// +inf or NaN.
template <typename T, int N> __device__ __forceinline__ void online_update(float& m, float& s, const float (&x)[N]) {
  float mx = m;
#pragma unroll
  for (int k = 0; k < N; ++k) mx = fmaxf(mx, x[k]);
  const float ref = ce_ref(mx);
  s *= ce_exp<T>(m - ref);
#pragma unroll
  for (int k = 0; k < N; ++k) s += ce_exp<T>(x[k] - ref);
  m = mx;
}

// stats_out (optional): per row {max, sumexp(at max), target_logit or 0 if target outside [v0, v0+V)}
template <typename T>
__global__ void __launch_bounds__(CE_THREADS) ce_fwd_kernel(const T* __restrict__ logits, const long long* __restrict__ targets,
                                                            float* __restrict__ loss, float* __restrict__ lse_out, float* __restrict__ stats_out,
                                                            int V, long long ld, long long vocab_start, long long ignore_index) {
  __shared__ float scratch[32];
  const long long row = blockIdx.x;
  const T* lr = logits + row * ld;
  constexpr int VN = Vec16<T>::N;
  float m = -INFINITY, s = 0.f;
  const int nvec = V / VN;
  for (int j = threadIdx.x; j < nvec; j += CE_THREADS) {
    const Vec16<T> t = ld16(lr + j * VN);
    float x[VN];
#pragma unroll
    for (int k = 0; k < VN; ++k) x[k] = to_f32(t.v[k]);
    online_update<T, VN>(m, s, x);
  }
  for (int j = nvec * VN + threadIdx.x; j < V; j += CE_THREADS) {
    const float x[1] = {to_f32(lr[j])};
    online_update<T, 1>(m, s, x);
  }
  const float gmax = block_max(m, scratch);
  const float gref = ce_ref(gmax);
  const float gsum = block_sum(s * ce_exp<T>(m - gref), scratch);  // a thread without a finite value adds its 0 or NaN
  if (threadIdx.x == 0) {
    const long long tgt = targets[row];
    const long long local = tgt - vocab_start;
    const bool mine = tgt != ignore_index && local >= 0 && local < V;
    const float tl = mine ? to_f32(lr[local]) : 0.f;
    const float lse = gref + ce_log<T>(gsum);
    if (lse_out != nullptr) lse_out[row] = lse;
    if (loss != nullptr) loss[row] = (tgt == ignore_index) ? 0.f : (lse - tl);
    if (stats_out != nullptr) {
      stats_out[row * 3 + 0] = gmax;
      stats_out[row * 3 + 1] = gsum;
      stats_out[row * 3 + 2] = tl;
    }
  }
}

// dlogits[row, j] = (exp(logit - lse[row]) - [j == target]) * gscale[row-independent scalar] * gout[row or scalar]
template <typename T>
__global__ void __launch_bounds__(CE_THREADS) ce_bwd_kernel(const T* __restrict__ logits, const long long* __restrict__ targets,
                                                            const float* __restrict__ lse, const float* __restrict__ grad_out, int grad_is_scalar,
                                                            float scale, T* __restrict__ dlogits, int V, long long ld,
                                                            long long vocab_start, long long ignore_index) {
  const long long row = blockIdx.x;
  const T* lr = logits + row * ld;
  T* dr = dlogits + row * ld;
  constexpr int VN = Vec16<T>::N;
  const long long tgt = targets[row];
  const float g = (tgt == ignore_index) ? 0.f : scale * (grad_is_scalar ? grad_out[0] : grad_out[row]);
  const float l = lse[row];
  const long long local = tgt - vocab_start;
  const int nvec = V / VN;
  for (int j = threadIdx.x; j < nvec; j += CE_THREADS) {
    const Vec16<T> t = ld16(lr + j * VN);
    Vec16<T> o;
#pragma unroll
    for (int k = 0; k < VN; ++k) {
      float p = ce_exp<T>(to_f32(t.v[k]) - l);
      if (j * VN + k == local) p -= 1.f;
      o.v[k] = from_f32<T>(p * g);
    }
    st16(dr + j * VN, o);
  }
  for (int j = nvec * VN + threadIdx.x; j < V; j += CE_THREADS) {
    float p = ce_exp<T>(to_f32(lr[j]) - l);
    if (j == local) p -= 1.f;
    dr[j] = from_f32<T>(p * g);
  }
}

}  // namespace fsb

// logits: [rows, V] of dtype FSB_BF16 or FSB_F32 with row stride ld; rows start on 16-byte boundaries.
FSB_API int fsb_ce_fwd_dtype(const void* logits, int dtype, const long long* targets, float* loss, float* lse, float* stats, long long rows,
                             int V, long long ld, long long vocab_start, long long ignore_index, cudaStream_t stream) {
  using namespace fsb;
  if (rows <= 0) return 0;
  const dim3 grid(static_cast<unsigned>(rows));
  if (dtype == FSB_BF16 && ld % 8 == 0)
    ce_fwd_kernel<__nv_bfloat16><<<grid, CE_THREADS, 0, stream>>>(static_cast<const __nv_bfloat16*>(logits), targets, loss, lse, stats, V, ld,
                                                                  vocab_start, ignore_index);
  else if (dtype == FSB_F32 && ld % 4 == 0)
    ce_fwd_kernel<float><<<grid, CE_THREADS, 0, stream>>>(static_cast<const float*>(logits), targets, loss, lse, stats, V, ld, vocab_start, ignore_index);
  else return -1;
  return static_cast<int>(cudaGetLastError());
}

FSB_API int fsb_ce_bwd_dtype(const void* logits, int dtype, const long long* targets, const float* lse, const float* grad_out, int grad_is_scalar,
                             float scale, void* dlogits, long long rows, int V, long long ld, long long vocab_start,
                             long long ignore_index, cudaStream_t stream) {
  using namespace fsb;
  if (rows <= 0) return 0;
  const dim3 grid(static_cast<unsigned>(rows));
  if (dtype == FSB_BF16 && ld % 8 == 0)
    ce_bwd_kernel<__nv_bfloat16><<<grid, CE_THREADS, 0, stream>>>(static_cast<const __nv_bfloat16*>(logits), targets, lse, grad_out, grad_is_scalar,
                                                                  scale, static_cast<__nv_bfloat16*>(dlogits), V, ld, vocab_start, ignore_index);
  else if (dtype == FSB_F32 && ld % 4 == 0)
    ce_bwd_kernel<float><<<grid, CE_THREADS, 0, stream>>>(static_cast<const float*>(logits), targets, lse, grad_out, grad_is_scalar, scale,
                                                          static_cast<float*>(dlogits), V, ld, vocab_start, ignore_index);
  else return -1;
  return static_cast<int>(cudaGetLastError());
}
