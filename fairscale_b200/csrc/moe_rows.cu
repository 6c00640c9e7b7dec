// Row movement of a mixture-of-experts layer inside one GPU's memory: tokens to expert slots and back.
//
//   pack    : int32 routing [4, S] (idx1, idx2, loc1, loc2) -> expert / slot (int64 [S, 2]) and keep (bool [S, 2])
//   claim   : expert, slot, keep -> flat (int32 [S, 2]) = expert * C + slot, or -1 for a choice that is not kept, and one
//             byte per row of the [E * C, M] buffer: does a token claim it?
//   scatter : out[flat[s, k], :] = x[s, :] (* w[s, k]);   rows of out that no token claimed are zeroed
//   gather  : out[s, :] = sum_k w[s, k] * buf[flat[s, k], :];   dots[s, k] = <buf[flat[s, k], :], g[s, :]>;
//             kept[s, k, :] = buf[flat[s, k], :] on the way (zero for a choice that is not kept), for a later gather without flat
//
// All three are bound by memory traffic: a warp moves one row with 16-byte accesses (four in flight per lane), scatter
// reads a token once for both of its slots, gather sums both choices in fp32 registers.  A choice is known to be dropped
// from its flat index alone, so nothing on the host depends on how many tokens were kept (the index_copy formulation
// compacts the kept rows first, which makes the host wait for the device twice per direction).  Flat indices and claims
// come from the route as the layer gets it - a gate may have changed what the routing kernels made.
// Layer forward + backward, 8192 tokens of 1024 bf16, 8 experts of 4096: 3740 us with index ops, 1224 us now (866 us of them the
// expert products); 820 tokens of 512, 4 experts of 2048: 2606 -> 1036 us.
//
// Replaces the dense einsum dispatch / combine of the reference (fairscale/nn/moe/moe_layer.py:77,88).

#include "common.cuh"

namespace fsb {

constexpr int MR_THREADS = 256;
constexpr int MR_WARPS = MR_THREADS / 32;

template <typename T, int VEC> struct alignas(VEC == 1 ? sizeof(T) : 16) RowVec { T v[VEC]; };
template <typename T, int VEC> __device__ __forceinline__ RowVec<T, VEC> row_ld(const T* p) {
  RowVec<T, VEC> r;
  if constexpr (VEC == 1) r.v[0] = *p;
  else *reinterpret_cast<uint4*>(r.v) = *reinterpret_cast<const uint4*>(p);
  return r;
}
template <typename T, int VEC> __device__ __forceinline__ void row_st(T* p, const RowVec<T, VEC>& x) {
  if constexpr (VEC == 1) *p = x.v[0];
  else *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(x.v);
}

__global__ void __launch_bounds__(MR_THREADS) moe_route_pack_kernel(const int* __restrict__ route, int S, int C, long long* __restrict__ expert,
                                                                    long long* __restrict__ slot, unsigned char* __restrict__ keep) {
  const int i = blockIdx.x * MR_THREADS + threadIdx.x;  // (token, choice)
  if (i >= 2 * S) return;
  const int s = i >> 1, k = i & 1;
  const int l = route[(2 + k) * S + s];
  expert[i] = route[k * S + s];
  slot[i] = l < C ? l : 0;
  keep[i] = l < C ? 1 : 0;
}

// `claimed` is all zero before the launch
__global__ void __launch_bounds__(MR_THREADS) moe_claim_rows_kernel(const long long* __restrict__ expert, const long long* __restrict__ slot,
                                                                    const unsigned char* __restrict__ keep, long long choices, long long E, long long C,
                                                                    int* __restrict__ flat, unsigned char* __restrict__ claimed) {
  const long long i = static_cast<long long>(blockIdx.x) * MR_THREADS + threadIdx.x;
  if (i >= choices) return;
  const long long row = expert[i] * C + slot[i];
  const bool kept = keep[i] != 0 && row >= 0 && row < E * C;
  flat[i] = kept ? static_cast<int>(row) : -1;
  if (kept) claimed[row] = 1;
}

// Warps 0 .. S-1 (in grid-stride order) each move one token; warps S .. S + E * C - 1 each look at one row of `out`.
template <typename T, int VEC>
__global__ void __launch_bounds__(MR_THREADS) moe_scatter_local_kernel(const T* __restrict__ x, const int* __restrict__ flat, const float* __restrict__ w,
                                                                       long long S, int M, T* __restrict__ out, const unsigned char* __restrict__ claimed,
                                                                       long long rows) {
  const int lane = threadIdx.x & 31;
  const long long warps = static_cast<long long>(gridDim.x) * MR_WARPS;
  for (long long i = static_cast<long long>(blockIdx.x) * MR_WARPS + (threadIdx.x >> 5); i < S + rows; i += warps) {
    if (i < S) {
      const int r0 = flat[2 * i], r1 = flat[2 * i + 1];
      if (r0 < 0 && r1 < 0) continue;
      const float w0 = w != nullptr ? w[2 * i] : 1.f, w1 = w != nullptr ? w[2 * i + 1] : 1.f;
      const T* src = x + i * M;
      T* d0 = out + static_cast<long long>(r0) * M;
      T* d1 = out + static_cast<long long>(r1) * M;
#pragma unroll 4
      for (int j = lane * VEC; j < M; j += 32 * VEC) {
        const RowVec<T, VEC> v = row_ld<T, VEC>(src + j);
        if (w == nullptr) {
          if (r0 >= 0) row_st<T, VEC>(d0 + j, v);
          if (r1 >= 0) row_st<T, VEC>(d1 + j, v);
        } else {
          RowVec<T, VEC> a, b;
#pragma unroll
          for (int k = 0; k < VEC; ++k) {
            const float f = to_f32(v.v[k]);
            a.v[k] = from_f32<T>(f * w0);
            b.v[k] = from_f32<T>(f * w1);
          }
          if (r0 >= 0) row_st<T, VEC>(d0 + j, a);
          if (r1 >= 0) row_st<T, VEC>(d1 + j, b);
        }
      }
    } else {
      const long long r = i - S;
      if (claimed[r]) continue;
      RowVec<T, VEC> z;
#pragma unroll
      for (int k = 0; k < VEC; ++k) z.v[k] = from_f32<T>(0.f);
      for (int j = lane * VEC; j < M; j += 32 * VEC) row_st<T, VEC>(out + r * M + j, z);
    }
  }
}

template <typename T, int VEC>
__global__ void __launch_bounds__(MR_THREADS) moe_gather_local_kernel(const T* __restrict__ buf, const int* __restrict__ flat, const float* __restrict__ w,
                                                                      long long S, int M, T* __restrict__ out, const T* __restrict__ g,
                                                                      float* __restrict__ dots, T* __restrict__ kept) {
  const int lane = threadIdx.x & 31;
  const long long warps = static_cast<long long>(gridDim.x) * MR_WARPS;
  for (long long s = static_cast<long long>(blockIdx.x) * MR_WARPS + (threadIdx.x >> 5); s < S; s += warps) {
    const int r0 = flat != nullptr ? flat[2 * s] : static_cast<int>(2 * s), r1 = flat != nullptr ? flat[2 * s + 1] : static_cast<int>(2 * s + 1);
    const float w0 = w != nullptr ? w[2 * s] : 1.f, w1 = w != nullptr ? w[2 * s + 1] : 1.f;
    const T* b0 = buf + static_cast<long long>(r0) * M;
    const T* b1 = buf + static_cast<long long>(r1) * M;
    float dot0 = 0.f, dot1 = 0.f;
#pragma unroll 4
    for (int j = lane * VEC; j < M; j += 32 * VEC) {
      RowVec<T, VEC> a, b, gv;
#pragma unroll
      for (int k = 0; k < VEC; ++k) a.v[k] = b.v[k] = gv.v[k] = from_f32<T>(0.f);
      if (r0 >= 0) a = row_ld<T, VEC>(b0 + j);
      if (r1 >= 0) b = row_ld<T, VEC>(b1 + j);
      if (kept != nullptr) {
        row_st<T, VEC>(kept + 2 * s * M + j, a);
        row_st<T, VEC>(kept + (2 * s + 1) * M + j, b);
      }
      if (dots != nullptr) {
        gv = row_ld<T, VEC>(g + s * M + j);
#pragma unroll
        for (int k = 0; k < VEC; ++k) {
          const float f = to_f32(gv.v[k]);
          dot0 = fmaf(to_f32(a.v[k]), f, dot0);
          dot1 = fmaf(to_f32(b.v[k]), f, dot1);
        }
      }
      if (out != nullptr) {
        RowVec<T, VEC> o;
#pragma unroll
        for (int k = 0; k < VEC; ++k) {
          float acc = 0.f;
          if (r0 >= 0) acc = to_f32(a.v[k]) * w0;
          if (r1 >= 0) acc = fmaf(to_f32(b.v[k]), w1, acc);
          o.v[k] = from_f32<T>(acc);
        }
        row_st<T, VEC>(out + s * M + j, o);
      }
    }
    if (dots != nullptr) {
      dot0 = warp_sum(dot0);
      dot1 = warp_sum(dot1);
      if (lane == 0) {
        dots[2 * s] = r0 >= 0 ? dot0 : 0.f;
        dots[2 * s + 1] = r1 >= 0 ? dot1 : 0.f;
      }
    }
  }
}

}  // namespace fsb

static int mr_grid(long long items) {
  const long long blocks = (items + fsb::MR_WARPS - 1) / fsb::MR_WARPS;
  return static_cast<int>(blocks < 148LL * 8 ? blocks : 148LL * 8);
}
// 16-byte accesses need whole vectors per row and aligned bases; a row length or a view that breaks that moves element by element
static bool mr_vec(int M, int size, const void* a, const void* b, const void* c) {
  const uintptr_t ptrs = reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c);
  return (static_cast<long long>(M) * size) % 16 == 0 && (ptrs & 15u) == 0;
}

// route int32 [4, S]; expert / slot int64 [S, 2]; keep bool [S, 2].
FSB_API int fsb_moe_route_pack(const int* route, int S, int C, long long* expert, long long* slot, unsigned char* keep, cudaStream_t stream) {
  using namespace fsb;
  if (S <= 0) return 0;
  moe_route_pack_kernel<<<(2 * S + MR_THREADS - 1) / MR_THREADS, MR_THREADS, 0, stream>>>(route, S, C, expert, slot, keep);
  return static_cast<int>(cudaGetLastError());
}

// expert / slot int64 [S, 2], keep bool [S, 2]; flat int32 [S, 2]; claimed [E * C] bytes.  E * C must fit 31 bits.
FSB_API int fsb_moe_claim_rows(const long long* expert, const long long* slot, const unsigned char* keep, long long S, long long E, long long C, int* flat,
                               unsigned char* claimed, cudaStream_t stream) {
  using namespace fsb;
  if (E * C > 0x7fffffffll) return -1;
  if (E * C > 0) {
    const cudaError_t e = cudaMemsetAsync(claimed, 0, static_cast<size_t>(E * C), stream);
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  if (S <= 0) return 0;
  moe_claim_rows_kernel<<<static_cast<unsigned>((2 * S + MR_THREADS - 1) / MR_THREADS), MR_THREADS, 0, stream>>>(expert, slot, keep, 2 * S, E, C, flat, claimed);
  return static_cast<int>(cudaGetLastError());
}

template <typename T>
static void moe_scatter_t(const void* x, const int* flat, const float* w, long long S, int M, void* out, const unsigned char* claimed, long long rows,
                          cudaStream_t stream) {
  using namespace fsb;
  const int grid = mr_grid(S + rows);
  if (mr_vec(M, sizeof(T), x, out, nullptr))
    moe_scatter_local_kernel<T, 16 / sizeof(T)><<<grid, MR_THREADS, 0, stream>>>(static_cast<const T*>(x), flat, w, S, M, static_cast<T*>(out), claimed, rows);
  else
    moe_scatter_local_kernel<T, 1><<<grid, MR_THREADS, 0, stream>>>(static_cast<const T*>(x), flat, w, S, M, static_cast<T*>(out), claimed, rows);
}

// x [S, M], out [rows, M] (fp32 / fp16 / bf16); w fp32 [S, 2] or null; flat and claimed from fsb_moe_claim_rows.
FSB_API int fsb_moe_scatter_local(const void* x, int dtype, const int* flat, const float* w, long long S, int M, void* out, const unsigned char* claimed,
                                  long long rows, cudaStream_t stream) {
  if (S + rows <= 0 || M <= 0) return 0;
  if (dtype == FSB_F32) moe_scatter_t<float>(x, flat, w, S, M, out, claimed, rows, stream);
  else if (dtype == FSB_F16) moe_scatter_t<__half>(x, flat, w, S, M, out, claimed, rows, stream);
  else if (dtype == FSB_BF16) moe_scatter_t<__nv_bfloat16>(x, flat, w, S, M, out, claimed, rows, stream);
  else return -1;
  return static_cast<int>(cudaGetLastError());
}

template <typename T>
static void moe_gather_t(const void* buf, const int* flat, const float* w, long long S, int M, void* out, const void* g, float* dots, void* kept,
                         cudaStream_t stream) {
  using namespace fsb;
  const int grid = mr_grid(S);
  auto launch = [&](auto kernel) {
    kernel<<<grid, MR_THREADS, 0, stream>>>(static_cast<const T*>(buf), flat, w, S, M, static_cast<T*>(out), static_cast<const T*>(g), dots,
                                            static_cast<T*>(kept));
  };
  if (mr_vec(M, sizeof(T), buf, out, g) && mr_vec(M, sizeof(T), kept, nullptr, nullptr)) launch(moe_gather_local_kernel<T, 16 / sizeof(T)>);
  else launch(moe_gather_local_kernel<T, 1>);
}

// buf [rows, M] with flat from fsb_moe_claim_rows, or [2 * S, M] with flat null: the rows of choice (s, k) are row 2 * s + k.  out
// [S, M] or null; g [S, M] and dots fp32 [S, 2], or both null; kept [2 * S, M] or null.
FSB_API int fsb_moe_gather_local(const void* buf, int dtype, const int* flat, const float* w, long long S, int M, void* out, const void* g, float* dots,
                                 void* kept, cudaStream_t stream) {
  if (S <= 0) return 0;
  if ((g == nullptr) != (dots == nullptr) || 2 * S > 0x7fffffffll) return -1;
  if (dtype == FSB_F32) moe_gather_t<float>(buf, flat, w, S, M, out, g, dots, kept, stream);
  else if (dtype == FSB_F16) moe_gather_t<__half>(buf, flat, w, S, M, out, g, dots, kept, stream);
  else if (dtype == FSB_BF16) moe_gather_t<__nv_bfloat16>(buf, flat, w, S, M, out, g, dots, kept, stream);
  else return -1;
  return static_cast<int>(cudaGetLastError());
}
