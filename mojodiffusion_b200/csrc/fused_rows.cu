// Row kernels around attention: scaled softmax of a score matrix. fp32 arithmetic, 16-byte accesses.
//
// Reference behaviour: serenitymojo/ops/attention.mojo:18-180 (math-mode softmax), serenitymojo/models/dit/ltx2_dit.mojo:518-652
// (norm over the inner dimension, split rotation, 2 * sigmoid head gates).
#include "common.cuh"
#include "kernels_api.h"

namespace mdb {

__device__ __forceinline__ float fr_warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float fr_warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
template <int THREADS, bool MAX>
__device__ __forceinline__ float fr_block(float v, float* red) {
  v = MAX ? fr_warp_max(v) : fr_warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  const int l = threadIdx.x & 31;
  float t = l < THREADS / 32 ? red[l] : (MAX ? -INFINITY : 0.f);
  return MAX ? fr_warp_max(t) : fr_warp_sum(t);
}

// P[r, :] = softmax(S[r, :] * scale) (fp32 scores, bf16 probabilities). One block per row; up to 16384 columns stay in registers
// (CACHED), so the scores are read once; longer rows are read three times, from L2 after the first. Bound by HBM: 6 bytes per
// score. The row maximum ignores NaN scores, their exponentials carry the NaN into the sum and so into the whole row.
constexpr int SM_THREADS = 512, SM_VEC = 8;
template <bool CACHED>
__global__ void __launch_bounds__(SM_THREADS)
softmax_rows_kernel(const float* __restrict__ s, __nv_bfloat16* __restrict__ p, int cols, long long lds, long long ldp, float scale_log2) {
  __shared__ float red[32];
  const float4* sr = reinterpret_cast<const float4*>(s + static_cast<size_t>(blockIdx.x) * lds);
  uint2* pr = reinterpret_cast<uint2*>(p + static_cast<size_t>(blockIdx.x) * ldp);
  const int nv = (cols + 3) >> 2;
  auto load = [&](int i) {                       // scaled scores, columns past the end are -inf
    float4 v = sr[i];
    const int c = i * 4;
    // __fmul_rn: a product fused with the subtraction of the (rounded) maximum would be off by the maximum's rounding
    v.x = __fmul_rn(v.x, scale_log2);
    v.y = c + 1 < cols ? __fmul_rn(v.y, scale_log2) : -INFINITY;
    v.z = c + 2 < cols ? __fmul_rn(v.z, scale_log2) : -INFINITY;
    v.w = c + 3 < cols ? __fmul_rn(v.w, scale_log2) : -INFINITY;
    return v;
  };
  float4 v[CACHED ? SM_VEC : 1];
  float m = -INFINITY;
  if (CACHED) {
#pragma unroll
    for (int k = 0; k < SM_VEC; ++k) {
      const int i = threadIdx.x + k * SM_THREADS;
      v[k] = i < nv ? load(i) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
      m = fmaxf(fmaxf(fmaxf(v[k].x, v[k].y), fmaxf(v[k].z, v[k].w)), m);
    }
  } else {
    for (int i = threadIdx.x; i < nv; i += SM_THREADS) {
      const float4 t = load(i);
      m = fmaxf(fmaxf(fmaxf(t.x, t.y), fmaxf(t.z, t.w)), m);
    }
  }
  m = fr_block<SM_THREADS, true>(m, red);
  float sum = 0.f;
  auto ex = [&](float4 t) { return make_float4(exp2f(t.x - m), exp2f(t.y - m), exp2f(t.z - m), exp2f(t.w - m)); };
  if (CACHED) {
#pragma unroll
    for (int k = 0; k < SM_VEC; ++k) {
      if (threadIdx.x + k * SM_THREADS < nv) {
        v[k] = ex(v[k]);
        sum += (v[k].x + v[k].y) + (v[k].z + v[k].w);
      }
    }
  } else {
    for (int i = threadIdx.x; i < nv; i += SM_THREADS) {
      const float4 t = ex(load(i));
      sum += (t.x + t.y) + (t.z + t.w);
    }
  }
  sum = fr_block<SM_THREADS, false>(sum, red);
  const float inv = 1.f / sum;
  auto put = [&](int i, float4 t) { pr[i] = make_uint2(pack_bf16x2(t.x * inv, t.y * inv), pack_bf16x2(t.z * inv, t.w * inv)); };
  if (CACHED) {
#pragma unroll
    for (int k = 0; k < SM_VEC; ++k) {
      const int i = threadIdx.x + k * SM_THREADS;
      if (i < nv) put(i, v[k]);
    }
  } else {
    for (int i = threadIdx.x; i < nv; i += SM_THREADS) put(i, ex(load(i)));
  }
}

}  // namespace mdb

using namespace mdb;
typedef __nv_bfloat16 bf16;

extern "C" int mdb_softmax_rows(const float* s, void* p, long long rows, int cols, long long lds, long long ldp, float scale, cudaStream_t st) {
  if (cols <= 0 || lds % 4 || ldp % 4 || lds < (cols + 3) / 4 * 4 || ldp < (cols + 3) / 4 * 4 || rows > 2147483647ll) return -1;
  if ((reinterpret_cast<uintptr_t>(s) & 15) || (reinterpret_cast<uintptr_t>(p) & 7)) return -1;
  if (rows <= 0) return 0;
  const float k = scale * 1.4426950408889634f;
  if (cols <= 4 * SM_THREADS * SM_VEC) softmax_rows_kernel<true><<<(unsigned)rows, SM_THREADS, 0, st>>>(s, (bf16*)p, cols, lds, ldp, k);
  else softmax_rows_kernel<false><<<(unsigned)rows, SM_THREADS, 0, st>>>(s, (bf16*)p, cols, lds, ldp, k);
  return (int)cudaGetLastError();
}
