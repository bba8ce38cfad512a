// build: precise-math
// Row kernels that replace chains of elementwise passes around attention: scaled softmax of a score matrix, full-width
// RMSNorm + rotary embedding of packed q and k in place, per-head output gates. bf16 tensors, fp32 arithmetic, 16-byte
// accesses; each element crosses memory once per direction. Built without fast math: the torch operations that these kernels
// replace use the precise exponential and division.
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

// P[r, :] = softmax(S[r, :] * scale) (fp32 scores, bf16 probabilities and, when asked for, what their rounding left as a second bf16
// row: two terms hold a probability to 2^-17). One block per row; up to 16384 columns stay in registers
// (CACHED), so the scores are read once; longer rows are read three times, from L2 after the first. Bound by HBM: 6 bytes per
// score. The row maximum ignores NaN scores, their exponentials carry the NaN into the sum and so into the whole row.
constexpr int SM_THREADS = 512, SM_VEC = 8;
template <bool CACHED>
__global__ void __launch_bounds__(SM_THREADS)
softmax_rows_kernel(const float* __restrict__ s, __nv_bfloat16* __restrict__ p, __nv_bfloat16* __restrict__ low, int cols, long long lds, long long ldp,
                    float scale_log2) {
  __shared__ float red[32];
  const float* sr = s + static_cast<size_t>(blockIdx.x) * lds;
  __nv_bfloat16* pr = p + static_cast<size_t>(blockIdx.x) * ldp;
  __nv_bfloat16* lr = low ? low + static_cast<size_t>(blockIdx.x) * ldp : nullptr;
  const int nv = (cols + 3) >> 2;
  auto load = [&](int i) {                       // scaled scores; columns past the end are not touched and count as -inf
    const int c = i * 4;
    float4 v;
    if (c + 3 < cols) {
      v = *reinterpret_cast<const float4*>(sr + c);
    } else {
      v = make_float4(sr[c], -INFINITY, -INFINITY, -INFINITY);
      if (c + 1 < cols) v.y = sr[c + 1];
      if (c + 2 < cols) v.z = sr[c + 2];
    }
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
  auto store = [&](__nv_bfloat16* row, int c, uint2 q) {
    if (c + 3 < cols) {
      *reinterpret_cast<uint2*>(row + c) = q;
    } else {
      const __nv_bfloat162 *h0 = reinterpret_cast<const __nv_bfloat162*>(&q.x), *h1 = reinterpret_cast<const __nv_bfloat162*>(&q.y);
      row[c] = h0->x;
      if (c + 1 < cols) row[c + 1] = h0->y;
      if (c + 2 < cols) row[c + 2] = h1->x;
    }
  };
  auto put = [&](int i, float4 t) {
    t = make_float4(t.x * inv, t.y * inv, t.z * inv, t.w * inv);
    const uint2 q = make_uint2(pack_bf16x2(t.x, t.y), pack_bf16x2(t.z, t.w));
    store(pr, i * 4, q);
    if (lr) {
      const float2 a = unpack_bf16x2(q.x), b = unpack_bf16x2(q.y);
      store(lr, i * 4, make_uint2(pack_bf16x2(t.x - a.x, t.y - a.y), pack_bf16x2(t.z - b.x, t.w - b.y)));
    }
  };
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

// In place on a packed projection row: RMSNorm over all D columns of q (blockIdx.y 0) and k (1), times a weight, then the
// split-half rotation inside each head of Dh columns. A work item is 8 columns of a head's first half with the 8 columns Dh / 2
// further, so both halves of a rotation are in one thread; a row of 4096 columns is one item per thread. Replaces two norms
// into fresh buffers, two copies back into the packed rows and a rotation pass (six passes over q and k: 232 us per layer at
// 6144 x 4096) by one: 119 us with room for four items per thread, 61 where one is enough (201 MB: 3.3 TB/s, bound by the chain of
// load, two barriers and store of a row; 52 us under ncu from cold caches).
// A block has as many threads as the row has items, up to 256 (rows of 256 columns: 16 items; a block of 256 threads for them made
// the pass slower than the separate operations, 238 against 206 us for an attention of 6144 tokens).
constexpr int NR_THREADS = 256, NR_ITEMS = 4;
template <int THREADS, int ITEMS>
__global__ void __launch_bounds__(THREADS)
rms_rope_rows_kernel(__nv_bfloat16* __restrict__ buf, const __nv_bfloat16* __restrict__ wq, const __nv_bfloat16* __restrict__ wk,
                     const float* __restrict__ cosv, const float* __restrict__ sinv, long long ld, int D, int Dh, int q_off, int k_off,
                     int rows_per_batch, float eps) {
  __shared__ float red[32];
  const long long row = blockIdx.x;
  const __nv_bfloat16* w = blockIdx.y ? wk : wq;
  __nv_bfloat16* x = buf + row * ld + (blockIdx.y ? k_off : q_off);
  const int half = Dh >> 1, per_head = half >> 3, items = D >> 4;
  float a[ITEMS][8], b[ITEMS][8];
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const int i = threadIdx.x + k * THREADS;
    if (i < items) {
      const int c = (i / per_head) * Dh + (i % per_head) * 8;
      const uint4 u = *reinterpret_cast<const uint4*>(x + c), t = *reinterpret_cast<const uint4*>(x + c + half);
      const uint32_t u4[4] = {u.x, u.y, u.z, u.w}, t4[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(u4[j]), g = unpack_bf16x2(t4[j]);
        a[k][2 * j] = f.x; a[k][2 * j + 1] = f.y;
        b[k][2 * j] = g.x; b[k][2 * j + 1] = g.y;
        ss += f.x * f.x + f.y * f.y + g.x * g.x + g.y * g.y;
      }
    }
  }
  ss = fr_block<THREADS, false>(ss, red);
  const float rstd = rsqrtf(ss / D + eps);
  const size_t tok = static_cast<size_t>(row % rows_per_batch) * half;
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const int i = threadIdx.x + k * THREADS;
    if (i < items) {
      const int h0 = (i % per_head) * 8, c = (i / per_head) * Dh + h0;
      const uint4 wa = *reinterpret_cast<const uint4*>(w + c), wb = *reinterpret_cast<const uint4*>(w + c + half);
      const float4 c0 = *reinterpret_cast<const float4*>(cosv + tok + h0), c1 = *reinterpret_cast<const float4*>(cosv + tok + h0 + 4);
      const float4 s0 = *reinterpret_cast<const float4*>(sinv + tok + h0), s1 = *reinterpret_cast<const float4*>(sinv + tok + h0 + 4);
      const float cs[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w}, sn[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
      const uint32_t wa4[4] = {wa.x, wa.y, wa.z, wa.w}, wb4[4] = {wb.x, wb.y, wb.z, wb.w};
      uint32_t u4[4], t4[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 fa = unpack_bf16x2(wa4[j]), fb = unpack_bf16x2(wb4[j]);
        const float a0 = a[k][2 * j] * rstd * fa.x, a1 = a[k][2 * j + 1] * rstd * fa.y;
        const float b0 = b[k][2 * j] * rstd * fb.x, b1 = b[k][2 * j + 1] * rstd * fb.y;
        u4[j] = pack_bf16x2(a0 * cs[2 * j] - b0 * sn[2 * j], a1 * cs[2 * j + 1] - b1 * sn[2 * j + 1]);
        t4[j] = pack_bf16x2(b0 * cs[2 * j] + a0 * sn[2 * j], b1 * cs[2 * j + 1] + a1 * sn[2 * j + 1]);
      }
      *reinterpret_cast<uint4*>(x + c) = make_uint4(u4[0], u4[1], u4[2], u4[3]);
      *reinterpret_cast<uint4*>(x + c + half) = make_uint4(t4[0], t4[1], t4[2], t4[3]);
    }
  }
}

// o[row, h, :] *= 2 * sigmoid(logit[row, h]), in place; one 16-byte vector per thread step
__global__ void __launch_bounds__(256)
head_gate_kernel(__nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ logit, long long vecs, int H, int Dh, long long ld_logit) {
  const int hv = Dh >> 3, rv = H * hv;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < vecs; i += gridDim.x * 256ll) {
    const long long row = i / rv;
    const int h = static_cast<int>(i - row * rv) / hv;
    const float g = 2.f * (1.f / (1.f + expf(-__bfloat162float(logit[row * ld_logit + h]))));
    uint4* q = reinterpret_cast<uint4*>(o) + i;
    const uint4 u = *q;
    uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16x2(w[j]);
      w[j] = pack_bf16x2(f.x * g, f.y * g);
    }
    *q = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

}  // namespace mdb

using namespace mdb;
typedef __nv_bfloat16 bf16;

extern "C" int mdb_softmax_rows(const float* s, void* p, void* low, long long rows, int cols, long long lds, long long ldp, float scale, cudaStream_t st) {
  if (cols <= 0 || lds % 4 || ldp % 4 || lds < cols || ldp < cols || rows > 2147483647ll) return -1;
  if ((reinterpret_cast<uintptr_t>(s) & 15) || ((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(low)) & 7)) return -1;
  if (rows <= 0) return 0;
  const float k = scale * 1.4426950408889634f;
  if (cols <= 4 * SM_THREADS * SM_VEC) softmax_rows_kernel<true><<<(unsigned)rows, SM_THREADS, 0, st>>>(s, (bf16*)p, (bf16*)low, cols, lds, ldp, k);
  else softmax_rows_kernel<false><<<(unsigned)rows, SM_THREADS, 0, st>>>(s, (bf16*)p, (bf16*)low, cols, lds, ldp, k);
  return (int)cudaGetLastError();
}

extern "C" int mdb_rms_rope_rows(void* buf, const void* wq, const void* wk, const float* cosv, const float* sinv, long long rows, long long ld, int D,
                                 int Dh, int q_off, int k_off, int rows_per_batch, float eps, cudaStream_t st) {
  if (D % Dh || Dh % 16 || (D >> 4) > NR_THREADS * NR_ITEMS || ld % 8 || q_off % 8 || k_off % 8 || (reinterpret_cast<uintptr_t>(buf) & 15) ||
      ((reinterpret_cast<uintptr_t>(wq) | reinterpret_cast<uintptr_t>(wk) | reinterpret_cast<uintptr_t>(cosv) | reinterpret_cast<uintptr_t>(sinv)) & 15) ||
      rows_per_batch <= 0 || rows > 2147483647ll)
    return -1;
  if (rows <= 0) return 0;
  const int items = D >> 4;
  auto kern = items <= 32    ? rms_rope_rows_kernel<32, 1>
              : items <= 64  ? rms_rope_rows_kernel<64, 1>
              : items <= 128 ? rms_rope_rows_kernel<128, 1>
              : items <= 256 ? rms_rope_rows_kernel<NR_THREADS, 1>
                             : rms_rope_rows_kernel<NR_THREADS, NR_ITEMS>;
  const int threads = items <= 32 ? 32 : items <= 64 ? 64 : items <= 128 ? 128 : NR_THREADS;
  kern<<<dim3((unsigned)rows, 2), threads, 0, st>>>((bf16*)buf, (const bf16*)wq, (const bf16*)wk, cosv, sinv, ld, D, Dh, q_off, k_off, rows_per_batch, eps);
  return (int)cudaGetLastError();
}

extern "C" int mdb_head_gate(void* o, const void* logit, long long rows, int H, int Dh, long long ld_logit, cudaStream_t st) {
  if (Dh % 8 || (reinterpret_cast<uintptr_t>(o) & 15)) return -1;
  const long long vecs = rows * H * (Dh / 8);
  if (vecs <= 0) return 0;
  long long blocks = (vecs + 255) / 256;
  const long long cap = 16ll * device_sm_count();
  head_gate_kernel<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, st>>>((bf16*)o, (const bf16*)logit, vecs, H, Dh, ld_logit);
  return (int)cudaGetLastError();
}
