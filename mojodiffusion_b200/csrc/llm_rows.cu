// build: precise-math
// Row kernels of the decoder stack around its projections: per-head RMSNorm + rotary embedding of q and k with the cache append,
// and attention of one query per sequence over that cache. bf16 storage, fp32 arithmetic.
//
// Both work on a few rows, so they are bound by latency: what they save is launches (the same steps as elementwise torch
// operations were 67 launches a layer, and the host could not issue them as fast as the GPU ran them). Exponentials, divisions and
// roundings are the precise ones that those operations use; sums of products are written as fmaf where it matters for time.
//
// Reference behaviour: serenitymojo/llm/decoder.mojo:1-150, serenitymojo/llm/sqa.mojo:1-116.
#include "common.cuh"
#include "kernels_api.h"

namespace mdb {

__device__ __forceinline__ float lr_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// x += y (when y is given), then h = x * rsqrt(mean(x^2) + eps) * w, bf16 rows of up to 16384 columns, one block per row, x in
// place. Sums are fp32; the sum, the normalised value and its product with w are rounded to bf16 one after the other, as the
// separate additions and multiplications of the stack round them.
constexpr int LR_THREADS = 256, LR_VEC = 8;
__device__ __forceinline__ float lr_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
__global__ void __launch_bounds__(LR_THREADS)
add_rms_rows_kernel(__nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ w,
                    __nv_bfloat16* __restrict__ h, int D, float eps) {
  __shared__ float red[LR_THREADS / 32];
  uint4* xr = reinterpret_cast<uint4*>(x + static_cast<size_t>(blockIdx.x) * D);
  const uint4* yr = y ? reinterpret_cast<const uint4*>(y + static_cast<size_t>(blockIdx.x) * D) : nullptr;
  const int nv = D >> 3;
  float ss = 0.f;
  uint4 v[LR_VEC];
#pragma unroll
  for (int k = 0; k < LR_VEC; ++k) {
    const int i = threadIdx.x + k * LR_THREADS;
    if (i < nv) {
      v[k] = xr[i];
      uint32_t* q = reinterpret_cast<uint32_t*>(&v[k]);
      if (yr) {
        const uint4 t = yr[i];
        const uint32_t t4[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = unpack_bf16x2(q[j]), g = unpack_bf16x2(t4[j]);
          q[j] = pack_bf16x2(f.x + g.x, f.y + g.y);
        }
        xr[i] = v[k];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) { const float2 f = unpack_bf16x2(q[j]); ss += f.x * f.x + f.y * f.y; }
    }
  }
  ss = lr_sum(ss);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  ss = 0.f;
#pragma unroll
  for (int i = 0; i < LR_THREADS / 32; ++i) ss += red[i];
  const float rstd = rsqrtf(ss / D + eps);
  uint4* o = reinterpret_cast<uint4*>(h + static_cast<size_t>(blockIdx.x) * D);
  const uint4* wv = reinterpret_cast<const uint4*>(w);
#pragma unroll
  for (int k = 0; k < LR_VEC; ++k) {
    const int i = threadIdx.x + k * LR_THREADS;
    if (i < nv) {
      const uint4 u = wv[i];
      const uint32_t u4[4] = {u.x, u.y, u.z, u.w};
      uint32_t* q = reinterpret_cast<uint32_t*>(&v[k]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(q[j]), g = unpack_bf16x2(u4[j]);
        q[j] = pack_bf16x2(lr_round(f.x * rstd) * g.x, lr_round(f.y * rstd) * g.y);
      }
      o[i] = v[k];
    }
  }
}

// qkv [rows, (H + 2 Hkv) * Dh] (q | k | v), one row per sequence. One warp per (row, head): q heads are normalised and rotated in
// place, k heads go normalised and rotated to k_cache[row, h, pos], v heads as they are to v_cache. Rotation pairs element i with
// i + Dh / 2; table rows are positions ([positions, Dh], bf16).
__global__ void __launch_bounds__(128)
qkv_rope_cache_kernel(__nv_bfloat16* __restrict__ qkv, const __nv_bfloat16* __restrict__ qn, const __nv_bfloat16* __restrict__ kn,
                      const __nv_bfloat16* __restrict__ cosv, const __nv_bfloat16* __restrict__ sinv, __nv_bfloat16* __restrict__ kc,
                      __nv_bfloat16* __restrict__ vc, long long rows, int H, int Hkv, int Dh, int T, int pos, float eps) {
  const int heads = H + 2 * Hkv, lane = threadIdx.x & 31;
  const long long item = blockIdx.x * 4ll + (threadIdx.x >> 5);
  if (item >= rows * heads) return;
  const long long row = item / heads;
  const int h = static_cast<int>(item - row * heads);
  __nv_bfloat16* x = qkv + row * heads * Dh + static_cast<long long>(h) * Dh;
  const int half = Dh >> 1;
  if (h >= H + Hkv) {
    __nv_bfloat16* o = vc + ((row * Hkv + (h - H - Hkv)) * T + pos) * Dh;
    for (int i = lane; i < Dh; i += 32) o[i] = x[i];
    return;
  }
  const __nv_bfloat16* w = h < H ? qn : kn;
  float a[4], c[4], ss = 0.f;                       // Dh <= 256: at most four pairs per lane
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int i = lane + 32 * k;
    a[k] = i < half ? __bfloat162float(x[i]) : 0.f;
    c[k] = i < half ? __bfloat162float(x[i + half]) : 0.f;
    ss += a[k] * a[k] + c[k] * c[k];
  }
  const float rstd = rsqrtf(lr_sum(ss) / Dh + eps);
  __nv_bfloat16* o = h < H ? x : kc + ((row * Hkv + (h - H)) * T + pos) * Dh;
  const __nv_bfloat16 *ct = cosv + static_cast<long long>(pos) * Dh, *st = sinv + static_cast<long long>(pos) * Dh;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int i = lane + 32 * k;
    if (i < half) {
      // rounded to bf16 after each product, as the separate multiplications round
      const float u = lr_round(lr_round(a[k] * rstd) * __bfloat162float(w[i]));
      const float v = lr_round(lr_round(c[k] * rstd) * __bfloat162float(w[i + half]));
      o[i] = __float2bfloat16_rn(lr_round(u * __bfloat162float(ct[i])) - lr_round(v * __bfloat162float(st[i])));
      o[i + half] = __float2bfloat16_rn(lr_round(v * __bfloat162float(ct[i + half])) + lr_round(u * __bfloat162float(st[i + half])));
    }
  }
}

// ---- many rows (a prompt). The stack computes each norm as x.float().pow(2).mean(-1), then scale, round, weight, and every bit of
// a prompt's features depends on the order in which that mean is summed, so the mean stays the torch reduction it was; what is
// fused is what surrounds it, value by value as before: 66 launches a layer become 24. Launches bound it: the prompt of 45 tokens and 36
// layers took 27 ms to issue and 10 to run (prompt and eight tokens: 46.7 -> 37.5 ms on a B200).

// x += y (when y is given, rounded to bf16), sq = x^2 in fp32; n8 groups of eight
__global__ void __launch_bounds__(256)
add_square_kernel(uint4* __restrict__ x, const uint4* __restrict__ y, float4* __restrict__ sq, long long n8) {
  const long long i = blockIdx.x * 256ll + threadIdx.x;
  if (i >= n8) return;
  uint4 v = x[i];
  uint32_t* q = reinterpret_cast<uint32_t*>(&v);
  if (y) {
    const uint4 t = y[i];
    const uint32_t t4[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16x2(q[j]), g = unpack_bf16x2(t4[j]);
      q[j] = pack_bf16x2(f.x + g.x, f.y + g.y);
    }
    x[i] = v;
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const float2 f = unpack_bf16x2(q[2 * j]), g = unpack_bf16x2(q[2 * j + 1]);
    sq[2 * i + j] = make_float4(f.x * f.x, f.y * f.y, g.x * g.x, g.y * g.y);
  }
}

// h = x * rsqrt(mean + eps) rounded, times w rounded; one block per row
__global__ void __launch_bounds__(128)
rms_scale_kernel(const uint4* __restrict__ x, const float* __restrict__ mean, const uint4* __restrict__ w, uint4* __restrict__ h, int nv, float eps) {
  const float rstd = rsqrtf(mean[blockIdx.x] + eps);
  const size_t base = static_cast<size_t>(blockIdx.x) * nv;
  for (int i = threadIdx.x; i < nv; i += 128) {
    uint4 v = x[base + i];
    const uint4 u = w[i];
    const uint32_t u4[4] = {u.x, u.y, u.z, u.w};
    uint32_t* q = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16x2(q[j]), g = unpack_bf16x2(u4[j]);
      q[j] = pack_bf16x2(lr_round(f.x * rstd) * g.x, lr_round(f.y * rstd) * g.y);
    }
    h[base + i] = v;
  }
}

// squares of the q and k heads of packed rows [rows, (H + 2 Hkv) * Dh] -> sq_q [rows, H * Dh], sq_k [rows, Hkv * Dh]; n pairs
__global__ void __launch_bounds__(256)
square_heads_kernel(const uint32_t* __restrict__ qkv, float2* __restrict__ sq_q, float2* __restrict__ sq_k, long long n, int q2, int kv2) {
  const long long i = blockIdx.x * 256ll + threadIdx.x;
  if (i >= n) return;
  const long long row = i / (q2 + kv2);
  const int c = static_cast<int>(i - row * (q2 + kv2));
  const float2 f = unpack_bf16x2(qkv[row * (q2 + 2 * kv2) + c]);
  const float2 s = make_float2(f.x * f.x, f.y * f.y);
  if (c < q2) sq_q[row * q2 + c] = s; else sq_k[row * kv2 + c - q2] = s;
}

// packed rows of a prompt (row = b * S + s), one warp per (row, head): q normalised and rotated -> qo [rows, H, Dh]; k normalised and
// rotated, v as it is -> caches [B, Hkv, T, Dh] at position s, and once per query head of the group -> kr, vr [B, H, S, Dh]
__global__ void __launch_bounds__(128)
prompt_rope_cache_kernel(const __nv_bfloat16* __restrict__ qkv, const float* __restrict__ mean_q, const float* __restrict__ mean_k,
                         const __nv_bfloat16* __restrict__ qn, const __nv_bfloat16* __restrict__ kn, const __nv_bfloat16* __restrict__ cosv,
                         const __nv_bfloat16* __restrict__ sinv, __nv_bfloat16* __restrict__ qo, __nv_bfloat16* __restrict__ kr,
                         __nv_bfloat16* __restrict__ vr, __nv_bfloat16* __restrict__ kc, __nv_bfloat16* __restrict__ vc, long long rows, int S, int H,
                         int Hkv, int Dh, int T, float eps) {
  const int heads = H + 2 * Hkv, lane = threadIdx.x & 31, half = Dh >> 1, rep = H / Hkv;
  const long long item = blockIdx.x * 4ll + (threadIdx.x >> 5);
  if (item >= rows * heads) return;
  const long long row = item / heads, b = row / S;
  const int h = static_cast<int>(item - row * heads), s = static_cast<int>(row - b * S);
  const __nv_bfloat16* x = qkv + row * heads * Dh + static_cast<long long>(h) * Dh;
  const bool is_v = h >= H + Hkv;
  const int g = is_v ? h - H - Hkv : h - H;                       // key / value head
  if (is_v) {
    for (int i = lane; i < Dh; i += 32) {
      const __nv_bfloat16 v = x[i];
      vc[((b * Hkv + g) * T + s) * Dh + i] = v;
      for (int r = 0; r < rep; ++r) vr[((b * H + g * rep + r) * S + s) * Dh + i] = v;
    }
    return;
  }
  const __nv_bfloat16* w = h < H ? qn : kn;
  const float rstd = rsqrtf((h < H ? mean_q[row * H + h] : mean_k[row * Hkv + g]) + eps);
  const __nv_bfloat16 *ct = cosv + static_cast<long long>(s) * Dh, *st = sinv + static_cast<long long>(s) * Dh;
  for (int i = lane; i < half; i += 32) {
    const float u = lr_round(lr_round(__bfloat162float(x[i]) * rstd) * __bfloat162float(w[i]));
    const float v = lr_round(lr_round(__bfloat162float(x[i + half]) * rstd) * __bfloat162float(w[i + half]));
    const __nv_bfloat16 lo = __float2bfloat16_rn(lr_round(u * __bfloat162float(ct[i])) - lr_round(v * __bfloat162float(st[i])));
    const __nv_bfloat16 hi = __float2bfloat16_rn(lr_round(v * __bfloat162float(ct[i + half])) + lr_round(u * __bfloat162float(st[i + half])));
    if (h < H) {
      __nv_bfloat16* o = qo + (row * H + h) * Dh;
      o[i] = lo;
      o[i + half] = hi;
    } else {
      __nv_bfloat16* o = kc + ((b * Hkv + g) * T + s) * Dh;
      o[i] = lo;
      o[i + half] = hi;
      for (int r = 0; r < rep; ++r) {
        __nv_bfloat16* k = kr + ((b * H + g * rep + r) * S + s) * Dh;
        k[i] = lo;
        k[i + half] = hi;
      }
    }
  }
}

// One query per (sequence, head) over the first ``len`` cache rows of its key / value head: scores and probabilities in fp32 in
// shared memory, sums in fp32. Eight lanes share a key (16-byte loads), so a block of 16 warps scores 64 keys at a time; for the
// weighted sum Dh / 8 lanes cover a value row and the remaining groups of threads split the keys.
constexpr int DA_THREADS = 512;
__global__ void __launch_bounds__(DA_THREADS)
decode_attention_kernel(const __nv_bfloat16* __restrict__ q, long long ldq, const __nv_bfloat16* __restrict__ kc, const __nv_bfloat16* __restrict__ vc,
                        __nv_bfloat16* __restrict__ o, int H, int Hkv, int Dh, int T, int len, float scale) {
  extern __shared__ float da_sm[];                  // [len rounded up to 4] probabilities, then [groups][Dh] partial sums
  __shared__ float red[DA_THREADS / 32];
  const int h = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long b = blockIdx.y;
  const long long kv = (b * Hkv + h / (H / Hkv)) * static_cast<long long>(T) * Dh;
  const __nv_bfloat16* qr = q + b * ldq + static_cast<long long>(h) * Dh;
  const int sub = lane & 7;
  float qf[4][8];                                   // Dh <= 256: vectors sub, sub + 8, ... of the query
  const int nv = Dh >> 3;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int v = sub + 8 * k;
    const uint4 u = v < nv ? *reinterpret_cast<const uint4*>(qr + v * 8) : make_uint4(0, 0, 0, 0);
    const uint32_t u4[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) { const float2 f = unpack_bf16x2(u4[j]); qf[k][2 * j] = f.x; qf[k][2 * j + 1] = f.y; }
  }
  float m = -INFINITY;
  const int rounds = (len + DA_THREADS / 8 - 1) / (DA_THREADS / 8);
  for (int r = 0; r < rounds; ++r) {                // whole warps take part in the shuffles
    const int t = r * (DA_THREADS / 8) + warp * 4 + (lane >> 3);
    float acc = 0.f;
    if (t < len) {
      const __nv_bfloat16* kr = kc + kv + static_cast<long long>(t) * Dh;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int v = sub + 8 * k;
        if (v < nv) {
          const uint4 u = *reinterpret_cast<const uint4*>(kr + v * 8);
          const uint32_t u4[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) { const float2 f = unpack_bf16x2(u4[j]); acc = fmaf(qf[k][2 * j], f.x, acc); acc = fmaf(qf[k][2 * j + 1], f.y, acc); }
        }
      }
    }
    acc += __shfl_xor_sync(0xffffffffu, acc, 4);
    acc += __shfl_xor_sync(0xffffffffu, acc, 2);
    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
    acc *= scale;
    if (t < len) {
      m = fmaxf(m, acc);
      if (sub == 0) da_sm[t] = acc;
    }
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, s));
  if (lane == 0) red[warp] = m;
  __syncthreads();
  m = red[0];
#pragma unroll
  for (int i = 1; i < DA_THREADS / 32; ++i) m = fmaxf(m, red[i]);
  __syncthreads();
  float sum = 0.f;
  for (int t = threadIdx.x; t < len; t += DA_THREADS) {
    const float e = expf(da_sm[t] - m);
    da_sm[t] = e;
    sum += e;
  }
  sum = lr_sum(sum);
  if (lane == 0) red[warp] = sum;
  __syncthreads();
  sum = 0.f;
#pragma unroll
  for (int i = 0; i < DA_THREADS / 32; ++i) sum += red[i];
  const float inv = 1.f / sum;
  const int groups = DA_THREADS / nv, g = threadIdx.x / nv, v = threadIdx.x % nv;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (g < groups) {
#pragma unroll 4
    for (int t = g; t < len; t += groups) {
      const uint4 u = *reinterpret_cast<const uint4*>(vc + kv + static_cast<long long>(t) * Dh + v * 8);
      const float p = da_sm[t];
      const uint32_t u4[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) { const float2 f = unpack_bf16x2(u4[j]); acc[2 * j] = fmaf(p, f.x, acc[2 * j]); acc[2 * j + 1] = fmaf(p, f.y, acc[2 * j + 1]); }
    }
    float* part = da_sm + ((len + 3) & ~3) + g * Dh + v * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) part[j] = acc[j];
  }
  __syncthreads();
  for (int d = threadIdx.x; d < Dh; d += DA_THREADS) {
    float t = 0.f;
    for (int i = 0; i < groups; ++i) t += da_sm[((len + 3) & ~3) + i * Dh + d];
    o[(b * H + h) * Dh + d] = __float2bfloat16_rn(t * inv);
  }
}

}  // namespace mdb

using namespace mdb;
typedef __nv_bfloat16 bf16;

extern "C" int mdb_add_rms_rows(void* x, const void* y, const void* w, void* h, long long rows, int D, float eps, cudaStream_t st) {
  if (D % 8 || D <= 0 || D > 8 * LR_THREADS * LR_VEC || rows > 2147483647ll ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(w)) & 15))
    return -1;
  if (rows <= 0) return 0;
  add_rms_rows_kernel<<<(unsigned)rows, LR_THREADS, 0, st>>>((bf16*)x, (const bf16*)y, (const bf16*)w, (bf16*)h, D, eps);
  return (int)cudaGetLastError();
}

extern "C" int mdb_qkv_rope_cache(void* qkv, const void* qn, const void* kn, const void* cosv, const void* sinv, void* kc, void* vc, long long rows, int H,
                                  int Hkv, int Dh, int T, int pos, float eps, cudaStream_t st) {
  if (Dh % 2 || Dh > 256 || Dh <= 0 || Hkv <= 0 || pos < 0 || pos >= T || !qn || !kn) return -1;
  const long long blocks = (rows * (H + 2 * Hkv) + 3) / 4;
  if (blocks <= 0) return 0;
  if (blocks > 2147483647ll) return -1;
  qkv_rope_cache_kernel<<<(unsigned)blocks, 128, 0, st>>>((bf16*)qkv, (const bf16*)qn, (const bf16*)kn, (const bf16*)cosv, (const bf16*)sinv, (bf16*)kc,
                                                          (bf16*)vc, rows, H, Hkv, Dh, T, pos, eps);
  return (int)cudaGetLastError();
}

extern "C" int mdb_add_square(void* x, const void* y, float* sq, long long n, cudaStream_t st) {
  if (n % 8 || n / 2048 >= 2147483647ll || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(sq)) & 15)) return -1;
  if (n <= 0) return 0;
  add_square_kernel<<<(unsigned)((n / 8 + 255) / 256), 256, 0, st>>>((uint4*)x, (const uint4*)y, (float4*)sq, n / 8);
  return (int)cudaGetLastError();
}
extern "C" int mdb_rms_scale(const void* x, const float* mean, const void* w, void* h, long long rows, int D, float eps, cudaStream_t st) {
  if (D % 8 || D <= 0 || rows > 2147483647ll || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(h)) & 15)) return -1;
  if (rows <= 0) return 0;
  rms_scale_kernel<<<(unsigned)rows, 128, 0, st>>>((const uint4*)x, mean, (const uint4*)w, (uint4*)h, D / 8, eps);
  return (int)cudaGetLastError();
}
extern "C" int mdb_square_heads(const void* qkv, float* sq_q, float* sq_k, long long rows, int H, int Hkv, int Dh, cudaStream_t st) {
  const long long n = rows * (H + Hkv) * (Dh / 2);
  if (Dh % 2 || Dh <= 0 || n / 256 >= 2147483647ll) return -1;
  if (n <= 0) return 0;
  square_heads_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>((const uint32_t*)qkv, (float2*)sq_q, (float2*)sq_k, n, H * Dh / 2, Hkv * Dh / 2);
  return (int)cudaGetLastError();
}
extern "C" int mdb_prompt_rope_cache(const void* qkv, const float* mean_q, const float* mean_k, const void* qn, const void* kn, const void* cosv,
                                     const void* sinv, void* qo, void* kr, void* vr, void* kc, void* vc, int B, int S, int H, int Hkv, int Dh, int T,
                                     float eps, cudaStream_t st) {
  if (Dh % 2 || Dh <= 0 || Hkv <= 0 || H % Hkv || S > T || !qn || !kn) return -1;
  const long long rows = static_cast<long long>(B) * S, blocks = (rows * (H + 2 * Hkv) + 3) / 4;
  if (blocks <= 0) return 0;
  if (blocks > 2147483647ll) return -1;
  prompt_rope_cache_kernel<<<(unsigned)blocks, 128, 0, st>>>((const bf16*)qkv, mean_q, mean_k, (const bf16*)qn, (const bf16*)kn, (const bf16*)cosv,
                                                             (const bf16*)sinv, (bf16*)qo, (bf16*)kr, (bf16*)vr, (bf16*)kc, (bf16*)vc, rows, S, H, Hkv, Dh, T, eps);
  return (int)cudaGetLastError();
}

// shared memory one block needs; a cache longer than MDB_DECODE_ATTENTION_MAX rows stays on the torch statement
extern "C" int mdb_decode_attention(const void* q, long long ldq, const void* kc, const void* vc, void* o, int B, int H, int Hkv, int Dh, int T, int len,
                                    float scale, cudaStream_t st) {
  if (Dh % 8 || Dh > 256 || Dh <= 0 || Hkv <= 0 || H % Hkv || len <= 0 || len > T || len > MDB_DECODE_ATTENTION_MAX || ldq % 8 || B > 65535) return -1;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(kc) | reinterpret_cast<uintptr_t>(vc)) & 15) return -1;
  if (B <= 0) return 0;
  const int groups = DA_THREADS / (Dh / 8);
  const size_t smem = (((len + 3) & ~3) + static_cast<size_t>(groups) * Dh) * sizeof(float);
  decode_attention_kernel<<<dim3(H, B), DA_THREADS, smem, st>>>((const bf16*)q, ldq, (const bf16*)kc, (const bf16*)vc, (bf16*)o, H, Hkv, Dh, T, len, scale);
  return (int)cudaGetLastError();
}
