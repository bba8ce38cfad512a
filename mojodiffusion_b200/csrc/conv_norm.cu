// NHWC image kernels around the implicit-GEMM convolution: GroupNorm fused with SiLU, nearest 2x upsample,
// pixel shuffle / unshuffle, 2x2 average pool. 128-bit accesses, fp32 statistics.
//
// Reference behaviour: serenitymojo/ops/norm.mojo:855-1049 (NHWC GroupNorm(32)), serenitymojo/models/vae/upsample.mojo
// (nearest 2x), serenitymojo/ops/pixelshuffle.mojo:144-770, serenitymojo/models/vae/decoder2d.mojo:150-362 (how the
// ResnetBlock uses GN -> SiLU -> conv).
#include "common.cuh"
#include "kernels_api.h"

namespace mdb {

// stats[n, g] = (mean, rstd) over H*W*(C/G) elements. One block per (n, g).
__global__ void __launch_bounds__(256)
group_norm_stats_kernel(const __nv_bfloat16* __restrict__ x, float* __restrict__ stats, int HW, int C, int G, float eps) {
  const int n = blockIdx.x / G, g = blockIdx.x % G;
  const int cpg = C / G;
  const __nv_bfloat16* base = x + static_cast<size_t>(n) * HW * C + g * cpg;
  const int vec = cpg >> 3;  // cpg is a multiple of 8 on the vector path, else scalar
  float s = 0.f, ss = 0.f;
  if (vec > 0 && (cpg & 7) == 0) {
    const long long total = static_cast<long long>(HW) * vec;
    for (long long i = threadIdx.x; i < total; i += blockDim.x) {
      const int p = static_cast<int>(i / vec), v = static_cast<int>(i % vec);
      const uint4 u = *reinterpret_cast<const uint4*>(base + static_cast<size_t>(p) * C + v * 8);
      const uint32_t w4[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 f = unpack_bf16x2(w4[k]);
        s += f.x + f.y;
        ss += f.x * f.x + f.y * f.y;
      }
    }
  } else {
    const long long total = static_cast<long long>(HW) * cpg;
    for (long long i = threadIdx.x; i < total; i += blockDim.x) {
      const float f = __bfloat162float(base[(i / cpg) * C + (i % cpg)]);
      s += f;
      ss += f * f;
    }
  }
  __shared__ float rs[8], rss[8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    ss += __shfl_xor_sync(0xffffffffu, ss, o);
  }
  if ((threadIdx.x & 31) == 0) {
    rs[threadIdx.x >> 5] = s;
    rss[threadIdx.x >> 5] = ss;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float a = 0.f, b = 0.f;
    for (int i = 0; i < 8; ++i) {
      a += rs[i];
      b += rss[i];
    }
    const float cnt = static_cast<float>(HW) * cpg;
    const float mean = a / cnt;
    const float var = fmaxf(b / cnt - mean * mean, 0.f);
    stats[2 * blockIdx.x] = mean;
    stats[2 * blockIdx.x + 1] = rsqrtf(var + eps);
  }
}

// Statistics over many blocks: a block takes a range of pixels of one sample for a slab of ``sv`` 8-channel vectors that ends
// on a group boundary (all channels up to 2048 of them; each thread owns one vector and strides over the pixels: 128-bit
// coalesced loads, four in flight). Its per-channel partials are reduced in a fixed order (over the pixel lanes, then over the
// channels of a group) and written to part[n, chunk, g] = (sum, sum of squares); a second kernel adds the chunks, one warp per
// group, and turns them into (mean, rstd). No atomics: the result does not depend on scheduling. One block per (sample,
// group), as the kernel above, leaves most of the device idle for a 1024 x 1024 x 128 image (32 blocks, and 4 channels per
// group defeat its vector path).
__global__ void __launch_bounds__(256)
group_norm_partial_kernel(const __nv_bfloat16* __restrict__ x, float* __restrict__ part, int HW, int C, int G, int ppb, int sv) {
  extern __shared__ float gsm[];                 // [256][16] per-thread channel partials, then [8 * sv][2] channel sums
  const int n = blockIdx.y, cpg = C / G, v0 = blockIdx.z * sv;
  const int cv = min(sv, (C >> 3) - v0);         // vectors of this slab
  const int lanes = blockDim.x / cv;
  float s[8], ss[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) s[k] = ss[k] = 0.f;
  if (static_cast<int>(threadIdx.x) < lanes * cv) {
    const int v = threadIdx.x % cv, pl = threadIdx.x / cv;
    const int p0 = blockIdx.x * ppb, p1 = min(p0 + ppb, HW);
    const __nv_bfloat16* base = x + (static_cast<size_t>(n) * HW) * C + (v0 + v) * 8;
#pragma unroll 4
    for (int p = p0 + pl; p < p1; p += lanes) {
      const uint4 u = *reinterpret_cast<const uint4*>(base + static_cast<size_t>(p) * C);
      const uint32_t w4[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 f = unpack_bf16x2(w4[k]);
        s[2 * k] += f.x; ss[2 * k] += f.x * f.x;
        s[2 * k + 1] += f.y; ss[2 * k + 1] += f.y * f.y;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) { gsm[threadIdx.x * 16 + k] = s[k]; gsm[threadIdx.x * 16 + 8 + k] = ss[k]; }
  __syncthreads();
  float* csum = gsm + 256 * 16;
  for (int c = threadIdx.x; c < 8 * cv; c += blockDim.x) {
    const int v = c >> 3, k = c & 7;
    float a = 0.f, b = 0.f;
    for (int pl = 0; pl < lanes; ++pl) { a += gsm[(pl * cv + v) * 16 + k]; b += gsm[(pl * cv + v) * 16 + 8 + k]; }
    csum[2 * c] = a; csum[2 * c + 1] = b;
  }
  __syncthreads();
  float* out = part + (static_cast<size_t>(n) * gridDim.x + blockIdx.x) * 2 * G;
  const int g0 = v0 * 8 / cpg;
  for (int g = threadIdx.x; g < cv * 8 / cpg; g += blockDim.x) {
    float a = 0.f, b = 0.f;
    for (int c = g * cpg; c < (g + 1) * cpg; ++c) { a += csum[2 * c]; b += csum[2 * c + 1]; }
    out[2 * (g0 + g)] = a; out[2 * (g0 + g) + 1] = b;
  }
}
// stats[n, g] = (mean, rstd) (or, with cnt <= 0, the raw sums) from the chunk partials: one warp per (sample, group), each lane
// adds every 32nd chunk, the lanes are joined in a fixed order. (One thread per group walked up to 592 chunks one load after
// the other: 38 us per call on the 1024 x 1024 decoder, as long as the pass over the image.)
__global__ void __launch_bounds__(256)
group_norm_finalize_kernel(const float* __restrict__ part, float* __restrict__ stats, int N, int G, int chunks, int stride,
                           float cnt, float eps) {
  const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (i >= N * G) return;
  const int n = i / G, g = i % G;
  float a = 0.f, b = 0.f;
#pragma unroll 4
  for (int c = lane; c < chunks; c += 32) {
    const float* p = part + (static_cast<size_t>(n) * chunks + c) * stride + 2 * g;
    a += p[0]; b += p[1];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if (lane != 0) return;
  if (cnt > 0.f) {
    const float mean = a / cnt;
    const float var = fmaxf(b / cnt - mean * mean, 0.f);
    stats[2 * i] = mean;
    stats[2 * i + 1] = rsqrtf(var + eps);
  } else {
    stats[2 * i] = a;
    stats[2 * i + 1] = b;
  }
}

// y = act((x - mean) * rstd * w[c] + b[c]); act 0 none, 2 SiLU. A thread keeps one 8-channel vector (its mean, rstd, w and b
// in registers) and walks the pixels, four loads in flight, so the loop is one 16-byte load, three operations per channel, the
// activation and one store. rstd and w are not multiplied beforehand: their product can overflow where no result does. (The earlier form re-derived channel, group and sample by division for every element: 99 us per
// call on the 1024 x 1024 decoder where the bytes need about 45.)
__global__ void __launch_bounds__(256)
group_norm_apply_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y,
                        const float* __restrict__ stats, const __nv_bfloat16* __restrict__ w,
                        const __nv_bfloat16* __restrict__ b, int HW, int C, int G, int act, int ppb, int sv) {
  const int n = blockIdx.y, cpg = C / G, v0 = blockIdx.z * sv;
  const int cv = min(sv, (C >> 3) - v0), lanes = blockDim.x / cv;
  if (static_cast<int>(threadIdx.x) >= lanes * cv) return;
  const int v = v0 + threadIdx.x % cv, p0 = blockIdx.x * ppb, p1 = min(p0 + ppb, HW), first = p0 + threadIdx.x / cv;
  const size_t base = (static_cast<size_t>(n) * HW) * C + v * 8;
  auto load = [&](int p) { return *reinterpret_cast<const uint4*>(x + base + static_cast<size_t>(p) * C); };
  // a small image is one vector per thread: requested before the parameters, its pass is one memory latency shorter
  const bool single = ppb <= lanes;
  const uint4 u0 = single && first < p1 ? load(first) : make_uint4(0, 0, 0, 0);
  float mean[8], rstd[8], mul[8], add[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int c = v * 8 + k, g = c / cpg;
    mean[k] = stats[2 * (n * G + g)];
    rstd[k] = stats[2 * (n * G + g) + 1];
    mul[k] = w ? __bfloat162float(w[c]) : 1.f;
    add[k] = w && b ? __bfloat162float(b[c]) : 0.f;
  }
  auto put = [&](int p, uint4 u) {
    const uint32_t w4[4] = {u.x, u.y, u.z, u.w};
    uint32_t o4[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 f = unpack_bf16x2(w4[k]);
      float t0 = (f.x - mean[2 * k]) * rstd[2 * k] * mul[2 * k] + add[2 * k];
      float t1 = (f.y - mean[2 * k + 1]) * rstd[2 * k + 1] * mul[2 * k + 1] + add[2 * k + 1];
      if (act == 2) { t0 = silu_f(t0); t1 = silu_f(t1); }
      o4[k] = pack_bf16x2(t0, t1);
    }
    *reinterpret_cast<uint4*>(y + base + static_cast<size_t>(p) * C) = make_uint4(o4[0], o4[1], o4[2], o4[3]);
  };
  if (single) {
    if (first < p1) put(first, u0);
    return;
  }
#pragma unroll 4
  for (int p = first; p < p1; p += lanes) put(p, load(p));
}

// ---- GroupNorm backward -------------------------------------------------------------------------------------------------
// With xh = (x - mean) * rstd, z = xh * w + b, y = act(z) and g = dy * act'(z) * w:
//   dx = rstd * (g - mean_group(g) - xh * mean_group(g * xh)),   dw[c] = sum dy act'(z) xh,   db[c] = sum dy act'(z)
// (serenitymojo/ops/norm_backward.mojo:951,1080). Pass 1 (one block per sample and group) forms the two group means and,
// when asked, adds the per-channel sums into fp32 dw / db; pass 2 is elementwise.
__device__ __forceinline__ float gn_dact(float z, int act) {
  if (act != 2) return 1.f;
  const float sg = 1.f / (1.f + __expf(-z));
  return sg * (1.f + z * (1.f - sg));
}
__global__ void __launch_bounds__(256)
group_norm_bwd_sums_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy, const float* __restrict__ stats,
                           const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ b, float* __restrict__ sums,
                           float* __restrict__ dw, float* __restrict__ db, int HW, int C, int G, int act) {
  const int n = blockIdx.x / G, g = blockIdx.x % G;
  const int cpg = C / G;
  const size_t base = static_cast<size_t>(n) * HW * C + g * cpg;
  const float mean = stats[2 * blockIdx.x], rstd = stats[2 * blockIdx.x + 1];
  float s1 = 0.f, s2 = 0.f;
  // each thread keeps to one channel of the group while it walks the pixels, so its dw / db partials are per channel;
  // blockDim / cpg pixel lanes per channel, the threads beyond lanes * cpg idle
  const int lanes = blockDim.x / cpg;
  if (static_cast<int>(threadIdx.x) < lanes * cpg) {
    const int c = threadIdx.x % cpg, pl = threadIdx.x / cpg;
    const float wc = w ? __bfloat162float(w[g * cpg + c]) : 1.f, bc = b ? __bfloat162float(b[g * cpg + c]) : 0.f;
    float a1 = 0.f, a2 = 0.f;
    for (int p = pl; p < HW; p += lanes) {
      const size_t off = base + static_cast<size_t>(p) * C + c;
      const float xh = (__bfloat162float(x[off]) - mean) * rstd;
      const float dz = __bfloat162float(dy[off]) * gn_dact(xh * wc + bc, act);
      a1 += dz;
      a2 += dz * xh;
    }
    if (dw) atomicAdd(&dw[g * cpg + c], a2);
    if (db) atomicAdd(&db[g * cpg + c], a1);
    s1 = a1 * wc;
    s2 = a2 * wc;
  }
  __shared__ float r1[8], r2[8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  if ((threadIdx.x & 31) == 0) { r1[threadIdx.x >> 5] = s1; r2[threadIdx.x >> 5] = s2; }
  __syncthreads();
  if (threadIdx.x == 0) {
    float a = 0.f, c2 = 0.f;
    for (int i = 0; i < 8; ++i) { a += r1[i]; c2 += r2[i]; }
    const float cnt = static_cast<float>(HW) * cpg;
    sums[2 * blockIdx.x] = a / cnt;
    sums[2 * blockIdx.x + 1] = c2 / cnt;
  }
}
// many-block form of the sums above (same decomposition and ordered reductions as group_norm_partial_kernel). part[n, chunk]
// holds per group (sum g, sum g * xh) and, when weight gradients are wanted, per channel (sum dz * xh, sum dz) after the
// 2 * G group values; group_norm_finalize_kernel / group_norm_wgrad_kernel add the chunks in order.
__global__ void __launch_bounds__(256)
group_norm_bwd_partial_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy, const float* __restrict__ stats,
                              const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ b, float* __restrict__ part,
                              int wgrad, int HW, int C, int G, int act, int ppb, int sv) {
  extern __shared__ float gsm[];                 // [256][16], then [C][2]
  const int n = blockIdx.y, cpg = C / G, v0 = blockIdx.z * sv;
  const int cv = min(sv, (C >> 3) - v0);
  const int lanes = blockDim.x / cv;
  float a1[8], a2[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) a1[k] = a2[k] = 0.f;
  if (static_cast<int>(threadIdx.x) < lanes * cv) {
    const int v = threadIdx.x % cv, pl = threadIdx.x / cv;
    const int p0 = blockIdx.x * ppb, p1 = min(p0 + ppb, HW);
    float wc[8], bc[8], mean[8], rstd[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int c = (v0 + v) * 8 + k, g = c / cpg;
      wc[k] = w ? __bfloat162float(w[c]) : 1.f;
      bc[k] = b ? __bfloat162float(b[c]) : 0.f;
      mean[k] = stats[2 * (n * G + g)];
      rstd[k] = stats[2 * (n * G + g) + 1];
    }
    const size_t base = (static_cast<size_t>(n) * HW) * C + (v0 + v) * 8;
#pragma unroll 2
    for (int p = p0 + pl; p < p1; p += lanes) {
      const uint4 ux = *reinterpret_cast<const uint4*>(x + base + static_cast<size_t>(p) * C);
      const uint4 ud = *reinterpret_cast<const uint4*>(dy + base + static_cast<size_t>(p) * C);
      const uint32_t x4[4] = {ux.x, ux.y, ux.z, ux.w}, d4[4] = {ud.x, ud.y, ud.z, ud.w};
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float2 fx = unpack_bf16x2(x4[k >> 1]), fd = unpack_bf16x2(d4[k >> 1]);
        const float xh = (((k & 1) ? fx.y : fx.x) - mean[k]) * rstd[k];
        const float dz = ((k & 1) ? fd.y : fd.x) * gn_dact(xh * wc[k] + bc[k], act);
        a1[k] += dz;
        a2[k] += dz * xh;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) { gsm[threadIdx.x * 16 + k] = a1[k]; gsm[threadIdx.x * 16 + 8 + k] = a2[k]; }
  __syncthreads();
  float* csum = gsm + 256 * 16;                  // [C][2] = (sum dz, sum dz * xh)
  const int stride = 2 * G + (wgrad ? 2 * C : 0);
  float* out = part + (static_cast<size_t>(n) * gridDim.x + blockIdx.x) * stride;
  for (int c = threadIdx.x; c < 8 * cv; c += blockDim.x) {
    const int v = c >> 3, k = c & 7;
    float a = 0.f, bsum = 0.f;
    for (int pl = 0; pl < lanes; ++pl) { a += gsm[(pl * cv + v) * 16 + k]; bsum += gsm[(pl * cv + v) * 16 + 8 + k]; }
    csum[2 * c] = a; csum[2 * c + 1] = bsum;
    if (wgrad) { out[2 * G + 2 * (8 * v0 + c)] = bsum; out[2 * G + 2 * (8 * v0 + c) + 1] = a; }
  }
  __syncthreads();
  const int g0 = v0 * 8 / cpg;
  for (int g = threadIdx.x; g < cv * 8 / cpg; g += blockDim.x) {
    float a = 0.f, bsum = 0.f;
    for (int c = g * cpg; c < (g + 1) * cpg; ++c) {
      const float wc = w ? __bfloat162float(w[8 * v0 + c]) : 1.f;
      a += csum[2 * c] * wc; bsum += csum[2 * c + 1] * wc;
    }
    out[2 * (g0 + g)] = a; out[2 * (g0 + g) + 1] = bsum;
  }
}
// dw[c] / db[c] += over samples and chunks, in order
__global__ void group_norm_wgrad_kernel(const float* __restrict__ part, float* __restrict__ dw, float* __restrict__ db, int N, int C, int G,
                                        int chunks) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  const int stride = 2 * G + 2 * C;
  float a = 0.f, b = 0.f;
  for (int i = 0; i < N * chunks; ++i) { a += part[static_cast<size_t>(i) * stride + 2 * G + 2 * c]; b += part[static_cast<size_t>(i) * stride + 2 * G + 2 * c + 1]; }
  dw[c] += a;
  db[c] += b;
}
// one thread per 8-channel vector over a range of pixels, as group_norm_apply_kernel
__global__ void __launch_bounds__(256)
group_norm_bwd_apply_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy,
                            __nv_bfloat16* __restrict__ dx, const float* __restrict__ stats, const float* __restrict__ sums,
                            const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ b,
                            int HW, int C, int G, int act, float sum_scale, int ppb, int sv) {
  const int n = blockIdx.y, cpg = C / G, v0 = blockIdx.z * sv;
  const int cv = min(sv, (C >> 3) - v0), lanes = blockDim.x / cv;
  if (static_cast<int>(threadIdx.x) >= lanes * cv) return;
  const int v = v0 + threadIdx.x % cv, p0 = blockIdx.x * ppb, p1 = min(p0 + ppb, HW), first = p0 + threadIdx.x / cv;
  const size_t base = (static_cast<size_t>(n) * HW) * C + v * 8;
  auto load = [&](const __nv_bfloat16* t, int p) { return *reinterpret_cast<const uint4*>(t + base + static_cast<size_t>(p) * C); };
  const bool single = ppb <= lanes;
  const uint4 ux0 = single && first < p1 ? load(x, first) : make_uint4(0, 0, 0, 0), ud0 = single && first < p1 ? load(dy, first) : make_uint4(0, 0, 0, 0);
  float mean[8], rstd[8], m1[8], m2[8], wc[8], bc[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int c = v * 8 + k, i = n * G + c / cpg;
    mean[k] = stats[2 * i]; rstd[k] = stats[2 * i + 1];
    m1[k] = sums[2 * i] * sum_scale; m2[k] = sums[2 * i + 1] * sum_scale;
    wc[k] = w ? __bfloat162float(w[c]) : 1.f;
    bc[k] = b ? __bfloat162float(b[c]) : 0.f;
  }
  auto put = [&](int p, uint4 ux, uint4 ud) {
    const uint32_t x4[4] = {ux.x, ux.y, ux.z, ux.w}, d4[4] = {ud.x, ud.y, ud.z, ud.w};
    float o[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float2 fx = unpack_bf16x2(x4[k >> 1]), fd = unpack_bf16x2(d4[k >> 1]);
      const float xh = (((k & 1) ? fx.y : fx.x) - mean[k]) * rstd[k];
      const float gg = ((k & 1) ? fd.y : fd.x) * gn_dact(xh * wc[k] + bc[k], act) * wc[k];
      o[k] = rstd[k] * (gg - m1[k] - xh * m2[k]);
    }
    *reinterpret_cast<uint4*>(dx + base + static_cast<size_t>(p) * C) =
        make_uint4(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]), pack_bf16x2(o[4], o[5]), pack_bf16x2(o[6], o[7]));
  };
  if (single) {
    if (first < p1) put(first, ux0, ud0);
    return;
  }
#pragma unroll 2
  for (int p = first; p < p1; p += lanes) put(p, load(x, p), load(dy, p));
}

// nearest-neighbour 2x upsample, NHWC
__global__ void upsample2x_kernel(const uint4* __restrict__ x, uint4* __restrict__ y, int N, int H, int W, int cv) {
  const long long total = static_cast<long long>(N) * H * 2 * W * 2 * cv;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int c = static_cast<int>(i % cv);
    long long r = i / cv;
    const int ow = static_cast<int>(r % (2 * W));
    r /= 2 * W;
    const int oh = static_cast<int>(r % (2 * H));
    const int n = static_cast<int>(r / (2 * H));
    y[i] = x[((static_cast<long long>(n) * H + (oh >> 1)) * W + (ow >> 1)) * cv + c];
  }
}

// Channels zero-padded to Cp (a multiple of 8): x [N, H, W, C] with any element strides -> contiguous [N, H, W, Cp], one 16-byte vector a
// thread. Bound by the bytes written; the concatenation with zeros it stands in for walked a planar image (NCHW seen as NHWC) element by
// element: 0.51 ms for three planar 488 x 712 images, the whole encode 6.67 -> 6.32 ms with this kernel (B200).
__global__ void pad_channels_kernel(const __nv_bfloat16* __restrict__ x, uint4* __restrict__ y, unsigned total, int H, int W, int C, unsigned chunks,
                                    long long s0, long long s1, long long s2, long long s3) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const unsigned pixel = i / chunks;
  const int c0 = static_cast<int>(i - pixel * chunks) * 8;
  uint32_t v[4] = {0u, 0u, 0u, 0u};
  if (c0 < C) {
    const unsigned r = pixel / W, n = r / H;
    const __nv_bfloat16* p = x + n * s0 + (r - n * H) * s1 + (pixel - r * W) * s2;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (c0 + j < C) v[j >> 1] |= static_cast<uint32_t>(__bfloat16_as_ushort(p[(c0 + j) * s3])) << (16 * (j & 1));
  }
  y[i] = make_uint4(v[0], v[1], v[2], v[3]);
}

// 2x2 average pool, NHWC (down-sampling path of encoders when no strided conv is used)
__global__ void avgpool2x_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y, int N, int H, int W,
                                 int C) {
  const int Ho = H / 2, Wo = W / 2;
  const long long total = static_cast<long long>(N) * Ho * Wo * C;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int c = static_cast<int>(i % C);
    long long r = i / C;
    const int ow = static_cast<int>(r % Wo);
    r /= Wo;
    const int oh = static_cast<int>(r % Ho);
    const int n = static_cast<int>(r / Ho);
    const __nv_bfloat16* p = x + ((static_cast<long long>(n) * H + 2 * oh) * W + 2 * ow) * C + c;
    const float s = __bfloat162float(p[0]) + __bfloat162float(p[C]) + __bfloat162float(p[static_cast<long long>(W) * C]) +
                    __bfloat162float(p[static_cast<long long>(W) * C + C]);
    y[i] = __float2bfloat16_rn(0.25f * s);
  }
}

static inline int grid_for(long long n, int threads) {
  long long b = (n + threads - 1) / threads;
  const long long cap = static_cast<long long>(mdb::device_sm_count()) * 16;
  return static_cast<int>(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace mdb

using namespace mdb;
typedef __nv_bfloat16 bf16;

// Slab of channel vectors per block: a whole number of groups, at most 256 vectors (one per thread). Returns 0 when a group
// alone is wider (the block-per-group kernels take those statistics).
static int gn_slab(int C, int G) {
  const int cpg = C / G;
  int unit = cpg;                                               // lcm(cpg, 8) / 8 vectors
  for (int d = 8; d > 1; d >>= 1)
    if (cpg % d == 0) { unit = cpg / d; break; }
  if (unit > 256) return 0;
  const int cv = C / 8, most = 256 / unit * unit, slabs = (cv + most - 1) / most;
  return (cv / unit + slabs - 1) / slabs * unit;
}
// How the elementwise passes split a sample: any slab of up to 256 vectors, about eight blocks per SM, at least four pixels per
// thread, or one where that leaves SMs without a block
static void gn_apply_split(int N, int HW, int C, int* sv, dim3* grid, int* ppb) {
  const int cv = C / 8, slabs = (cv + 255) / 256;
  *sv = (cv + slabs - 1) / slabs;
  const int lanes = 256 / *sv;
  long long want = 8ll * mdb::device_sm_count() / (static_cast<long long>(N) * slabs);
  if (want < 1) want = 1;
  long long pp = (HW + want - 1) / want;
  if (pp < 4 * lanes) pp = (HW + 4 * lanes - 1) / (4 * lanes) * static_cast<long long>(N) * slabs < mdb::device_sm_count() ? lanes : 4 * lanes;
  *ppb = static_cast<int>(pp);
  *grid = dim3(static_cast<unsigned>((HW + pp - 1) / pp), N, slabs);
}
// How the many-block kernels split a sample for the forward statistics or the backward sums: chunk count and pixels per chunk (0 chunks: use
// the block-per-group kernels)
static void gn_chunks(int N, int HW, int C, int G, bool backward, int* chunks, int* ppb) {
  const int sms = mdb::device_sm_count(), sv = gn_slab(C, G);
  *chunks = 0;
  *ppb = 0;
  if (sv == 0 || N * G >= 4 * sms || N > 65535) return;
  // wide tensors of a few pixels: one block per group reads its share at once (1 x 8 x 8 x 2560: 5.4 us against 9.7 for the chunks
  // and their finish, backward sums 12.7 against 20.3; 2 x 247 pixels: 9.4 against 11.2, but backward 31.6 against 22.8)
  if (C > 2048 && HW < (backward ? 160 : 512)) return;
  const int slabs = (C / 8 + sv - 1) / sv;
  int ch = (4 * sms + N * slabs - 1) / (N * slabs);             // about four blocks per SM over all samples
  int pp = (HW + ch - 1) / ch;
  const int lanes = 256 / sv;
  if (pp < 4 * lanes) pp = 4 * lanes;                           // at least a few pixels per thread
  *ppb = pp;
  *chunks = (HW + pp - 1) / pp;
}
// fp32 elements of scratch the forward (wgrad < 0) or the backward (wgrad 0 / 1) needs
extern "C" long long mdb_group_norm_scratch_floats(int N, int HW, int C, int G, int wgrad) {
  int chunks, chunks_bwd, ppb;
  gn_chunks(N, HW, C, G, false, &chunks, &ppb);
  gn_chunks(N, HW, C, G, true, &chunks_bwd, &ppb);
  const long long base = (wgrad < 0 ? 2ll : 4ll) * N * G;
  const long long fwd = 2ll * G * N * chunks;
  const long long bwd = (2ll * G + (wgrad > 0 ? 2ll * C : 0)) * N * chunks_bwd;
  return base + (wgrad < 0 ? fwd : (fwd > bwd ? fwd : bwd));
}
static void launch_finalize(const float* part, float* stats, int N, int G, int chunks, int stride, float cnt, float eps, cudaStream_t st) {
  group_norm_finalize_kernel<<<(N * G + 7) / 8, 256, 0, st>>>(part, stats, N, G, chunks, stride, cnt, eps);
}
// (mean, rstd) per (sample, group) into stats; ``part`` is scratch for the chunk partials
static int launch_group_stats(const void* x, float* stats, float* part, int N, int HW, int C, int G, float eps, cudaStream_t st) {
  int chunks, ppb;
  gn_chunks(N, HW, C, G, false, &chunks, &ppb);
  if (chunks == 0) {
    group_norm_stats_kernel<<<N * G, 256, 0, st>>>((const bf16*)x, stats, HW, C, G, eps);
    return (int)cudaGetLastError();
  }
  const int sv = gn_slab(C, G), slabs = (C / 8 + sv - 1) / sv;
  const size_t smem = (256 * 16 + 16 * sv) * sizeof(float);
  group_norm_partial_kernel<<<dim3(chunks, N, slabs), 256, smem, st>>>((const bf16*)x, part, HW, C, G, ppb, sv);
  launch_finalize(part, stats, N, G, chunks, 2 * G, static_cast<float>(HW) * (C / G), eps, st);
  return (int)cudaGetLastError();
}
static int launch_group_apply(const void* x, void* y, const float* stats, const void* w, const void* b, int N, int HW, int C, int G, int act,
                              cudaStream_t st) {
  int sv, ppb;
  dim3 grid;
  for (int n0 = 0; n0 < N; n0 += 65535) {                       // grid.y limit
    const int n = N - n0 < 65535 ? N - n0 : 65535;
    gn_apply_split(n, HW, C, &sv, &grid, &ppb);
    const size_t off = static_cast<size_t>(n0) * HW * C;
    group_norm_apply_kernel<<<grid, 256, 0, st>>>((const bf16*)x + off, (bf16*)y + off, stats + 2ll * n0 * G, (const bf16*)w, (const bf16*)b, HW, C,
                                                  G, act, ppb, sv);
  }
  return (int)cudaGetLastError();
}

// stats: [N * G, 2] scratch (mean, rstd), sums: [N * G, 2] scratch; dw / db: fp32 [C] accumulators (zeroed by the caller) or null
extern "C" int mdb_group_norm_bwd(const void* x, const void* dy, void* dx, float* scratch, const void* w, const void* b, float* dw,
                                  float* db, int N, int HW, int C, int G, float eps, int act, cudaStream_t st) {
  if (C % G || C % 8 || (act != 0 && act != 2) || (C / G) > 256) return -1;
  if (N == 0) return 0;
  float* stats = scratch;
  float* sums = scratch + 2ll * N * G;
  float* part = scratch + 4ll * N * G;
  if (int rc = launch_group_stats(x, stats, part, N, HW, C, G, eps, st)) return rc;
  int chunks, ppb;
  gn_chunks(N, HW, C, G, true, &chunks, &ppb);
  if (chunks == 0) {
    group_norm_bwd_sums_kernel<<<N * G, 256, 0, st>>>((const bf16*)x, (const bf16*)dy, stats, (const bf16*)w, (const bf16*)b, sums, dw, db,
                                                      HW, C, G, act);
  } else {
    const int wgrad = dw != nullptr ? 1 : 0;
    const int sv = gn_slab(C, G), slabs = (C / 8 + sv - 1) / sv;
    const size_t smem = (256 * 16 + 16 * sv) * sizeof(float);
    group_norm_bwd_partial_kernel<<<dim3(chunks, N, slabs), 256, smem, st>>>((const bf16*)x, (const bf16*)dy, stats, (const bf16*)w,
                                                                             (const bf16*)b, part, wgrad, HW, C, G, act, ppb, sv);
    if (wgrad) group_norm_wgrad_kernel<<<(C + 255) / 256, 256, 0, st>>>(part, dw, db, N, C, G, chunks);
    // raw group sums (cnt <= 0), chunks added in order
    launch_finalize(part, sums, N, G, chunks, 2 * G + (wgrad ? 2 * C : 0), -1.f, 0.f, st);
  }
  const float sum_scale = chunks == 0 ? 1.f : 1.f / (static_cast<float>(HW) * (C / G));
  int sv, ppb2;
  dim3 grid;
  for (int n0 = 0; n0 < N; n0 += 65535) {                       // grid.y limit
    gn_apply_split(N - n0 < 65535 ? N - n0 : 65535, HW, C, &sv, &grid, &ppb2);
    const size_t off = static_cast<size_t>(n0) * HW * C;
    group_norm_bwd_apply_kernel<<<grid, 256, 0, st>>>((const bf16*)x + off, (const bf16*)dy + off, (bf16*)dx + off, stats + 2ll * n0 * G,
                                                      sums + 2ll * n0 * G, (const bf16*)w, (const bf16*)b, HW, C, G, act, sum_scale, ppb2, sv);
  }
  return (int)cudaGetLastError();
}
extern "C" int mdb_group_norm(const void* x, void* y, float* stats, const void* w, const void* b, int N, int HW, int C,
                              int G, float eps, int act, cudaStream_t st) {
  if (C % 8 || C % G) return -1;
  if (N <= 0 || HW <= 0) return 0;
  if (int rc = launch_group_stats(x, stats, stats + 2ll * N * G, N, HW, C, G, eps, st)) return rc;
  return launch_group_apply(x, y, stats, w, b, N, HW, C, G, act, st);
}
extern "C" int mdb_upsample2x(const void* x, void* y, int N, int H, int W, int C, cudaStream_t st) {
  if (C % 8) return -1;
  const long long total = static_cast<long long>(N) * H * W * 4 * (C / 8);
  if (total <= 0) return 0;
  upsample2x_kernel<<<grid_for(total, 256), 256, 0, st>>>((const uint4*)x, (uint4*)y, N, H, W, C / 8);
  return (int)cudaGetLastError();
}
extern "C" int mdb_pad_channels(const void* x, void* y, int N, int H, int W, int C, int Cp, const long long* strides, cudaStream_t st) {
  const long long total = static_cast<long long>(N) * H * W * (Cp / 8);
  if (Cp % 8 || Cp < C || total >= (1ll << 31)) return -1;
  if (total <= 0) return 0;
  pad_channels_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, st>>>((const bf16*)x, (uint4*)y, static_cast<unsigned>(total), H, W, C,
                                                                                   static_cast<unsigned>(Cp / 8), strides[0], strides[1], strides[2], strides[3]);
  return (int)cudaGetLastError();
}
extern "C" int mdb_avgpool2x(const void* x, void* y, int N, int H, int W, int C, cudaStream_t st) {
  const long long total = static_cast<long long>(N) * (H / 2) * (W / 2) * C;
  if (total <= 0) return 0;
  avgpool2x_kernel<<<grid_for(total, 256), 256, 0, st>>>((const bf16*)x, (bf16*)y, N, H, W, C);
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------------------------
// GroupNorm with a built-in workspace (see the declaration for the contract a caller relies on).
// The statistics buffer is a file-scope device array, so the address is fixed for the life of the module on each device
// and the call has nothing to allocate or free.
// ---------------------------------------------------------------------------------------------------------------
#include <cstdio>

static __device__ __align__(256) float g_group_norm_static_stats[2 * MDB_GROUP_NORM_STATIC_MAX_GROUPS];

namespace {
constexpr int kMaxDevices = 64;
float* g_static_stats_addr[kMaxDevices];   // per device; written once, always with the same value for that device

// Address of the array on the current device. cudaGetSymbolAddress answers for whichever device is current, so the
// cache is indexed by device ordinal. Two threads that get here together store the same pointer.
int static_stats_ptr(float** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (dev < 0 || dev >= kMaxDevices) return -21;
  float* p = g_static_stats_addr[dev];
  if (p == nullptr) {
    void* sym = nullptr;
    e = cudaGetSymbolAddress(&sym, g_group_norm_static_stats);
    if (e != cudaSuccess) return static_cast<int>(e);
    p = static_cast<float*>(sym);
    g_static_stats_addr[dev] = p;
  }
  *out = p;
  return 0;
}
}  // namespace

extern "C" int mdb_group_norm_static_ws(const void* x, void* y, const void* w, const void* b, int N, int HW, int C,
                                        int G, float eps, int act, cudaStream_t st) {
  if (G <= 0 || C <= 0 || C % 8 || C % G) return -1;
  if (N <= 0 || HW <= 0) return 0;
  const long long groups = static_cast<long long>(N) * G;
  if (groups > MDB_GROUP_NORM_STATIC_MAX_GROUPS) {
    fprintf(stderr,
            "mdb_group_norm_static_ws: N * G = %lld exceeds the built-in workspace of %d (sample, group) pairs; "
            "split the batch or call mdb_group_norm with a buffer of your own\n",
            groups, MDB_GROUP_NORM_STATIC_MAX_GROUPS);
    return MDB_ERR_STATIC_WS_TOO_SMALL;
  }
  float* stats = nullptr;
  const int rc = static_stats_ptr(&stats);
  if (rc) return rc;
  // same two launches as mdb_group_norm; the first fills stats[0 .. 2 * N * G), the second reads exactly that range
  group_norm_stats_kernel<<<N * G, 256, 0, st>>>((const bf16*)x, stats, HW, C, G, eps);
  return launch_group_apply(x, y, stats, w, b, N, HW, C, G, act, st);
}
