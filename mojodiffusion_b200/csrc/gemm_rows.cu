// Few-row GEMM: out[M, N] = epi(sum_seg A_seg[M, K_seg] * B_seg[N, K_seg]^T) for M <= 8, bf16 operands, fp32 sums.
//
// For few rows and for small weights (choose_form in gemm_tcgen05.cu has the measured line).
// What bounds it: the weights are read once and used for at most eight multiply-adds per element, so the time is that of
// streaming B from HBM. The 128-row tensor-core tiles read the same bytes from only N / 128 CTAs, and one SM takes in about
// 64 bytes per clock: a 1 x 3072 x 9216 projection kept 72 SMs waiting for 47 us where the weights need 9 us.
// Here every warp owns C whole columns (rows of B): a lane reads 16 bytes of each of its columns per step and issues eight
// such loads together (4 KB per warp in flight; with two, a 2560 x 9728 weight streamed at 2.3 TB/s); A (a few KB) comes from L1.
// C is 4, 2 or 1, the widest that still gives every SM two blocks. No shared memory, no split of K: a column's sum is 32 lane
// sums joined in a fixed order, so the result does not depend on scheduling.
//
// Role in the reference: the single-token and modulation-vector matrix-vector products, serenitymojo/ops/linear.mojo:40-180.
#include "common.cuh"
#include "gemm_api.h"

#include <string.h>

namespace mdb {

constexpr int ROWS_WARPS = 8;

struct RowsParams {
  const __nv_bfloat16* A[MDB_GEMM_MAX_SEG];
  const __nv_bfloat16* B[MDB_GEMM_MAX_SEG];
  const __nv_bfloat16* B2[MDB_GEMM_MAX_SEG];      // paired mode: row c of B2 is the second half of column c
  long long lda[MDB_GEMM_MAX_SEG], ldb[MDB_GEMM_MAX_SEG];
  int K[MDB_GEMM_MAX_SEG];
  int num_seg, M, N, pair_offset, act, act_on_second, out_fp32, accumulate, round_halves;
  float alpha;
  const __nv_bfloat16 *bias, *residual, *gate;
  int ld_res, gate_stride, rows_per_group, ld_out;
  void* out;
};

__device__ __forceinline__ float rows_act(int act, float x) {
  switch (act) {
    case MDB_ACT_GELU_TANH: return gelu_tanh_f(x);
    case MDB_ACT_SILU: return silu_f(x);
    case MDB_ACT_GELU_ERF: return gelu_erf_f(x);
    default: return x;
  }
}
// SiLU for results that are rounded to bf16 and used again: this file is built with fast math, whose exponential is off by up to
// 2^-17 at |x| of 60 (the product x log2(e) is rounded before 2^y is taken) and flips that rounding where the torch operation does
// not. Here the product's remainder y_low is carried: e^x = 2^y (1 + y_low ln 2). In double precision the same cost the decode
// step's gated MLP 2 us of 20.
__device__ __forceinline__ float rows_silu_exact(float x) {
  constexpr float log2e = 1.44269502f, log2e_low = 1.92596299e-8f;          // log2(e) in two terms
  const float y = __fmul_rn(-x, log2e);
  const float low = __fmaf_rn(-x, log2e_low, __fmaf_rn(-x, log2e, -y));
  float e = exp2f(y);
  if (fabsf(y) < 128.f) e = __fmaf_rn(e, low * 0.693147181f, e);            // beyond, e is 0 or infinite for the quotient
  return __fdiv_rn(x, 1.f + e);
}
__device__ __forceinline__ uint4 ldg_stream(const uint4* p) {   // weights: read once, not kept in L1
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void dot8(float& acc, const float (&a)[8], const uint4& b) {
  const float2 b0 = unpack_bf16x2(b.x), b1 = unpack_bf16x2(b.y), b2 = unpack_bf16x2(b.z), b3 = unpack_bf16x2(b.w);
  acc = fmaf(a[0], b0.x, acc); acc = fmaf(a[1], b0.y, acc); acc = fmaf(a[2], b1.x, acc); acc = fmaf(a[3], b1.y, acc);
  acc = fmaf(a[4], b2.x, acc); acc = fmaf(a[5], b2.y, acc); acc = fmaf(a[6], b3.x, acc); acc = fmaf(a[7], b3.y, acc);
}

// MR rows (M rounded up to 1, 2, 4, 8; the surplus repeats the last row), C columns per warp, PAIR: a column is row c of B and
// row c of B2 (SwiGLU / GEGLU).
template <int MR, int C, bool PAIR>
__global__ void __launch_bounds__(ROWS_WARPS * 32)
gemm_rows_kernel(const __grid_constant__ RowsParams p) {
  constexpr int W = PAIR ? 2 * C : C;             // rows of B a warp reads
  constexpr int U = 8 / W;                        // steps of K issued together: eight 16-byte loads in flight per lane
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = (blockIdx.x * ROWS_WARPS + warp) * C;
  if (n0 >= p.N) return;
  float acc[MR][W];
#pragma unroll
  for (int m = 0; m < MR; ++m)
#pragma unroll
    for (int c = 0; c < W; ++c) acc[m][c] = 0.f;
  for (int s = 0; s < p.num_seg; ++s) {
    const uint4* b[W];
    const uint4* a[MR];
#pragma unroll
    for (int c = 0; c < W; ++c) {
      const int col = min(n0 + (PAIR ? c >> 1 : c), p.N - 1);
      b[c] = reinterpret_cast<const uint4*>((PAIR && (c & 1) ? p.B2[s] : p.B[s]) + static_cast<size_t>(col) * p.ldb[s]);
    }
#pragma unroll
    for (int m = 0; m < MR; ++m) a[m] = reinterpret_cast<const uint4*>(p.A[s] + static_cast<size_t>(min(m, p.M - 1)) * p.lda[s]);
    const int kv = p.K[s] >> 3;                   // 16-byte vectors
    for (int i = lane; i < kv; i += 32 * U) {
      uint4 v[U][W];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int c = 0; c < W; ++c) v[u][c] = i + 32 * u < kv ? ldg_stream(b[c] + i + 32 * u) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (i + 32 * u >= kv) break;
#pragma unroll
        for (int m = 0; m < MR; ++m) {
          const uint4 t = __ldg(a[m] + i + 32 * u);
          const float2 x0 = unpack_bf16x2(t.x), x1 = unpack_bf16x2(t.y), x2 = unpack_bf16x2(t.z), x3 = unpack_bf16x2(t.w);
          const float f[8] = {x0.x, x0.y, x1.x, x1.y, x2.x, x2.y, x3.x, x3.y};
#pragma unroll
          for (int c = 0; c < W; ++c) dot8(acc[m][c], f, v[u][c]);
        }
      }
    }
  }
#pragma unroll
  for (int m = 0; m < MR; ++m)
#pragma unroll
    for (int c = 0; c < W; ++c)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[m][c] += __shfl_xor_sync(0xffffffffu, acc[m][c], o);
#pragma unroll
  for (int m = 0; m < MR; ++m)
#pragma unroll
    for (int c = 0; c < C; ++c) {
      if (lane != m * C + c) continue;            // MR * C <= 32: one lane per result
      const int col = n0 + c;
      if (m >= p.M || col >= p.N) continue;
      float x = acc[m][PAIR ? 2 * c : c] * p.alpha;
      if (p.bias) x += __bfloat162float(p.bias[col]);
      if (PAIR) {
        float y = acc[m][PAIR ? 2 * c + 1 : c] * p.alpha;
        if (p.bias) y += __bfloat162float(p.bias[col + p.pair_offset]);
        if (p.round_halves) {
          // both projections and the SiLU rounded to bf16, as separate operations round them
          x = __bfloat162float(__float2bfloat16_rn(x));
          y = __bfloat162float(__float2bfloat16_rn(y));
          x = __bfloat162float(__float2bfloat16_rn(rows_silu_exact(x))) * y;
        } else {
          x = p.act_on_second ? x * rows_act(p.act, y) : rows_act(p.act, x) * y;
        }
      } else {
        x = rows_act(p.act, x);
      }
      if (p.gate) x *= __bfloat162float(p.gate[static_cast<size_t>(m / p.rows_per_group) * p.gate_stride + col]);
      if (p.residual) x += __bfloat162float(p.residual[static_cast<size_t>(m) * p.ld_res + col]);
      if (p.out_fp32) {
        float* o = reinterpret_cast<float*>(p.out) + static_cast<size_t>(m) * p.ld_out + col;
        *o = p.accumulate ? *o + x : x;
      } else {
        reinterpret_cast<__nv_bfloat16*>(p.out)[static_cast<size_t>(m) * p.ld_out + col] = __float2bfloat16_rn(x);
      }
    }
}

template <int MR, bool PAIR>
static int launch_rows(const RowsParams& p, int sms, cudaStream_t st) {
  // widest column group that still leaves two blocks per SM (four columns of eight rows is one result per lane)
  const long long want = 2ll * sms * ROWS_WARPS;
  const int c = p.N >= 4 * want && !PAIR ? 4 : p.N >= 2 * want ? 2 : 1;
  const int blocks = (p.N + ROWS_WARPS * c - 1) / (ROWS_WARPS * c);
  if (!PAIR && c == 4) gemm_rows_kernel<MR, 4, false><<<blocks, ROWS_WARPS * 32, 0, st>>>(p);
  else if (c == 2) gemm_rows_kernel<MR, 2, PAIR><<<blocks, ROWS_WARPS * 32, 0, st>>>(p);
  else gemm_rows_kernel<MR, 1, PAIR><<<blocks, ROWS_WARPS * 32, 0, st>>>(p);
  return static_cast<int>(cudaGetLastError());
}

static int launch_rows_any(const RowsParams& p, int sms, bool pair, cudaStream_t st) {
  if (p.M == 1) return pair ? launch_rows<1, true>(p, sms, st) : launch_rows<1, false>(p, sms, st);
  if (p.M == 2) return pair ? launch_rows<2, true>(p, sms, st) : launch_rows<2, false>(p, sms, st);
  if (p.M <= 4) return pair ? launch_rows<4, true>(p, sms, st) : launch_rows<4, false>(p, sms, st);
  return pair ? launch_rows<8, true>(p, sms, st) : launch_rows<8, false>(p, sms, st);
}

}  // namespace mdb

// True when the few-row kernel computes exactly what mdb_gemm_launch was asked for. It reads whole 16-byte vectors along K
// and rows of 16-byte alignment (what the tensor maps of the tiled kernel also ask for); everything with a scale, a routed /
// gathered / reduced operand, an MN-major operand, a caller-chosen tile or split_k != 0 (1: one accumulator per output, as a
// longer input has it, while the sums here are joined from 32 lanes) stays on the tiled kernels.
extern "C" int mdb_gemm_rows_ok(const MdbGemmArgs* a) {
  if (a->M > MDB_GEMM_ROWS_MAX || a->kind != 0 || a->a_mn || a->b_mn || a->bn != 0 || a->conv_taps > 0 || a->split_k != 0 ||
      a->gather_world > 1 || a->route_owner_cols > 0 || a->reduce_rows_per_owner > 0 || a->row_scale || a->col_scale || a->prof)
    return 0;
  for (int s = 0; s < a->num_seg; ++s) {
    if (a->K[s] % 8 || a->K[s] <= 0 || a->K[s] > (1ll << 30) || a->lda[s] % 8 || a->ldb[s] % 8) return 0;
    if ((reinterpret_cast<uintptr_t>(a->A[s]) | reinterpret_cast<uintptr_t>(a->B[s])) & 15) return 0;
  }
  return 1;
}

extern "C" int mdb_gemm_rows(const MdbGemmArgs* a, cudaStream_t st) {
  using namespace mdb;
  RowsParams p;
  memset(&p, 0, sizeof(p));
  for (int s = 0; s < a->num_seg; ++s) {
    p.A[s] = reinterpret_cast<const __nv_bfloat16*>(a->A[s]);
    p.B[s] = reinterpret_cast<const __nv_bfloat16*>(a->B[s]);
    p.B2[s] = p.B[s] + static_cast<size_t>(a->pair_offset > 0 ? a->pair_offset : 0) * a->ldb[s];
    p.lda[s] = a->lda[s];
    p.ldb[s] = a->ldb[s];
    p.K[s] = static_cast<int>(a->K[s]);
  }
  p.num_seg = a->num_seg; p.M = a->M; p.N = a->N; p.pair_offset = a->pair_offset;
  p.act = a->act; p.act_on_second = a->act_on_second; p.alpha = a->alpha;
  p.bias = reinterpret_cast<const __nv_bfloat16*>(a->bias);
  p.residual = reinterpret_cast<const __nv_bfloat16*>(a->residual);
  p.gate = reinterpret_cast<const __nv_bfloat16*>(a->gate);
  p.ld_res = a->ld_res; p.gate_stride = a->gate_stride; p.rows_per_group = a->rows_per_group > 0 ? a->rows_per_group : 1;
  p.out = a->out; p.ld_out = a->ld_out; p.out_fp32 = a->out_fp32; p.accumulate = a->accumulate_out;
  return launch_rows_any(p, a->num_sms > 0 ? a->num_sms : device_sm_count(), a->pair_offset > 0, st);
}

// silu(x w1^T) * (x w2^T) with the two halves in weights of their own, each half and the activation rounded to bf16 before they
// meet, M <= MDB_GEMM_ROWS_MAX rows; everything contiguous bf16
extern "C" int mdb_glu_rows(const void* x, const void* w1, const void* w2, void* out, int M, int N, int K, cudaStream_t st) {
  using namespace mdb;
  if (M <= 0 || M > MDB_GEMM_ROWS_MAX || N <= 0 || K <= 0 || K % 8 ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w1) | reinterpret_cast<uintptr_t>(w2)) & 15))
    return -1;
  RowsParams p;
  memset(&p, 0, sizeof(p));
  p.A[0] = reinterpret_cast<const __nv_bfloat16*>(x);
  p.B[0] = reinterpret_cast<const __nv_bfloat16*>(w1);
  p.B2[0] = reinterpret_cast<const __nv_bfloat16*>(w2);
  p.lda[0] = p.ldb[0] = p.K[0] = K;
  p.num_seg = 1; p.M = M; p.N = N; p.act = MDB_ACT_SILU; p.alpha = 1.f; p.rows_per_group = 1; p.out = out; p.ld_out = N;
  p.round_halves = 1;
  return launch_rows_any(p, device_sm_count(), true, st);
}
