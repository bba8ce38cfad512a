// Persistent warp-specialised GEMM for sm_100a: TMA (128-byte swizzle) -> shared memory ring ->
// tcgen05.mma with the accumulator in TMEM (double buffered, so the epilogue of tile i overlaps the
// main loop of tile i+1) -> tcgen05.ld epilogue with fused bias / activation / gated residual /
// paired (SwiGLU, GEGLU) / dequant-scale math. bf16 rows leave as tiled bulk stores (BulkEpilogue) where they are local and start on
// 16 bytes, else by stores of the lanes.
//
//   out[M,N] = epi( sum_seg  A_seg[M,K_seg] * B_seg[N,K_seg]^T )
//
// Up to three K segments share one accumulator. That is how a LoRA up-projection (A2 = x*down^T,
// B2 = up), a split input (FLUX single-block linear2 over [attn | gelu(mlp)]) or a beta=1
// accumulate are folded into one launch without a concat.
//
// Operand majors: K-major (row-major [rows,K], the forward layout of x and of nn.Linear weights) and
// MN-major (the same buffers read transposed: dx = dY*W uses W MN-major, dW = dY^T*x uses both).
// Element kinds: bf16 (kind::f16) and fp8 e4m3 (kind::f8f6f4, scales applied in the epilogue).
//
// Covers the role of the reference's cuBLAS call + bias/cast kernels (serenitymojo/ops/linear.mojo:40-180,182,404),
// its GEMM backward calls (serenitymojo/ops/linalg_backward.mojo:99-124) and its weight-only fp8 kernel
// (serenitymojo/ops/fp8_gemm.mojo:28-73).
#include "common.cuh"
#include "gemm_api.h"

#include <cudaTypedefs.h>
#include <atomic>
#include <cmath>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

namespace mdb {

constexpr int BM = 128;
constexpr int BK_BYTES = 128;  // one swizzle atom row: 64 bf16 or 128 fp8
constexpr int GATHER_STAGES = 2;          // shared-memory stages of the fused all-gather (bulk copies)
constexpr int GATHER_PIECE = 16384;       // bytes per stage
constexpr int NUM_THREADS = 224;  // warps: 0 TMA, 1 UMMA issue, 2-5 epilogue, 6 peer gather (all-gather fused GEMM)
constexpr int CONV_TW = 16, CONV_TH = 8;  // conv mode: one M tile = 8 rows x 16 columns of output pixels

struct alignas(64) GemmMaps {
  CUtensorMap a[MDB_GEMM_MAX_SEG];
  CUtensorMap b[MDB_GEMM_MAX_SEG];
  CUtensorMap out;   // GemmParams::bulk_out only
};

// Kernel parameters are __grid_constant__: the run-time index into route_out otherwise makes the compiler copy all 416 bytes of them
// into each thread's local memory, which with 227 KB of shared memory in use lives in L2 (epilogue of a 128 x 128 tile 7000
// cycles, 5600 without the copy; 8192 x 5120 x 640 94.8 -> 67.9 us).
struct GemmParams {
  int M, N;
  int num_seg;
  int kblocks[MDB_GEMM_MAX_SEG];
  int pair_offset;  // paired mode (>0): second half of the B tile comes from rows n0 + pair_offset
  int act;          // MDB_ACT_*
  int act_on_second;  // paired mode: 0 -> act(first)*second (SwiGLU), 1 -> first*act(second) (GEGLU)
  float alpha;
  const float* row_scale;          // [M] or null
  const float* col_scale;          // [N(+pair)] or null
  const __nv_bfloat16* bias;       // [N(+pair)] or null
  const __nv_bfloat16* residual;   // [M, ld_res] or null
  const __nv_bfloat16* gate;       // [groups, gate_stride] or null; group = row / rows_per_group
  int ld_res, gate_stride, rows_per_group;
  void* out;
  int ld_out;
  int out_fp32;
  int accumulate_out;  // out += result (fp32 out only)
  int bulk_out;        // the output is a local, 16-byte aligned bf16 matrix (or image): rows leave through maps.out, see BulkEpilogue
  int* status;
  long long* prof;  // optional [grid, 8] cycle counters (profiling builds of the caller)
  long long* trace;  // optional per-K-block time line of CTAs 0 and 1: [2 CTAs][3 roles][trace_len] clock64 values
  int trace_len;
  // peer-routed output (sequence-parallel all-to-all in the epilogue): see MdbGemmArgs
  void* route_out[MDB_GEMM_MAX_PEERS];
  int route_owner_cols, route_part_cols, route_row_offset, route_rows_per_batch, route_batch_rows;
  int route_split, route_row_offset_b;
  // all-gather fused into the GEMM (gather_world > 1): operand A (gather_operand 0) or B (1) lives in a local
  // buffer of `gather_world` equal row chunks; chunk r is rank r's shard. Warp 6 of every CTA copies its slice of
  // each remote chunk from the owner's memory (peer loads) and bumps ready[chunk]; the TMA producer waits for
  // ready[chunk] == gridDim.x before it loads a tile of that chunk. Tiles are visited local chunk first.
  const void* gather_src[MDB_GEMM_MAX_PEERS];
  void* gather_dst;
  int* gather_ready;
  long long gather_chunk_bytes;
  int gather_world, gather_rank, gather_operand, gather_chunk_rows;
  // reduce-scatter fused into the epilogue (route_owner_cols == 0 && reduce_rows_per_owner > 0): fp32 partial
  // results are added (red.global.add) into the row owner's fp32 buffer route_out[row / reduce_rows_per_owner]
  int reduce_rows_per_owner;
  int reduce_src_rank;   // staged bf16 variant: slot of the owner's staging buffer this rank writes
  // implicit-GEMM convolution (conv_taps > 0): A is an NHWC image read through a 4-D tensor map, one 16x8 pixel
  // patch per M tile, one shifted box per filter tap; rows outside the image are skipped by the epilogue
  int conv_taps, conv_kw, conv_pad_h, conv_pad_w, conv_h, conv_w, conv_tiles_h, conv_tiles_w, conv_cblocks, conv_tiles_m;
  int conv_stride, conv_off_h, conv_off_w;   // pair kernel: input pixel of tap (kh, kw) = output pixel * stride + (kh, kw) + off
};

__device__ __forceinline__ float apply_act_rt(int act, float x) {
  switch (act) {
    case MDB_ACT_GELU_TANH: return gelu_tanh_f(x);
    case MDB_ACT_SILU: return silu_f(x);
    case MDB_ACT_GELU_ERF: return gelu_erf_f(x);
    default: return x;
  }
}

// 32 consecutive bf16 -> fp32 (64 bytes, 16-byte aligned)
__device__ __forceinline__ void load32_bf16(const __nv_bfloat16* p, float (&f)[32]) {
  const uint4* q = reinterpret_cast<const uint4*>(p);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint4 u = q[i];
    const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
    f[i * 8 + 0] = a.x; f[i * 8 + 1] = a.y; f[i * 8 + 2] = b.x; f[i * 8 + 3] = b.y;
    f[i * 8 + 4] = c.x; f[i * 8 + 5] = c.y; f[i * 8 + 6] = d.x; f[i * 8 + 7] = d.y;
  }
}
__device__ __forceinline__ void load32_f32(const float* p, float (&f)[32]) {
  const float4* q = reinterpret_cast<const float4*>(p);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float4 u = q[i];
    f[i * 4 + 0] = u.x; f[i * 4 + 1] = u.y; f[i * 4 + 2] = u.z; f[i * 4 + 3] = u.w;
  }
}

template <int ACT>
__device__ __forceinline__ void act32(float (&v)[32]) {
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    if (ACT == MDB_ACT_GELU_TANH) v[j] = gelu_tanh_f(v[j]);
    if (ACT == MDB_ACT_SILU) v[j] = silu_f(v[j]);
    if (ACT == MDB_ACT_GELU_ERF) v[j] = gelu_erf_f(v[j]);
  }
}
__device__ __forceinline__ void act32_rt(int act, float (&v)[32]) {
  // the flag is tested once per 32 values; each case is a tight unrolled loop
  if (act == MDB_ACT_GELU_TANH) act32<MDB_ACT_GELU_TANH>(v);
  else if (act == MDB_ACT_SILU) act32<MDB_ACT_SILU>(v);
  else if (act == MDB_ACT_GELU_ERF) act32<MDB_ACT_GELU_ERF>(v);
}

// Where a 32-column slab of output row `row` starting at column `col0` goes. Plain GEMM: the local output.
// Routed mode: columns are (part, owner, local) blocks; the slab is stored into the owner rank's buffer at
// row  batch * route_batch_rows + route_row_offset + row_in_batch  and column  part * owner_cols + local.
__device__ __forceinline__ void* out_slab_ptr(const GemmParams& p, int row, int col0, int esz) {
  if (p.reduce_rows_per_owner > 0) {
    const int owner = row / p.reduce_rows_per_owner;
    size_t orow = static_cast<size_t>(row - owner * p.reduce_rows_per_owner);
    if (!p.out_fp32) orow += static_cast<size_t>(p.reduce_src_rank) * p.reduce_rows_per_owner;
    return reinterpret_cast<char*>(p.route_out[owner]) + (orow * p.ld_out + col0) * esz;
  }
  if (p.route_owner_cols <= 0)
    return reinterpret_cast<char*>(p.out) + (static_cast<size_t>(row) * p.ld_out + col0) * esz;
  const int part = col0 / p.route_part_cols;
  const int within = col0 - part * p.route_part_cols;
  const int owner = within / p.route_owner_cols;
  const int lcol = part * p.route_owner_cols + (within - owner * p.route_owner_cols);
  const int b = row / p.route_rows_per_batch;
  const int rin = row - b * p.route_rows_per_batch;
  const int off = (p.route_split > 0 && rin >= p.route_split) ? p.route_row_offset_b + (rin - p.route_split) : p.route_row_offset + rin;
  const size_t orow = static_cast<size_t>(b) * p.route_batch_rows + off;
  return reinterpret_cast<char*>(p.route_out[owner]) + (orow * p.ld_out + lcol) * esz;
}

// Ragged edge (fewer than 32 columns left, or an unaligned pointer): scalar, rarely taken.
__device__ __noinline__ void epilogue_row32_slow(const GemmParams& p, int row, int col0, int ncols, const uint32_t* r,
                                                 const uint32_t* r2, bool paired) {
  const float rs = (p.row_scale ? p.row_scale[row] : 1.f) * p.alpha;
  for (int j = 0; j < ncols; ++j) {
    const int col = col0 + j;
    float x = __uint_as_float(r[j]) * rs;
    if (p.col_scale) x *= p.col_scale[col];
    if (p.bias) x += __bfloat162float(p.bias[col]);
    if (paired) {
      float y = __uint_as_float(r2[j]) * rs;
      if (p.col_scale) y *= p.col_scale[col + p.pair_offset];
      if (p.bias) y += __bfloat162float(p.bias[col + p.pair_offset]);
      x = p.act_on_second ? x * apply_act_rt(p.act, y) : apply_act_rt(p.act, x) * y;
    } else {
      x = apply_act_rt(p.act, x);
    }
    if (p.gate) x *= __bfloat162float(p.gate[static_cast<size_t>(row / p.rows_per_group) * p.gate_stride + col]);
    if (p.residual) x += __bfloat162float(p.residual[static_cast<size_t>(row) * p.ld_res + col]);
    if (p.out_fp32) {
      float* o = reinterpret_cast<float*>(out_slab_ptr(p, row, col0, 4)) + j;
      if (p.reduce_rows_per_owner > 0) atomicAdd(o, x);   // fp32 reduce mode
      else *o = p.accumulate_out ? *o + x : x;
    } else {
      reinterpret_cast<__nv_bfloat16*>(out_slab_ptr(p, row, col0, 2))[j] = __float2bfloat16_rn(x);
    }
  }
}

// One 32-column slab of one output row. r[] holds the raw accumulators (r2[] the paired half).
// stage_row (optional): this lane's 256-byte row of the warp's shared-memory staging buffer; the packed bf16 slab then
// goes there (16-byte chunks stage_chunk0 .. +3, XOR-swizzled by the lane so that neither the row-wise writes nor the
// later chunk-wise reads conflict) instead of to global memory.
__device__ __forceinline__ void epilogue_row32(const GemmParams& p, int row, int col0, const uint32_t (&r)[32],
                                               const uint32_t (&r2)[32], bool paired, bool aligned,
                                               uint4* stage_row = nullptr, int stage_chunk0 = 0, int swz = 0) {
  if (row >= p.M || col0 >= p.N) return;
  const int ncols = min(32, p.N - col0);
  if (ncols < 32 || !aligned) {
    // copies live in local memory only on this branch, so the fast path keeps its accumulators in registers
    uint32_t t0[32], t1[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      t0[j] = r[j];
      t1[j] = paired ? r2[j] : 0u;
    }
    epilogue_row32_slow(p, row, col0, ncols, t0, t1, paired);
    return;
  }
  float v[32];
  const float rs = (p.row_scale ? p.row_scale[row] : 1.f) * p.alpha;
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]) * rs;
  if (p.col_scale) {
    float t[32];
    load32_f32(p.col_scale + col0, t);
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] *= t[j];
  }
  if (p.bias) {
    float t[32];
    load32_bf16(p.bias + col0, t);
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] += t[j];
  }
  if (paired) {
    float w[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) w[j] = __uint_as_float(r2[j]) * rs;
    if (p.col_scale) {
      float t[32];
      load32_f32(p.col_scale + col0 + p.pair_offset, t);
#pragma unroll
      for (int j = 0; j < 32; ++j) w[j] *= t[j];
    }
    if (p.bias) {
      float t[32];
      load32_bf16(p.bias + col0 + p.pair_offset, t);
#pragma unroll
      for (int j = 0; j < 32; ++j) w[j] += t[j];
    }
    if (p.act_on_second) act32_rt(p.act, w); else act32_rt(p.act, v);
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] *= w[j];
  } else if (p.act != MDB_ACT_NONE) {
    act32_rt(p.act, v);
  }
  if (p.gate) {
    float t[32];
    load32_bf16(p.gate + static_cast<size_t>(row / p.rows_per_group) * p.gate_stride + col0, t);
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] *= t[j];
  }
  if (p.residual) {
    float t[32];
    load32_bf16(p.residual + static_cast<size_t>(row) * p.ld_res + col0, t);
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] += t[j];
  }
  if (p.out_fp32) {
    float4* o = reinterpret_cast<float4*>(out_slab_ptr(p, row, col0, 4));
    if (p.reduce_rows_per_owner > 0) {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(o + j), "f"(v[4 * j]), "f"(v[4 * j + 1]),
                     "f"(v[4 * j + 2]), "f"(v[4 * j + 3])
                     : "memory");
    } else if (p.accumulate_out) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float4 old = o[j];
        o[j] = make_float4(old.x + v[4 * j], old.y + v[4 * j + 1], old.z + v[4 * j + 2], old.w + v[4 * j + 3]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    }
  } else {
    uint4* o = stage_row ? stage_row : reinterpret_cast<uint4*>(out_slab_ptr(p, row, col0, 2));
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint4 t;
      t.x = pack_bf16x2(v[8 * j + 0], v[8 * j + 1]);
      t.y = pack_bf16x2(v[8 * j + 2], v[8 * j + 3]);
      t.z = pack_bf16x2(v[8 * j + 4], v[8 * j + 5]);
      t.w = pack_bf16x2(v[8 * j + 6], v[8 * j + 7]);
      o[stage_row ? ((stage_chunk0 + j) ^ swz) : j] = t;
    }
  }
}

// Epilogue of one accumulator tile for one warp (its 32 TMEM lanes = 32 output rows), each lane storing its own row.
__device__ __forceinline__ void epilogue_direct(const GemmParams& p, uint32_t taddr, int pair_col_off, int row, int n0, int out_cols,
                                                bool paired, bool aligned) {
#pragma unroll 1
  for (int c = 0; c < out_cols / 32; ++c) {
    uint32_t r0[32], r1[32];
    tmem_ld_32x32b_x32(taddr + c * 32, r0);
    if (paired) tmem_ld_32x32b_x32(taddr + pair_col_off + c * 32, r1);
    tmem_wait_ld();
    epilogue_row32(p, row, n0 + c * 32, r0, r1, paired, aligned);
  }
}

// The same with row segments staged for peers. bf16 outputs whose tile lies fully
// inside the matrix go through a per-warp staging buffer in shared memory (32 rows of GW = 128 columns), GW columns at a time: every
// lane packs its row's slabs into the buffer, then the warp stores whole row segments of 2 * GW bytes (GW / 8 lanes x 16 bytes
// per row). Local stores become full cache lines and peer-routed stores (sequence-parallel scatter, staged reduce-scatter) cross
// NVLink as 128- or 256-byte writes instead of 64-byte fragments of 32 different rows. Everything else (fp32 outputs, ragged
// edges, unaligned pointers) keeps the direct per-lane stores.
__device__ __forceinline__ void epilogue_tile(const GemmParams& p, uint32_t taddr, int pair_col_off, int row, int n0,
                                              int out_cols, bool paired, bool aligned, uint8_t* stage_warp, int lane) {
  constexpr int GW = 128, CH = GW / 8;                          // columns of a staged row, its 16-byte chunks
  const bool staged = stage_warp != nullptr && aligned && !p.out_fp32 && out_cols % GW == 0 && n0 + out_cols <= p.N;
  if (!staged) {
    epilogue_direct(p, taddr, pair_col_off, row, n0, out_cols, paired, aligned);
    return;
  }
  uint4* my_row = reinterpret_cast<uint4*>(stage_warp + lane * (2 * GW));
  const int swz = lane & (CH - 1);
#pragma unroll 1
  for (int g = 0; g < out_cols / GW; ++g) {
#pragma unroll 1
    for (int c = 0; c < GW / 32; ++c) {
      uint32_t r0[32], r1[32];
      tmem_ld_32x32b_x32(taddr + g * GW + c * 32, r0);
      if (paired) tmem_ld_32x32b_x32(taddr + pair_col_off + g * GW + c * 32, r1);
      tmem_wait_ld();
      epilogue_row32(p, row, n0 + g * GW + c * 32, r0, r1, paired, true, my_row, c * 4, swz);
    }
    __syncwarp();
    const int chunk = lane & (CH - 1);
#pragma unroll 4
    for (int i = 0; i < CH; ++i) {
      const int rl = (32 / CH) * i + lane / CH;                 // row of the warp this lane copies in this pass
      const int rr = __shfl_sync(0xffffffffu, row, rl);         // its global output row (p.M or more: not stored)
      const uint4 v = reinterpret_cast<const uint4*>(stage_warp + rl * (2 * GW))[chunk ^ (rl & (CH - 1))];
      if (rr < p.M) *reinterpret_cast<uint4*>(out_slab_ptr(p, rr, n0 + g * GW + chunk * 8, 2)) = v;
    }
    __syncwarp();
  }
}

// eight bf16 terms of the epilogue, kept packed until they are used; n of them exist, the rest reads as `fill`
__device__ __noinline__ uint4 load_terms_tail(const __nv_bfloat16* p, int n, uint32_t fill) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t lo = 2 * i < n ? reinterpret_cast<const uint16_t*>(p)[2 * i] : fill & 0xffffu;
    const uint32_t hi = 2 * i + 1 < n ? reinterpret_cast<const uint16_t*>(p)[2 * i + 1] : fill >> 16;
    w[i] = lo | hi << 16;
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ uint4 load_terms(const __nv_bfloat16* p, int n, uint32_t fill) {
  return n >= 8 ? *reinterpret_cast<const uint4*>(p) : load_terms_tail(p, n, fill);
}
// wait for the TMEM loads of this thread; r is tied to it, so that nothing computed from r moves above
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                 "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]),
                 "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]),
                 "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}

// Epilogue of one accumulator tile for one warp when the output is a local bf16 matrix (GemmParams::bulk_out). What bounds it is
// latency: a warp is alone on its scheduler and next to 227 KB of shared memory there is no L1 to speak of, so every global load
// in the loop over the columns costs 350 to 700 cycles, every run-time flag 40. A tile of 256 columns took 10 000 cycles (15 000
// with a bias, 21 000 with GELU, 29 000 with gate and residual): bias and residual were loaded per 32-column slab, and the staged
// rows were copied out with a division-laden address per 16 bytes. Here it takes 6 000, 6 000, 11 500 and 12 200: 8192 x 5120 x 640
// with bias 91 -> 51 us, with GELU 121 -> 80, with gate and residual 159 -> 94 (B200, cold L2). Eight warps instead of four take no less
// (TMEM reads and shuffles are shared) and spill.
//  - load() runs before the accumulator is complete: each lane holds eight of the tile's columns of bias, gate and scales, which a
//    slab gets by warp shuffles, and the first 64 columns of its row's residual (the next 64 are always on their way);
//  - a missing term is replaced by its neutral value (-0 added, 1 multiplied: exact) instead of a branch; run() is compiled with and
//    without gate and residual (TERMS), and in the pair kernel for no activation and both GELUs by themselves;
//  - the next slab's TMEM load is in flight while one is computed;
//  - 64 columns of the warp's 32 rows leave as one tiled bulk store from a swizzled 4 KB buffer (two per warp), which also clips
//    ragged rows, columns and image edges.
// The arithmetic per element is that of epilogue_row32, which rounds each product before it adds: hence __fmul_rn here, where no branch
// keeps the compiler from contracting scale * value + bias or gate * value + residual.
constexpr uint32_t TERM_ZERO = 0x80008000u, TERM_ONE = 0x3f803f80u;     // bf16 pairs: -0 and 1
template <int KIND>
struct BulkEpilogue {
  const GemmParams& p;
  int row, n0, out_cols, lane;      // row: this lane's output row (for residual, gate and row scale); p.M or more is not stored
  bool paired;
  uint4 bias, bias2, gate;
  uint4 res[8];
  float scale[KIND == 1 ? 8 : 1], scale2[KIND == 1 ? 8 : 1];
  bool gate_shared;                 // the warp's rows have one gate

  __device__ __forceinline__ BulkEpilogue(const GemmParams& p_, int row_, int n0_, int out_cols_, int lane_, bool paired_)
      : p(p_), row(row_), n0(n0_), out_cols(out_cols_), lane(lane_), paired(paired_), gate_shared(true) {}
  __device__ __forceinline__ int term_row() const { return row < p.M ? row : p.M - 1; }
  __device__ __forceinline__ const __nv_bfloat16* gate_row() const { return p.gate + static_cast<size_t>(term_row() / p.rows_per_group) * p.gate_stride; }
  __device__ __forceinline__ void load_residual(int col, uint4 (&d)[8]) const {
    const __nv_bfloat16* r = p.residual + static_cast<size_t>(term_row()) * p.ld_res + col;
#pragma unroll
    for (int i = 0; i < 8; ++i) d[i] = load_terms(r + 8 * i, p.N - col - 8 * i, TERM_ZERO);
  }
  __device__ __forceinline__ void load() {
    const int c = n0 + lane * 8, n = lane * 8 < out_cols ? p.N - c : 0;
    bias = bias2 = make_uint4(TERM_ZERO, TERM_ZERO, TERM_ZERO, TERM_ZERO);
    gate = make_uint4(TERM_ONE, TERM_ONE, TERM_ONE, TERM_ONE);
    if (p.bias) {
      bias = load_terms(p.bias + c, n, TERM_ZERO);
      if (paired) bias2 = load_terms(p.bias + c + p.pair_offset, n, TERM_ZERO);
    }
    if (p.gate) {
      const int g = term_row() / p.rows_per_group;
      gate_shared = __all_sync(0xffffffffu, g == __shfl_sync(0xffffffffu, g, 0));
      if (gate_shared) gate = load_terms(gate_row() + c, n, TERM_ONE);
    }
    if (KIND == 1) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        scale[j] = p.col_scale && j < n ? p.col_scale[c + j] : 1.f;
        scale2[j] = p.col_scale && paired && j < n ? p.col_scale[c + p.pair_offset + j] : 1.f;
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) res[i] = make_uint4(TERM_ZERO, TERM_ZERO, TERM_ZERO, TERM_ZERO);
    if (p.residual) load_residual(n0, res);
  }
  // v op= the terms of slab s, eight columns per lane from lanes 4 s .. 4 s + 3
  template <bool MUL>
  __device__ __forceinline__ void columns(const uint4& u, int s, float (&v)[32]) const {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const uint32_t mine = (k & 3) == 0 ? u.x : (k & 3) == 1 ? u.y : (k & 3) == 2 ? u.z : u.w;
      const float2 f = unpack_bf16x2(__shfl_sync(0xffffffffu, mine, 4 * s + (k >> 2)));
      v[2 * k] = MUL ? __fmul_rn(v[2 * k], f.x) : v[2 * k] + f.x;
      v[2 * k + 1] = MUL ? __fmul_rn(v[2 * k + 1], f.y) : v[2 * k + 1] + f.y;
    }
  }
  __device__ __forceinline__ void scales(const float* sc, int s, float (&v)[32]) const {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __fmul_rn(v[j], __shfl_sync(0xffffffffu, sc[j & 7], 4 * s + (j >> 3)));
  }
  // turn: bulk stores this warp has issued, which take the staging buffers in turn; release(): called once the accumulator has been
  // read; store(buffer, column): issues the bulk store of 64 columns
  template <bool PAIRED, int ACT, bool TERMS, int BUFFERS, typename Release, typename Store>
  __device__ __forceinline__ void run_mode(uint32_t taddr, int pair_col_off, uint8_t* stage, int& turn, Release release, Store store) {
    const float rs = (KIND == 1 && p.row_scale ? p.row_scale[term_row()] : 1.f) * p.alpha;
    uint32_t r[32], r2[32];
    tmem_ld_32x32b_x32(taddr, r);
    if (PAIRED) tmem_ld_32x32b_x32(taddr + pair_col_off, r2);
    const int groups = min(out_cols, p.N - n0 + 63) / 64;            // those with a column of the matrix: every group is stored
#pragma unroll 1
    for (int g = 0; g < groups; ++g) {
      uint4 now[8];
      if (TERMS) {
#pragma unroll
        for (int i = 0; i < 8; ++i) now[i] = res[i];
        if (p.residual && g + 1 < groups) load_residual(n0 + g * 64 + 64, res);
      }
      uint8_t* buf = stage + (turn++ % BUFFERS) * 4096;
      uint4* my_row = reinterpret_cast<uint4*>(buf + lane * 128);
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int s = 2 * g + half;
        float v[32], w[32];
        tmem_wait_ld(r);
        if (PAIRED) tmem_wait_ld(r2);
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          v[j] = KIND == 1 ? __fmul_rn(__uint_as_float(r[j]), rs) : __uint_as_float(r[j]);      // bf16 operands: rs is 1
          if (PAIRED) w[j] = KIND == 1 ? __fmul_rn(__uint_as_float(r2[j]), rs) : __uint_as_float(r2[j]);
        }
        if (half == 0 || g + 1 < groups) {
          tmem_ld_32x32b_x32(taddr + (s + 1) * 32, r);
          if (PAIRED) tmem_ld_32x32b_x32(taddr + pair_col_off + (s + 1) * 32, r2);
        } else {
          release();
        }
        if (KIND == 1) scales(scale, s, v);
        columns<false>(bias, s, v);
        if (PAIRED) {
          if (KIND == 1) scales(scale2, s, w);
          columns<false>(bias2, s, w);
          if (p.act_on_second) {
#pragma unroll
            for (int j = 0; j < 32; ++j) { const float x = v[j]; v[j] = w[j]; w[j] = x; }
          }
        }
        if (ACT < 0) act32_rt(p.act, v);
        else act32<ACT>(v);
        if (PAIRED) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] *= w[j];
        }
        if (TERMS) {
          if (gate_shared) {
            columns<true>(gate, s, v);
          } else {
            const int col = n0 + s * 32;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint4 u = load_terms(gate_row() + col + 8 * i, p.N - col - 8 * i, TERM_ONE);
              const uint32_t x[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const float2 f = unpack_bf16x2(x[k]);
                v[8 * i + 2 * k] = __fmul_rn(v[8 * i + 2 * k], f.x);
                v[8 * i + 2 * k + 1] = __fmul_rn(v[8 * i + 2 * k + 1], f.y);
              }
            }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t x[4] = {now[4 * half + i].x, now[4 * half + i].y, now[4 * half + i].z, now[4 * half + i].w};
#pragma unroll
            for (int k = 0; k < 4; ++k) { const float2 f = unpack_bf16x2(x[k]); v[8 * i + 2 * k] += f.x; v[8 * i + 2 * k + 1] += f.y; }
          }
        }
        if (half == 0) {
          if (lane == 0) tma_store_wait_read<BUFFERS - 1>();      // the store that used this buffer last has read it
          __syncwarp();
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
          my_row[(half * 4 + j) ^ (lane & 7)] = make_uint4(pack_bf16x2(v[8 * j], v[8 * j + 1]), pack_bf16x2(v[8 * j + 2], v[8 * j + 3]),
                                                           pack_bf16x2(v[8 * j + 4], v[8 * j + 5]), pack_bf16x2(v[8 * j + 6], v[8 * j + 7]));
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        store(buf, n0 + g * 64);
        tma_store_commit();
      }
    }
  }
  template <bool PAIRED, bool FIXED, int BUFFERS, typename Release, typename Store>
  __device__ __forceinline__ void run(uint32_t taddr, int pair_col_off, uint8_t* stage, int& turn, Release release, Store store) {
    const bool terms = !PAIRED && (p.gate || p.residual);
#define MDB_RUN(ACT_, TERMS_) run_mode<PAIRED, ACT_, TERMS_, BUFFERS>(taddr, pair_col_off, stage, turn, release, store)
    if (!PAIRED && terms && p.act == MDB_ACT_NONE) MDB_RUN(MDB_ACT_NONE, !PAIRED);
    else if (!PAIRED && terms) MDB_RUN(-1, !PAIRED);
    else if (!PAIRED && p.act == MDB_ACT_NONE) MDB_RUN(MDB_ACT_NONE, false);
    else if (FIXED && p.act == MDB_ACT_GELU_TANH) MDB_RUN(FIXED ? MDB_ACT_GELU_TANH : -1, false);
    else if (FIXED && p.act == MDB_ACT_GELU_ERF) MDB_RUN(FIXED ? MDB_ACT_GELU_ERF : -1, false);
    else MDB_RUN(-1, false);
#undef MDB_RUN
  }
};

__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Tile -> (m block, n block). Plain GEMM: m fastest. With a fused all-gather the gathered operand's blocks are
// visited starting at the local chunk (already present), then in the order the gather warps fetch the peers.
__device__ __forceinline__ int tile_m_index(const GemmParams& p, int tile, int tiles_m, int tiles_n) {
  if (p.gather_world > 1 && p.gather_operand == 1) return tile % tiles_m;
  int m = tile % tiles_m;
  if (p.gather_world > 1) {
    const int shift = (p.gather_rank * p.gather_chunk_rows) / BM;
    m = (m + shift) % tiles_m;
  }
  return m;
}
__device__ __forceinline__ int tile_n_index(const GemmParams& p, int tile, int tiles_m, int tiles_n) {
  int n = tile / tiles_m;
  if (p.gather_world > 1 && p.gather_operand == 1) {
    const int bn_rows = (p.N + tiles_n - 1) / tiles_n;
    const int shift = (p.gather_rank * p.gather_chunk_rows) / max(bn_rows, 1);
    n = (n + shift) % tiles_n;
  }
  return n;
}

// KIND: 0 = bf16 operands (kind::f16), 1 = fp8 e4m3 operands (kind::f8f6f4)
// BULK: GemmParams::bulk_out
template <int BN, int STAGES, bool A_MN, bool B_MN, int KIND, bool BULK>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_tcgen05_kernel(const __grid_constant__ GemmMaps maps, const __grid_constant__ GemmParams p) {
  constexpr int A_BYTES = BM * BK_BYTES;
  constexpr int B_BYTES = BN * BK_BYTES;
  constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr int TMEM_COLS = (2 * BN < 32) ? 32 : 2 * BN;
  constexpr int KSTEPS = 4;  // 128-byte rows / 32 bytes per UMMA K step
  static_assert(!(KIND == 1 && (A_MN || B_MN)), "fp8 operands are K-major only");

  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full_bar[STAGES];
  __shared__ uint64_t empty_bar[STAGES];
  __shared__ uint64_t tfull_bar[2];
  __shared__ uint64_t tempty_bar[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;
  __shared__ uint64_t gather_bar[GATHER_STAGES];

  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&tfull_bar[s], 1);
      mbar_init(&tempty_bar[s], 4);
    }
    for (int s = 0; s < GATHER_STAGES; ++s) mbar_init(&gather_bar[s], 1);
    abort_s = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(&tmem_base_s, TMEM_COLS);
    tmem_relinquish();
  }
  if (warp == 0 && lane == 0) {
    for (int s = 0; s < p.num_seg; ++s) {
      tma_prefetch_desc(&maps.a[s]);
      tma_prefetch_desc(&maps.b[s]);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_s;

  const int tiles_m = p.conv_taps > 0 ? p.conv_tiles_m : (p.M + BM - 1) / BM;
  const int tiles_n = (p.N + (p.pair_offset > 0 ? BN / 2 : BN) - 1) / (p.pair_offset > 0 ? BN / 2 : BN);
  const int num_tiles = tiles_m * tiles_n;
  int total_kb = 0;
  for (int s = 0; s < p.num_seg; ++s) total_kb += p.kblocks[s];
  constexpr int K_ELEMS = (KIND == 0) ? 64 : 128;  // elements per 128-byte row

  if (warp == 0) {
    // ------------------------------- TMA producer -------------------------------
    // The whole warp runs the loop (waits included) and elect.sync picks the lane that issues: tcgen05 / TMA instructions
    // issued from a convergent warp cost about 120 cycles each, from inside a one-lane branch about 190 (measured), which
    // is more than the 128 cycles a 128 x 256 x 16 MMA takes.
    {
      int stage = 0;
      uint32_t phase = 0;
      int last_stage = -1;
      uint32_t last_phase = 0;
      bool ok = true;
      long long t_wait = 0;
      unsigned chunk_seen = 1u << p.gather_rank;   // chunks whose arrival this CTA has already observed
      int n_trace = 0;
      for (int tile = blockIdx.x; ok && tile < num_tiles; tile += gridDim.x) {
        const int m0 = tile_m_index(p, tile, tiles_m, tiles_n) * BM;
        const int nblk = tile_n_index(p, tile, tiles_m, tiles_n);
        const int n0 = p.pair_offset > 0 ? nblk * (BN / 2) : nblk * BN;
        if (p.gather_world > 1) {
          // every chunk this tile touches must have landed (a tile may straddle two chunks)
          const int r0 = p.gather_operand == 0 ? m0 : n0;
          const int r1 = r0 + (p.gather_operand == 0 ? BM : BN) - 1;
          const int c_lo = min(r0 / p.gather_chunk_rows, p.gather_world - 1);
          const int c_hi = min(r1 / p.gather_chunk_rows, p.gather_world - 1);
          for (int c = c_lo; ok && c <= c_hi; ++c) {
            if (chunk_seen & (1u << c)) continue;
            const uint64_t t0 = globaltimer_ns();
            uint32_t spins = 0;
            bool mine = true;
            while (ld_acquire_gpu(p.gather_ready + c) < static_cast<int>(gridDim.x)) {
              if ((++spins & 0xffu) == 0 && (abort_s || globaltimer_ns() - t0 > MDB_WAIT_LIMIT_NS)) {
                abort_s = 1;
                mine = false;
                break;
              }
            }
            if (!__all_sync(0xffffffffu, mine)) {
              if (lane == 0) report_status(p.status, STATUS_TIMEOUT, 5, c);
              ok = false;
              break;
            }
            chunk_seen |= 1u << c;
          }
          if (!ok) break;
          asm volatile("fence.proxy.async.global;" ::: "memory");   // peer-copied bytes -> visible to the TMA reads
        }
        for (int s = 0; ok && s < p.num_seg; ++s) {
          for (int kb = 0; kb < p.kblocks[s]; ++kb) {
            const long long tw0 = p.prof ? clock64() : 0;
            if (!__all_sync(0xffffffffu, mbar_wait(&empty_bar[stage], phase ^ 1u, &abort_s))) {
              if (lane == 0) report_status(p.status, STATUS_TIMEOUT, 1, stage);
              ok = false;
              break;
            }
            if (p.prof) t_wait += clock64() - tw0;
            if (p.trace && lane == 0 && blockIdx.x < 2 && n_trace < p.trace_len) p.trace[(blockIdx.x * 3 + 0) * p.trace_len + n_trace++] = clock64();
            uint8_t* sa = smem + stage * STAGE_BYTES;
            uint8_t* sb = sa + A_BYTES;
            int k0 = kb * K_ELEMS;
            if (elect_one()) {
              mbar_expect_tx(&full_bar[stage], STAGE_BYTES);
              if (p.conv_taps > 0) {
                // tile -> (image, patch row, patch col); k block -> (filter tap, channel block)
                const int mt = tile % tiles_m;
                const int tw = mt % p.conv_tiles_w, th = (mt / p.conv_tiles_w) % p.conv_tiles_h;
                const int img = mt / (p.conv_tiles_w * p.conv_tiles_h);
                const int tap = kb / p.conv_cblocks, cb = kb - tap * p.conv_cblocks;
                const int kh = tap / p.conv_kw, kw = tap - kh * p.conv_kw;
                tma_load_4d(sa, &maps.a[s], &full_bar[stage], cb * K_ELEMS, tw * CONV_TW + kw - p.conv_pad_w,
                            th * CONV_TH + kh - p.conv_pad_h, img);
                k0 = (tap * p.conv_cblocks + cb) * K_ELEMS;
              } else if (!A_MN) {
                tma_load_2d(sa, &maps.a[s], &full_bar[stage], k0, m0);
              } else {
                // boxes [64 m-elements][64 k-rows], 8 KB each
                tma_load_2d(sa, &maps.a[s], &full_bar[stage], m0, k0);
                tma_load_2d(sa + 8192, &maps.a[s], &full_bar[stage], m0 + 64, k0);
              }
              if (!B_MN) {
                constexpr int HALF_ROWS = BN / 2;
                const int n1 = p.pair_offset > 0 ? n0 + p.pair_offset : n0 + HALF_ROWS;
                tma_load_2d(sb, &maps.b[s], &full_bar[stage], k0, n0);
                tma_load_2d(sb + HALF_ROWS * BK_BYTES, &maps.b[s], &full_bar[stage], k0, n1);
              } else {
#pragma unroll
                for (int j = 0; j < BN / 64; ++j)
                  tma_load_2d(sb + j * 8192, &maps.b[s], &full_bar[stage], n0 + j * 64, k0);
              }
            }
            __syncwarp();
            last_stage = stage;
            last_phase = phase;
            if (++stage == STAGES) {
              stage = 0;
              phase ^= 1u;
            }
          }
        }
      }
      if (p.prof && lane == 0) p.prof[blockIdx.x * 8 + 1] = t_wait;
      if (!ok && last_stage >= 0) {
        // abandoned: let the copies already in flight land before the CTA goes away (bounded)
        uint64_t t0 = globaltimer_ns();
        while (!mbar_try_wait(&full_bar[last_stage], last_phase) && globaltimer_ns() - t0 < 5000000ull) {
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------- UMMA issuer --------------------------------
    // whole warp in the loop, elect.sync for the issuing lane (see the producer)
    {
      constexpr uint32_t idesc =
          (KIND == 0) ? make_idesc(1, UMMA_BF16, UMMA_BF16, A_MN ? 1u : 0u, B_MN ? 1u : 0u, BM, BN)
                      : make_idesc(1, UMMA_E4M3, UMMA_E4M3, 0u, 0u, BM, BN);
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      bool ok = true;
      long long t_full = 0, t_tempty = 0;
      int n_trace = 0;
      const long long t_begin = p.prof ? clock64() : 0;
      for (int tile = blockIdx.x; ok && tile < num_tiles; tile += gridDim.x, ++it) {
        const int acc = it & 1;
        const uint32_t acc_phase = (it >> 1) & 1;
        const long long te0 = p.prof ? clock64() : 0;
        if (!__all_sync(0xffffffffu, mbar_wait(&tempty_bar[acc], acc_phase ^ 1u, &abort_s))) {
          if (lane == 0) report_status(p.status, STATUS_TIMEOUT, 2, acc);
          break;
        }
        if (p.prof) t_tempty += clock64() - te0;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < total_kb; ++kb) {
          const long long tf0 = p.prof ? clock64() : 0;
          if (!__all_sync(0xffffffffu, mbar_wait(&full_bar[stage], phase, &abort_s))) {
            if (lane == 0) report_status(p.status, STATUS_TIMEOUT, 3, stage);
            ok = false;
            break;
          }
          if (p.prof) t_full += clock64() - tf0;
          if (p.trace && lane == 0 && blockIdx.x < 2 && n_trace < p.trace_len) p.trace[(blockIdx.x * 3 + 1) * p.trace_len + n_trace++] = clock64();
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * STAGE_BYTES);
          const uint32_t sb = sa + A_BYTES;
          const uint64_t da = A_MN ? make_desc_mnmajor_sw128(sa, 8192) : make_desc_kmajor_sw128(sa);
          const uint64_t db = B_MN ? make_desc_mnmajor_sw128(sb, 8192) : make_desc_kmajor_sw128(sb);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < KSTEPS; ++k) {
              // K-major: 32 bytes along the row per step; MN-major: 16 K-rows of 128 B per step
              const uint64_t a_k = da + static_cast<uint64_t>(A_MN ? (k * 2048) >> 4 : (k * 32) >> 4);
              const uint64_t b_k = db + static_cast<uint64_t>(B_MN ? (k * 2048) >> 4 : (k * 32) >> 4);
              if (KIND == 0)
                umma_f16_ss(d_tmem, a_k, b_k, idesc, (kb | k) != 0 ? 1u : 0u);
              else
                umma_f8_ss(d_tmem, a_k, b_k, idesc, (kb | k) != 0 ? 1u : 0u);
            }
            umma_commit(&empty_bar[stage]);  // smem slot free once these UMMAs have read it
            if (kb == total_kb - 1) umma_commit(&tfull_bar[acc]);
          }
          __syncwarp();
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      if (p.prof && lane == 0) {
        p.prof[blockIdx.x * 8 + 0] = clock64() - t_begin;
        p.prof[blockIdx.x * 8 + 2] = t_full;
        p.prof[blockIdx.x * 8 + 3] = t_tempty;
        p.prof[blockIdx.x * 8 + 6] = it;
      }
    }
    __syncwarp();
  } else if (warp == 6) {
    // ------------------------------- peer gather (all-gather fused GEMM) --------
    if (p.gather_world > 1 && lane == 0) {
      // One thread streams this CTA's share of every peer chunk through two 16 KB shared-memory stages with bulk copies:
      // peer memory -> shared (completion on an mbarrier), shared -> the local gathered buffer (bulk group). 32 KB are in
      // flight per CTA, which keeps NVLink busy from all SMs together; nothing passes through registers.
      uint8_t* gs = smem + STAGES * STAGE_BYTES;
      const long long pieces = (p.gather_chunk_bytes + GATHER_PIECE - 1) / GATHER_PIECE;
      uint32_t ph[GATHER_STAGES] = {0, 0};
      bool ok = true;
      for (int i = 1; i < p.gather_world && ok; ++i) {
        const int c = (p.gather_rank + i) % p.gather_world;
        const char* src = reinterpret_cast<const char*>(p.gather_src[c]);
        char* dst = reinterpret_cast<char*>(p.gather_dst) + c * p.gather_chunk_bytes;
        const long long mine = blockIdx.x < pieces ? (pieces - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
        auto piece_off = [&](long long k) { return (static_cast<long long>(blockIdx.x) + k * gridDim.x) * GATHER_PIECE; };
        auto piece_len = [&](long long k) {
          const long long rem = p.gather_chunk_bytes - piece_off(k);
          return static_cast<uint32_t>(rem < GATHER_PIECE ? rem : GATHER_PIECE);
        };
        auto issue = [&](long long k) {
          const int sgi = static_cast<int>(k % GATHER_STAGES);
          mbar_expect_tx(&gather_bar[sgi], piece_len(k));
          bulk_load_g2s(gs + sgi * GATHER_PIECE, src + piece_off(k), piece_len(k), &gather_bar[sgi]);
        };
        long long issued = 0;
        for (; issued < mine && issued < GATHER_STAGES; ++issued) issue(issued);
        for (long long k = 0; k < mine; ++k) {
          const int sgi = static_cast<int>(k % GATHER_STAGES);
          if (!mbar_wait(&gather_bar[sgi], ph[sgi], &abort_s)) {
            report_status(p.status, STATUS_TIMEOUT, 70, c);
            ok = false;
            // bounded drain of the loads still in flight (jobs k .. issued-1), so that nothing lands in shared memory
            // after this CTA has left
            for (long long j = k; j < issued; ++j) {
              const int sj = static_cast<int>(j % GATHER_STAGES);
              const uint64_t t0 = globaltimer_ns();
              while (!mbar_try_wait(&gather_bar[sj], ph[sj]) && globaltimer_ns() - t0 < MDB_WAIT_LIMIT_NS) {}
            }
            break;
          }
          ph[sgi] ^= 1;
          bulk_store_s2g(dst + piece_off(k), gs + sgi * GATHER_PIECE, piece_len(k));
          tma_store_commit();
          if (issued < mine) {
            tma_store_wait_read<0>();                      // the stage has been read out: it may be refilled
            issue(issued++);
          }
        }
        tma_store_wait<0>();                               // this CTA's share of chunk c is in the gathered buffer
        if (!ok) break;
        __threadfence();
        atomicAdd(p.gather_ready + c, 1);
      }
    }
  } else {
    // ------------------------------- epilogue (4 warps) -------------------------
    const int quad = warp & 3;  // TMEM lane quadrant this warp may access
    const bool paired = p.pair_offset > 0;
    // the vector epilogue needs 16-byte aligned rows in every tensor it touches (columns advance in 64-byte steps)
    const int esz = p.out_fp32 ? 4 : 2;
    bool aligned = ((reinterpret_cast<uintptr_t>(p.out) | static_cast<uintptr_t>(static_cast<size_t>(p.ld_out) * esz)) & 15) == 0;
    if (p.bias) aligned = aligned && ((reinterpret_cast<uintptr_t>(p.bias) | static_cast<uintptr_t>(p.pair_offset * 2)) & 15) == 0;
    if (p.col_scale) aligned = aligned && ((reinterpret_cast<uintptr_t>(p.col_scale) | static_cast<uintptr_t>(p.pair_offset * 4)) & 15) == 0;
    if (p.gate) aligned = aligned && ((reinterpret_cast<uintptr_t>(p.gate) | static_cast<uintptr_t>(p.gate_stride * 2)) & 15) == 0;
    if (p.residual) aligned = aligned && ((reinterpret_cast<uintptr_t>(p.residual) | static_cast<uintptr_t>(static_cast<size_t>(p.ld_res) * 2)) & 15) == 0;
    int it = 0, turn = 0;
    long long t_twait = 0, t_work = 0;
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x, ++it) {
      const int acc = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1;
      const int m0 = tile_m_index(p, tile, tiles_m, tiles_n) * BM;
      const int nblk = tile_n_index(p, tile, tiles_m, tiles_n);
      const int n0 = paired ? nblk * (BN / 2) : nblk * BN;
      const int out_cols = paired ? BN / 2 : BN;
      int row = m0 + quad * 32 + lane, img = 0, ow0 = 0, oh0 = 0;
      if (p.conv_taps > 0) {
        const int mt = tile % tiles_m;
        const int tw = mt % p.conv_tiles_w, th = (mt / p.conv_tiles_w) % p.conv_tiles_h;
        img = mt / (p.conv_tiles_w * p.conv_tiles_h);
        ow0 = tw * CONV_TW;
        oh0 = th * CONV_TH + quad * (32 / CONV_TW);
        const int oh = oh0 + lane / CONV_TW, ow = ow0 + lane % CONV_TW;
        row = (oh < p.conv_h && ow < p.conv_w) ? (img * p.conv_h + oh) * p.conv_w + ow : p.M;  // p.M = skipped
      }
      BulkEpilogue<KIND> bulk(p, row, n0, out_cols, lane, paired);
      if (BULK) bulk.load();
      const long long tq0 = p.prof ? clock64() : 0;
      // warp-uniform decision: the TMEM loads below are warp-collective
      const bool got = __all_sync(0xffffffffu, mbar_wait(&tfull_bar[acc], acc_phase, &abort_s));
      if (!got) {
        if (lane == 0) report_status(p.status, STATUS_TIMEOUT, 4, acc);
        break;
      }
      tc_fence_after();
      const long long tq1 = p.prof ? clock64() : 0;
      t_twait += tq1 - tq0;
      if (p.trace && blockIdx.x < 2 && warp == 2 && lane == 0 && 2 * it + 1 < p.trace_len) p.trace[(blockIdx.x * 3 + 2) * p.trace_len + 2 * it] = clock64();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + acc * BN;
      uint8_t* stages = smem + STAGES * STAGE_BYTES;
      auto release = [&] {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty_bar[acc]);
      };
      if constexpr (BULK) {
        auto store = [&](const uint8_t* buf, int col) {
          if (p.conv_taps > 0) {
            if (oh0 < p.conv_h) tma_store_4d(&maps.out, buf, col, ow0, oh0, img);
          } else if (m0 + quad * 32 < p.M) {
            tma_store_2d(&maps.out, buf, col, m0 + quad * 32);
          }
        };
        if (BN == 256 && paired) bulk.template run<BN == 256, false, 2>(taddr, BN / 2, stages + quad * 8192, turn, release, store);
        else bulk.template run<false, false, 2>(taddr, 0, stages + quad * 8192, turn, release, store);
      } else {
        // the staging buffers share their 32 KB with the stages of the fused all-gather, which therefore stores directly
        epilogue_tile(p, taddr, BN / 2, row, n0, out_cols, paired, aligned, p.gather_world > 1 ? nullptr : stages + quad * 8192, lane);
        release();
      }
      if (p.prof) t_work += clock64() - tq1;
      if (p.trace && blockIdx.x < 2 && warp == 2 && lane == 0 && 2 * it + 1 < p.trace_len) p.trace[(blockIdx.x * 3 + 2) * p.trace_len + 2 * it + 1] = clock64();
    }
    if (BULK && lane == 0) tma_store_wait<0>();   // the rows are out before the staging buffers go away
    if (p.prof && warp == 2 && lane == 0) {
      p.prof[blockIdx.x * 8 + 4] = t_twait;
      p.prof[blockIdx.x * 8 + 5] = t_work;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------------
// CTA-pair variant: one 256 x 256 output tile per cluster of two CTAs (tcgen05 cta_group::2). Each CTA stages its
// own 128 rows of A and its own 128 rows of B per K block (32 KB instead of the 48 KB a lone 128 x 256 CTA needs for
// the same MMA time), so the shared-memory fill rate, which bounds the one-CTA kernel on DiT shapes, drops by a third
// and the ring is 6 stages deep. The even CTA issues the MMAs for both; each CTA reads its own 128 x 256 fp32
// accumulator from its own TMEM and runs the same fused epilogue. bf16 operands of any majors or K-major fp8 (KIND 1),
// paired (GLU) mode, routed / staged-reduce epilogues; no fused gather or convolution (the gather stays on the
// one-CTA kernel, 3 x 3 convolutions have a pair kernel of their own below).
// ---------------------------------------------------------------------------------
constexpr int PAIR_THREADS = 192;  // warps: 0 TMA, 1 UMMA issue (leader only), 2-5 epilogue

template <int STAGES, bool A_MN, bool B_MN, int KIND, bool BULK>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1)
gemm_tcgen05_pair_kernel(const __grid_constant__ GemmMaps maps, const __grid_constant__ GemmParams p) {
  constexpr int BN = 256;               // accumulator columns per CTA (the whole tile width)
  constexpr int BNH = 128;              // B rows staged by one CTA
  constexpr int A_BYTES = BM * BK_BYTES;
  constexpr int B_BYTES = BNH * BK_BYTES;
  constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr int TMEM_COLS = 2 * BN;
  constexpr int KSTEPS = 4;
  constexpr int K_ELEMS = (KIND == 0) ? 64 : 128;
  static_assert(!(KIND == 1 && (A_MN || B_MN)), "fp8 operands are K-major only");

  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full_bar[STAGES];    // used in the leader: both CTAs' loads of a stage have landed
  __shared__ uint64_t empty_bar[STAGES];   // in each CTA: the MMAs that read this stage are done
  __shared__ uint64_t tfull_bar[2];        // in each CTA: accumulator complete
  __shared__ uint64_t tempty_bar[2];       // used in the leader: 8 epilogue warps (4 per CTA) have drained the accumulator
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;

  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&tfull_bar[s], 1);
      mbar_init(&tempty_bar[s], 8);
    }
    abort_s = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(&tmem_base_s, TMEM_COLS);
    tmem_relinquish_pair();
  }
  if (warp == 0 && lane == 0) {
    for (int s = 0; s < p.num_seg; ++s) {
      tma_prefetch_desc(&maps.a[s]);
      tma_prefetch_desc(&maps.b[s]);
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_arrive();   // the peer's barriers exist before anything is sent to them
  cluster_wait();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_s;
  const uint32_t peer_abort = mapa_shared(smem_u32(&abort_s), rank ^ 1u);

  const bool paired = p.pair_offset > 0;
  const int tiles_m = (p.M + 2 * BM - 1) / (2 * BM);
  const int tiles_n = (p.N + (paired ? BNH : BN) - 1) / (paired ? BNH : BN);
  const int num_tiles = tiles_m * tiles_n;
  const int cluster_id = blockIdx.x >> 1, num_clusters = gridDim.x >> 1;
  int total_kb = 0;
  for (int s = 0; s < p.num_seg; ++s) total_kb += p.kblocks[s];

  if (warp == 0) {
    // ------------------------------- TMA producer (both CTAs) -------------------
    // whole warp in the loop, elect.sync for the issuing lane (see the one-CTA kernel)
    {
      int stage = 0;
      uint32_t phase = 0;
      int last_stage = -1;
      bool ok = true;
      long long t_wait = 0;
      int n_trace = 0;
      for (int tile = cluster_id; ok && tile < num_tiles; tile += num_clusters) {
        const int m0 = (tile % tiles_m) * (2 * BM) + static_cast<int>(rank) * BM;
        const int nblk = tile / tiles_m;
        // this CTA's 128 rows of B: the lower / upper half of the tile, or in paired mode the first / second operand
        const int n0 = paired ? nblk * BNH + (leader ? 0 : p.pair_offset) : nblk * BN + static_cast<int>(rank) * BNH;
        for (int s = 0; ok && s < p.num_seg; ++s) {
          for (int kb = 0; kb < p.kblocks[s]; ++kb) {
            const long long tw0 = p.prof ? clock64() : 0;
            if (!__all_sync(0xffffffffu, mbar_wait(&empty_bar[stage], phase ^ 1u, &abort_s))) {
              if (lane == 0) {
                report_status(p.status, STATUS_TIMEOUT, 21, stage);
                st_shared_cluster_u32(peer_abort, 1u);
              }
              ok = false;
              break;
            }
            if (p.prof) t_wait += clock64() - tw0;
            if (p.trace && lane == 0 && blockIdx.x < 2 && n_trace < p.trace_len) p.trace[(blockIdx.x * 3 + 0) * p.trace_len + n_trace++] = clock64();
            uint8_t* sa = smem + stage * STAGE_BYTES;
            uint8_t* sb = sa + A_BYTES;
            const uint32_t bar = mapa_shared(smem_u32(&full_bar[stage]), 0u);
            const int k0 = kb * K_ELEMS;
            if (elect_one()) {
              if (leader) mbar_expect_tx(&full_bar[stage], 2 * STAGE_BYTES);
              if (!A_MN) {
                tma_load_2d_pair(sa, &maps.a[s], bar, k0, m0);
              } else {
                tma_load_2d_pair(sa, &maps.a[s], bar, m0, k0);
                tma_load_2d_pair(sa + 8192, &maps.a[s], bar, m0 + 64, k0);
              }
              if (!B_MN) {
                tma_load_2d_pair(sb, &maps.b[s], bar, k0, n0);
              } else {
                tma_load_2d_pair(sb, &maps.b[s], bar, n0, k0);
                tma_load_2d_pair(sb + 8192, &maps.b[s], bar, n0 + 64, k0);
              }
            }
            __syncwarp();
            last_stage = stage;
            if (++stage == STAGES) {
              stage = 0;
              phase ^= 1u;
            }
          }
        }
      }
      if (p.prof && lane == 0) p.prof[blockIdx.x * 8 + 1] = t_wait;
      if (!ok && last_stage >= 0) {
        // abandoned: give the copies already in flight time to land before the CTA goes away (bounded)
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 2000000ull) {
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------- UMMA issuer (leader CTA only) --------------
    if (leader) {
      constexpr uint32_t idesc = (KIND == 0) ? make_idesc(1, UMMA_BF16, UMMA_BF16, A_MN ? 1u : 0u, B_MN ? 1u : 0u, 2 * BM, BN)
                                             : make_idesc(1, UMMA_E4M3, UMMA_E4M3, 0u, 0u, 2 * BM, BN);
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      bool ok = true;
      long long t_full = 0, t_tempty = 0;
      int n_trace = 0;
      const long long t_begin = p.prof ? clock64() : 0;
      for (int tile = cluster_id; ok && tile < num_tiles; tile += num_clusters, ++it) {
        const int acc = it & 1;
        const uint32_t acc_phase = (it >> 1) & 1;
        const long long te0 = p.prof ? clock64() : 0;
        if (!__all_sync(0xffffffffu, mbar_wait(&tempty_bar[acc], acc_phase ^ 1u, &abort_s))) {
          if (lane == 0) {
            report_status(p.status, STATUS_TIMEOUT, 22, acc);
            st_shared_cluster_u32(peer_abort, 1u);
          }
          break;
        }
        if (p.prof) t_tempty += clock64() - te0;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < total_kb; ++kb) {
          const long long tf0 = p.prof ? clock64() : 0;
          if (!__all_sync(0xffffffffu, mbar_wait(&full_bar[stage], phase, &abort_s))) {
            if (lane == 0) {
              report_status(p.status, STATUS_TIMEOUT, 23, stage);
              st_shared_cluster_u32(peer_abort, 1u);
            }
            ok = false;
            break;
          }
          if (p.prof) t_full += clock64() - tf0;
          if (p.trace && lane == 0 && blockIdx.x < 2 && n_trace < p.trace_len) p.trace[(blockIdx.x * 3 + 1) * p.trace_len + n_trace++] = clock64();
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * STAGE_BYTES);
          const uint32_t sb = sa + A_BYTES;
          const uint64_t da = A_MN ? make_desc_mnmajor_sw128(sa, 8192) : make_desc_kmajor_sw128(sa);
          const uint64_t db = B_MN ? make_desc_mnmajor_sw128(sb, 8192) : make_desc_kmajor_sw128(sb);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < KSTEPS; ++k) {
              const uint64_t a_k = da + static_cast<uint64_t>(A_MN ? (k * 2048) >> 4 : (k * 32) >> 4);
              const uint64_t b_k = db + static_cast<uint64_t>(B_MN ? (k * 2048) >> 4 : (k * 32) >> 4);
              if (KIND == 0)
                umma_f16_ss_pair(d_tmem, a_k, b_k, idesc, (kb | k) != 0 ? 1u : 0u);
              else
                umma_f8_ss_pair(d_tmem, a_k, b_k, idesc, (kb | k) != 0 ? 1u : 0u);
            }
            umma_commit_pair(&empty_bar[stage], 3);   // the stage is free in both CTAs once these MMAs have read it
            if (kb == total_kb - 1) umma_commit_pair(&tfull_bar[acc], 3);
          }
          __syncwarp();
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      if (p.prof && lane == 0) {
        p.prof[blockIdx.x * 8 + 0] = clock64() - t_begin;
        p.prof[blockIdx.x * 8 + 2] = t_full;
        p.prof[blockIdx.x * 8 + 3] = t_tempty;
        p.prof[blockIdx.x * 8 + 6] = it;
      }
    }
    __syncwarp();
  } else {
    // ------------------------------- epilogue (4 warps per CTA) -----------------
    const int quad = warp & 3;
    const int esz = p.out_fp32 ? 4 : 2;
    bool aligned = ((reinterpret_cast<uintptr_t>(p.out) | static_cast<uintptr_t>(static_cast<size_t>(p.ld_out) * esz)) & 15) == 0;
    if (p.bias) aligned = aligned && ((reinterpret_cast<uintptr_t>(p.bias) | static_cast<uintptr_t>(p.pair_offset * 2)) & 15) == 0;
    if (p.col_scale) aligned = aligned && ((reinterpret_cast<uintptr_t>(p.col_scale) | static_cast<uintptr_t>(p.pair_offset * 4)) & 15) == 0;
    if (p.gate) aligned = aligned && ((reinterpret_cast<uintptr_t>(p.gate) | static_cast<uintptr_t>(p.gate_stride * 2)) & 15) == 0;
    if (p.residual) aligned = aligned && ((reinterpret_cast<uintptr_t>(p.residual) | static_cast<uintptr_t>(static_cast<size_t>(p.ld_res) * 2)) & 15) == 0;
    int it = 0, turn = 0;
    long long t_twait = 0, t_work = 0;
    for (int tile = cluster_id; tile < num_tiles; tile += num_clusters, ++it) {
      const int acc = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1;
      const int m0 = (tile % tiles_m) * (2 * BM) + static_cast<int>(rank) * BM;
      const int nblk = tile / tiles_m;
      const int n0 = paired ? nblk * BNH : nblk * BN;
      const int out_cols = paired ? BNH : BN;
      const int row = m0 + quad * 32 + lane;
      BulkEpilogue<KIND> bulk(p, row, n0, out_cols, lane, paired);
      if (BULK) bulk.load();
      const long long tq0 = p.prof ? clock64() : 0;
      const bool got = __all_sync(0xffffffffu, mbar_wait(&tfull_bar[acc], acc_phase, &abort_s));
      if (!got) {
        if (lane == 0) {
          report_status(p.status, STATUS_TIMEOUT, 24, acc);
          st_shared_cluster_u32(peer_abort, 1u);
        }
        break;
      }
      tc_fence_after();
      const long long tq1 = p.prof ? clock64() : 0;
      t_twait += tq1 - tq0;
      if (p.trace && blockIdx.x < 2 && warp == 2 && lane == 0 && 2 * it + 1 < p.trace_len) p.trace[(blockIdx.x * 3 + 2) * p.trace_len + 2 * it] = clock64();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + acc * BN;
      uint8_t* stages = smem + STAGES * STAGE_BYTES;
      auto release = [&] {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&tempty_bar[acc]), 0u));
      };
      if constexpr (BULK) {
        auto store = [&](const uint8_t* buf, int col) {
          if (m0 + quad * 32 < p.M) tma_store_2d(&maps.out, buf, col, m0 + quad * 32);
        };
        if (paired) bulk.template run<true, true, 2>(taddr, BNH, stages + quad * 8192, turn, release, store);
        else bulk.template run<false, true, 2>(taddr, 0, stages + quad * 8192, turn, release, store);
      } else {
        epilogue_tile(p, taddr, BNH, row, n0, out_cols, paired, aligned, stages + quad * 8192, lane);
        release();
      }
      if (p.prof) t_work += clock64() - tq1;
      if (p.trace && blockIdx.x < 2 && warp == 2 && lane == 0 && 2 * it + 1 < p.trace_len) p.trace[(blockIdx.x * 3 + 2) * p.trace_len + 2 * it + 1] = clock64();
    }
    if (BULK && lane == 0) tma_store_wait<0>();   // the rows are out before the staging buffers go away
    if (p.prof && warp == 2 && lane == 0) {
      p.prof[blockIdx.x * 8 + 4] = t_twait;
      p.prof[blockIdx.x * 8 + 5] = t_work;
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_arrive();   // neither CTA frees TMEM or leaves while its partner may still signal or read
  cluster_wait();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------------
// 3 x 3 convolution on CTA pairs: each CTA owns one 8 x 16 patch of output pixels (128 rows of the implicit GEMM), the pair
// shares a 256- or 128-channel tile of the filter (half of its rows staged by each CTA, cta_group::2).
// What bounds the convolution is how many bytes an SM takes in per multiply-add: about 64 bytes per clock, while a lone CTA
// re-reads its 16 KB patch for every filter tap next to 32 KB of filter (726 cycles per 128 x 256 x 64 step where the tensor
// core needs 512). Here the three vertical taps of a column kw share one staged box of 10 x 16 pixels: tap kh starts
// kh * 16 rows (2048 bytes, a whole number of swizzle atoms) into it. Per three taps a CTA takes in 20 KB of pixels instead
// of 48, and half of the filter tile. With HALO = false (stride 2, where neighbouring taps share no pixels) every tap
// loads its own box through a tensor map with element strides.
// Measured (B200), convolutions alone: 1024 x 1024 decode 13.4 -> 7.2 ms (1.42 PFLOP/s), encode of three 488 x 712 images 8.4 -> 3.8 ms.
// RESIDENT (up to 128 input and output channels): all nine taps of the filter fit beside the pixel ring (147 KB per CTA) and are
// loaded once per CTA instead of once per tile; with them a pair took in 528 KB per tile of 256 pixels and the L2 was the bound
// (128 -> 128 at 1024 x 1024: 440 -> 355 us).
// Work order: channel tiles of one pair of patches are neighbours in the tile order, so the patch comes from L2 once.
// ---------------------------------------------------------------------------------
template <int BN, bool HALO, bool RESIDENT>
struct ConvPairShape {
  static_assert(!RESIDENT || (HALO && BN == 128), "the resident filter is that of one 128-channel tile");
  static constexpr int BNH = BN / 2;                                   // filter rows staged by one CTA
  static constexpr int TAPS = HALO ? 3 : 1;                            // taps served by one staged pixel box
  static constexpr int A_BYTES = (HALO ? CONV_TH + 2 : CONV_TH) * CONV_TW * BK_BYTES;
  static constexpr int B_BYTES = BNH * BK_BYTES;
  static constexpr int A_STAGES = RESIDENT ? 3 : HALO ? (BN == 256 ? 3 : 5) : 5;
  static constexpr int B_STAGES = RESIDENT ? 18 : HALO ? (BN == 256 ? 7 : 8) : 6;
  static constexpr int BUFFERS = RESIDENT ? 1 : 2;                     // 4 KB staging buffers of an epilogue warp
  static constexpr int SMEM = A_STAGES * A_BYTES + B_STAGES * B_BYTES + 4 * BUFFERS * 4096 + 1024;
  static_assert(SMEM <= 227 * 1024, "pipeline exceeds the shared memory of an SM");
  static_assert(B_BYTES % 1024 == 0 && A_BYTES % 1024 == 0, "stages start on swizzle atoms");
};

template <int BN, bool HALO, bool RESIDENT, bool BULK>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1)
conv_tcgen05_pair_kernel(const __grid_constant__ GemmMaps maps, const __grid_constant__ GemmParams p) {
  using S = ConvPairShape<BN, HALO, RESIDENT>;
  constexpr int TMEM_COLS = 2 * BN;
  constexpr int KSTEPS = 4, K_ELEMS = 64;

  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t a_full[S::A_STAGES], b_full[S::B_STAGES];      // used in the leader: both CTAs' loads have landed
  __shared__ uint64_t a_empty[S::A_STAGES], b_empty[S::B_STAGES];    // in each CTA: the MMAs that read the stage are done
  __shared__ uint64_t tfull_bar[2], tempty_bar[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;

  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem_a = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  uint8_t* smem_b = smem_a + S::A_STAGES * S::A_BYTES;
  uint8_t* smem_st = smem_b + S::B_STAGES * S::B_BYTES;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::A_STAGES; ++s) { mbar_init(&a_full[s], 1); mbar_init(&a_empty[s], 1); }
    for (int s = 0; s < S::B_STAGES; ++s) { mbar_init(&b_full[s], 1); mbar_init(&b_empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&tfull_bar[s], 1); mbar_init(&tempty_bar[s], 8); }
    abort_s = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(&tmem_base_s, TMEM_COLS);
    tmem_relinquish_pair();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&maps.a[0]);
    tma_prefetch_desc(&maps.b[0]);
  }
  tc_fence_before();
  __syncthreads();
  cluster_arrive();   // the peer's barriers exist before anything is sent to them
  cluster_wait();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_s;
  const uint32_t peer_abort = mapa_shared(smem_u32(&abort_s), rank ^ 1u);

  const int tiles_n = (p.N + BN - 1) / BN;
  const int num_tiles = ((p.conv_tiles_m + 1) / 2) * tiles_n;
  const int cluster_id = blockIdx.x >> 1, num_clusters = gridDim.x >> 1;
  const int groups = p.conv_cblocks * 3 * (3 / S::TAPS);              // pixel boxes per tile

  if (warp == 0) {
    // ------------------------------- TMA producer (both CTAs) -------------------
    int as = 0, bs = 0;
    uint32_t aph = 0, bph = 0;
    bool ok = true, issued = false;
    for (int tile = cluster_id; ok && tile < num_tiles; tile += num_clusters) {
      const int n0 = (tile % tiles_n) * BN + static_cast<int>(rank) * S::BNH;
      const int mt = (tile / tiles_n) * 2 + static_cast<int>(rank);   // past the last patch: image index past the batch, zeros
      const int tw = mt % p.conv_tiles_w, th = (mt / p.conv_tiles_w) % p.conv_tiles_h;
      const int img = mt / (p.conv_tiles_w * p.conv_tiles_h);
      for (int g = 0; ok && g < groups; ++g) {
        // pixel box g: (channel block, kw) with all kh, or (channel block, kw, kh)
        const int cb = g / (groups / p.conv_cblocks), r = g - cb * (groups / p.conv_cblocks);
        const int kw = HALO ? r : r / 3, kh0 = HALO ? 0 : r - (r / 3) * 3;
        if (!__all_sync(0xffffffffu, mbar_wait(&a_empty[as], aph ^ 1u, &abort_s))) {
          if (lane == 0) { report_status(p.status, STATUS_TIMEOUT, 31, as); st_shared_cluster_u32(peer_abort, 1u); }
          ok = false;
          break;
        }
        if (elect_one()) {
          if (leader) mbar_expect_tx(&a_full[as], 2 * S::A_BYTES);
          tma_load_4d_pair(smem_a + as * S::A_BYTES, &maps.a[0], mapa_shared(smem_u32(&a_full[as]), 0u), cb * K_ELEMS,
                           tw * CONV_TW * p.conv_stride + kw + p.conv_off_w, th * CONV_TH * p.conv_stride + kh0 + p.conv_off_h, img);
        }
        __syncwarp();
        issued = true;
        if (++as == S::A_STAGES) { as = 0; aph ^= 1u; }
        if (RESIDENT && tile != cluster_id) continue;                // the filter is there since the first tile
        for (int t = 0; t < S::TAPS; ++t) {
          const int k0 = (((kh0 + t) * 3 + kw) * p.conv_cblocks + cb) * K_ELEMS;
          if (!RESIDENT && !__all_sync(0xffffffffu, mbar_wait(&b_empty[bs], bph ^ 1u, &abort_s))) {
            if (lane == 0) { report_status(p.status, STATUS_TIMEOUT, 32, bs); st_shared_cluster_u32(peer_abort, 1u); }
            ok = false;
            break;
          }
          if (elect_one()) {
            if (leader) mbar_expect_tx(&b_full[bs], 2 * S::B_BYTES);
            tma_load_2d_pair(smem_b + bs * S::B_BYTES, &maps.b[0], mapa_shared(smem_u32(&b_full[bs]), 0u), k0, n0);
          }
          __syncwarp();
          if (++bs == S::B_STAGES) { bs = 0; bph ^= 1u; }
        }
      }
    }
    if (!ok && issued) {
      // abandoned: give the copies already in flight time to land before the CTA goes away (bounded)
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 2000000ull) {
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------- UMMA issuer (leader CTA only) --------------
    if (leader) {
      constexpr uint32_t idesc = make_idesc(1, UMMA_BF16, UMMA_BF16, 0u, 0u, 2 * BM, BN);
      int as = 0, bs = 0, it = 0;
      uint32_t aph = 0, bph = 0;
      bool ok = true;
      for (int tile = cluster_id; ok && tile < num_tiles; tile += num_clusters, ++it) {
        const int acc = it & 1;
        if (!__all_sync(0xffffffffu, mbar_wait(&tempty_bar[acc], ((it >> 1) & 1) ^ 1u, &abort_s))) {
          if (lane == 0) { report_status(p.status, STATUS_TIMEOUT, 33, acc); st_shared_cluster_u32(peer_abort, 1u); }
          break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int g = 0; ok && g < groups; ++g) {
          bool got = mbar_wait(&a_full[as], aph, &abort_s);
          if (RESIDENT) { bs = g * S::TAPS; bph = 0; }               // stage = position in the tile, filled once
          for (int t = 0; t < S::TAPS; ++t) {
            if (!__all_sync(0xffffffffu, got && mbar_wait(&b_full[bs], bph, &abort_s))) {
              if (lane == 0) { report_status(p.status, STATUS_TIMEOUT, 34, bs); st_shared_cluster_u32(peer_abort, 1u); }
              ok = false;
              break;
            }
            tc_fence_after();
            const uint64_t da = make_desc_kmajor_sw128(smem_u32(smem_a + as * S::A_BYTES) + t * (CONV_TW * BK_BYTES));
            const uint64_t db = make_desc_kmajor_sw128(smem_u32(smem_b + bs * S::B_BYTES));
            if (elect_one()) {
#pragma unroll
              for (int k = 0; k < KSTEPS; ++k)
                umma_f16_ss_pair(d_tmem, da + static_cast<uint64_t>((k * 32) >> 4), db + static_cast<uint64_t>((k * 32) >> 4), idesc,
                                 (g | t | k) != 0 ? 1u : 0u);
              if (!RESIDENT) umma_commit_pair(&b_empty[bs], 3);   // the stages are free in both CTAs once these MMAs have read them
              if (t == S::TAPS - 1) {
                umma_commit_pair(&a_empty[as], 3);
                if (g == groups - 1) umma_commit_pair(&tfull_bar[acc], 3);
              }
            }
            __syncwarp();
            if (++bs == S::B_STAGES) { bs = 0; bph ^= 1u; }
          }
          if (++as == S::A_STAGES) { as = 0; aph ^= 1u; }
        }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------- epilogue (4 warps per CTA) -----------------
    const int quad = warp & 3;
    bool aligned = ((reinterpret_cast<uintptr_t>(p.out) | static_cast<uintptr_t>(static_cast<size_t>(p.ld_out) * 2)) & 15) == 0;
    if (p.bias) aligned = aligned && (reinterpret_cast<uintptr_t>(p.bias) & 15) == 0;
    if (p.residual) aligned = aligned && ((reinterpret_cast<uintptr_t>(p.residual) | static_cast<uintptr_t>(static_cast<size_t>(p.ld_res) * 2)) & 15) == 0;
    int it = 0, turn = 0;
    for (int tile = cluster_id; tile < num_tiles; tile += num_clusters, ++it) {
      const int acc = it & 1;
      const int n0 = (tile % tiles_n) * BN;
      const int mt = (tile / tiles_n) * 2 + static_cast<int>(rank);
      const int tw = mt % p.conv_tiles_w, th = (mt / p.conv_tiles_w) % p.conv_tiles_h;
      const int img = mt / (p.conv_tiles_w * p.conv_tiles_h);
      const int ow0 = tw * CONV_TW, oh0 = th * CONV_TH + quad * (32 / CONV_TW);
      const int oh = oh0 + lane / CONV_TW, ow = ow0 + lane % CONV_TW;
      const int row = (mt < p.conv_tiles_m && oh < p.conv_h && ow < p.conv_w) ? (img * p.conv_h + oh) * p.conv_w + ow : p.M;   // p.M = skipped
      BulkEpilogue<0> bulk(p, row, n0, BN, lane, false);
      if (BULK) bulk.load();
      const bool got = __all_sync(0xffffffffu, mbar_wait(&tfull_bar[acc], (it >> 1) & 1, &abort_s));
      if (!got) {
        if (lane == 0) { report_status(p.status, STATUS_TIMEOUT, 35, acc); st_shared_cluster_u32(peer_abort, 1u); }
        break;
      }
      tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + acc * BN;
      auto release = [&] {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&tempty_bar[acc]), 0u));
      };
      if constexpr (BULK) {
        auto store = [&](const uint8_t* buf, int col) {
          if (mt < p.conv_tiles_m && oh0 < p.conv_h) tma_store_4d(&maps.out, buf, col, ow0, oh0, img);
        };
        bulk.template run<false, false, S::BUFFERS>(taddr, 0, smem_st + quad * (S::BUFFERS * 4096), turn, release, store);
      } else {
        epilogue_direct(p, taddr, 0, row, n0, BN, false, aligned);
        release();
      }
    }
    if (BULK && lane == 0) tma_store_wait<0>();   // the rows are out before the staging buffers go away
  }

  tc_fence_before();
  __syncthreads();
  cluster_arrive();   // neither CTA frees TMEM or leaves while its partner may still signal or read
  cluster_wait();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------
static PFN_cuTensorMapEncodeTiled_v12000 get_encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
  }
  return fn;
}

}  // namespace mdb

extern "C" int mdb_make_tmap(void* out_map, const void* ptr, int elem_bytes, int rank, const int64_t* extents,
                             const int64_t* strides_bytes, const int* box, int swizzle128) {
  return mdb_make_tmap_strided(out_map, ptr, elem_bytes, rank, extents, strides_bytes, box, nullptr, swizzle128);
}
extern "C" int mdb_make_tmap_strided(void* out_map, const void* ptr, int elem_bytes, int rank, const int64_t* extents,
                                     const int64_t* strides_bytes, const int* box, const int* elem_strides, int swizzle128) {
  auto fn = mdb::get_encode_fn();
  if (!fn) return -1;
  // The encode call is a driver-API entry and needs a current context. A thread that has not made a runtime call yet
  // (an autograd worker whose first node is one of our backward kernels) has none: bind the primary context once.
  static thread_local bool ctx_bound = false;
  if (!ctx_bound) {
    cudaFree(nullptr);
    ctx_bound = true;
  }
  cuuint64_t gdim[5];
  cuuint64_t gstr[5];
  cuuint32_t bdim[5];
  cuuint32_t estr[5];
  for (int i = 0; i < rank; ++i) {
    gdim[i] = static_cast<cuuint64_t>(extents[i]);
    bdim[i] = static_cast<cuuint32_t>(box[i]);
    estr[i] = elem_strides ? static_cast<cuuint32_t>(elem_strides[i]) : 1;
    if (i > 0) gstr[i - 1] = static_cast<cuuint64_t>(strides_bytes[i]);
  }
  CUtensorMapDataType dt = elem_bytes == 1   ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                           : elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                             : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  CUresult r = fn(reinterpret_cast<CUtensorMap*>(out_map), dt, rank, const_cast<void*>(ptr), gdim, gstr, bdim, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : static_cast<int>(r);
}

namespace mdb {

template <int BN, int STAGES, bool A_MN, bool B_MN, int KIND, bool BULK>
static int launch_variant(const GemmMaps& maps, const GemmParams& p, int num_sms, cudaStream_t stream) {
  constexpr int STAGE_BYTES = BM * BK_BYTES + BN * BK_BYTES;
  // operand ring + 32 KB that serve as the epilogue's staging buffers (4 warps x 8 KB) or, with a fused all-gather, as its
  // two bulk-copy stages
  constexpr int SMEM_GATHER = STAGES * STAGE_BYTES + 1024 + GATHER_STAGES * GATHER_PIECE;
  static_assert(GATHER_STAGES * GATHER_PIECE == 4 * 8192, "staging buffers and gather stages share one region");
  static_assert(SMEM_GATHER <= 227 * 1024, "pipeline + staging exceed the shared memory of an SM");
  const int SMEM = SMEM_GATHER;
  auto kern = gemm_tcgen05_kernel<BN, STAGES, A_MN, B_MN, KIND, BULK>;
  static bool attr_done = false;
  if (!attr_done) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_GATHER);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_done = true;
  }
  const int tiles_m = p.conv_taps > 0 ? p.conv_tiles_m : (p.M + BM - 1) / BM;
  const int bn_eff = p.pair_offset > 0 ? BN / 2 : BN;
  const int tiles_n = (p.N + bn_eff - 1) / bn_eff;
  int grid = tiles_m * tiles_n;
  if (grid > num_sms) grid = num_sms;
  if (grid < 1) return 0;
  kern<<<grid, NUM_THREADS, SMEM, stream>>>(maps, p);
  return static_cast<int>(cudaGetLastError());
}

// How many CTA pairs the device can hold at once: an SM whose partner in the same TPC is not available cannot host half
// a pair, so the number differs from chip to chip. A persistent grid must not exceed it (surplus pairs would run their
// whole tile list after the others finish) and the tile-shape choice uses it as the pair kernel's width.
static int pair_capacity(int num_sms) {
  static int cached = 0;
  if (cached > 0) return cached;
  constexpr int SMEM = 6 * (BM * BK_BYTES + 128 * BK_BYTES) + 4 * 8192 + 1024;
  auto kern = gemm_tcgen05_pair_kernel<6, false, false, 0, true>;
  int n = 0;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) == cudaSuccess) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(static_cast<unsigned>(num_sms & ~1), 1, 1);
    cfg.blockDim = dim3(PAIR_THREADS, 1, 1);
    cfg.dynamicSmemBytes = SMEM;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) n = 0;
  }
  cudaGetLastError();
  if (n < 1 || n > num_sms / 2) n = num_sms / 2;
  cached = n;
  return cached;
}

template <int STAGES, bool A_MN, bool B_MN, int KIND, bool BULK>
static int launch_pair_variant(const GemmMaps& maps, const GemmParams& p, int num_sms, cudaStream_t stream) {
  constexpr int SMEM = STAGES * (BM * BK_BYTES + 128 * BK_BYTES) + 4 * 8192 + 1024;   // ring + epilogue staging (4 warps x 8 KB)
  static_assert(SMEM <= 227 * 1024, "pipeline exceeds the shared memory of an SM");
  auto kern = gemm_tcgen05_pair_kernel<STAGES, A_MN, B_MN, KIND, BULK>;
  static bool attr_done = false;
  if (!attr_done) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_done = true;
  }
  const int tiles_m = (p.M + 2 * BM - 1) / (2 * BM);
  const int tiles_n = (p.N + (p.pair_offset > 0 ? 128 : 256) - 1) / (p.pair_offset > 0 ? 128 : 256);
  const int max_pairs = pair_capacity(num_sms);
  int clusters = tiles_m * tiles_n;
  if (clusters > max_pairs) clusters = max_pairs;
  if (clusters < 1) return 0;
  kern<<<2 * clusters, PAIR_THREADS, SMEM, stream>>>(maps, p);
  return static_cast<int>(cudaGetLastError());
}

template <int BN, bool HALO, bool RESIDENT>
static int launch_conv_pair(const GemmMaps& maps, const GemmParams& p, int num_sms, cudaStream_t stream) {
  constexpr int SMEM = ConvPairShape<BN, HALO, RESIDENT>::SMEM;
  auto kern = p.bulk_out ? conv_tcgen05_pair_kernel<BN, HALO, RESIDENT, true> : conv_tcgen05_pair_kernel<BN, HALO, RESIDENT, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
  if (e != cudaSuccess) return static_cast<int>(e);
  const long long tiles = static_cast<long long>((p.conv_tiles_m + 1) / 2) * ((p.N + BN - 1) / BN);
  const int max_pairs = pair_capacity(num_sms);
  const int clusters = static_cast<int>(tiles < max_pairs ? tiles : max_pairs);
  kern<<<2 * clusters, PAIR_THREADS, SMEM, stream>>>(maps, p);
  return static_cast<int>(cudaGetLastError());
}

#include "gemm_splitk.cuh"

}  // namespace mdb

extern "C" int mdb_gemm_pair_capacity(int num_sms) { return mdb::pair_capacity(num_sms > 0 ? num_sms : mdb::device_sm_count()); }

// MDB200_GEMM_PAIR=0 keeps every automatically tiled GEMM on the one-CTA kernel (A/B measurements); default: choose.
static int pair_mode() {
  static int mode = -1;
  if (mode < 0) {
    const char* e = getenv("MDB200_GEMM_PAIR");
    mode = (e != nullptr && e[0] == '0') ? 0 : 1;
  }
  return mode;
}

namespace mdb {
// The form of a bf16 GEMM that is left to the launch: few-row kernel, one CTA or CTA pair per tile, or clusters that share a tile's
// reduction. Every form is estimated in microseconds and the lowest one taken.
//
// The terms are fitted to measured times of all forms over 1457 calls (M 1 to 65536, N and K 16 to 21504, the three operand
// layouts, with and without epilogue terms; B200, weights from HBM). Over them the choice is 1.4 % above the best form of each
// (geometric mean; 18 of them more than 20 %). They were measured with the epilogue whose lanes store their rows; bf16 rows that leave
// as bulk stores take about half of its time, and ragged ones no more than others. Over the whole-K times measured since, the choice is 2.3 %
// above the best form, with refitted terms (epilogues 1 to 2.1 us) 1.6 %. The terms stay all the same, because a form is also an order of
// sums: a training step passes a changed order through its optimizer into single gradient entries (up to 0.9 of their root mean square
// after one step of an SDXL adapter). What they say, of the former epilogue where they speak of one:
//  - a 64-wide K step takes 0.32 / 0.34 / 0.46 us of a lone CTA with 64 / 128 / 256 columns (what an SM takes in bounds it) and
//    0.34 of a pair;
//  - a tile's epilogue takes 1.6 to 3 us, three times that with activation, gate or residual, and hides behind the next tile's
//    steps only; rows that end off 32 columns left its vector path (N = 16: 8 us more; still so for fp32 and unaligned rows);
//  - a cluster's tile starts, meets in shared memory and ends in 6 to 9 us, and finishing its rows costs a CTA 2.2 to 7.2 us / splits
//    (six times that with epilogue terms): it pays for long reductions only, and never for tiles that come in many waves
//    (65536 x 128 x 128: 65 us in clusters of one, 17 on the persistent tiles). 15 % are added for it, so that it wins clear cases;
//  - the few-row kernel streams weights at 5 to 6 TB/s for one row, but unpacks A once per column and row: at eight rows it is at
//    1.7 (8 x 18432 x 3072: 65 us, tiles 33), and each column costs a warp its reduction over the lanes.
struct GemmForm {
  int bn, splits;          // splits 0: whole reductions; otherwise CTAs (or pairs) per cluster
  bool pair, rows;
};
static GemmForm choose_form(const MdbGemmArgs* a, int sms, bool pairs, bool rows_ok) {
  const bool paired = a->pair_offset > 0, whole_only = a->split_k != 0 || paired || (a->a_mn && !a->b_mn) || !pairs;
  double kb = 0, k_all = 0;
  for (int s = 0; s < a->num_seg; ++s) { kb += static_cast<double>((a->K[s] + 63) / 64); k_all += static_cast<double>(a->K[s]); }
  const double n_all = paired ? 2.0 * a->N : a->N;                           // rows of B
  const double memory = 2.0 * (a->M * k_all + n_all * k_all + static_cast<double>(a->M) * a->N) / 3.6e6;
  const bool heavy = a->act != 0 || a->gate || a->residual || paired;
  const double whole_terms = heavy ? 3.0 : a->bias ? 1.4 : 1.0, split_terms = heavy ? 6.2 : a->bias ? 2.1 : 1.0;
  auto ceil_div = [](double x, double y) { return std::ceil(x / y); };
  auto with_memory = [&](double t) { return std::sqrt(std::sqrt(t * t * t * t + memory * memory * memory * memory)); };   // neither hides wholly behind the other
  auto tiles = [&](double tm, double tn) { return ceil_div(a->M, tm) * ceil_div(a->N, tn); };
  auto step = [](int w) { return w == 64 ? 0.32 : w == 128 ? 0.34 : 0.46; };
  GemmForm best = {256, 0, false, false};
  double best_us = 1e30;
  auto offer = [&](double us, GemmForm f) { if (us < best_us) { best_us = us; best = f; } };

  auto whole = [&](double n_tiles, int width, double step_us, double epilogue) {
    const double e = epilogue * whole_terms + (a->N % 32 != 0 && a->N < 256 ? 8.0 : 0.0), main = kb * step_us;
    return with_memory(5.0 + ceil_div(n_tiles, width) * (main > e ? main : e) + e);
  };
  offer(whole(tiles(BM, paired ? 128 : 256), sms, step(256), 3.0), {256, 0, false, false});
  if (!paired) {
    offer(whole(tiles(BM, 128), sms, step(128), 2.1), {128, 0, false, false});
    offer(whole(tiles(BM, 64), sms, step(64), 1.6), {64, 0, false, false});
  }
  if (pairs && a->M > BM) offer(whole(tiles(2 * BM, paired ? 128 : 256), pair_capacity(sms), 0.34, 2.9), {256, 0, true, false});
  if (!whole_only) {
    for (int w = 128; w >= 64; w -= 64)
      for (int sp = 1; sp <= SPLIT_MAX && (sp == 1 || kb / sp >= 4); ++sp) {
        const int cap = w == 128 ? split_capacity<128>(sp, sms) : split_capacity<64>(sp, sms);
        const double fixed = w == 128 ? 7.0 + 3.55 * split_terms / sp : 5.9 + 2.2 * split_terms / sp;
        offer(with_memory(1.15 * ceil_div(tiles(BM, w), cap) * (ceil_div(kb, sp) * step(w) + fixed)), {w, sp, false, false});
      }
    for (int sp = 2; sp <= PSPLIT_MAX && kb / sp >= 4 && !a->a_mn && a->M > BM; ++sp)
      offer(with_memory(1.15 * ceil_div(tiles(2 * BM, 256), pair_split_capacity(sp, sms)) * (ceil_div(kb, sp) * 0.34 + 9.0 + 7.2 * split_terms / sp)), {256, sp, true, false});
  }
  if (rows_ok) {
    const int r = a->M == 1 ? 0 : a->M == 2 ? 1 : a->M <= 4 ? 2 : 3;          // rows rounded up to 1, 2, 4, 8
    static const double base[4] = {2.5, 2.7, 3.3, 4.0}, per_k[4] = {0.83e-3, 1.0e-3, 1.3e-3, 1.8e-3}, per_column[4] = {0.16e-3, 0.27e-3, 0.95e-3, 1.75e-3};
    static const double per_mb_one[4] = {0.2, 0.28, 0.38, 0.7}, per_mb[4] = {0.165, 0.2, 0.32, 0.46};     // one column per warp, several
    const bool one = n_all < 32.0 * sms || (paired && r == 3);
    const double stream = n_all * k_all * 2e-6 * (one ? per_mb_one[r] : per_mb[r]), lane = k_all * per_k[r];
    const double columns = a->N * per_column[r] * (heavy && !paired ? 2.0 : 1.0), both = std::sqrt(stream * stream + columns * columns);
    offer(base[r] + (lane > both ? lane : both), {0, 0, false, true});
  }
  return best;
}
}  // namespace mdb

extern "C" int mdb_gemm_launch(const MdbGemmArgs* a, cudaStream_t stream) {
  using namespace mdb;
  if (a->M <= 0 || a->N <= 0 || a->num_seg < 1 || a->num_seg > MDB_GEMM_MAX_SEG || a->split_k > 1) return -2;
  MdbGemmArgs flat;
  if (a->conv_taps == 1 && a->conv_stride <= 1 && a->conv_pad_h == 0 && a->conv_pad_w == 0 && a->kind == 0) {
    // a 1 x 1 convolution is a plain GEMM over the pixels: no patches that hang over the image's edge, all tilings open
    flat = *a;
    flat.conv_taps = 0;
    a = &flat;
  }
  const int eb = a->kind == 1 ? 1 : 2;
  const int k_elems = BK_BYTES / eb;
  const bool paired = a->pair_offset > 0;
  const int sms = a->num_sms > 0 ? a->num_sms : device_sm_count();
  int bn = a->bn;
  // bn == 512 asks for the CTA-pair kernel (256 x 256 tile over two SMs); it shares the tensor maps of the 128 x 256 tile
  const bool pair_ok = a->conv_taps <= 0 && a->gather_world <= 1;
  bool use_pair = bn == 512 && pair_ok;
  if (bn == 512) bn = 256;
  const bool auto_tile = bn != 64 && bn != 128 && bn != 256;
  int splits = 0;
  bool pair_split = false;
  const bool plain = a->kind == 0 && a->conv_taps <= 0 && a->gather_world <= 1 && !a->row_scale && !a->col_scale && a->route_owner_cols <= 0 &&
                     a->reduce_rows_per_owner <= 0 && !a->prof;
  if (auto_tile && plain) {
    const GemmForm f = choose_form(a, sms, pair_mode() != 0, mdb_gemm_rows_ok(a) != 0);
    if (f.rows) return mdb_gemm_rows(a, stream);
    bn = f.bn;
    splits = f.splits;
    use_pair = f.pair && f.splits == 0;
    pair_split = f.pair && f.splits > 0;
  } else if (auto_tile) {
    // default tile choice: 128x256 unless the narrower 128x128 tile fills the machine noticeably better
    // (fewer idle SMs in the last wave); 128x64 only for very skinny outputs
    const int tm = (a->M + BM - 1) / BM;
    auto wave_eff = [&](int w) {
      const long long tiles = static_cast<long long>(tm) * ((a->N + w - 1) / w);
      const long long waves = (tiles + sms - 1) / sms;
      return static_cast<double>(tiles) / static_cast<double>(waves * sms);
    };
    bn = 256;
    if (!paired && wave_eff(128) > 1.12 * wave_eff(256)) bn = 128;
    if (!paired && a->N <= 64) bn = 64;
  }
  if (paired && bn != 256) bn = 256;
  if (auto_tile && !plain && pair_ok && a->M > BM && pair_mode() != 0) {
    // CTA pair (256 x 256 tile on two SMs) or lone CTAs? Compare waves x time per tile. A lone CTA's 128 x 256 tile moves
    // 96 KB through shared memory per K block (48 KB written by TMA, 48 KB read by the tensor core): 726 cycles measured,
    // bound by the 128 B/clk of shared memory. A pair tile moves 64 KB per SM and runs at the tensor rate: 523 cycles.
    const int n_tile = paired ? 128 : 256;
    const long long t2 = static_cast<long long>((a->M + 2 * BM - 1) / (2 * BM)) * ((a->N + n_tile - 1) / n_tile);
    const int pairs = pair_capacity(sms);
    const long long w2 = (t2 + pairs - 1) / pairs;
    const long long t1 = static_cast<long long>((a->M + BM - 1) / BM) * ((a->N + (paired ? 128 : bn) - 1) / (paired ? 128 : bn));
    const long long w1 = (t1 + sms - 1) / sms;
    const double cost1 = static_cast<double>(w1) * (bn == 256 ? 1.0 : bn == 128 ? 0.55 : 0.32);
    const double cost2 = static_cast<double>(w2) * 0.72;
    if (cost2 <= cost1) {
      use_pair = true;
      bn = 256;
    }
  }
  // 3 x 3 convolutions: waves x time of one 64-wide K step (726 cycles of a lone CTA's 128 x 256 tile = 1; a pair's tile of two
  // patches x 256 channels takes 533). The 128-wide pair tile serves layers of up to 128 channels only: with its filter
  // resident it takes 355 us against 440 for 128 -> 128 at 1024 x 1024, no more because a pair's 128-wide MMAs (64 cycles each) leave shared memory no room beside them; small images stay on lone CTAs.
  bool conv_pair = false;
  const int conv_stride = a->conv_taps > 0 && a->conv_stride > 1 ? a->conv_stride : 1;
  if (a->conv_taps > 0) {
    if (conv_stride > 1 && (conv_stride != 2 || a->conv_taps != 9 || a->conv_kw != 3)) return -11;
    const long long patches = static_cast<long long>(a->conv_n) * ((a->conv_h + CONV_TH - 1) / CONV_TH) * ((a->conv_w + CONV_TW - 1) / CONV_TW);
    const int pairs = pair_capacity(sms);
    const int wide = a->N > 128 || conv_stride > 1 ? 256 : 128;
    const long long t_pair = (patches + 1) / 2 * ((a->N + wide - 1) / wide), t_lone = patches * ((a->N + bn - 1) / bn);
    const double pair = static_cast<double>((t_pair + pairs - 1) / pairs) * (wide == 256 ? 0.73 : 0.62);
    const double lone = static_cast<double>((t_lone + sms - 1) / sms) * (bn == 256 ? 1.0 : bn == 128 ? 0.83 : 0.62);
    conv_pair = conv_stride > 1 ||
                (a->conv_taps == 9 && a->conv_kw == 3 && auto_tile && a->kind == 0 && !a->out_fp32 && pair_mode() != 0 && pair <= lone);
    if (conv_pair) bn = wide;    // filter box: half of the tile's rows
  }
  GemmMaps maps;
  GemmParams p;
  memset(&p, 0, sizeof(p));
  p.M = a->M;
  p.N = a->N;
  p.num_seg = a->num_seg;
  const int n_rows_total = paired ? a->N + a->pair_offset : a->N;  // rows of B that exist
  for (int s = 0; s < a->num_seg; ++s) {
    const int64_t K = a->K[s];
    if (K <= 0) return -3;
    p.kblocks[s] = static_cast<int>((K + k_elems - 1) / k_elems);
    // A
    {
      int64_t ext[2], str[2];
      int box[2];
      if (a->conv_taps > 0) {
        if (s != 0 || a->a_mn || a->kind != 0) return -6;
        const int64_t cin = a->conv_cin;
        const int64_t in_h = conv_stride > 1 ? a->conv_in_h : a->conv_h, in_w = conv_stride > 1 ? a->conv_in_w : a->conv_w;
        int64_t e4[4] = {cin, in_w, in_h, a->conv_n};
        int64_t s4[4] = {eb, cin * eb, in_w * cin * eb, in_h * in_w * cin * eb};
        // stride 1 on the pair kernel: two more rows of pixels serve all three vertical taps; stride 2: every second pixel
        int b4[4] = {k_elems, CONV_TW * conv_stride, conv_pair && conv_stride == 1 ? CONV_TH + 2 : CONV_TH * conv_stride, 1};
        int st4[4] = {1, conv_stride, conv_stride, 1};
        int r = mdb_make_tmap_strided(&maps.a[s], a->A[s], eb, 4, e4, s4, b4, st4, 1);
        if (r) return 1000 + r;
        p.kblocks[s] = a->conv_taps * static_cast<int>((cin + k_elems - 1) / k_elems);
      } else
      if (!a->a_mn) {  // [M rows][K] row-major
        ext[0] = K; ext[1] = a->M; str[0] = eb; str[1] = a->lda[s] * eb; box[0] = k_elems; box[1] = BM;
      } else {  // stored [K rows][M]
        ext[0] = a->M; ext[1] = K; str[0] = eb; str[1] = a->lda[s] * eb; box[0] = 64; box[1] = 64;
      }
      if (a->conv_taps <= 0) {
        int r = mdb_make_tmap(&maps.a[s], a->A[s], eb, 2, ext, str, box, 1);
        if (r) return 1000 + r;
      }
    }
    {
      int64_t ext[2], str[2];
      int box[2];
      if (!a->b_mn) {  // [N rows][K]
        ext[0] = K; ext[1] = n_rows_total; str[0] = eb; str[1] = a->ldb[s] * eb; box[0] = k_elems; box[1] = bn / 2;
      } else {  // stored [K rows][N]
        ext[0] = a->N; ext[1] = K; str[0] = eb; str[1] = a->ldb[s] * eb; box[0] = 64; box[1] = 64;
      }
      int r = mdb_make_tmap(&maps.b[s], a->B[s], eb, 2, ext, str, box, 1);
      if (r) return 2000 + r;
    }
  }
  p.pair_offset = a->pair_offset;
  p.act = a->act;
  p.act_on_second = a->act_on_second;
  p.alpha = a->alpha;
  p.row_scale = a->row_scale;
  p.col_scale = a->col_scale;
  p.bias = reinterpret_cast<const __nv_bfloat16*>(a->bias);
  p.residual = reinterpret_cast<const __nv_bfloat16*>(a->residual);
  p.gate = reinterpret_cast<const __nv_bfloat16*>(a->gate);
  p.ld_res = a->ld_res;
  p.gate_stride = a->gate_stride;
  p.rows_per_group = a->rows_per_group > 0 ? a->rows_per_group : 1;
  p.out = a->out;
  p.ld_out = a->ld_out;
  p.out_fp32 = a->out_fp32;
  p.accumulate_out = a->accumulate_out;
  p.status = a->status;
  p.prof = a->prof;
  p.trace = a->trace;
  p.trace_len = a->trace_len;
  for (int i = 0; i < MDB_GEMM_MAX_PEERS; ++i) p.route_out[i] = a->route_out[i];
  for (int i = 0; i < MDB_GEMM_MAX_PEERS; ++i) p.gather_src[i] = a->gather_src[i];
  p.gather_dst = a->gather_dst;
  p.gather_ready = a->gather_ready;
  p.gather_chunk_bytes = a->gather_chunk_bytes;
  p.gather_world = a->gather_world;
  p.gather_rank = a->gather_rank;
  p.gather_operand = a->gather_operand;
  p.gather_chunk_rows = a->gather_chunk_rows > 0 ? a->gather_chunk_rows : 1;
  p.reduce_rows_per_owner = a->reduce_rows_per_owner;
  if (a->gather_world > 1) {
    if (a->gather_ready == nullptr || a->gather_dst == nullptr || (a->gather_chunk_bytes & 15) || a->conv_taps > 0) return -8;
    cudaError_t e = cudaMemsetAsync(a->gather_ready, 0, sizeof(int) * MDB_GEMM_MAX_PEERS, stream);
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  p.reduce_src_rank = a->reduce_src_rank;
  if (a->reduce_rows_per_owner > 0 && !a->out_fp32 && (a->reduce_src_rank < 0 || a->reduce_src_rank >= MDB_GEMM_MAX_PEERS)) return -9;
  p.conv_taps = a->conv_taps;
  if (a->conv_taps > 0) {
    if (a->conv_cin % k_elems) return -7;
    p.conv_kw = a->conv_kw; p.conv_pad_h = a->conv_pad_h; p.conv_pad_w = a->conv_pad_w;
    p.conv_h = a->conv_h; p.conv_w = a->conv_w;
    p.conv_stride = conv_stride;
    p.conv_off_h = (conv_stride > 1 ? a->conv_offset : 0) - a->conv_pad_h;
    p.conv_off_w = (conv_stride > 1 ? a->conv_offset : 0) - a->conv_pad_w;
    p.conv_tiles_h = (a->conv_h + CONV_TH - 1) / CONV_TH;
    p.conv_tiles_w = (a->conv_w + CONV_TW - 1) / CONV_TW;
    p.conv_cblocks = a->conv_cin / k_elems;
    p.conv_tiles_m = a->conv_n * p.conv_tiles_h * p.conv_tiles_w;
  }
  // a local bf16 output whose rows and terms start on 16 bytes leaves through a tensor map (32 rows x 64 columns, or 2 x 16 pixels
  // x 64 channels, a store); the rest (fp32, peers' buffers, odd strides) is written by the lanes, as are the few products of bf16 operands
  // with another factor than 1: a rounded product by itself in every epilogue took a guided SDXL step from 29.9 to 30.6 ms
  auto fits = [](const void* ptr, int64_t stride_bytes) { return ((reinterpret_cast<uintptr_t>(ptr) | static_cast<uintptr_t>(stride_bytes)) & 15) == 0; };
  p.bulk_out = !a->out_fp32 && a->route_owner_cols <= 0 && a->reduce_rows_per_owner <= 0 && a->gather_world <= 1 && splits == 0 &&
               fits(a->out, static_cast<int64_t>(a->ld_out) * 2) && fits(a->bias, a->pair_offset > 0 ? a->pair_offset * 2 : 0) &&
               !(a->pair_offset > 0 && (a->gate || a->residual)) && (a->kind == 1 || (!a->row_scale && !a->col_scale && a->alpha == 1.f)) && (!a->gate || fits(a->gate, static_cast<int64_t>(a->gate_stride) * 2)) &&
               (!a->residual || fits(a->residual, static_cast<int64_t>(a->ld_res) * 2));
  if (p.bulk_out) {
    int r;
    if (a->conv_taps > 0) {
      const int64_t row = static_cast<int64_t>(a->ld_out) * 2;
      const int64_t e4[4] = {a->N, a->conv_w, a->conv_h, a->conv_n}, s4[4] = {2, row, row * a->conv_w, row * a->conv_w * a->conv_h};
      const int b4[4] = {64, CONV_TW, 32 / CONV_TW, 1};
      r = mdb_make_tmap(&maps.out, a->out, 2, 4, e4, s4, b4, 1);
    } else {
      const int64_t e2[2] = {a->N, a->M}, s2[2] = {2, static_cast<int64_t>(a->ld_out) * 2};
      const int b2[2] = {64, 32};
      r = mdb_make_tmap(&maps.out, a->out, 2, 2, e2, s2, b2, 1);
    }
    if (r) return 3000 + r;
  }
  p.route_owner_cols = a->route_owner_cols;
  p.route_part_cols = a->route_part_cols > 0 ? a->route_part_cols : a->N;
  p.route_row_offset = a->route_row_offset;
  p.route_rows_per_batch = a->route_rows_per_batch > 0 ? a->route_rows_per_batch : a->M;
  p.route_batch_rows = a->route_batch_rows;
  p.route_split = a->route_split;
  p.route_row_offset_b = a->route_row_offset_b;
  if (a->route_owner_cols > 0 && ((a->route_owner_cols % 32) || (p.route_part_cols % a->route_owner_cols))) return -5;

  if (conv_pair) {
    if (conv_stride > 1) return launch_conv_pair<256, false, false>(maps, p, sms, stream);
    if (bn == 256) return launch_conv_pair<256, true, false>(maps, p, sms, stream);
    return p.conv_cblocks <= 2 ? launch_conv_pair<128, true, true>(maps, p, sms, stream) : launch_conv_pair<128, true, false>(maps, p, sms, stream);
  }
  if (pair_split) return a->b_mn ? launch_pair_split<true>(maps, p, splits, stream) : launch_pair_split<false>(maps, p, splits, stream);
  if (splits > 0) {
    if (!a->a_mn && !a->b_mn) return bn == 128 ? launch_split<128, false, false>(maps, p, splits, stream) : launch_split<64, false, false>(maps, p, splits, stream);
    if (!a->a_mn) return bn == 128 ? launch_split<128, false, true>(maps, p, splits, stream) : launch_split<64, false, true>(maps, p, splits, stream);
    return bn == 128 ? launch_split<128, true, true>(maps, p, splits, stream) : launch_split<64, true, true>(maps, p, splits, stream);
  }
#define MDB_LAUNCH(BN_, ST_, AMN_, BMN_, KIND_) \
  return p.bulk_out ? launch_variant<BN_, ST_, AMN_, BMN_, KIND_, true>(maps, p, sms, stream) : launch_variant<BN_, ST_, AMN_, BMN_, KIND_, false>(maps, p, sms, stream)
#define MDB_LAUNCH_PAIR(AMN_, BMN_, KIND_) \
  return p.bulk_out ? launch_pair_variant<6, AMN_, BMN_, KIND_, true>(maps, p, sms, stream) : launch_pair_variant<6, AMN_, BMN_, KIND_, false>(maps, p, sms, stream)
  if (use_pair) {
    if (a->kind == 1) {
      if (a->a_mn || a->b_mn) return -4;
      MDB_LAUNCH_PAIR(false, false, 1);
    }
    if (!a->a_mn && !a->b_mn) MDB_LAUNCH_PAIR(false, false, 0);
    if (!a->a_mn && a->b_mn) MDB_LAUNCH_PAIR(false, true, 0);
    if (a->a_mn && a->b_mn) MDB_LAUNCH_PAIR(true, true, 0);
    MDB_LAUNCH_PAIR(true, false, 0);
  }
  if (a->kind == 1) {
    if (a->a_mn || a->b_mn) return -4;
    if (bn == 256) MDB_LAUNCH(256, 4, false, false, 1);
    if (bn == 128) MDB_LAUNCH(128, 6, false, false, 1);
    MDB_LAUNCH(64, 8, false, false, 1);
  }
  if (!a->a_mn && !a->b_mn) {
    if (bn == 256) MDB_LAUNCH(256, 4, false, false, 0);
    if (bn == 128) MDB_LAUNCH(128, 6, false, false, 0);
    MDB_LAUNCH(64, 8, false, false, 0);
  }
  if (!a->a_mn && a->b_mn) {
    if (bn == 256) MDB_LAUNCH(256, 4, false, true, 0);
    if (bn == 128) MDB_LAUNCH(128, 6, false, true, 0);
    MDB_LAUNCH(64, 8, false, true, 0);
  }
  if (a->a_mn && a->b_mn) {
    if (bn == 256) MDB_LAUNCH(256, 4, true, true, 0);
    if (bn == 128) MDB_LAUNCH(128, 6, true, true, 0);
    MDB_LAUNCH(64, 8, true, true, 0);
  }
  if (bn == 256) MDB_LAUNCH(256, 4, true, false, 0);
  if (bn == 128) MDB_LAUNCH(128, 6, true, false, 0);
  MDB_LAUNCH(64, 8, true, false, 0);
#undef MDB_LAUNCH
#undef MDB_LAUNCH_PAIR
}

MDB_DEFINE_WAIT_LIMIT_SETTER(mdb_set_wait_limit_gemm)
