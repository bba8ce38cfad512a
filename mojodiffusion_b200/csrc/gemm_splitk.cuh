// Split-K GEMM over a thread-block cluster (included by gemm_tcgen05.cu, inside namespace mdb). One output tile of 128 x BN
// belongs to a cluster of S CTAs; each runs a contiguous share of the K blocks (over all segments) into its own TMEM
// accumulator, the parts meet in distributed shared memory and every CTA finishes 128 / S rows of the tile.
//
// Two forms: single CTAs with 128 x 128 / 128 x 64 tiles, and CTA pairs (cta_group::2) with 256 x 256 tiles, which take in half
// the bytes per multiply-add and serve the larger outputs (512 x 3072 x 15360: 84 us on clusters of four single CTAs, 56 on clusters
// of two pairs, 80 on pairs that keep whole reductions).
//
// What it is for: outputs with fewer tiles than the GPU has SMs (a few hundred token rows, LoRA down-projections and their
// gradients). There one SM takes in about 64 bytes per clock, so a tile of a long reduction takes kblocks x 600 cycles
// (128 x 128, 32 KB a block) whatever the other SMs do; S CTAs cut that by S. The parts are added in CTA order in fp32, once, before the
// epilogue and the only rounding: no zero-filled fp32 output, no atomics, no cast pass, and a result that does not depend on
// scheduling.

template <int BN>
struct SplitShape {
  static constexpr int STAGE_BYTES = BM * BK_BYTES + BN * BK_BYTES;
  static constexpr int STAGES = BN == 128 ? 6 : 8;
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024;
  static_assert(BM * BN * 4 <= STAGES * STAGE_BYTES, "the fp32 part of a tile reuses the operand ring");
  static_assert(SMEM <= 227 * 1024, "pipeline exceeds the shared memory of an SM");
};
constexpr int SPLIT_THREADS = 192;        // warps: 0 TMA, 1 UMMA issue, 2-5 accumulator read-out; all warps finish rows
constexpr int SPLIT_MAX = 8;

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// v = sum over s < splits (in that order) of the eight floats at o0 / o1 of CTA s * stride + first; every part's loads are issued
// before the first is used (one remote latency per item instead of one per part)
template <int MAX>
__device__ __forceinline__ void split_sum8(uint32_t o0, uint32_t o1, int splits, uint32_t stride, uint32_t first, float (&v)[8]) {
  float4 a[MAX], b[MAX];
#pragma unroll
  for (int s = 0; s < MAX; ++s)
    if (s < splits) {
      a[s] = ld_cluster_f4(mapa_shared(o0, s * stride + first));
      b[s] = ld_cluster_f4(mapa_shared(o1, s * stride + first));
    }
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = 0.f;
#pragma unroll
  for (int s = 0; s < MAX; ++s)
    if (s < splits) {
      v[0] += a[s].x; v[1] += a[s].y; v[2] += a[s].z; v[3] += a[s].w;
      v[4] += b[s].x; v[5] += b[s].y; v[6] += b[s].z; v[7] += b[s].w;
    }
}

// eight columns col0.. of one output row, summed parts in v
__device__ __forceinline__ void split_store8(const GemmParams& p, int row, int col0, float (&v)[8], bool aligned) {
  const int n = min(8, p.N - col0);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (j >= n) break;
    const int col = col0 + j;
    float x = v[j] * p.alpha;
    if (p.bias) x += __bfloat162float(p.bias[col]);
    x = apply_act_rt(p.act, x);
    if (p.gate) x *= __bfloat162float(p.gate[static_cast<size_t>(row / p.rows_per_group) * p.gate_stride + col]);
    if (p.residual) x += __bfloat162float(p.residual[static_cast<size_t>(row) * p.ld_res + col]);
    v[j] = x;
  }
  if (p.out_fp32) {
    float* o = reinterpret_cast<float*>(p.out) + static_cast<size_t>(row) * p.ld_out + col0;
    for (int j = 0; j < n; ++j) o[j] = p.accumulate_out ? o[j] + v[j] : v[j];
    return;
  }
  __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.out) + static_cast<size_t>(row) * p.ld_out + col0;
  if (n == 8 && aligned) {
    *reinterpret_cast<uint4*>(o) = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
  } else {
    for (int j = 0; j < n; ++j) o[j] = __float2bfloat16_rn(v[j]);
  }
}

template <int BN, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(SPLIT_THREADS, 1)
gemm_splitk_kernel(const __grid_constant__ GemmMaps maps, const __grid_constant__ GemmParams p, const int splits) {
  using S = SplitShape<BN>;
  constexpr int A_BYTES = BM * BK_BYTES;
  constexpr int TMEM_COLS = BN;
  constexpr int K_ELEMS = 64, KSTEPS = 4;
  constexpr int CHUNKS = BN / 4;                    // 16-byte fp32 chunks of a row

  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full_bar[S::STAGES], empty_bar[S::STAGES], done_bar;
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;

  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int part = static_cast<int>(cluster_ctarank());
  const int tile = blockIdx.x / splits;
  const int tiles_m = (p.M + BM - 1) / BM;
  const int m0 = (tile % tiles_m) * BM, n0 = (tile / tiles_m) * BN;
  int total_kb = 0;
  for (int s = 0; s < p.num_seg; ++s) total_kb += p.kblocks[s];
  const int kb_lo = static_cast<int>(static_cast<long long>(part) * total_kb / splits);
  const int kb_hi = static_cast<int>(static_cast<long long>(part + 1) * total_kb / splits);

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(&done_bar, 1);
    abort_s = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(&tmem_base_s, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_s;

  if (warp == 0) {
    int stage = 0, last_stage = -1;
    uint32_t phase = 0, last_phase = 0;
    bool ok = true;
    int s = 0, base = 0;
    for (int kb = kb_lo; ok && kb < kb_hi; ++kb) {
      while (kb - base >= p.kblocks[s]) base += p.kblocks[s++];
      const int k0 = (kb - base) * K_ELEMS;
      if (!__all_sync(0xffffffffu, mbar_wait(&empty_bar[stage], phase ^ 1u, &abort_s))) {
        if (lane == 0) report_status(p.status, STATUS_TIMEOUT, 41, stage);
        ok = false;
        break;
      }
      uint8_t* sa = smem + stage * S::STAGE_BYTES;
      uint8_t* sb = sa + A_BYTES;
      if (elect_one()) {
        mbar_expect_tx(&full_bar[stage], S::STAGE_BYTES);
        if (!A_MN) {
          tma_load_2d(sa, &maps.a[s], &full_bar[stage], k0, m0);
        } else {
          tma_load_2d(sa, &maps.a[s], &full_bar[stage], m0, k0);
          tma_load_2d(sa + 8192, &maps.a[s], &full_bar[stage], m0 + 64, k0);
        }
        if (!B_MN) {
          tma_load_2d(sb, &maps.b[s], &full_bar[stage], k0, n0);
          tma_load_2d(sb + (BN / 2) * BK_BYTES, &maps.b[s], &full_bar[stage], k0, n0 + BN / 2);
        } else {
#pragma unroll
          for (int j = 0; j < BN / 64; ++j) tma_load_2d(sb + j * 8192, &maps.b[s], &full_bar[stage], n0 + j * 64, k0);
        }
      }
      __syncwarp();
      last_stage = stage;
      last_phase = phase;
      if (++stage == S::STAGES) { stage = 0; phase ^= 1u; }
    }
    if (!ok && last_stage >= 0) {
      // abandoned: let the copies already in flight land (bounded)
      const uint64_t t0 = globaltimer_ns();
      while (!mbar_try_wait(&full_bar[last_stage], last_phase) && globaltimer_ns() - t0 < 5000000ull) {
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc(1, UMMA_BF16, UMMA_BF16, A_MN ? 1u : 0u, B_MN ? 1u : 0u, BM, BN);
    int stage = 0;
    uint32_t phase = 0;
    for (int kb = kb_lo; kb < kb_hi; ++kb) {
      if (!__all_sync(0xffffffffu, mbar_wait(&full_bar[stage], phase, &abort_s))) {
        if (lane == 0) report_status(p.status, STATUS_TIMEOUT, 42, stage);
        break;
      }
      tc_fence_after();
      const uint32_t sa = smem_u32(smem + stage * S::STAGE_BYTES), sb = sa + A_BYTES;
      const uint64_t da = A_MN ? make_desc_mnmajor_sw128(sa, 8192) : make_desc_kmajor_sw128(sa);
      const uint64_t db = B_MN ? make_desc_mnmajor_sw128(sb, 8192) : make_desc_kmajor_sw128(sb);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < KSTEPS; ++k)
          umma_f16_ss(tmem_base, da + static_cast<uint64_t>(A_MN ? (k * 2048) >> 4 : (k * 32) >> 4),
                      db + static_cast<uint64_t>(B_MN ? (k * 2048) >> 4 : (k * 32) >> 4), idesc, (kb != kb_lo || k != 0) ? 1u : 0u);
        umma_commit(&empty_bar[stage]);
        if (kb == kb_hi - 1) umma_commit(&done_bar);
      }
      __syncwarp();
      if (++stage == S::STAGES) { stage = 0; phase ^= 1u; }
    }
    __syncwarp();
  } else {
    // the accumulator goes to the operand ring (every MMA that read it is complete) as fp32 rows; chunks are XOR-swizzled by
    // the row so that the row-per-lane writes and the chunk-per-lane reads below both spread over the banks
    const int quad = warp & 3, row = quad * 32 + lane;
    if (__all_sync(0xffffffffu, mbar_wait(&done_bar, 0, &abort_s))) {
      tc_fence_after();
      float4* mine = reinterpret_cast<float4*>(smem) + row * CHUNKS;
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + c * 32, r);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 8; ++j)
          mine[(c * 8 + j) ^ (row & 15)] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]),
                                                       __uint_as_float(r[4 * j + 3]));
      }
    } else if (lane == 0) {
      report_status(p.status, STATUS_TIMEOUT, 43, 0);
    }
    tc_fence_before();
  }
  __syncwarp();
  cluster_arrive();   // all parts are in shared memory
  cluster_wait();
  {
    bool aligned = ((reinterpret_cast<uintptr_t>(p.out) | static_cast<uintptr_t>(static_cast<size_t>(p.ld_out) * 2)) & 15) == 0;
    const int row_lo = part * BM / splits, row_hi = (part + 1) * BM / splits;
    const int cols = min(BN, p.N - n0), groups = (cols + 7) / 8;
    const int rows = min(row_hi, p.M - m0) - row_lo;
    const uint32_t base = smem_u32(smem);
    for (int i = threadIdx.x; i < rows * groups; i += SPLIT_THREADS) {
      const int row = row_lo + i / groups, g = i % groups;
      float v[8];
      const uint32_t o0 = base + (row * CHUNKS + ((2 * g) ^ (row & 15))) * 16, o1 = base + (row * CHUNKS + ((2 * g + 1) ^ (row & 15))) * 16;
      split_sum8<SPLIT_MAX>(o0, o1, splits, 1u, 0u, v);
      split_store8(p, m0 + row, n0 + g * 8, v, aligned);
    }
  }
  __syncwarp();
  cluster_arrive();   // no CTA leaves while another still reads its part
  cluster_wait();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ---- pairs: one 256 x 256 tile per cluster of S pairs (2 S CTAs). A pair runs its share of the K blocks exactly as
// gemm_tcgen05_pair_kernel does (each CTA stages 128 rows of A and of B, the even CTA issues for both); afterwards every CTA
// holds a 128 x 256 fp32 part in its own TMEM, the S parts of a row half meet in distributed shared memory, and pair i finishes
// 128 / S rows of each half.
constexpr int PSPLIT_STAGES = 6, PSPLIT_STAGE_BYTES = 2 * BM * BK_BYTES, PSPLIT_MAX = 4;
constexpr int PSPLIT_SMEM = PSPLIT_STAGES * PSPLIT_STAGE_BYTES + 1024;
static_assert(BM * 256 * 4 <= PSPLIT_STAGES * PSPLIT_STAGE_BYTES, "the fp32 part of a tile reuses the operand ring");

template <bool B_MN>
__global__ void __launch_bounds__(SPLIT_THREADS, 1)
gemm_pair_splitk_kernel(const __grid_constant__ GemmMaps maps, const __grid_constant__ GemmParams p, const int splits) {
  constexpr int BN = 256, BNH = 128, TMEM_COLS = 256, K_ELEMS = 64, KSTEPS = 4, CHUNKS = BN / 4;
  constexpr int A_BYTES = BM * BK_BYTES;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full_bar[PSPLIT_STAGES];    // used in the even CTA: both CTAs' loads of a stage have landed
  __shared__ uint64_t empty_bar[PSPLIT_STAGES];   // in each CTA: the MMAs that read this stage are done
  __shared__ uint64_t done_bar;                   // in each CTA: accumulator complete
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;

  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t crank = cluster_ctarank(), rank = crank & 1u, lead = crank & ~1u;
  const bool leader = rank == 0;
  const int part = static_cast<int>(crank >> 1);
  const int tile = blockIdx.x / (2 * splits);
  const int tiles_m = (p.M + 2 * BM - 1) / (2 * BM);
  const int m0 = (tile % tiles_m) * (2 * BM) + static_cast<int>(rank) * BM, n0 = (tile / tiles_m) * BN;
  int total_kb = 0;
  for (int s = 0; s < p.num_seg; ++s) total_kb += p.kblocks[s];
  const int kb_lo = static_cast<int>(static_cast<long long>(part) * total_kb / splits);
  const int kb_hi = static_cast<int>(static_cast<long long>(part + 1) * total_kb / splits);

  if (threadIdx.x == 0) {
    for (int s = 0; s < PSPLIT_STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(&done_bar, 1);
    abort_s = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(&tmem_base_s, TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_arrive();   // the peer's barriers exist before anything is sent to them
  cluster_wait();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_s;
  const uint32_t peer_abort = mapa_shared(smem_u32(&abort_s), crank ^ 1u);

  if (warp == 0) {
    int stage = 0, s = 0, base = 0;
    uint32_t phase = 0;
    bool ok = true, issued = false;
    for (int kb = kb_lo; kb < kb_hi; ++kb) {
      while (kb - base >= p.kblocks[s]) base += p.kblocks[s++];
      const int k0 = (kb - base) * K_ELEMS;
      if (!__all_sync(0xffffffffu, mbar_wait(&empty_bar[stage], phase ^ 1u, &abort_s))) {
        if (lane == 0) { report_status(p.status, STATUS_TIMEOUT, 61, stage); st_shared_cluster_u32(peer_abort, 1u); }
        ok = false;
        break;
      }
      uint8_t* sa = smem + stage * PSPLIT_STAGE_BYTES;
      uint8_t* sb = sa + A_BYTES;
      const uint32_t bar = mapa_shared(smem_u32(&full_bar[stage]), lead);
      const int nb = n0 + static_cast<int>(rank) * BNH;
      if (elect_one()) {
        if (leader) mbar_expect_tx(&full_bar[stage], 2 * PSPLIT_STAGE_BYTES);
        tma_load_2d_pair(sa, &maps.a[s], bar, k0, m0);
        if (!B_MN) {
          tma_load_2d_pair(sb, &maps.b[s], bar, k0, nb);
        } else {
          tma_load_2d_pair(sb, &maps.b[s], bar, nb, k0);
          tma_load_2d_pair(sb + 8192, &maps.b[s], bar, nb + 64, k0);
        }
      }
      __syncwarp();
      issued = true;
      if (++stage == PSPLIT_STAGES) { stage = 0; phase ^= 1u; }
    }
    if (!ok && issued) {
      // abandoned: give the copies already in flight time to land (bounded)
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 2000000ull) {
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (leader) {
      constexpr uint32_t idesc = make_idesc(1, UMMA_BF16, UMMA_BF16, 0u, B_MN ? 1u : 0u, 2 * BM, BN);
      const uint16_t mask = static_cast<uint16_t>(3u << lead);
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb_lo; kb < kb_hi; ++kb) {
        if (!__all_sync(0xffffffffu, mbar_wait(&full_bar[stage], phase, &abort_s))) {
          if (lane == 0) { report_status(p.status, STATUS_TIMEOUT, 62, stage); st_shared_cluster_u32(peer_abort, 1u); }
          break;
        }
        tc_fence_after();
        const uint32_t sa = smem_u32(smem + stage * PSPLIT_STAGE_BYTES), sb = sa + A_BYTES;
        const uint64_t da = make_desc_kmajor_sw128(sa);
        const uint64_t db = B_MN ? make_desc_mnmajor_sw128(sb, 8192) : make_desc_kmajor_sw128(sb);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < KSTEPS; ++k)
            umma_f16_ss_pair(tmem_base, da + static_cast<uint64_t>((k * 32) >> 4), db + static_cast<uint64_t>(B_MN ? (k * 2048) >> 4 : (k * 32) >> 4),
                             idesc, (kb != kb_lo || k != 0) ? 1u : 0u);
          umma_commit_pair(&empty_bar[stage], mask);
          if (kb == kb_hi - 1) umma_commit_pair(&done_bar, mask);
        }
        __syncwarp();
        if (++stage == PSPLIT_STAGES) { stage = 0; phase ^= 1u; }
      }
    }
    __syncwarp();
  } else {
    const int quad = warp & 3, row = quad * 32 + lane;
    if (__all_sync(0xffffffffu, mbar_wait(&done_bar, 0, &abort_s))) {
      tc_fence_after();
      float4* mine = reinterpret_cast<float4*>(smem) + row * CHUNKS;
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + c * 32, r);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 8; ++j)
          mine[(c * 8 + j) ^ (row & 15)] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]),
                                                       __uint_as_float(r[4 * j + 3]));
      }
    } else if (lane == 0) {
      report_status(p.status, STATUS_TIMEOUT, 63, 0);
      st_shared_cluster_u32(peer_abort, 1u);
    }
    tc_fence_before();
  }
  __syncwarp();
  cluster_arrive();   // all parts are in shared memory
  cluster_wait();
  {
    const bool aligned = ((reinterpret_cast<uintptr_t>(p.out) | static_cast<uintptr_t>(static_cast<size_t>(p.ld_out) * 2)) & 15) == 0;
    const int row_lo = part * BM / splits, row_hi = (part + 1) * BM / splits;
    const int groups = (min(BN, p.N - n0) + 7) / 8;
    const int rows = min(row_hi, p.M - m0) - row_lo;
    const uint32_t base = smem_u32(smem);
    for (int i = threadIdx.x; i < rows * groups; i += SPLIT_THREADS) {
      const int row = row_lo + i / groups, g = i % groups;
      float v[8];
      const uint32_t o0 = base + (row * CHUNKS + ((2 * g) ^ (row & 15))) * 16, o1 = base + (row * CHUNKS + ((2 * g + 1) ^ (row & 15))) * 16;
      split_sum8<PSPLIT_MAX>(o0, o1, splits, 2u, rank, v);
      split_store8(p, m0 + row, n0 + g * 8, v, aligned);
    }
  }
  __syncwarp();
  cluster_arrive();   // no CTA frees TMEM or leaves while another still reads its part
  cluster_wait();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

template <typename Kernel>
static cudaError_t cluster_config(Kernel kern, int smem, int ctas, int cluster, cudaStream_t stream, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr) {
  memset(cfg, 0, sizeof(*cfg));
  cfg->gridDim = dim3(static_cast<unsigned>(ctas), 1, 1);
  cfg->blockDim = dim3(SPLIT_THREADS, 1, 1);
  cfg->dynamicSmemBytes = smem;
  cfg->stream = stream;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = cluster;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cfg->attrs = attr;
  cfg->numAttrs = 1;
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}
// clusters of `cluster` CTAs the device holds at once (one CTA per SM; a cluster lives inside one GPC)
template <typename Kernel>
static int cluster_capacity(Kernel kern, int smem, int cluster, int num_sms, std::atomic<int>* cached) {
  int n = cached->load(std::memory_order_relaxed);
  if (n > 0) return n;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  if (cluster_config(kern, smem, num_sms / cluster * cluster, cluster, nullptr, &cfg, &attr) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess)
    n = 0;
  cudaGetLastError();
  if (n < 1 || n > num_sms / cluster) n = num_sms / cluster > 0 ? num_sms / cluster : 1;
  cached->store(n, std::memory_order_relaxed);
  return n;
}
template <int BN>
static int split_capacity(int splits, int num_sms) {
  static std::atomic<int> cached[SPLIT_MAX + 1];
  return cluster_capacity(gemm_splitk_kernel<BN, false, false>, SplitShape<BN>::SMEM, splits, num_sms, &cached[splits]);
}
static int pair_split_capacity(int splits, int num_sms) {
  static std::atomic<int> cached[PSPLIT_MAX + 1];
  return cluster_capacity(gemm_pair_splitk_kernel<false>, PSPLIT_SMEM, 2 * splits, num_sms, &cached[splits]);
}

template <int BN, bool A_MN, bool B_MN>
static int launch_split(const GemmMaps& maps, const GemmParams& p, int splits, cudaStream_t stream) {
  const long long tiles = static_cast<long long>((p.M + BM - 1) / BM) * ((p.N + BN - 1) / BN);
  auto kern = gemm_splitk_kernel<BN, A_MN, B_MN>;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  cudaError_t e = cluster_config(kern, SplitShape<BN>::SMEM, static_cast<int>(tiles * splits), splits, stream, &cfg, &attr);
  return static_cast<int>(e != cudaSuccess ? e : cudaLaunchKernelEx(&cfg, kern, maps, p, splits));
}
template <bool B_MN>
static int launch_pair_split(const GemmMaps& maps, const GemmParams& p, int splits, cudaStream_t stream) {
  const long long tiles = static_cast<long long>((p.M + 2 * BM - 1) / (2 * BM)) * ((p.N + 255) / 256);
  auto kern = gemm_pair_splitk_kernel<B_MN>;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  cudaError_t e = cluster_config(kern, PSPLIT_SMEM, static_cast<int>(tiles * 2 * splits), 2 * splits, stream, &cfg, &attr);
  return static_cast<int>(e != cudaSuccess ? e : cudaLaunchKernelEx(&cfg, kern, maps, p, splits));
}
