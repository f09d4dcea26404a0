// bfloat16 matrix product for a few hundred tokens (short prompts, prompt portions beside decoding requests):
//   D[t, n] = sum_k X[t, k] * W[n, k]      (both operands K-major, float32 accumulation)
//
// What bounds it: between the decode products, which the weights' way from memory bounds, and those of whole prompts,
// which the tensor cores bound, it is the operands' way from L2 into shared memory.  About 10.6 TB/s arrive there, while
// the tensor cores at full clock would take 18 from tiles of 256 x 256.  So the weights are the 256 rows of an MMA
// on a pair of SMs (tcgen05.mma.cta_group::2, each block loads 128 rows) and ALL tokens of a group, up to 512 in two
// accumulators of up to 256 columns, its N side: a pair loads every weight byte of its tile once, whatever the token
// count, and the columns follow the token count in steps of 16 (32 above 256) instead of filling tiles of 256.
// Half of the columns' rows come from either block.
//
// Few weight rows leave pairs idle, so K is split over up to four pairs, which form one thread-block cluster of up to
// eight blocks: every block stages its float32 sums in the shared memory that the operands leave, and every pair adds up
// its share of the tokens over distributed shared memory, in the order of the splits, and stores bfloat16.  The host picks
// groups, splits and (where whole rounds of the pairs leave a few tiles over) a second launch for those with more splits
// by the estimate in plan_rows.
//
// Every wait on an mbarrier is bounded, reports kErrWait and lets the block leave through the common exit, which
// meets the cluster at a barrier before tensor memory is freed.  Every block loads for itself.
#include <math.h>

#include "tcgen05_utils.cuh"
#include "entry_points.cuh"

namespace tk {

constexpr int kGkBM = 128;           // weight rows per block; the pair's tile has 256
constexpr int kGkBK = 64;
constexpr int kGkThreads = 320;      // warp 0: TMA, warp 1: MMA (first block of the pair only), warps 2..9: epilogue
constexpr int kGkEpiThreads = kGkThreads - 64;
constexpr int kGkMaxStages = 8;
constexpr int kGkMaxSplits = 4;
constexpr uint32_t kGkRingBytes = 208u * 1024u;
constexpr uint32_t kGkWBytes = kGkBM * kGkBK * 2;

struct GemmTokensParams {
  void* out;
  int* err;
  int tokens, rows, k;
  long long ld_out;
  int tile0;              // first 256-row tile of this launch
  int width;              // columns of a group: n_acc * acc_n
  int acc_n;              // columns of one accumulator: a multiple of 16 up to 256
  int n_acc;              // 1 or 2
  int n_splits;
  int n_stages;
  int chunk;              // columns that are staged at a time
  int mode;               // 0: bf16 [tokens, rows]; 1, 2: gated activation, bf16 [tokens, rows / 2]; 3..6: unary_act(sum, mode - 3)
};

// Sums over S splits of the four floats at `addr` in the blocks first, first + 2, ..., for U tokens `step` bytes apart (from
// the token `there` on the last one again), all requested before the first is used: a load over the cluster's network takes
// the better part of a microsecond.
template <int S, int U>
__device__ __forceinline__ void gk_sums(uint32_t addr, uint32_t step, uint32_t first, int there, float4 (&out)[U]) {
  float4 v[S][U];
#pragma unroll
  for (int j = 0; j < S; ++j) {
    uint32_t at = addr;
    if (S > 1) asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(at) : "r"(addr), "r"(first + 2u * (uint32_t)j));
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t from = at + (uint32_t)min(u, there - 1) * step;
      if (S == 1) {
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n"
                     : "=f"(v[j][u].x), "=f"(v[j][u].y), "=f"(v[j][u].z), "=f"(v[j][u].w) : "r"(from) : "memory");
      } else {
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n"
                     : "=f"(v[j][u].x), "=f"(v[j][u].y), "=f"(v[j][u].z), "=f"(v[j][u].w) : "r"(from) : "memory");
      }
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    out[u] = v[0][u];
#pragma unroll
    for (int j = 1; j < S; ++j) {
      out[u].x += v[j][u].x; out[u].y += v[j][u].y; out[u].z += v[j][u].z; out[u].w += v[j][u].w;
    }
  }
}

// The staged columns [c_begin, c_end) that fall to this split, added up over S splits, through the activation and out.
template <int S>
__device__ __forceinline__ void gk_store(const GemmTokensParams& p, uint32_t base, int tile, int tok0, int c_begin, int c_end,
                                         int split, uint32_t half, int et) {
  __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.out);
  const int last = min(c_end, p.tokens - tok0);          // the group's tokens end here
  if (p.mode == 1 || p.mode == 2) {
    // four neighbouring outputs of the tile's 64 a thread: gate in rows j.., up in rows 64 + j..
    constexpr int U = S > 2 ? 2 : (S == 2 ? 3 : 4);
    const int j4 = (et & 15) * 4, inter = p.rows >> 1;
    const int oc = (tile * 2 + (int)half) * 64 + j4;
    if (oc >= inter) return;       // inter is a multiple of 64: all four outputs exist
    constexpr int kStep = S * (kGkEpiThreads / 16);
    for (int c = c_begin + split + S * (et >> 4); c < last; c += U * kStep) {
      const int there = min(U, (last - c + kStep - 1) / kStep);
      const uint32_t at = base + (uint32_t)(((c - c_begin) * kGkBM + j4) * 4);
      float4 g[U], u[U];
      gk_sums<S, U>(at, kStep * kGkBM * 4, half, there, g);
      gk_sums<S, U>(at + 64 * 4, kStep * kGkBM * 4, half, there, u);
#pragma unroll
      for (int i = 0; i < U; ++i) {
        if (i >= there) continue;
        uint2 packed;
        *reinterpret_cast<__nv_bfloat162*>(&packed.x) =
            __floats2bfloat162_rn(glu_act(g[i].x, p.mode - 1) * u[i].x, glu_act(g[i].y, p.mode - 1) * u[i].y);
        *reinterpret_cast<__nv_bfloat162*>(&packed.y) =
            __floats2bfloat162_rn(glu_act(g[i].z, p.mode - 1) * u[i].z, glu_act(g[i].w, p.mode - 1) * u[i].w);
        *reinterpret_cast<uint2*>(out + (size_t)(tok0 + c + i * kStep) * p.ld_out + oc) = packed;
      }
    }
    return;
  }
  // a warp takes a token, its lanes four neighbouring rows each; rows are a multiple of 8
  constexpr int U = S > 2 ? 4 : 8;
  const int r4 = (et & 31) * 4, row = tile * 2 * kGkBM + (int)half * kGkBM + r4;
  if (row >= p.rows) return;
  constexpr int kStep = S * (kGkEpiThreads / 32);
  for (int c = c_begin + split + S * (et >> 5); c < last; c += U * kStep) {
    const int there = min(U, (last - c + kStep - 1) / kStep);
    float4 s[U];
    gk_sums<S, U>(base + (uint32_t)(((c - c_begin) * kGkBM + r4) * 4), kStep * kGkBM * 4, half, there, s);
#pragma unroll
    for (int i = 0; i < U; ++i) {
      if (i >= there) continue;
      if (p.mode >= 3) {
        const int act = p.mode - 3;
        s[i] = make_float4(unary_act(s[i].x, act), unary_act(s[i].y, act), unary_act(s[i].z, act), unary_act(s[i].w, act));
      }
      uint2 packed;
      *reinterpret_cast<__nv_bfloat162*>(&packed.x) = __floats2bfloat162_rn(s[i].x, s[i].y);
      *reinterpret_cast<__nv_bfloat162*>(&packed.y) = __floats2bfloat162_rn(s[i].z, s[i].w);
      *reinterpret_cast<uint2*>(out + (size_t)(tok0 + c + i * kStep) * p.ld_out + row) = packed;
    }
  }
}

// grid: x the blocks of a cluster (2 * n_splits), y groups of tokens (neighbours share a weight tile in L2), z row tiles.
__global__ void __launch_bounds__(kGkThreads, 1)
gemm_tokens_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                   GemmTokensParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t raw = gt_smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;         // the same offset in all blocks
  unsigned char* smem = smem_raw + (base - raw);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kGkRingBytes);
  uint64_t* empty_bar = full_bar + kGkMaxStages;
  uint64_t* acc_full = empty_bar + kGkMaxStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const uint32_t half = rank & 1u;
  const int split = (int)(rank >> 1);
  const int tile = p.tile0 + (int)blockIdx.z;
  const int tok0 = (int)blockIdx.y * p.width;
  const int kb_total = (p.k + kGkBK - 1) / kGkBK;
  const int kb_per = (kb_total + p.n_splits - 1) / p.n_splits;
  const int kb_begin = split * kb_per;
  const int n_kb = min(kb_begin + kb_per, kb_total) - kb_begin;      // at least one (the host sees to it)
  const uint32_t x_acc_bytes = (uint32_t)(p.acc_n >> 1) * kGkBK * 2;   // this block's rows of one accumulator's columns
  const uint32_t stage_bytes = kGkWBytes + (uint32_t)p.n_acc * x_acc_bytes;
  const int w_row = tile * 2 * kGkBM + (int)half * kGkBM;
  const int x_row = tok0 + (int)half * (p.acc_n >> 1);
  const uint32_t tmem_cols = p.n_acc == 2 ? 512u : (p.acc_n <= 32 ? 32u : p.acc_n <= 64 ? 64u : p.acc_n <= 128 ? 128u : 256u);

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.n_stages; ++s) {
      mbar_init(gt_smem_u32(&full_bar[s]), 1);
      mbar_init(gt_smem_u32(&empty_bar[s]), 1);
    }
    mbar_init(gt_smem_u32(acc_full), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n"
                 ::"r"(gt_smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();            // all blocks' barriers exist before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // only now may later kernels begin: none of them can take tensor memory before this block has its own
  pdl_trigger();

  if (warp == 0) {
    // ---- TMA producer of this block's halves ---------------------------------------------------
    if (elect_one()) {
      const int first = min(n_kb, p.n_stages);
      // the weights of the first ring, which no kernel writes, before the wait for the kernel in front
      for (int i = 0; i < first; ++i) {
        const uint32_t full = gt_smem_u32(&full_bar[i]);
        if (half == 0) mbar_expect_tx(full, 2 * stage_bytes);        // both blocks' halves land here
        tma_load_2d_pair(base + (uint32_t)i * stage_bytes, &map_w, (kb_begin + i) * kGkBK, w_row, full);
      }
      pdl_wait();
      for (int i = 0; i < first; ++i) {
        const uint32_t full = gt_smem_u32(&full_bar[i]);
        const uint32_t dst = base + (uint32_t)i * stage_bytes + kGkWBytes;
        for (int a = 0; a < p.n_acc; ++a) {
          tma_load_2d_pair(dst + (uint32_t)a * x_acc_bytes, &map_x, (kb_begin + i) * kGkBK, x_row + a * p.acc_n, full);
        }
      }
      int s = 0;
      uint32_t parity = 0;
      for (int i = first; i < n_kb; ++i) {
        if (!mbar_wait(gt_smem_u32(&empty_bar[s]), parity, abort_flag)) {
          set_error(p.err, kErrWait, 24, i, s);
          *abort_flag = 1;
          break;
        }
        const uint32_t full = gt_smem_u32(&full_bar[s]);
        if (half == 0) mbar_expect_tx(full, 2 * stage_bytes);
        const uint32_t dst = base + (uint32_t)s * stage_bytes;
        tma_load_2d_pair(dst, &map_w, (kb_begin + i) * kGkBK, w_row, full);
        for (int a = 0; a < p.n_acc; ++a) {
          tma_load_2d_pair(dst + kGkWBytes + (uint32_t)a * x_acc_bytes, &map_x, (kb_begin + i) * kGkBK, x_row + a * p.acc_n, full);
        }
        if (++s == p.n_stages) { s = 0; parity ^= 1u; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---- MMA issuer: the pair's first block only --------------------------------------------------
    if (half == 0 && elect_one()) {
      // bf16 x bf16 -> f32, K-major operands, M = 256 over the pair, N = acc_n
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.acc_n >> 3) << 17) |
                             ((uint32_t)(256 >> 4) << 24);
      const uint16_t mask = (uint16_t)(3u << rank);
      bool ok = true;
      int s = 0;
      uint32_t parity = 0;
      for (int i = 0; i < n_kb; ++i) {
        if (!mbar_wait(gt_smem_u32(&full_bar[s]), parity, abort_flag)) {
          set_error(p.err, kErrWait, 25, i, s);
          *abort_flag = 1;
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t w_addr = base + (uint32_t)s * stage_bytes;
        const uint64_t desc_a = umma_desc_sw128(w_addr);
        for (int a = 0; a < p.n_acc; ++a) {
          const uint64_t desc_b = umma_desc_sw128(w_addr + kGkWBytes + (uint32_t)a * x_acc_bytes);
#pragma unroll
          for (int k = 0; k < kGkBK / 16; ++k) {
            umma_bf16_pair(tmem_base + (uint32_t)(a * 256), desc_a + (uint64_t)(2 * k), desc_b + (uint64_t)(2 * k), idesc,
                        (i > 0 || k > 0) ? 1u : 0u);
          }
        }
        umma_commit_pair(gt_smem_u32(&empty_bar[s]), mask);      // both blocks may refill the stage
        if (++s == p.n_stages) { s = 0; parity ^= 1u; }
      }
      if (ok) umma_commit_pair(gt_smem_u32(acc_full), mask);     // both blocks may read their accumulators
    }
    __syncwarp();
  }

  // ---- epilogue: warps 2..9 of all blocks, two to a quarter of the accumulator's lanes ------------
  const int et = (int)threadIdx.x - 64;
  const int quarter = warp & 3;
  bool ok = true;
  if (warp >= 2) {
    pdl_wait();                  // nothing is stored before the kernels in front are done with the output
    ok = __all_sync(0xffffffffu, mbar_wait(gt_smem_u32(acc_full), 0u, abort_flag));
    if (!ok && lane == 0) { set_error(p.err, kErrWait, 26, (int)rank, 0); *abort_flag = 1; }
    tc_fence_after();
  }
  float* stage = reinterpret_cast<float*>(smem);       // [chunk][128]: the ring, which the products are done with
  for (int c_begin = 0; c_begin < p.width; c_begin += p.chunk) {
    const int c_end = min(c_begin + p.chunk, p.width);
    if (c_begin > 0) {
      // the columns before these have been read by everyone
      if (p.n_splits > 1) cluster_sync_all(); else __syncthreads();
    }
    if (warp >= 2) {
      // columns 16 by 16, the quarter's two warps in turn, two blocks on the way at a time; a block of 16 lies in
      // one accumulator
      for (int c0 = c_begin + 16 * ((warp - 2) >> 2); c0 < c_end; c0 += 64) {
        uint32_t v[2][16];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c = c0 + 32 * h, a = c >= p.acc_n ? 1 : 0;
          if (ok && c < c_end) {
            tmem_ld16(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(a * 256 + c - a * p.acc_n), v[h]);
          } else {
#pragma unroll
            for (int e = 0; e < 16; ++e) v[h][e] = 0u;
          }
        }
        tmem_wait_ld();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (c0 + 32 * h < c_end) {
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              stage[(c0 + 32 * h - c_begin + e) * kGkBM + quarter * 32 + lane] = __uint_as_float(v[h][e]);
            }
          }
        }
      }
    }
    if (p.n_splits > 1) cluster_sync_all(); else __syncthreads();
    if (warp >= 2) {
      switch (p.n_splits) {
        case 1: gk_store<1>(p, base, tile, tok0, c_begin, c_end, split, half, et); break;
        case 2: gk_store<2>(p, base, tile, tok0, c_begin, c_end, split, half, et); break;
        case 3: gk_store<3>(p, base, tile, tok0, c_begin, c_end, split, half, et); break;
        default: gk_store<4>(p, base, tile, tok0, c_begin, c_end, split, half, et); break;
      }
    }
    __syncwarp();
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();            // no block leaves while another may still reach into it
  if (warp == 2) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
  }
}

// ---- host side ------------------------------------------------------------------------------

static int make_tokens_map(CUtensorMap* map, const void* ptr, long long rows, long long k, long long ld, int box_rows) {
  const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kGkBK, (cuuint32_t)box_rows};
  return make_bf16_map(map, ptr, 2, dims, strides, box);
}

constexpr size_t kGkSmemBytes = kGkRingBytes + 1024 /* alignment */ + 256 /* barriers */;

// How many clusters of n_splits pairs the device holds at a time (0: the device did not say).
static int resident_clusters(int n_splits) {
  static int known[64][kGkMaxSplits + 1] = {{0}};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (known[dev][n_splits] == 0) {
    if (cudaFuncSetAttribute(gemm_tokens_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGkSmemBytes) != cudaSuccess) return 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * n_splits, 1, 148);
    cfg.blockDim = dim3(kGkThreads);
    cfg.dynamicSmemBytes = kGkSmemBytes;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2 * n_splits; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_tokens_kernel, &cfg) != cudaSuccess || n < 1) return 0;
    known[dev][n_splits] = n;
  }
  return known[dev][n_splits];
}

struct TokensPlan { int groups, splits, width, tail_tiles, tail_splits; float us; };

static int group_width(int tokens, int groups) {
  const int w = (tokens + groups - 1) / groups;
  return w <= 256 ? (w + 15) / 16 * 16 : (w + 31) / 32 * 32;
}

// Microseconds that `tiles` row tiles take with these groups and splits; negative: not possible.  Measured (B200, products
// one after another): a k block takes what the tensor cores need at 1.73 GHz, what its operands need from L2 (10.6 TB/s for
// all blocks together) or 0.2 us to issue, whichever is longest; a round of blocks begins and ends in 4.4 us and 1.1 us for
// every 96 columns it stages, adds up and stores.
static float estimate(int tiles, int kb_total, int groups, int splits, int width, int slots) {
  const int kb = (kb_total + splits - 1) / splits;
  if (slots < 1 || (splits - 1) * kb >= kb_total) return -1.0f;
  const int clusters = tiles * groups, rounds = (clusters + slots - 1) / slots;
  const float blocks = 2.0f * (float)splits * (float)(clusters < slots ? clusters : slots);
  const float mma = 2.0f * (float)width / 1730.0f, load = blocks * (16384.0f + 64.0f * (float)width) / 10.6e6f;
  const float per_kb = fmaxf(fmaxf(mma, load), 0.2f);
  return (float)rounds * (per_kb * (float)kb + 4.4f + 0.0115f * (float)width + (splits > 1 ? 0.4f + 0.003f * (float)width : 0.0f));
}

// Groups of tokens and K splits of least estimated time.  Where a number of whole rounds leaves tiles over, those may
// run as a launch of their own with more splits.
static TokensPlan plan_rows(int tokens, int rows, int k) {
  const int tiles = (rows + 255) / 256, kb_total = (k + kGkBK - 1) / kGkBK;
  TokensPlan best = {0, 0, 0, 0, 0, 1e30f};
  const int g_min = (tokens + 511) / 512;
  int slots[kGkMaxSplits + 1];
  for (int s = 1; s <= kGkMaxSplits; ++s) slots[s] = resident_clusters(s);
  for (int g = g_min; g <= g_min + 7 && g <= 64; ++g) {
    const int width = group_width(tokens, g);
    if (width > 512 || (g > g_min && width < 32)) continue;
    for (int s = 1; s <= kGkMaxSplits; ++s) {
      const float whole = estimate(tiles, kb_total, g, s, width, slots[s]);
      if (whole >= 0.0f && whole < best.us) best = {g, s, width, 0, 0, whole};
      if (whole < 0.0f || slots[s] < g) continue;
      const int per_round = slots[s] / g, left = tiles % per_round;
      if (left == 0 || left == tiles) continue;
      const float head = estimate(tiles - left, kb_total, g, s, width, slots[s]) - 1.0f;     // the tail begins early
      for (int s2 = s + 1; s2 <= kGkMaxSplits; ++s2) {
        const float tail = estimate(left, kb_total, g, s2, width, slots[s2]);
        if (tail >= 0.0f && head + tail < best.us) best = {g, s, width, left, s2, head + tail};
      }
    }
  }
  return best;
}

static int launch_tokens(const void* x, const void* w, GemmTokensParams p, long long ld_x, long long ld_w, int groups, int tiles,
                         int splits, int width, int tile0, int* launches, cudaStream_t stream) {
  if (tiles <= 0) return 0;
  const int kb_total = (p.k + kGkBK - 1) / kGkBK, kb = splits > 0 ? (kb_total + splits - 1) / splits : 0;
  if (splits < 1 || splits > kGkMaxSplits || (splits - 1) * kb >= kb_total || groups < 1 || groups > 65535 || tiles > 65535 ||
      width < 16 || width > 512 || width % (width > 256 ? 32 : 16) != 0 || (long long)groups * width < p.tokens) {
    return (int)cudaErrorInvalidValue;
  }
  p.n_acc = width > 256 ? 2 : 1;
  p.acc_n = width / p.n_acc;
  p.width = width;
  p.n_splits = splits;
  p.tile0 = tile0;
  const unsigned stage_bytes = kGkWBytes + (unsigned)p.n_acc * (unsigned)(p.acc_n / 2) * kGkBK * 2;
  int stages = (int)(kGkRingBytes / stage_bytes);
  if (stages > kGkMaxStages) stages = kGkMaxStages;
  p.n_stages = stages;
  p.chunk = (int)(kGkRingBytes / (kGkBM * 4)) / 32 * 32;       // whole steps of the two warps of a quarter
  CUtensorMap map_w, map_x;
  int rc = make_tokens_map(&map_w, w, p.rows, p.k, ld_w, kGkBM);
  if (rc != 0) return rc;
  rc = make_tokens_map(&map_x, x, p.tokens, p.k, ld_x, p.acc_n / 2);
  if (rc != 0) return rc;
  if (resident_clusters(splits) < 1) return (int)cudaErrorLaunchOutOfResources;
  rc = (int)launch_cluster(gemm_tokens_kernel, dim3(2 * splits, groups, tiles), dim3(kGkThreads), kGkSmemBytes, stream,
                           dim3(2 * splits, 1, 1), map_w, map_x, p);
  if (rc == 0 && launches != nullptr) ++*launches;
  return rc;
}

}  // namespace tk

// out = x * w^T for up to a few hundred tokens.  x: [tokens, k] bf16 (row stride ld_x), w: [rows, k] bf16 (row stride ld_w).
// mode 0: out is bf16 [tokens, rows]; modes 1 and 2 (rows a multiple of 128, gate and up rows of w alternating in blocks of
// 64): out is bf16 [tokens, rows / 2] = act(gate) * up with silu or the tanh form of gelu; modes 3 to 6: bf16 [tokens, rows] =
// unary_act(sum, mode - 3).  groups = 0: the plan is the function's own; otherwise that many groups of tokens and K splits,
// in one launch.  launches: null, or counted up by the kernels launched (one or two).
TK_API int tk_gemm_bf16_tokens(const void* x, const void* w, void* out, int* err, int tokens, int rows, int k,
                               long long ld_x, long long ld_w, long long ld_out, int mode, int groups, int splits,
                               int* launches, cudaStream_t stream) {
  if (tokens <= 0 || rows <= 0) return 0;
  const bool glu = mode == 1 || mode == 2;
  if (k <= 0 || k % 8 != 0 || rows % 8 != 0 || ld_out % 8 != 0 || mode < 0 || mode > 6 || (glu && rows % 128 != 0) ||
      ((uintptr_t)out & 15u) != 0 || groups < 0) {
    return (int)cudaErrorInvalidValue;
  }
  tk::GemmTokensParams p = {};
  p.out = out; p.err = err; p.tokens = tokens; p.rows = rows; p.k = k; p.ld_out = ld_out; p.mode = mode;
  const int tiles = (rows + 255) / 256;
  if (groups > 0) {
    return tk::launch_tokens(x, w, p, ld_x, ld_w, groups, tiles, splits, tk::group_width(tokens, groups), 0, launches,
                             stream);
  }
  const tk::TokensPlan plan = tk::plan_rows(tokens, rows, k);
  if (plan.groups == 0) return (int)cudaErrorInvalidValue;
  const int head = tiles - plan.tail_tiles;
  int rc = tk::launch_tokens(x, w, p, ld_x, ld_w, plan.groups, head, plan.splits, plan.width, 0, launches, stream);
  if (rc != 0) return rc;
  return tk::launch_tokens(x, w, p, ld_x, ld_w, plan.groups, plan.tail_tiles, plan.tail_splits, plan.width, head, launches,
                           stream);
}
