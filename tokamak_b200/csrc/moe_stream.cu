// The experts' products in steps of few tokens (bfloat16) on the 5th-generation tensor cores.
//
//   D[t, n] = sum_k X[t, k] * W_e[n, k]     for every expert e that some token of the step chose
//
// The bound is the stream of the chosen experts' weights from memory, each byte once.  So, as in gemm_tcgen05.cu, a
// weight is the 128-row operand of the MMA and the step's tokens (at most 64) are its N side: a block takes one
// (128-row tile of an expert, K split), the splits of a tile form a cluster that adds the partial sums up over
// distributed shared memory.  All tokens are multiplied with every chosen expert (the tensor cores
// have nothing else to do) and the columns of tokens that did not choose it are not stored; a column's sum does not
// depend on the others.  Nor does it depend on the number of splits, which follows from the tokens of the step: k is cut
// into as many segments as its size alone says, each has sums of its own in tensor memory, and the segments' sums are
// added as a binary tree whose lower levels lie in a block and whose upper levels lie in the cluster.  Which experts
// those are is read on the device by every block for itself from the router's choice: the n-th block row takes the n-th
// chosen expert in ascending order, and leaves at once where there is none.
//
// The first product stores act(gate) * up or act(up) as bfloat16 rows of the (token, choice) pairs, expert by expert,
// in the order of the tokens; the second one takes an expert's stretch of these rows as its N side and stores
// every pair's float32 sums or, for a reader of partial sums, its share of the weighted sum.  Nothing else (no sorting
// kernel, no gathered or padded rows) is needed.
//
// Measured at 8 experts of 4,096 x 2,048, two a token (B200, both products and the weighted sum, us; in parentheses the
// experts chosen and the time of their bytes at 6.54 TB/s), beside the grouped product on pairs of SMs over rows
// padded to 256 an expert (and its gathering kernel) and beside moe_small_kernel on the CUDA cores:
//   1 token (2, 15.4): 25.3 / 70.8 / 31.0      4 tokens (4, 30.8): 43.4 / 99.3 / 66.7
//   8 tokens (7, 53.9): 76.0 / 156 / 144      64 tokens (8, 61.6): 94 / 162
// One sum over all of k instead of the segments' tree, with splits that changed the bits: the same to 32 tokens, 88 at 64.
// From the float64 result 1.7e-3 (relative, 2-norm) like moe_small_kernel, against 2.3e-3 on pairs of SMs, which
// rounds the second product's rows to bfloat16.
#include "tcgen05_utils.cuh"

namespace tk {

constexpr int kMsBM = 128;            // weight rows of a block = UMMA M
constexpr int kMsBK = 64;             // k elements of a stage = one 128-byte swizzle span
constexpr int kMsThreads = 192;       // warp 0: TMA, warp 1: MMA, warps 2..5: epilogue
constexpr int kMsMaxTokens = 64;
constexpr int kMsMaxPairs = 1024;
constexpr int kMsMaxExperts = 1024;

enum MsMode : int { kMsSums = 0, kMsUnary = 1, kMsGated = 2 };      // as MoeProduct in moe.cu

struct MoeStreamParams {
  const int* chosen;      // [n_tokens, per]: expert of every pair, -1 for none; a token names an expert once at most
  void* out;              // kMsSums: float [pairs, n_rows]; else bf16 [pairs in the order of their experts, n_out]
  const float* weights;   // kMsSums: null, or [n_tokens, per]: out is float [per, n_tokens, n_rows], sums times weight
  int* err;
  int n_tokens, per, experts;
  int n_rows;             // weight rows of an expert (gated: 2 n_out, in blocks of 64 gate and 64 up rows in turn)
  int k, n_stages, n_splits, mode, act;
  int per_block;          // segments of k that a block takes: 1, 2 or 4
  int seg_kb;             // k blocks of a segment
  int choice_is_there;    // the kernel in front is the first product of the same choice
};

// The sum over the cluster's n (1, 2, 4, 8) blocks of the four floats at one shared-memory address of each, as a binary tree.
__device__ __forceinline__ float4 ms_cluster_tree(uint32_t addr, int n) {
  float4 v[8];
#pragma unroll
  for (int rk = 0; rk < 8; ++rk) {
    if (rk < n) v[rk] = ld_cluster_f32x4(addr, (uint32_t)rk);
  }
#pragma unroll
  for (int w = 1; w < 8; w <<= 1) {
#pragma unroll
    for (int rk = 0; rk + w < 8; rk += 2 * w) {
      if (rk + w < n) { v[rk].x += v[rk + w].x; v[rk].y += v[rk + w].y; v[rk].z += v[rk + w].z; v[rk].w += v[rk + w].w; }
    }
  }
  return v[0];
}

__device__ __forceinline__ void ms_add16(uint32_t (&a)[16], const uint32_t (&b)[16]) {
#pragma unroll
  for (int e = 0; e < 16; ++e) a[e] = __float_as_uint(__uint_as_float(a[e]) + __uint_as_float(b[e]));
}

// BN: columns of the N side, 16, 32 or 64.  A block of four segments has an accumulator each, or at 64 columns two that it
// uses twice (four would leave an SM room for two blocks instead of three: 64 tokens 88 -> 98 us at the case above): the
// sum of the first two segments waits in registers, and the products with the third begin once it is there.
template <int BN>
__global__ void __launch_bounds__(kMsThreads, BN == 64 ? 3 : 4)
moe_stream_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, MoeStreamParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ unsigned bits_s[kMsMaxExperts / 32];
  __shared__ short pair_of_s[kMsMaxTokens];       // the expert's pairs, in the order of their tokens
  __shared__ int expert_s, before_s, count_s;
  const uint32_t raw = gt_smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* smem = smem_raw + (base - raw);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x, rank = blockIdx.y, split = blockIdx.z;
  const uint32_t w_bytes = kMsBM * kMsBK * 2;
  constexpr uint32_t x_bytes = (uint32_t)BN * kMsBK * 2;
  const bool two_rounds = BN == 64 && p.per_block == 4;
  const uint32_t stage_bytes = w_bytes + ((x_bytes + 1023u) & ~1023u);
  const uint32_t tmem_cols = max(32u, (uint32_t)(BN * (two_rounds ? 2 : p.per_block)));      // a power of two, 128 at most
  unsigned char* ctrl = smem + (size_t)p.n_stages * stage_bytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(ctrl);
  uint64_t* empty_bar = full_bar + p.n_stages;
  uint64_t* accum_bar = empty_bar + p.n_stages;
  uint64_t* half_bar = accum_bar + 1;           // two rounds: the first two segments are complete, and have been read
  uint64_t* read_bar = half_bar + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(read_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.n_stages; ++s) {
      mbar_init(gt_smem_u32(&full_bar[s]), 1);
      mbar_init(gt_smem_u32(&empty_bar[s]), 1);
    }
    mbar_init(gt_smem_u32(accum_bar), 1);
    mbar_init(gt_smem_u32(half_bar), 1);
    mbar_init(gt_smem_u32(read_bar), 4);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n"
                 ::"r"(gt_smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (threadIdx.x < kMsMaxExperts / 32) bits_s[threadIdx.x] = 0u;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // Only now may later kernels begin: none of them can take tensor memory before this block has its own, and the second
  // product reads the router's choice before it waits for the first: a block of the first lets it begin only once the
  // router is through.
  if (!p.choice_is_there) pdl_wait();
  pdl_trigger();

  // ---- the expert of this block, and where its pairs lie ---------------------------------------
  const int pairs = p.n_tokens * p.per;
  for (int i = threadIdx.x; i < pairs; i += kMsThreads) {
    const int e = __ldcg(p.chosen + i);        // (not through L1: the choice may be read before the wait)
    if (e >= 0 && e < p.experts) atomicOr(&bits_s[e >> 5], 1u << (e & 31));
  }
  __syncthreads();
  if (warp == 0) {
    unsigned word = bits_s[lane];
    const int c = __popc(word);
    int upto = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += up;
    }
    int nth = rank - (upto - c);              // of this lane's experts, if it is among them
    const bool here = nth >= 0 && nth < c;
    if (lane == 31 && upto <= rank) expert_s = -1;
    if (here) {
      for (; nth > 0; --nth) word &= word - 1u;
      expert_s = lane * 32 + __ffs(word) - 1;
    }
    __syncwarp();
    const int e = expert_s;
    int count = 0, before = 0;
    for (int i0 = 0; i0 < pairs && e >= 0; i0 += 32) {
      const int other = i0 + lane < pairs ? __ldcg(p.chosen + i0 + lane) : -1;
      const unsigned mine = __ballot_sync(0xffffffffu, other == e);
      before += __popc(__ballot_sync(0xffffffffu, other >= 0 && other < e));
      if (other == e) {
        const int place = count + __popc(mine & ((1u << lane) - 1u));
        if (place < kMsMaxTokens) pair_of_s[place] = (short)(i0 + lane);
      }
      count += __popc(mine);
    }
    if (lane == 0) { before_s = before; count_s = count; }
  }
  __syncthreads();
  const int expert = expert_s;
  if (expert < 0) {                           // the whole cluster leaves: its blocks share the rank
    if (p.choice_is_there) pdl_wait();
    if (warp == 2) {
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    }
    return;
  }
  const int before = before_s;

  const int kb_total = (p.k + kMsBK - 1) / kMsBK;
  const int kb_per = p.per_block * p.seg_kb;
  const int kb_begin = split * kb_per;
  const int n_kb = max(min(kb_begin + kb_per, kb_total) - kb_begin, 0);
  const int w_row = expert * p.n_rows + tile * kMsBM;
  const int x_row = p.mode == kMsSums ? before : 0;

  const auto load_w = [&](int i, int s) {
    const uint32_t full = gt_smem_u32(&full_bar[s]);
    mbar_expect_tx(full, w_bytes + x_bytes);
    tma_load_2d(base + (uint32_t)s * stage_bytes, &map_w, (kb_begin + i) * kMsBK, w_row, full);
  };
  const auto load_x = [&](int i, int s) {
    tma_load_2d(base + (uint32_t)s * stage_bytes + w_bytes, &map_x, (kb_begin + i) * kMsBK, x_row, gt_smem_u32(&full_bar[s]));
  };
  const int first = min(n_kb, p.n_stages);

  if (warp == 0 && elect_one()) {
    // ---- TMA producer ---------------------------------------------------------------------
    // the first ring's weights, which no kernel writes, then (where that was not waited for) the rows of the first product
    for (int i = 0; i < first; ++i) load_w(i, i);
    if (p.choice_is_there) pdl_wait();
    for (int i = 0; i < first; ++i) load_x(i, i);
    int s = 0;                                // the ring's stage and its phase
    uint32_t phase = 0;
    for (int i = first; i < n_kb; ++i) {
      if (!mbar_wait(gt_smem_u32(&empty_bar[s]), phase, abort_flag)) {
        set_error(p.err, kErrWait, 0, i, s);
        *abort_flag = 1;
        break;
      }
      load_w(i, s);
      load_x(i, s);
      if (++s == p.n_stages) { s = 0; phase ^= 1u; }
    }
  }
  if (warp == 1 && elect_one()) {
    // ---- MMA issuer -----------------------------------------------------------------------
    const uint32_t idesc = umma_idesc_bf16(BN);
    bool ok = true;
    uint32_t acc = tmem_base;
    int s = 0;
    uint32_t phase = 0;
    for (int i = 0, in_seg = 0; i < n_kb; ++i) {
      if (two_rounds && i == 2 * p.seg_kb) {
        umma_commit(gt_smem_u32(half_bar));
        if (!mbar_wait(gt_smem_u32(read_bar), 0u, abort_flag)) {
          set_error(p.err, kErrWait, 3, i, s);
          *abort_flag = 1;
          ok = false;
          break;
        }
        acc = tmem_base;
      }
      if (!mbar_wait(gt_smem_u32(&full_bar[s]), phase, abort_flag)) {
        set_error(p.err, kErrWait, 1, i, s);
        *abort_flag = 1;
        ok = false;
        break;
      }
      tc_fence_after();
      const uint32_t w_addr = base + (uint32_t)s * stage_bytes;
      const uint64_t desc_w = umma_desc_sw128(w_addr), desc_x = umma_desc_sw128(w_addr + w_bytes);
#pragma unroll
      for (int k = 0; k < kMsBK / 16; ++k) {
        umma_bf16(acc, desc_w + (uint64_t)(2 * k), desc_x + (uint64_t)(2 * k), idesc, (in_seg > 0 || k > 0) ? 1u : 0u);
      }
      if (++in_seg == p.seg_kb) { in_seg = 0; acc += (uint32_t)BN; }
      umma_commit(gt_smem_u32(&empty_bar[s]));
      if (++s == p.n_stages) { s = 0; phase ^= 1u; }
    }
    if (ok) umma_commit(gt_smem_u32(accum_bar));
  }
  if (warp >= 2) {
    if (p.choice_is_there) pdl_wait();        // nothing is stored before the kernels in front are done with the output
    // ---- accumulator -> shared memory, [column][row of the tile] ----------------------------------
    const int quarter = warp & 3;
    bool ok = n_kb > 0;
    const uint32_t acc = tmem_base + ((uint32_t)(quarter * 32) << 16);
    float* stage = reinterpret_cast<float*>(smem) + quarter * 32 + lane;
    uint32_t half[BN == 64 ? BN : 16];            // (the narrow forms never touch theirs)
    if (BN == 64 && two_rounds && ok) {
      ok = mbar_wait(gt_smem_u32(half_bar), 0u, abort_flag);
      if (!ok && lane == 0) { set_error(p.err, kErrWait, 4, 0, 0); *abort_flag = 1; }
      tc_fence_after();
      if (ok) {
#pragma unroll
        for (int c0 = 0; c0 < BN; c0 += 16) {
          uint32_t v[16], u[16];
          tmem_ld16(acc + (uint32_t)c0, v);
          tmem_ld16(acc + (uint32_t)(BN + c0), u);
          tmem_wait_ld();
          ms_add16(v, u);
#pragma unroll
          for (int e = 0; e < 16; ++e) half[BN == 64 ? c0 + e : e] = v[e];
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(gt_smem_u32(read_bar));
    }
    if (ok) {
      ok = mbar_wait(gt_smem_u32(accum_bar), 0u, abort_flag);
      if (!ok && lane == 0) { set_error(p.err, kErrWait, 2, 0, 0); *abort_flag = 1; }
    }
    tc_fence_after();
#pragma unroll
    for (int c0 = 0; c0 < BN; c0 += 16) {
      uint32_t v[16];
      if (ok) {
        tmem_ld16(acc + (uint32_t)c0, v);
        if (p.per_block > 1) {            // every segment holds k blocks then
          uint32_t u[16];
          tmem_ld16(acc + (uint32_t)(BN + c0), u);
          tmem_wait_ld();
          ms_add16(v, u);
          if (BN < 64 && p.per_block > 2) {
            uint32_t t[16];
            tmem_ld16(acc + (uint32_t)(2 * BN + c0), t);
            tmem_ld16(acc + (uint32_t)(3 * BN + c0), u);
            tmem_wait_ld();
            ms_add16(t, u);
            ms_add16(v, t);
          }
          if (BN == 64 && two_rounds) {
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              v[e] = __float_as_uint(__uint_as_float(half[BN == 64 ? c0 + e : e]) + __uint_as_float(v[e]));
            }
          }
        } else {
          tmem_wait_ld();
        }
      } else {
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = 0u;
      }
#pragma unroll
      for (int e = 0; e < 16; ++e) stage[(c0 + e) * kMsBM] = __uint_as_float(v[e]);
    }
    tc_fence_before();
  }
  cluster_sync_all();                         // every split has staged its sums
  if (warp >= 2) {
    // pair i of the expert belongs to block i mod splits of the cluster; a warp adds up one column at a time
    const uint32_t my_rank = p.n_splits > 1 ? cluster_ctarank() : 0u;
    const int mine = min(count_s, p.n_tokens);
    for (int i = (int)my_rank + p.n_splits * (warp - 2); i < mine; i += 4 * p.n_splits) {
      const int pair = pair_of_s[i], c = p.mode == kMsSums ? i : pair / p.per;
      const float4 v = ms_cluster_tree(base + (uint32_t)((c * kMsBM + 4 * lane) * 4), p.n_splits);
      if (p.mode == kMsGated) {
        // lanes 0..15 hold the gates of the tile's 64 outputs, lanes 16..31 the ups
        float4 u;
        u.x = __shfl_xor_sync(0xffffffffu, v.x, 16); u.y = __shfl_xor_sync(0xffffffffu, v.y, 16);
        u.z = __shfl_xor_sync(0xffffffffu, v.z, 16); u.w = __shfl_xor_sync(0xffffffffu, v.w, 16);
        if (lane < 16) {
          uint2 packed;
          *reinterpret_cast<__nv_bfloat162*>(&packed.x) =
              __floats2bfloat162_rn(glu_act(v.x, p.act) * u.x, glu_act(v.y, p.act) * u.y);
          *reinterpret_cast<__nv_bfloat162*>(&packed.y) =
              __floats2bfloat162_rn(glu_act(v.z, p.act) * u.z, glu_act(v.w, p.act) * u.w);
          *reinterpret_cast<uint2*>((__nv_bfloat16*)p.out + (size_t)(before + i) * (p.n_rows >> 1) + tile * 64 + 4 * lane) = packed;
        }
        continue;
      }
      const int row = tile * kMsBM + 4 * lane;          // rows are a multiple of 8: all four exist or none
      if (row >= p.n_rows) continue;
      if (p.mode == kMsUnary) {
        uint2 packed;
        *reinterpret_cast<__nv_bfloat162*>(&packed.x) = __floats2bfloat162_rn(unary_act(v.x, p.act), unary_act(v.y, p.act));
        *reinterpret_cast<__nv_bfloat162*>(&packed.y) = __floats2bfloat162_rn(unary_act(v.z, p.act), unary_act(v.w, p.act));
        *reinterpret_cast<uint2*>((__nv_bfloat16*)p.out + (size_t)(before + i) * p.n_rows + row) = packed;
      } else {
        size_t at = pair;
        float4 x = v;
        if (p.weights != nullptr) {           // a token's choices lie one array each: the reader of partial sums adds them up
          const float g = p.weights[pair];
          at = (size_t)(pair % p.per) * p.n_tokens + pair / p.per;
          x = g != 0.0f ? make_float4(g * v.x, g * v.y, g * v.z, g * v.w) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        *reinterpret_cast<float4*>((float*)p.out + at * p.n_rows + row) = x;
      }
    }
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  if (warp == 2) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n"
                 ::"r"(tmem_base), "r"(tmem_cols) : "memory");
  }
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");     // nobody reads this block's sums any more
}

// Segments of k whose sums are added as a tree: from k alone, four k blocks at least to a segment, and eight of them from k
// 4,096 on, where steps of one or two tokens want eight splits and large ones still give every SM work with two.  Steps of
// Tarivik, eight layers, with four segments there / with eight (tokens/s): experts of 4,096 x 2,048, one request 1,148 /
// 1,210, eight 7,321 / 7,324; of 6,144 x 4,096, one 700 / 700, eight 3,693 / 3,908.
static int moe_stream_segments(int kb_total) { return kb_total >= 64 ? 8 : kb_total >= 16 ? 4 : kb_total >= 8 ? 2 : 1; }

// K splits of a product: until the experts that the step is expected to choose (all choices alike) give 200 blocks, one
// segment at least for a block.  They change no bit of the result.
// Measured, us for both products with (first, second) splits, at 8 experts of 4,096 x 2,048, two a token: 1 token (2 experts)
// 47.7 (1, 1), 31.0 (1, 4), 32.5 (2, 2), 27.5 (2, 4); 2 tokens (4) 54.9 (1, 1), 44.3 (1, 2), 46.9 (2, 4); 8 tokens (6)
// 67.3 (1, 1), 56.6 (1, 2), 54.4 (1, 4), 63.8 (4, 4); at 64 of 1,408 x 2,048, six a token: 1 token (6) 33.2 (1, 1), 26.7
// (2, 4); 8 tokens (32) 100 (1, 1), 119 (2, 4).  More blocks than the SMs have room for only cost their starts.
static int moe_stream_splits(int n_tokens, int per, int experts, int tiles, int segments) {
  double missed = 1.0;
  for (int i = 0; i < n_tokens; ++i) missed *= 1.0 - (double)(per < experts ? per : experts) / experts;
  const double live = experts * (1.0 - missed);
  int splits = segments > 4 ? segments / 4 : 1;      // a block takes four segments at most
  while (splits < segments && live * tiles * splits < 200) splits *= 2;
  return splits;
}

template <int BN>
static cudaError_t launch_moe_stream(dim3 grid, size_t smem, cudaStream_t stream, const CUtensorMap& map_w,
                                     const CUtensorMap& map_x, const MoeStreamParams& p) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(moe_stream_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    configured = true;
  }
  return launch_cluster_z(moe_stream_kernel<BN>, grid, dim3(kMsThreads), smem, stream, (unsigned)p.n_splits, map_w, map_x, p);
}

}  // namespace tk

TK_API int tk_moe_stream_max_tokens() { return tk::kMsMaxTokens; }

// One product of the experts that the step's tokens chose.  w: [experts, n_rows, k] bfloat16.  mode kMsGated (w's rows
// are gate and up rows in turn, 64 at a time) and kMsUnary: x [n_tokens, k], out bf16 [pairs, n_rows / 2] or [pairs,
// n_rows], row by row in the order of the experts and, within one, of the tokens; kMsSums: x is such rows, out float32
// [pairs, n_rows] in the order of the pairs, or with weights [n_tokens, per] float32 [per, n_tokens, n_rows], the pairs'
// sums times their weights (every pair must have an expert).  n_splits: 0, or 1, 2, 4, 8 (the same bits up to the
// segments that k is cut into, 8 at most; a block takes four of them at most, so that 1 may become 2).  choice_is_there: the
// call before this one on the stream was the first product of the same choice, so that its experts' weights can be on their
// way before that product is through (8 tokens at the sizes above: the second product ends 20.3 us behind the first instead of 23.0).
TK_API int tk_moe_stream(const void* x, long long x_stride, const void* w, void* out, const int* chosen,
                         const float* weights, int* err, int n_tokens, int per, int experts, int n_rows, int k, int act,
                         int mode, int n_splits, int choice_is_there, cudaStream_t stream) {
  if (n_tokens <= 0 || per <= 0) return 0;
  const int pairs = n_tokens * per;
  if (n_tokens > tk::kMsMaxTokens || pairs > tk::kMsMaxPairs || experts < 1 || experts > tk::kMsMaxExperts || k < 8 ||
      k % 8 || n_rows < 8 || n_rows % 8 || mode < 0 || mode > 2 || (mode == tk::kMsGated && n_rows % 128) ||
      (weights != nullptr && mode != tk::kMsSums) ||
      (long long)experts * n_rows > 0x7fffffffLL || x_stride % 8) {
    return (int)cudaErrorInvalidValue;
  }
  const int bn = n_tokens <= 16 ? 16 : n_tokens <= 32 ? 32 : 64;
  const int tiles = (n_rows + tk::kMsBM - 1) / tk::kMsBM, kb_total = (k + tk::kMsBK - 1) / tk::kMsBK;
  int segments = tk::moe_stream_segments(kb_total);
  if (n_splits == 0) n_splits = tk::moe_stream_splits(n_tokens, per, experts, tiles, segments);
  if (n_splits != 1 && n_splits != 2 && n_splits != 4 && n_splits != 8) return (int)cudaErrorInvalidValue;
  if (segments < n_splits) segments = n_splits;
  if (segments > 4 * n_splits) n_splits = segments / 4;
  CUtensorMap map_w, map_x;
  const cuuint64_t w_dims[2] = {(cuuint64_t)k, (cuuint64_t)experts * (cuuint64_t)n_rows}, w_strides[1] = {(cuuint64_t)k * 2};
  const cuuint64_t x_dims[2] = {(cuuint64_t)k, (cuuint64_t)(mode == tk::kMsSums ? pairs : n_tokens)};
  const cuuint64_t x_strides[1] = {(cuuint64_t)x_stride * 2};
  const cuuint32_t w_box[2] = {tk::kMsBK, tk::kMsBM}, x_box[2] = {tk::kMsBK, (cuuint32_t)bn};
  int rc = tk::make_bf16_map(&map_w, w, 2, w_dims, w_strides, w_box);
  if (rc == 0) rc = tk::make_bf16_map(&map_x, x, 2, x_dims, x_strides, x_box);
  if (rc != 0) return rc;
  const unsigned stage_bytes = tk::kMsBM * tk::kMsBK * 2 + (((unsigned)bn * tk::kMsBK * 2 + 1023u) & ~1023u);
  // three stages let four blocks share an SM; the sums of a tile are staged in the same place
  int n_stages = 3;
  if ((unsigned)bn * tk::kMsBM * 4 > n_stages * stage_bytes) return (int)cudaErrorInvalidValue;
  const size_t smem = (size_t)n_stages * stage_bytes + 1024 + 256;
  tk::MoeStreamParams p;
  p.chosen = chosen; p.out = out; p.weights = weights; p.err = err; p.n_tokens = n_tokens; p.per = per;
  p.experts = experts; p.n_rows = n_rows; p.k = k; p.n_stages = n_stages; p.n_splits = n_splits; p.mode = mode; p.act = act;
  p.choice_is_there = choice_is_there != 0 ? 1 : 0;
  p.per_block = segments / n_splits; p.seg_kb = (kb_total + segments - 1) / segments;
  const dim3 grid((unsigned)tiles, (unsigned)(pairs < experts ? pairs : experts), (unsigned)n_splits);
  return (int)(bn == 16 ? tk::launch_moe_stream<16>(grid, smem, stream, map_w, map_x, p)
               : bn == 32 ? tk::launch_moe_stream<32>(grid, smem, stream, map_w, map_x, p)
                          : tk::launch_moe_stream<64>(grid, smem, stream, map_w, map_x, p));
}
