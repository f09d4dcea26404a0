// Attention of prompt portions over a latent cache on the 5th-generation tensor cores (see attention_latent.cu for the
// rows: all heads of a token are rows of one tile, the keys' leading DV elements are the values).
//
// A block takes 128 query rows and half of the value columns, so that their float32 sums (256 columns) and two tiles of
// scores fit tensor memory, and walks the keys 32 at a time: S = Q K^T into one of two score buffers, softmax by a thread a
// row, P written over S, O += P V with P from tensor memory and V the same shared-memory tile as K, read MN-major.
// Scores are formed by both halves (D products a key beside DV / 2).  Queries are converted to bfloat16 into shared memory
// once (128 x D, 147 KB at 576), key tiles come page by page by TMA into the two to four stages that this leaves.
//
// The output is rescaled only where a row's maximum grew by more than 2^8, so that a row's largest probability is not 1, as it
// is against its own maximum, but any number up to 256, and rounded to bfloat16 it would stay off.  So a probability is two
// bfloat16, its rounded value and what the rounding left, and O += P V a product of either: what remains of a result's error is its own
// rounding (2,000 tokens, rows of 576: 1.62e-3 of the result, as its rounding alone; 2.02e-3 with one).  It costs 0 to 3 %.
//
// Rows of a key tile that no query of the block sees (behind its last position, in front of its window) are zeroed once their scores
// are there: a page may hold anything in them.  A key that some of the block's 128 rows see and others do not must be finite, as
// must every key of a prompt.
//
// What bounds it: with N = 32 a product of scores reads 5 KB of shared memory for what takes the tensor cores 16 clocks, some
// 40 clocks each, 36 of them a tile at D = 576, and with two stages the way of a tile from L2 stands in the chain.
// B200, us, mma.sync kernel / this: 2,000 tokens of 16 heads, rows of 576 714 / 253, rows of 512 with a window of 1,024 467 / 166;
// 400 tokens 76 / 38, 64 tokens behind 8,000 1,147 / 452, 16 to 64 tokens alone 21 / 19; rows of 128 and 256 level.  With the
// products in a fixed order (S of the next tile, then P V of this one) 433, with the pairs as the grid's fastest dimension and
// four pieces of the queries on their way at a time 357.  (Before the probabilities' second half and the zeroed rows; behind a flushed
// L2 without / with these: 2,000 tokens 268 / 271 and 177 / 181, 400 tokens 46 / 48, 64 behind 8,000 501 / 505, 16 alone 24.6 / 24.6.)
//
// Every wait on an mbarrier is bounded and reports kErrWait.
#pragma once

#include "tcgen05_utils.cuh"

namespace tk {

constexpr int kLpRows = 128;
constexpr int kLpKeys = 32;
constexpr int kLpThreads = 192;        // warp 0: TMA, warp 1: MMA, warps 2..5: softmax and epilogue
constexpr int kLpMaxStages = 4;
constexpr int kLpAhead = 12;
constexpr uint32_t kLpQChunk = kLpRows * 128;      // 64 elements of the query rows
constexpr uint32_t kLpKChunk = kLpKeys * 128;      // 64 elements of a key tile
constexpr int kLpMaxSmem = 227 * 1024 - 1024 - 256;

// grid: x 128-row pieces of a pair's tokens x H rows, y halves of the value columns, z (request, 64-token tile) pairs, of which
// those with the most keys come first.
template <typename TQ>
__global__ void __launch_bounds__(kLpThreads, 1)
latent_prefill_kernel(const __grid_constant__ CUtensorMap map_k, LatentAttnParams p, int n_stages) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t raw = gt_smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* smem = smem_raw + (base - raw);
  const int D = p.D, H = p.H, chunks = D / 64;
  const uint32_t q_bytes = (uint32_t)chunks * kLpQChunk, k_bytes = (uint32_t)chunks * kLpKChunk;
  const uint32_t k_smem = base + q_bytes;
  uint64_t* k_full = reinterpret_cast<uint64_t*>(smem + q_bytes + (uint32_t)n_stages * k_bytes);
  uint64_t* k_empty = k_full + kLpMaxStages;
  uint64_t* s_full = k_empty + kLpMaxStages;
  uint64_t* p_full = s_full + 2;
  uint64_t* o_done = p_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < n_stages; ++s) {
      mbar_init(gt_smem_u32(&k_full[s]), 1);
      mbar_init(gt_smem_u32(&k_empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(gt_smem_u32(&s_full[b]), 1);
      mbar_init(gt_smem_u32(&p_full[b]), 4);
      mbar_init(gt_smem_u32(&o_done[b]), 1);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n"
                 ::"r"(gt_smem_u32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // only now may later kernels begin: none of them can take tensor memory before this block has its own
  pdl_trigger();
  pdl_wait();

  // ---- what this block works on
  const int work = blockIdx.z, r = p.tiles[2 * work], ti = p.tiles[2 * work + 1];
  int tokens = 0, kv_len = 0, q_len = 0;
  if (r < 0 || r >= p.n_reqs) {
    if (threadIdx.x == 0) set_error(p.err, kErrRequest, work, r, p.n_reqs);
  } else {
    q_len = p.req_q_len[r];
    kv_len = p.req_kv_len[r];
    tokens = min(64, q_len - ti * 64);
    if (tokens <= 0 || kv_len < q_len) {
      if (threadIdx.x == 0) set_error(p.err, kErrPosition, work, q_len, kv_len);
      tokens = 0;
    }
  }
  const int row_first = blockIdx.x * kLpRows, rows_here = min(kLpRows, tokens * H - row_first);
  if (rows_here > 0) {
    const int tok0 = p.req_q_start[r] + ti * 64, pos0 = kv_len - q_len + ti * 64;
    const int* table = p.block_table + (size_t)p.req_slot[r] * p.max_pages;
    const int pos_first = pos0 + row_first / H, pos_last = pos0 + (row_first + rows_here - 1) / H;
    const int lo_block = first_visible(pos_first, p.window, 0);
    const int first_kt = lo_block / kLpKeys, n_kt = pos_last / kLpKeys - first_kt + 1;
    const int half_cols = p.DV / 2, v_chunk0 = (int)blockIdx.y * (half_cols / 64);

    // the queries as bfloat16 rows in the swizzled layout that the products read (rows beyond the block's are zero)
    // kLpAhead pieces a thread on their way at a time
    const int pieces = D / 8;
    for (int i0 = threadIdx.x; i0 < kLpRows * pieces; i0 += kLpAhead * kLpThreads) {
      uint4 x[kLpAhead][sizeof(TQ) / 2];
#pragma unroll
      for (int u = 0; u < kLpAhead; ++u) {
        const int idx = i0 + u * kLpThreads, row = idx / pieces, c = idx - row * pieces;
        const bool in = row < rows_here;
        const int R = row_first + (in ? row : 0);
        const uint4* src = reinterpret_cast<const uint4*>((const TQ*)p.q + (size_t)(tok0 + R / H) * p.q_tok_stride +
                                                          (size_t)(R % H) * p.q_head_stride + c * 8);
#pragma unroll
        for (int e = 0; e < (int)sizeof(TQ) / 2; ++e) x[u][e] = in ? src[e] : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int u = 0; u < kLpAhead; ++u) {
        const int idx = i0 + u * kLpThreads, row = idx / pieces, c = idx - row * pieces;
        if (row >= kLpRows) continue;
        uint4 w = x[u][0];
        if (sizeof(TQ) == 4) {
          const uint4 a = x[u][0], b = x[u][sizeof(TQ) / 2 - 1];
          w = make_uint4(pack_bf16(__uint_as_float(a.x), __uint_as_float(a.y)), pack_bf16(__uint_as_float(a.z), __uint_as_float(a.w)),
                         pack_bf16(__uint_as_float(b.x), __uint_as_float(b.y)), pack_bf16(__uint_as_float(b.z), __uint_as_float(b.w)));
        }
        *reinterpret_cast<uint4*>(smem + (uint32_t)(c >> 3) * kLpQChunk + row * 128 + (((c & 7) ^ (row & 7)) << 4)) = w;
      }
    }
    fence_async_shared();
    __syncthreads();

    if (warp == 0) {
      // ---- producer: a copy is a page part (or a page) x 64 elements
      const int kpl = p.page_size < kLpKeys ? p.page_size : kLpKeys, parts = kLpKeys / kpl;
      int st = 0;
      uint32_t phase = 1;          // a fresh barrier counts as given back once
      for (int j = 0; j < n_kt; ++j) {
        if (!__all_sync(0xffffffffu, mbar_wait(gt_smem_u32(&k_empty[st]), phase, abort_flag))) {
          if (lane == 0) { set_error(p.err, kErrWait, 70, j, st); *abort_flag = 1; }
          break;
        }
        const uint32_t full = gt_smem_u32(&k_full[st]);
        if (lane == 0) mbar_expect_tx(full, k_bytes);
        __syncwarp();
        for (int i = lane; i < parts * chunks; i += 32) {
          const int u = i / chunks, c = i - u * chunks;
          int key0 = (first_kt + j) * kLpKeys + u * kpl;
          if (key0 + kpl - 1 < lo_block || key0 > pos_last) key0 = (pos_last / kpl) * kpl;       // nothing visible here
          const int pidx = key0 / p.page_size;
          int page = pidx < p.max_pages ? table[pidx] : -1;
          if (page < 0 || page >= p.num_pages) {
            set_error(p.err, kErrPage, tok0, pidx, page);
            page = 0;
          }
          tma_load_2d(k_smem + (uint32_t)st * k_bytes + (uint32_t)c * kLpKChunk + (uint32_t)(u * kpl * 128), &map_k, c * 64,
                      page * p.page_size + key0 % p.page_size, full);
        }
        if (++st == n_stages) { st = 0; phase ^= 1u; }
      }
    } else if (warp == 1) {
      // ---- MMA issuer
      if (elect_one()) {
        const uint32_t idesc_s = umma_idesc(kLpKeys, false), idesc_o = umma_idesc(half_cols, true);
        const uint64_t desc_q = umma_desc_sw128(base), desc_k = umma_desc_sw128(k_smem);
        const uint64_t desc_v = umma_desc_sw128_mn(k_smem + (uint32_t)v_chunk0 * kLpKChunk, kLpKChunk);
        const uint32_t tmem_s = tmem_base + 256u;
        // An event loop: whichever of the next tile's scores and the oldest tile's second product can go.  In a fixed
        // order the second product would wait for keys that wait for the stage it gives back.
        int st = 0, st_pv = 0, js = 0, jp = 0;          // tiles whose S, and whose O += P V, has been issued
        uint32_t phase = 0;
        unsigned idle = 0;
        while (jp < n_kt) {
          const int b = jp & 1;
          if (jp < js && mbar_test(gt_smem_u32(&p_full[b]), (uint32_t)(jp >> 1) & 1u)) {
            tc_fence_after();
            const uint64_t dv = desc_v + (uint64_t)((uint32_t)st_pv * (k_bytes >> 4));
#pragma unroll
            for (int k = 0; k < kLpKeys / 8; ++k) {          // the rounded probabilities, then what their rounding left
              umma_bf16_ts(tmem_base, tmem_s + (uint32_t)(b * kLpKeys + 8 * k),
                           dv + (uint64_t)(k % (kLpKeys / 16) * ((16 * 128) >> 4)), idesc_o, (jp > 0 || k > 0) ? 1u : 0u);
            }
            umma_commit(gt_smem_u32(&k_empty[st_pv]));
            umma_commit(gt_smem_u32(&o_done[b]));
            if (++st_pv == n_stages) st_pv = 0;
            ++jp;
            idle = 0;
          } else if (js < n_kt && js - jp < 2 && mbar_test(gt_smem_u32(&k_full[st]), phase)) {
            // the score buffer held the probabilities of two tiles before, whose second product has been issued
            tc_fence_after();
            const uint64_t dk = desc_k + (uint64_t)((uint32_t)st * (k_bytes >> 4));
            for (int c = 0; c < chunks; ++c) {
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                umma_bf16(tmem_s + (uint32_t)((js & 1) * kLpKeys), desc_q + (uint64_t)(c * (kLpQChunk >> 4) + 2 * k),
                          dk + (uint64_t)(c * (kLpKChunk >> 4) + 2 * k), idesc_s, (c > 0 || k > 0) ? 1u : 0u);
              }
            }
            umma_commit(gt_smem_u32(&s_full[js & 1]));
            if (++st == n_stages) { st = 0; phase ^= 1u; }
            ++js;
            idle = 0;
          } else if (++idle >= kGtSpinLimit || ((idle & 1023u) == 1023u && *abort_flag)) {
            if (idle >= kGtSpinLimit) {
              set_error(p.err, kErrWait, 71, js, jp);
              *abort_flag = 1;
            }
            break;
          }
        }
      }
      __syncwarp();
    } else {
      // ---- softmax and epilogue: row = lane of tensor memory
      const int quarter = warp & 3, row = quarter * 32 + lane, R = row_first + row;
      const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
      const uint32_t tmem_s = tmem_base + lane_addr + 256u, tmem_o = tmem_base + lane_addr;
      const bool live = row < rows_here;
      const int pos = live ? pos0 + R / H : -1, head = R % H, lo = live ? first_visible(pos, p.window, 0) : 0;
      float m_ref = -INFINITY, l = 0.0f;
      if (live && p.sinks != nullptr) { m_ref = p.sinks[head] * 1.4426950408889634f; l = 1.0f; }
      bool ok = true;
      int st = 0;                  // the stage that the tile lies in
      for (int j = 0; j < n_kt; ++j) {
        const int b = j & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(gt_smem_u32(&s_full[b]), (uint32_t)(j >> 1) & 1u, abort_flag));
        if (!ok) { if (lane == 0) { set_error(p.err, kErrWait, 73, j, quarter); *abort_flag = 1; } break; }
        tc_fence_after();
        uint32_t s[kLpKeys];
        tmem_ld32(tmem_s + (uint32_t)(b * kLpKeys), s);
        tmem_wait_ld();
        const int key0 = (first_kt + j) * kLpKeys;
        float x[kLpKeys], mx = -INFINITY;
        if (__all_sync(0xffffffffu, live && key0 >= lo && key0 + kLpKeys - 1 <= pos)) {
#pragma unroll
          for (int c = 0; c < kLpKeys; ++c) { x[c] = __uint_as_float(s[c]) * p.scale_log2; mx = fmaxf(mx, x[c]); }
        } else {
#pragma unroll
          for (int c = 0; c < kLpKeys; ++c) {
            x[c] = key0 + c <= pos && key0 + c >= lo ? __uint_as_float(s[c]) * p.scale_log2 : -INFINITY;
            mx = fmaxf(mx, x[c]);
          }
        }
        // a row's reference is moved only where its maximum grew by more than 2^8 (or where it has none yet)
        const bool grow = mx > m_ref + 8.0f;
        if (__any_sync(0xffffffffu, grow)) {
          const float m_new = grow ? mx : m_ref;
          // 0 where the row had no reference: a sink of -inf (or one that far down) is no term of the denominator
          const float f = grow ? exp2f(m_ref - m_new) : 1.0f;
          const bool summed = grow && m_ref != -INFINITY;      // without a reference there are no sums to rescale yet
          m_ref = m_new;
          l *= f;
          if (j > 0 && __any_sync(0xffffffffu, summed)) {
            const int i = j - 1;
            ok = __all_sync(0xffffffffu, mbar_wait(gt_smem_u32(&o_done[i & 1]), (uint32_t)(i >> 1) & 1u, abort_flag));
            if (!ok) { if (lane == 0) { set_error(p.err, kErrWait, 74, j, quarter); *abort_flag = 1; } break; }
            tc_fence_after();
            for (int c0 = 0; c0 < half_cols; c0 += 32) {
              uint32_t o[32];
              tmem_ld32(tmem_o + (uint32_t)c0, o);
              tmem_wait_ld();
#pragma unroll
              for (int c = 0; c < 32; ++c) o[c] = __float_as_uint(__uint_as_float(o[c]) * f);
              tmem_st32(tmem_o + (uint32_t)c0, o);
            }
            tmem_wait_st();
          }
        }
        const float m_use = m_ref == -INFINITY ? 0.0f : m_ref;
        // A probability as two bfloat16, the rounded value and what the rounding left: words 0..15 and 16..31.
        uint32_t packed[kLpKeys];
        float sum = 0.0f;
#pragma unroll
        for (int c = 0; c < kLpKeys; c += 2) {
          const float p0 = exp2f(x[c] - m_use), p1 = exp2f(x[c + 1] - m_use);
          const uint32_t hi = pack_bf16(p0, p1);
          packed[c / 2] = hi;
          packed[(kLpKeys + c) / 2] = pack_bf16(p0 - __uint_as_float(hi << 16), p1 - __uint_as_float(hi & 0xffff0000u));
          sum += p0 + p1;
        }
        l += sum;
        tmem_st32(tmem_s + (uint32_t)(b * kLpKeys), packed);
        if (key0 < lo_block || key0 + kLpKeys - 1 > pos_last) {
          // Rows that no query of the block sees become zeros as values (their scores are masked): a page may hold anything
          // there, and a probability of 0 does not undo an infinity or a NaN.
          unsigned char* tile = smem + q_bytes + (uint32_t)st * k_bytes + (uint32_t)v_chunk0 * kLpKChunk;
          for (int i = threadIdx.x - 64; i < kLpKeys * (half_cols / 8); i += kLpThreads - 64) {
            const int x = (i >> 3) % kLpKeys, c = (i >> 3) / kLpKeys;
            if (key0 + x >= lo_block && key0 + x <= pos_last) continue;
            *reinterpret_cast<uint4*>(tile + (uint32_t)c * kLpKChunk + x * 128 + (i & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
          }
          fence_async_shared();
        }
        if (++st == n_stages) st = 0;
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(gt_smem_u32(&p_full[b]));
      }
      if (ok) {
        const int i = n_kt - 1;
        ok = __all_sync(0xffffffffu, mbar_wait(gt_smem_u32(&o_done[i & 1]), (uint32_t)(i >> 1) & 1u, abort_flag));
        if (!ok && lane == 0) { set_error(p.err, kErrWait, 75, i, quarter); *abort_flag = 1; }
      }
      if (ok) {
        tc_fence_after();
        const float inv = live ? 1.0f / l : 0.0f;
        __nv_bfloat16* dst = p.out + ((size_t)(tok0 + R / H) * H + head) * p.DV + v_chunk0 * 64;
        for (int c0 = 0; c0 < half_cols; c0 += 32) {
          uint32_t o[32];
          tmem_ld32(tmem_o + (uint32_t)c0, o);
          tmem_wait_ld();
          if (live) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint4 v;
              uint32_t* w = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                w[e] = pack_bf16(__uint_as_float(o[q * 8 + 2 * e]) * inv, __uint_as_float(o[q * 8 + 2 * e + 1]) * inv);
              }
              *reinterpret_cast<uint4*>(dst + c0 + q * 8) = v;
            }
          }
        }
      }
      tc_fence_before();
    }
  }
  __syncthreads();
  tc_fence_after();
  if (warp == 2) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

// Whether the kernel takes these sizes: whole 64-element pieces of rows and of either half of the values, whole page parts in a
// tile of 32 keys, queries in 16-byte pieces, no more work items than a grid has planes.
static bool latent_prefill_takes(const LatentAttnParams& p, int q_size) {
  const bool pages = p.page_size == 8 || p.page_size == 16 || (p.page_size >= 32 && p.page_size % 32 == 0);
  return p.n_work <= 65535 && p.D % 64 == 0 && p.DV % 128 == 0 && p.DV <= 512 && p.D <= 576 && pages && ((uintptr_t)p.q & 15) == 0 &&
         ((uintptr_t)p.cache & 15) == 0 && ((uintptr_t)p.out & 15) == 0 && (p.q_tok_stride * q_size) % 16 == 0 &&
         (p.q_head_stride * q_size) % 16 == 0;
}

template <typename TQ>
static cudaError_t launch_latent_prefill(const LatentAttnParams& p, cudaStream_t stream) {
  const int chunks = p.D / 64;
  int stages = (kLpMaxSmem - chunks * (int)kLpQChunk) / (chunks * (int)kLpKChunk);
  if (stages > kLpMaxStages) stages = kLpMaxStages;
  const size_t smem = (size_t)chunks * kLpQChunk + (size_t)stages * chunks * kLpKChunk + 1024 /* alignment */ + 256 /* barriers */;
  static bool configured[64] = {false};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    e = cudaFuncSetAttribute(latent_prefill_kernel<TQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  CUtensorMap map_k;
  const cuuint64_t dims[2] = {(cuuint64_t)p.D, (cuuint64_t)p.num_pages * (cuuint64_t)p.page_size};
  const cuuint64_t strides[1] = {(cuuint64_t)p.D * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)(p.page_size < kLpKeys ? p.page_size : kLpKeys)};
  if (make_bf16_map(&map_k, p.cache, 2, dims, strides, box) != 0) return cudaErrorInvalidValue;
  const dim3 grid((unsigned)((64 * p.H + kLpRows - 1) / kLpRows), 2, (unsigned)p.n_work);
  return launch(latent_prefill_kernel<TQ>, grid, dim3(kLpThreads), smem, stream, map_k, p, stages);
}

}  // namespace tk
