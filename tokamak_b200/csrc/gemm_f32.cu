// True 32-bit matrix product for the float32 path: C[M,N] = A[M,K] * W[N,K]^T.
//
// Plain FFMA accumulation, no tensor cores, no TF32.  k is cut into segments, as many as its size alone says (one below 512, from
// there one for every 256 elements begun, eight at most, all of the same number of 32-element stages, of which the last may have fewer
// left); an output element is summed over a segment in ascending order by one thread, and the
// segments' sums are added in their order.  So the value of a row of C does not depend on how many other rows are in the
// batch: a difference between two ways of cutting the same tokens into steps then points at the cache or the batch, not at
// the matrix product.  For the same reason all tiles give the same bits, and so do the two ways to take the segments: one
// block after the other, or, where that leaves SMs idle, each by a block of its own in a cluster that adds the sums up over
// distributed shared memory.
//
// The bound is the FFMA rate (a loop of nothing else reaches 58 TFLOP/s; this kernel 45 at 2,000 x 6,144 x 1,024).
// A tile of A and one of W travel by cp.async into a ring of stages, rows as they lie in memory (k contiguous): a
// thread reads four k of a row with one 16-byte load, its rows lie a tile's thread count apart, and the padded pitch
// puts eight such rows on eight different bank groups.  Per four k a thread of a TM x TN micro-tile issues TM + TN
// loads for 4 TM TN multiply-adds.  (Micro-tiles of 8 x 8 in tiles of 64 x 64, 128 x 64 and 64 x 128 were measured slower:
// 254 x 6,144 x 1,024 takes 103 us with them and 91 with 8 x 4.)
#include "common.cuh"
#include "entry_points.cuh"

namespace tk {

constexpr int kF32BK = 32;                  // k elements of a stage
constexpr int kF32Pitch = kF32BK + 4;       // floats; an odd number of 16-byte pieces
constexpr int kF32Stages = 3;

struct GemmF32Params {
  const float* A;
  const float* W;
  float* C;
  int M, N, K, lda, ldw, ldc;
  long long batch_a, batch_w, batch_c;
  int seg_blocks;           // stages of k in a segment
  int splits;               // 1, or the segments, each a block of a cluster
};

// `bytes` of 16 (or of 4) from src, the rest of the piece zero; with bytes == 0 nothing is read.
template <bool kVec>
__device__ __forceinline__ void f32_cp_async(uint32_t dst, const float* src, int bytes) {
  if (kVec) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// Segments that k is cut into: from k alone.
static int f32_segments(int k) { return k < 512 ? 1 : k >= 2048 ? 8 : (k + 255) / 256; }

// kVec: 16-byte pieces (K and the row strides multiples of 4, the matrices on 16-byte boundaries).
template <int BM, int BN, int TM, int TN, bool kVec>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), 3) gemm_f32_kernel(GemmF32Params p) {
  constexpr int kTx = BN / TN, kTy = BM / TM, kThreads = kTx * kTy;
  constexpr int kRows = BM + BN;                       // rows of a stage: A's, then W's
  constexpr int kPiece = kVec ? 4 : 1;                 // floats of a copy
  constexpr int kPerRow = kF32BK / kPiece;
  extern __shared__ __align__(16) float f32_smem[];
  pdl_trigger();
  // a warp covers 8 threads of columns by 4 of rows: its loads of a fragment name 8 and 4 different pieces
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = (lane & 7) + 8 * (warp % (kTx / 8)), ty = (lane >> 3) + 4 * (warp / (kTx / 8));
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  // grid.z counts the products of a batch (one per head, say), each with its own A, W and C, and the segments of one
  const int seg = (int)blockIdx.z % p.splits, batch = (int)blockIdx.z / p.splits;
  const float* A = p.A + (size_t)batch * p.batch_a;
  const float* W = p.W + (size_t)batch * p.batch_w;
  float* C = p.C + (size_t)batch * p.batch_c;
  const uint32_t smem_u32 = (uint32_t)__cvta_generic_to_shared(f32_smem);
  pdl_wait();

  // this thread's piece of a row, and its first row of each operand; rows of a pass further on are a fixed way off
  constexpr int kPass = kThreads / kPerRow;
  const int x = (tid % kPerRow) * kPiece, row = tid / kPerRow;
  const float* a_src = A + (size_t)(m0 + row) * p.lda + x;
  const float* w_src = W + (size_t)(n0 + row) * p.ldw + x;
  auto stage = [&](int k0, int s) {
    const uint32_t dst = smem_u32 + (uint32_t)((s * kRows + row) * kF32Pitch + x) * 4u;
    const bool k_in = k0 + x < p.K;
#pragma unroll
    for (int i = 0; i < BM / kPass; ++i) {
      const bool in = k_in && m0 + row + i * kPass < p.M;
      f32_cp_async<kVec>(dst + (uint32_t)(i * kPass * kF32Pitch) * 4u, in ? a_src + (size_t)(i * kPass) * p.lda + k0 : A,
                         in ? 4 * kPiece : 0);
    }
#pragma unroll
    for (int i = 0; i < BN / kPass; ++i) {
      const bool in = k_in && n0 + row + i * kPass < p.N;
      f32_cp_async<kVec>(dst + (uint32_t)((BM + i * kPass) * kF32Pitch) * 4u, in ? w_src + (size_t)(i * kPass) * p.ldw + k0 : W,
                         in ? 4 * kPiece : 0);
    }
  };

  float acc[TM][TN], sum[TM][TN];          // of the segment; of the segments before it
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = sum[i][j] = 0.0f;
  const int all_k = (p.K + kF32BK - 1) / kF32BK;
  const int first_k = p.splits > 1 ? seg * p.seg_blocks : 0;
  const int n_k = p.splits > 1 ? max(min(p.seg_blocks, all_k - first_k), 0) : all_k;
#pragma unroll
  for (int s = 0; s < kF32Stages - 1; ++s) {
    if (s < n_k) stage((first_k + s) * kF32BK, s);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  int in_seg = 0;
  for (int kb = 0; kb < n_k; ++kb) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kF32Stages - 2) : "memory");
    __syncthreads();                      // stage kb is there, and everybody has left stage kb - 1
    if (kb + kF32Stages - 1 < n_k) stage((first_k + kb + kF32Stages - 1) * kF32BK, (kb + kF32Stages - 1) % kF32Stages);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    if (in_seg == p.seg_blocks) {
      in_seg = 0;
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) { sum[i][j] += acc[i][j]; acc[i][j] = 0.0f; }
    }
    ++in_seg;
    const float* sa = f32_smem + (kb % kF32Stages) * kRows * kF32Pitch + ty * kF32Pitch;
    const float* sw = f32_smem + (kb % kF32Stages) * kRows * kF32Pitch + (BM + tx) * kF32Pitch;
    // Columns beyond K are zero in both operands: fmaf(0, 0, acc) leaves every sum as it is.  The next four k are
    // loaded while these are multiplied: a small product leaves each scheduler a single warp.
    float4 a[2][TM], w[2][TN];
    auto load = [&](int kk, int b) {
#pragma unroll
      for (int i = 0; i < TM; ++i) a[b][i] = *reinterpret_cast<const float4*>(sa + i * kTy * kF32Pitch + kk);
#pragma unroll
      for (int j = 0; j < TN; ++j) w[b][j] = *reinterpret_cast<const float4*>(sw + j * kTx * kF32Pitch + kk);
    };
    load(0, 0);
#pragma unroll
    for (int q = 0; q < kF32BK / 4; ++q) {
      const int b = q & 1;
      if (q + 1 < kF32BK / 4) load(4 * (q + 1), b ^ 1);
#pragma unroll
      for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) {
            const float av = x == 0 ? a[b][i].x : x == 1 ? a[b][i].y : x == 2 ? a[b][i].z : a[b][i].w;
            const float wv = x == 0 ? w[b][j].x : x == 1 ? w[b][j].y : x == 2 ? w[b][j].z : w[b][j].w;
            acc[i][j] = fmaf(av, wv, acc[i][j]);
          }
    }
  }

  if (p.splits > 1) {
    // the cluster's blocks add their segments up, a share of the rows each, in the segments' order
    constexpr int kPitch = BN + 8;
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) f32_smem[(ty + i * kTy) * kPitch + tx + j * kTx] = acc[i][j];
    cluster_sync_all();
    const bool quads = (p.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
    for (int e = tid; e < BM * BN / 4; e += kThreads) {
      const int m = e / (BN / 4), c = (e % (BN / 4)) * 4;
      if (m % p.splits != seg || m0 + m >= p.M || n0 + c >= p.N) continue;
      const float4 v = cluster_sum_f32x4(smem_u32 + (uint32_t)(m * kPitch + c) * 4u, p.splits);
      float* dst = C + (size_t)(m0 + m) * p.ldc + n0 + c;
      if (quads && n0 + c + 3 < p.N) {
        *reinterpret_cast<float4*>(dst) = v;
      } else {
        const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (n0 + c + q < p.N) dst[q] = f[q];
        }
      }
    }
    cluster_sync_all();                   // nobody reads this block's sums any more
    return;
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty + i * kTy;
    if (m >= p.M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + j * kTx;
      if (n < p.N) C[(size_t)m * p.ldc + n] = sum[i][j] + acc[i][j];
    }
  }
}

template <int BM, int BN, int TM, int TN>
int launch_gemm_f32(const GemmF32Params& p, int batch, cudaStream_t stream) {
  const dim3 grid((unsigned)((p.N + BN - 1) / BN), (unsigned)((p.M + BM - 1) / BM), (unsigned)(batch * p.splits));
  if (grid.y > 65535 || (long long)batch * p.splits > 65535) return (int)cudaErrorInvalidValue;
  const dim3 block((BM / TM) * (BN / TN));
  constexpr size_t smem = (size_t)kF32Stages * (BM + BN) * kF32Pitch * sizeof(float);
  const bool vec = ((p.K | p.lda | p.ldw | p.batch_a | p.batch_w) & 3) == 0 &&
                   (((uintptr_t)p.A | (uintptr_t)p.W) & 15) == 0;
  auto kernel = vec ? gemm_f32_kernel<BM, BN, TM, TN, true> : gemm_f32_kernel<BM, BN, TM, TN, false>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  // Not launched early: while the kernel before it runs, the few blocks of a small product would gather on the
  // SMs that happen to be free and stay there.
  if (p.splits > 1) {
    return (int)launch_cluster_when(false, kernel, grid, block, smem, stream, dim3(1, 1, (unsigned)p.splits), p);
  }
  return (int)launch_in_order(kernel, grid, block, smem, stream, p);
}

// Tile number `tile` of three, or (0) the one that the sizes ask for.  Measured (B200, us; tiles of 16 x 64, 32 x 64 and
// 64 x 64, in parentheses their blocks), M x N x K:
//   254 x 6144 x 1024: 127 (1536), 96 (768), 86 (384)      254 x 1024 x 3072: 77 (256), 63 (128), 106 (64)
//   100 x 1024 x 2048: 33 (112), 42 (64), 71 (32)           40 x 4096 x 1024: 27 (192), 22 (128), 36 (64)
//    16 x 6144 x 1024: 17 (96), 22 (96), 34 (96)            1 x 151936 x 1024: 196, 251, 447
// so: the lowest tile while it is a block an SM at most or the rows fill no other, the highest from two blocks an SM on.
// One 64 x 64 tile with 4 x 4 outputs a thread and 16 k a stage, without a ring, took 197, 192, 127, 62, 81 and 709.
static int gemm_f32_tile(int m, int n, int batch, int sms) {
  const auto blocks = [&](int bm) { return (long long)((m + bm - 1) / bm) * ((n + 63) / 64) * batch; };
  return m <= 16 || blocks(16) <= sms ? 1 : m > 32 && blocks(64) >= 2LL * sms ? 3 : 2;
}

// The tile of a product whose segments are blocks of their own: the highest that gives two and a half blocks an SM.
static int gemm_f32_split_tile(int m, int n, int batch, int segments, int sms) {
  const auto blocks = [&](int bm) { return (long long)((m + bm - 1) / bm) * ((n + 63) / 64) * batch * segments; };
  return m <= 16 ? 1 : m > 32 && 2 * blocks(64) >= 5LL * sms ? 3 : 2 * blocks(32) >= 5LL * sms ? 2 : 1;
}

// tile 0: what the sizes ask for; 1 to 3: that tile, a block walks all segments; 9 to 11: the same tiles, a block a segment.
// Segments are blocks of their own where tiles of 64 rows would be fewer than three blocks for two SMs.  Measured (B200, us,
// one block for all segments as gemm_f32_tile has it / a block a segment), M x N x K:
//   1 x 1024 x 2048 35 / 12, x 3072 51 / 15, x 4096 x 1024 20 / 15      40 x 1024 x 3072 52 / 23, x 6144 x 1024 41 / 34
//   100 x 1024 x 3072 53 / 29, x 6144 x 1024 53 / 54 (192 blocks)       150 x 4096 x 1024 53 / 52 (192), x 6144 x 1024 66 / 73 (288)
//   254 x 1024 x 2048 45 / 37, x 3072 66 / 51, x 4096 x 1024 66 / 68 (256)      800 x 1024 x 3072 148 / 145 (208), 4096 x 1024 173 / 188
static int gemm_f32(GemmF32Params p, int batch, int tile, cudaStream_t stream) {
  const int segments = f32_segments(p.K), sms = device_sm_count();
  p.seg_blocks = ((p.K + kF32BK - 1) / kF32BK + segments - 1) / segments;
  if (p.seg_blocks < 1) p.seg_blocks = 1;
  bool split = segments > 1 && tile > 8;
  if (tile == 0) {
    split = segments > 1 && 2LL * ((p.M + 63) / 64) * ((p.N + 63) / 64) * batch < 3LL * sms;
    tile = split ? gemm_f32_split_tile(p.M, p.N, batch, segments, sms) : gemm_f32_tile(p.M, p.N, batch, sms);
  } else if (tile > 8) {
    tile -= 8;
  }
  p.splits = split ? segments : 1;
  switch (tile) {
    case 1: return launch_gemm_f32<16, 64, 2, 4>(p, batch, stream);
    case 2: return launch_gemm_f32<32, 64, 4, 4>(p, batch, stream);
    case 3: return launch_gemm_f32<64, 64, 8, 4>(p, batch, stream);
    default: return (int)cudaErrorInvalidValue;
  }
}

}  // namespace tk

// The tile that sizes get on a device of so many SMs where one block takes all of k.
TK_API int tk_gemm_f32_tile(int m, int n, int batch, int sms) { return tk::gemm_f32_tile(m, n, batch, sms); }

// `batch` products of the same sizes: product b reads A + b * batch_a and W + b * batch_w and writes
// C + b * batch_c (strides in elements).  `tile`: 0, or 1 to 3 for one tile whatever the sizes, 9 to 11
// for the same tiles with a block a segment of k (the same bits).
TK_API int tk_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int batch,
                       long long batch_a, long long batch_w, long long batch_c, int tile, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || batch <= 0) return 0;
  if (K < 0 || batch > 65535) return (int)cudaErrorInvalidValue;
  const tk::GemmF32Params p = {A, W, C, M, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c, 1, 1};
  return tk::gemm_f32(p, batch, tile, stream);
}
