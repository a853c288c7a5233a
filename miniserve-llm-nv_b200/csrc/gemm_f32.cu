// True float32 matrix product for the 32-bit path: C[M, N] = A[M, K] * W[N, K]^T with
// both operands stored K-major, as activations and `[out, in]` weights are.  Plain FFMA
// on the CUDA cores: no tensor cores and no reduced-precision mode, so a fault that
// bfloat16 rounding would hide shows up.  (Sums of 1,536 products and more are formed on the tensor
// cores from exact parts of the operands, see gemm_f32_tcgen05.cu.)  Each output element is one thread's sum over
// k in ascending order, whatever M is, so a row's result does not depend on the batch.
#include "common.cuh"

namespace ms {

// Large tiles.  What bounds it: the FMA pipes (74 TFLOP/s at 1.965 GHz).  A block owns a BM x BN tile, a thread TM x TN of it, taken in
// pieces of four rows and four columns so that the reads of shared memory are 16 bytes and a warp's addresses repeat.  The
// sums are packed pairs (one instruction for two multiply-adds, which leaves issue slots for the reads), so a slice of 16 k
// lies transposed, [k][row]: a pair of columns is two neighbours.  The next slice is in registers while this one is multiplied,
// and one barrier a slice orders the two buffers.  512 x 12,288 x 2,560: 670 us, 48 TFLOP/s (tiles of 128 x 128), where the ring
// below takes 842 and tiles of 64 x 64 with 4 x 4 a thread, whose every four multiply-adds wait for two reads, ran at 19 TFLOP/s.
template <int BM, int BN, int TM, int TN, bool WIDE>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_f32_large_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                int lda, int ldw, int ldc, long long batch_a, long long batch_w, long long batch_c) {
  grid_dependency_wait();
  grid_dependency_launch();
  constexpr int BK = 16, NT = (BM / TM) * (BN / TN), TX = BN / TN;
  constexpr int A_PIECES = (BM * BK / 4 + NT - 1) / NT, W_PIECES = (BN * BK / 4 + NT - 1) / NT;
  constexpr int RG = TM < 4 ? TM : 4;              // rows of a piece
  static_assert(TN % 4 == 0 && TM % RG == 0, "a thread's tile is made of pieces of four columns");
  A += (size_t)blockIdx.z * batch_a;     // one product per blockIdx.z (per head, for instance): operands `batch_*` apart
  W += (size_t)blockIdx.z * batch_w;
  C += (size_t)blockIdx.z * batch_c;
  __shared__ __align__(16) float As[2][BK][BM + 4];
  __shared__ __align__(16) float Ws[2][BK][BN + 4];
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  // (rows of a piece group lie RG * (BM / TM) apart, columns 4 * TX)
  auto row_of = [&](int i) { return (i / RG) * RG * (BM / TM) + ty * RG + i % RG; };
  auto col_of = [&](int j) { return (j / 4) * 4 * TX + tx * 4 + j % 4; };
  unsigned long long acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;

  float4 next_a[A_PIECES], next_w[W_PIECES];
  auto load4 = [&](const float* base, int ld, int row, int rows, int k) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row >= rows) return v;
    const float* p = base + (size_t)row * ld + k;
    if (WIDE) {                          // K, the row strides and the bases are multiples of four numbers
      if (k < K) v = *reinterpret_cast<const float4*>(p);
    } else {
      if (k < K) v.x = p[0];
      if (k + 1 < K) v.y = p[1];
      if (k + 2 < K) v.z = p[2];
      if (k + 3 < K) v.w = p[3];
    }
    return v;
  };
  auto fetch = [&](int k0) {
#pragma unroll
    for (int p = 0; p < A_PIECES; ++p) {
      const int piece = tid + p * NT;
      if (BM * BK / 4 % NT == 0 || piece < BM * BK / 4) next_a[p] = load4(A, lda, m0 + piece / (BK / 4), M, k0 + piece % (BK / 4) * 4);
    }
#pragma unroll
    for (int p = 0; p < W_PIECES; ++p) {
      const int piece = tid + p * NT;
      if (BN * BK / 4 % NT == 0 || piece < BN * BK / 4) next_w[p] = load4(W, ldw, n0 + piece / (BK / 4), N, k0 + piece % (BK / 4) * 4);
    }
  };
  auto stage = [&](int buffer) {
#pragma unroll
    for (int p = 0; p < A_PIECES; ++p) {
      const int piece = tid + p * NT, r = piece / (BK / 4), k = piece % (BK / 4) * 4;
      if (BM * BK / 4 % NT == 0 || piece < BM * BK / 4) {
        As[buffer][k][r] = next_a[p].x, As[buffer][k + 1][r] = next_a[p].y;
        As[buffer][k + 2][r] = next_a[p].z, As[buffer][k + 3][r] = next_a[p].w;
      }
    }
#pragma unroll
    for (int p = 0; p < W_PIECES; ++p) {
      const int piece = tid + p * NT, r = piece / (BK / 4), k = piece % (BK / 4) * 4;
      if (BN * BK / 4 % NT == 0 || piece < BN * BK / 4) {
        Ws[buffer][k][r] = next_w[p].x, Ws[buffer][k + 1][r] = next_w[p].y;
        Ws[buffer][k + 2][r] = next_w[p].z, Ws[buffer][k + 3][r] = next_w[p].w;
      }
    }
  };
  fetch(0);
  stage(0);
  __syncthreads();
  for (int k0 = 0, buffer = 0; k0 < K; k0 += BK, buffer ^= 1) {
    if (k0 + BK < K) fetch(k0 + BK);
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      unsigned long long a[TM], w[TN / 2];
#pragma unroll
      for (int i = 0; i < TM; i += RG) {
        float piece[RG];
        if (RG == 4) *reinterpret_cast<float4*>(piece) = *reinterpret_cast<const float4*>(&As[buffer][k][row_of(i)]);
        else
          for (int r = 0; r < RG; ++r) piece[r] = As[buffer][k][row_of(i + r)];
#pragma unroll
        for (int r = 0; r < RG; ++r) a[i + r] = pack2(piece[r], piece[r]);
      }
#pragma unroll
      for (int j = 0; j < TN; j += 4) {
        const ulonglong2 two = *reinterpret_cast<const ulonglong2*>(&Ws[buffer][k][col_of(j)]);
        w[j / 2] = two.x, w[j / 2 + 1] = two.y;
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = fma2(a[i], w[j], acc[i][j]);
    }
    if (k0 + BK < K) stage(buffer ^ 1);        // (its last readers passed the barrier before this slice)
    __syncthreads();
  }
  const bool wide_store = (ldc & 3) == 0 && (reinterpret_cast<size_t>(C) & 15) == 0;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + row_of(i);
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; j += 4) {
      const int n = n0 + col_of(j);
      float v[4];
      unpack2(acc[i][j / 2], v[0], v[1]);
      unpack2(acc[i][j / 2 + 1], v[2], v[3]);
      float* out = C + (size_t)m * ldc + n;
      if (wide_store && n + 4 <= N) {
        *reinterpret_cast<float4*>(out) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (n + e < N) out[e] = v[e];
      }
    }
  }
}

// Small tiles, for products whose large tiles would leave multiprocessors idle: what bounds them is the weight's way from memory, so
// slices arrive by cp.async in a ring of STAGES (STAGES - 1 on their way).  They lie in shared memory as they lie in memory, [row][k], rows
// four numbers apart from their neighbours' banks; a thread's TM x TN results lie a thread count apart, and TM + TN reads of sixteen
// bytes feed 4 TM TN multiply-adds.  1 x 2,048 x 6,144: 51 us (tiles of 8 x 16, three slices of 128 on their way) where a 64 x 64 tile
// without a ring takes 324; 389 x 2,048 x 6,144: 344 us (32 x 64) against 391 (64 x 128 of the kernel above).
template <int BM, int BN, int TM, int TN, int BK, int STAGES, bool WIDE>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_f32_ring_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                int lda, int ldw, int ldc, long long batch_a, long long batch_w, long long batch_c) {
  grid_dependency_wait();
  grid_dependency_launch();
  constexpr int NT = (BM / TM) * (BN / TN), TX = BN / TN, TY = BM / TM, LD = BK + 4, STAGE = (BM + BN) * LD;
  A += (size_t)blockIdx.z * batch_a;     // one product per blockIdx.z (per head, for instance): operands `batch_*` apart
  W += (size_t)blockIdx.z * batch_w;
  C += (size_t)blockIdx.z * batch_c;
  extern __shared__ __align__(16) float gemm_smem[];
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  auto copy_rows = [&](float* to, const float* base, int ld, int first, int rows, int total, int k0) {
    constexpr int PER = WIDE ? 4 : 1, PIECES = BK / PER;      // numbers a copy moves, copies a row takes
    for (int piece = tid; piece < rows * PIECES; piece += NT) {
      const int r = piece / PIECES, k = piece % PIECES * PER;
      const bool real = first + r < total && k0 + k < K;      // (WIDE: K is a multiple of four)
      const float* from = real ? base + (size_t)(first + r) * ld + k0 + k : base;
      const unsigned at = (unsigned)__cvta_generic_to_shared(to + r * LD + k);
      if (WIDE)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at), "l"(from), "r"(real ? 16 : 0) : "memory");
      else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(at), "l"(from), "r"(real ? 4 : 0) : "memory");
    }
  };
  auto fetch = [&](int slice) {
    if (slice * BK < K) {
      float* stage = gemm_smem + slice % STAGES * STAGE;
      copy_rows(stage, A, lda, m0, BM, M, slice * BK);
      copy_rows(stage + BM * LD, W, ldw, n0, BN, N, slice * BK);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) fetch(s);
  const int slices = (K + BK - 1) / BK;
  for (int slice = 0; slice < slices; ++slice) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                       // this slice is there, and the one before it has been read
    fetch(slice + STAGES - 1);
    const float* a_at = gemm_smem + slice % STAGES * STAGE + ty * LD;
    const float* w_at = gemm_smem + slice % STAGES * STAGE + BM * LD + tx * LD;
#pragma unroll
    for (int k = 0; k < BK; k += 4) {
      float4 w[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const float4*>(w_at + j * TX * LD + k);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(a_at + i * TY * LD + k);
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.x, w[j].x, acc[i][j]);
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.y, w[j].y, acc[i][j]);
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.z, w[j].z, acc[i][j]);
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.w, w[j].w, acc[i][j]);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty + i * TY;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + j * TX;
      if (n < N) C[(size_t)m * ldc + n] = acc[i][j];
    }
  }
}

// One launch; `wide`: rows, strides and bases let four numbers move at once.
template <typename Kernel>
static int launch_gemm_f32(Kernel kernel, int bm, int bn, int threads, int smem, const float* A, const float* W, float* C, int M, int N, int K,
                           int lda, int ldw, int ldc, int batch, long long batch_a, long long batch_w, long long batch_c,
                           cudaStream_t stream) {
  const int grid_m = (M + bm - 1) / bm, grid_n = (N + bn - 1) / bn;
  MS_REQUIRE(grid_m <= 65535 && batch <= 65535, "gemm_f32: %d rows or %d products in one launch is too many", M, batch);
  if (smem > 0) {
    const cudaError_t e = allow_shared(kernel, (size_t)smem);
    if (e != cudaSuccess) MS_FAIL("gemm_f32: %d bytes of shared memory refused: %s", smem, cudaGetErrorString(e));
  }
  ms::launch(kernel, dim3(grid_n, grid_m, batch), threads, smem, stream, A, W, C, M, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c);
  MS_CHECK_LAUNCH("gemm_f32");
  return 0;
}

// Which tile: the one with the least (r + start) * area / rate, r = ceil(tiles / multiprocessors) being the tiles of the busiest
// multiprocessor.  `rate` (1e3 results * k a microsecond and multiprocessor with many tiles) and `start` (what a lone tile takes longer,
// in tiles) are measured, one row per tile: with 64 tiles of 128 x 128 171 against 188 where each multiprocessor has three,
// with 64 of 16 x 32 26 against 74.  Every tile sums in the same order, so the choice changes no result.
struct GemmF32Tile { int rows, columns; double start, rate; };
static const GemmF32Tile kGemmF32Tiles[] = {{128, 128, 0.1, 188}, {64, 128, 0.34, 165}, {64, 64, 0.48, 132}, {32, 64, 0.72, 115},
                                            {16, 32, 1.85, 74},   {8, 32, 0.93, 40},    {8, 16, 1.2, 34}};

static int choose_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int batch,
                           long long batch_a, long long batch_w, long long batch_c, cudaStream_t stream) {
  constexpr long long kProcessors = 148;
  int best = 0;
  double least = 0.0;
  for (int t = 0; t < (int)(sizeof(kGemmF32Tiles) / sizeof(kGemmF32Tiles[0])); ++t) {
    const GemmF32Tile& tile = kGemmF32Tiles[t];
    const long long row_tiles = (M + tile.rows - 1) / tile.rows;
    if (row_tiles > 65535) continue;
    const long long tiles = row_tiles * ((N + tile.columns - 1) / tile.columns) * batch;
    const double cost = ((double)((tiles + kProcessors - 1) / kProcessors) + tile.start) * tile.rows * tile.columns / tile.rate;
    if (t == 0 || cost < least) best = t, least = cost;
  }
  const bool wide = ((K | lda | ldw) & 3) == 0 && ((batch_a | batch_w) & 3) == 0 &&
                    ((reinterpret_cast<size_t>(A) | reinterpret_cast<size_t>(W)) & 15) == 0;
#define MS_GEMM_F32_LARGE(BM, BN, TM, TN)                                                                                      \
  return launch_gemm_f32(wide ? gemm_f32_large_kernel<BM, BN, TM, TN, true> : gemm_f32_large_kernel<BM, BN, TM, TN, false>, BM, BN, \
                         (BM / TM) * (BN / TN), 0, A, W, C, M, N, K, lda, ldw, ldc, batch, batch_a, batch_w, batch_c, stream)
#define MS_GEMM_F32_RING(BM, BN, TM, TN, BK, STAGES)                                                                           \
  return launch_gemm_f32(                                                                                                      \
      wide ? gemm_f32_ring_kernel<BM, BN, TM, TN, BK, STAGES, true> : gemm_f32_ring_kernel<BM, BN, TM, TN, BK, STAGES, false>, BM, BN, \
      (BM / TM) * (BN / TN), STAGES * (BM + BN) * (BK + 4) * (int)sizeof(float), A, W, C, M, N, K, lda, ldw, ldc, batch, batch_a,  \
      batch_w, batch_c, stream)
  switch (best) {
    case 0: MS_GEMM_F32_LARGE(128, 128, 8, 8);
    case 1: MS_GEMM_F32_LARGE(64, 128, 8, 8);
    case 2: MS_GEMM_F32_RING(64, 64, 8, 4, 32, 4);
    case 3: MS_GEMM_F32_RING(32, 64, 4, 4, 32, 4);
    case 4: MS_GEMM_F32_RING(16, 32, 2, 4, 64, 4);
    case 5: MS_GEMM_F32_RING(8, 32, 1, 2, 64, 6);
    default: MS_GEMM_F32_RING(8, 16, 1, 1, 128, 4);
  }
#undef MS_GEMM_F32_LARGE
#undef MS_GEMM_F32_RING
}

}  // namespace ms

using namespace ms;

MS_EXPORT int ms_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                          cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  MS_REQUIRE(K > 0, "gemm_f32: inner size must be positive, got %d", K);
  MS_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm_f32: a row stride is smaller than its row (lda %d ldw %d ldc %d)",
             lda, ldw, ldc);
  return choose_gemm_f32(A, W, C, M, N, K, lda, ldw, ldc, 1, 0LL, 0LL, 0LL, stream);
}

// `batch` products of the same sizes in one launch: C_b[M, N] = A_b[M, K] * W_b[N, K]^T with X_b = X + b * batch_x
// (elements).  Rows may be strided (lda, ldw, ldc), so the operands can be slices of wider matrices: one head's
// columns of a projection, one head's rows of an output.
MS_EXPORT int ms_gemm_f32_batched(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                                  int batch, long long batch_a, long long batch_w, long long batch_c, cudaStream_t stream) {
  if (M == 0 || N == 0 || batch == 0) return 0;
  MS_REQUIRE(K > 0, "gemm_f32_batched: inner size must be positive, got %d", K);
  MS_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm_f32_batched: a row stride is smaller than its row (lda %d ldw %d ldc %d)",
             lda, ldw, ldc);
  return choose_gemm_f32(A, W, C, M, N, K, lda, ldw, ldc, batch, batch_a, batch_w, batch_c, stream);
}
