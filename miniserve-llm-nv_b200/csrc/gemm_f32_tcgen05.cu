// The float32 product C[M, N] = A[M, K] * W[N, K]^T on the fifth-generation tensor cores, as exact as the one on the CUDA cores: every
// operand is cut into three bfloat16 parts that add up to it exactly (x = hi + mid + lo: 24 bits in three times eight), and of the nine
// products of parts the six that reach a float32's last bit are summed (the other three are at most 2^-26 of a product each).  Numbers below
// 2^-110 are more than their parts, which end at 2^-133; see `as_it_is` for what comes of that.
//
// What the tensor cores do not do is round: an addition to an accumulator in tensor memory drops the bits behind its last, always
// towards zero, and over a sum of 2,048 that leaves five times the error of float32 additions (2.1e-6 against 4e-7, measured).  So a
// sum lives in tensor memory for one stage of 64 k only: the small products come first, while the accumulator is small, the product of
// the leading parts last, in four steps; the stage's sum is then read out and added in float32 registers, rounded to nearest, in
// ascending order of the stages.
//
// W is the MMA's A operand (128 rows of W are the lanes of tensor memory), a tile of up to 144 rows of A its B operand, so that the same kernel
// streams the weights for a single row and multiplies tiles for a prompt.  Where W has few rows its inner size is cut over a cluster of up to
// eight blocks, whose sums meet in distributed shared memory in the order of the ranks.  The cut depends on N and K alone, and a row's sum on
// nothing but itself: its bits do not depend on how many rows there are.
//
// One block a multiprocessor, 20 warps:
//   warps 0..7     a row of W a thread: 32 k of it from the ring (warps 0..3 the first half of a stage, 4..7 the second), cut into parts,
//                  stored to tensor memory;
//   warps 8..15    add the stages' sums up in registers (a row of W and every other piece of eight columns a thread), and store;
//   warp 16        fetches W by TMA into a ring of pieces of 32 k;
//   warps 17, 18   issue the MMAs, a stage in turn: a thread stands still while the tensor cores work on what it has issued, and a single one's
//                  waits for the next stage came on top of that (1.5 times the time);
//   warp 19        fetches the parts of A into a second ring.  A kernel before this one cuts A: every block would cut its rows again, which
//                  took as long as the MMAs.
//
// A sum that is not finite (an operand was not, or one of the products above has left the range that float32 has) or is very small is formed again by
// plain multiply-adds, so that infinities and NaNs are those of the plain product, and small operands count whole.
//
// Bound by the MMAs' operands: a stage of 144 rows takes 2,245 clocks, its 24 MMAs 1,730 when nothing else reads shared memory (16 rows:
// 1,800, an MMA of any width takes 65); the tensor pipe is busy for 62 % of the cycles at 389 x 12,288 x 2,048.  One row / 389 rows (us; the plain kernels in brackets): 12,288 x 2,048 44 / 110 (49 / 513), 2,048 x
// 6,144 30 / 93 (51 / 345), 2,048 x 2,048 19 / 54 (23 / 121), 21,888 x 2,560 97 / 257 (106 / 1,093).  Distance from 64 bits (2-norm,
// normal operands): K = 2,048 1.0e-7 to 1.3e-7 (plain 8.1e-7), K = 6,144 1.2e-7 (1.4e-6), K = 256 0.9e-7 (3e-7).
//
// Every wait on an mbarrier is bounded: a wait that does not finish sets the error flag that the host checks, all roles drain and
// tensor memory is freed on every path.
#include <algorithm>

#include "tcgen05.cuh"

namespace ms {
namespace t5f {
using namespace t5;

constexpr int kRows = 128;                   // of W a block
constexpr int kMost = 144;                   // rows of A a block, at most
constexpr int kStage = 64, kPiece = 32;      // k of a stage and of a piece of the ring (128 bytes of a float32 row)
constexpr int kThreads = 640;
constexpr int kMaxPieces = 12;               // of either ring
constexpr int kUnits = kMost / 16;           // pieces of eight columns that a summing thread has
constexpr int kAhead = 3;                    // pieces that it reads at a time
constexpr int kOperandColumns = 96;          // of tensor memory: three parts of a stage's W

__host__ __device__ constexpr unsigned rows_bytes(int tn) { return 3u * tn * 64u; }             // a piece's parts of A
constexpr unsigned kPieceBytes = kRows * 128;
__host__ __device__ constexpr int sum_columns(int tn) { return (tn + 31) / 32 * 32; }

struct Args {
  const float *A, *W;
  float* C;
  int M, N, K, lda, ldw, ldc;
  int tn, pieces, row_pieces, splits;
  int* error_flag;
};

// Whether a sum is taken as it is: finite, and zero or at least 2^-100.  What operands below 2^-110 lack in their parts is 2^-134 of the other operand at
// most, 2^-25 of such a sum while a row's magnitudes add up to less than 2^9.  Smaller sums are formed again (rows of 1e-36 times
// rows of ordinary numbers came out with 14 bits).
__device__ __forceinline__ bool as_it_is(float v) {
  const unsigned twice = __float_as_uint(v) << 1;          // (without the sign)
  return twice == 0u || (twice >= 27u << 24 && twice < 255u << 24);
}
// Descriptor of a K-major tile of 32 k: rows of 64 bytes with the 64-byte swizzle, groups of eight rows 512 bytes apart.
__device__ __forceinline__ uint64_t rows_desc(const void* smem_tile) {
  return (uint64_t)((smem_u32(smem_tile) & 0x3FFFF) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)4 << 61;
}

__device__ __forceinline__ float4 load_shared_of(unsigned cluster_address) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_address) : "memory");
  return v;
}

// What a block has stored in its rows of W and the columns c_first <= c < c_last of its tile and cannot stay as it is, by plain multiply-adds in ascending k.  All of
// its threads take part, with slices of 32 k in shared memory: 389 rows of NaNs, 2,048 x 6,144, take 1.8 ms (0.10 without); a thread for each such sum 32 ms.
constexpr int kAgain = 8, kAgainGroups = kThreads / kRows;       // columns a thread, threads a row of W
__device__ __noinline__ void plain_sums(const Args& p, float* room, int n0, int m0, int c_first, int c_last) {
  float *ws = room, *as = room + kRows * 36;                     // [128][36], [40][32]
  const int n = threadIdx.x % kRows, group = threadIdx.x / kRows;
#pragma unroll 1
  for (int c0 = c_first; c0 < c_last; c0 += kAgain * kAgainGroups) {
    const int mine = c0 + group * kAgain;
    unsigned bad = 0;
#pragma unroll
    for (int e = 0; e < kAgain; ++e)
      if (mine + e < c_last && m0 + mine + e < p.M && n0 + n < p.N && !as_it_is(p.C[(size_t)(m0 + mine + e) * p.ldc + n0 + n])) bad |= 1u << e;
    if (!__syncthreads_or(bad != 0u)) continue;
    const bool any = __any_sync(0xffffffffu, bad != 0u);
    float sum[kAgain];
#pragma unroll
    for (int e = 0; e < kAgain; ++e) sum[e] = 0.f;
#pragma unroll 1
    for (int k0 = 0; k0 < p.K; k0 += 32) {
      for (int i = threadIdx.x; i < (kRows + kAgain * kAgainGroups) * 8; i += kThreads) {
        const int row = i / 8, k = i % 8 * 4, c = c0 + row - kRows;
        const bool of_w = row < kRows, there = k0 + k < p.K && (of_w ? n0 + row < p.N : c < c_last && m0 + c < p.M);
        const float* from = of_w ? p.W + (size_t)(n0 + row) * p.ldw : p.A + (size_t)(m0 + c) * p.lda;
        const float4 v = there ? *reinterpret_cast<const float4*>(from + k0 + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        *reinterpret_cast<float4*>(of_w ? ws + row * 36 + k : as + (row - kRows) * 32 + k) = v;
      }
      __syncthreads();
      const int here = any ? min(32, p.K - k0) : 0;
      for (int k = 0; k < here; k += 4) {
        const float4 w = *reinterpret_cast<const float4*>(ws + n * 36 + k);
#pragma unroll
        for (int e = 0; e < kAgain; ++e) {
          const float4 a = *reinterpret_cast<const float4*>(as + (group * kAgain + e) * 32 + k);
          sum[e] = fmaf(a.w, w.w, fmaf(a.z, w.z, fmaf(a.y, w.y, fmaf(a.x, w.x, sum[e]))));
        }
      }
      __syncthreads();
    }
#pragma unroll
    for (int e = 0; e < kAgain; ++e)
      if (bad >> e & 1u) p.C[(size_t)(m0 + mine + e) * p.ldc + n0 + n] = sum[e];
  }
}

// [3][rows][ld] bfloat16 parts of rows of A, four numbers a thread.  Bound by memory: ten bytes a number.
__global__ void __launch_bounds__(256)
cut_rows_kernel(const float* __restrict__ A, int lda, int rows, int K, int ld, uint2* __restrict__ parts) {
  grid_dependency_wait();
  grid_dependency_launch();
  const unsigned per_row = K / 4, at = blockIdx.x * 256 + threadIdx.x;
  if (at >= per_row * (unsigned)rows) return;
  const unsigned row = at / per_row, k4 = at % per_row;
  const float4 v = *reinterpret_cast<const float4*>(A + (size_t)row * lda + 4 * k4);
  uint2 hi, mid, lo;
  cut(v.x, v.y, hi.x, mid.x, lo.x);
  cut(v.z, v.w, hi.y, mid.y, lo.y);
  uint2* to = parts + (size_t)row * (ld / 4) + k4;
  const size_t part = (size_t)rows * (ld / 4);
  to[0] = hi, to[part] = mid, to[2 * part] = lo;
}

__global__ void __launch_bounds__(kThreads, 1)
gemm_f32_tcgen05_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ Args p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t full[kMaxPieces], empty[kMaxPieces], rows_full[kMaxPieces], rows_empty[kMaxPieces], cut_full[2], cut_empty[2], sum_full[2], sum_empty[2];
  __shared__ unsigned tmem_base_s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tn = p.tn, pieces = p.pieces, row_pieces = p.row_pieces, splits = p.splits;
  const int rank = blockIdx.x % splits, n0 = blockIdx.x / splits * kRows, m0 = blockIdx.y * tn;
  const int all_stages = (p.K + kStage - 1) / kStage;
  const int first = (int)((long long)all_stages * rank / splits), stages = (int)((long long)all_stages * (rank + 1) / splits) - first;
  const unsigned columns = 2 * sum_columns(tn) + 2 * kOperandColumns <= 256 ? 256u : 512u;
  unsigned char* ring = smem + row_pieces * rows_bytes(tn);

  if (warp == 16 && lane == 0) {
    for (int s = 0; s < pieces; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 4);               // one arrival per cutting warp
    }
    for (int s = 0; s < row_pieces; ++s) {
      mbar_init(&rows_full[s], 1);
      mbar_init(&rows_empty[s], 1);
    }
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      mbar_init(&cut_full[s], 8);
      mbar_init(&cut_empty[s], 1);
      mbar_init(&sum_full[s], 1);
      mbar_init(&sum_empty[s], 8);                     // one arrival per summing warp
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 17) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  const unsigned tmem_base = tmem_base_s, operand_column = 2 * sum_columns(tn);
  grid_dependency_wait();
  grid_dependency_launch();

  float acc[kUnits][8];                      // of the summing warps
  bool fine = true;                          // what this thread has stored
  if (warp < 8) {
    // ---------------- rows of W into tensor memory: half a stage a warp
    const int half = warp >> 2;
    const unsigned row = threadIdx.x & 127, swizzle = row & 7;
    const unsigned to = tmem_base + ((unsigned)((warp & 3) * 32) << 16) + operand_column + half * 16;
    const unsigned char* from = ring + row * 128;
    bool ok = true;
    int piece = half;                        // (every other one: the ring has an even number)
    unsigned turn = 0;
    for (int s = 0; s < stages; ++s) {
      const int stage = s & 1;
      ok = mbar_wait(&full[piece], turn, p.error_flag, 51);
      if (!__all_sync(0xffffffffu, ok)) break;
      unsigned hi[16], mid[16], lo[16];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float4 v = *reinterpret_cast<const float4*>(from + piece * kPieceBytes + ((c ^ swizzle) << 4));
        cut(v.x, v.y, hi[2 * c], mid[2 * c], lo[2 * c]);
        cut(v.z, v.w, hi[2 * c + 1], mid[2 * c + 1], lo[2 * c + 1]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[piece]);
      if ((piece += 2) >= pieces) piece -= pieces, turn ^= 1;
      ok = mbar_wait(&cut_empty[stage], ((s >> 1) & 1) ^ 1, p.error_flag, 52);       // the MMAs have read what this replaces
      if (!__all_sync(0xffffffffu, ok)) break;
      tmem_fence_after();
      const unsigned at = to + stage * kOperandColumns;
      tmem_store_16(at, hi);
      tmem_store_16(at + 32, mid);
      tmem_store_16(at + 64, lo);
      tmem_store_wait();
      tmem_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&cut_full[stage]);
    }
  } else if (warp < 16) {
    // ---------------- the stages' sums: pieces of eight columns (warp - 8) / 4, + 2, ...
    const unsigned from = tmem_base + ((unsigned)((warp & 3) * 32) << 16);
    const int half = (warp - 8) >> 2;
#pragma unroll
    for (int u = 0; u < kUnits; ++u)
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[u][e] = 0.f;
    bool ok = true;
    for (int s = 0; s < stages; ++s) {
      const int buffer = s & 1;
      ok = mbar_wait(&sum_full[buffer], (s >> 1) & 1, p.error_flag, 55);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tmem_fence_after();
      const unsigned at = from + buffer * sum_columns(tn);
#pragma unroll
      for (int u = 0; u < kUnits; u += kAhead) {
        float v[kAhead][8];
        if ((2 * u + half) * 8 >= tn) break;
#pragma unroll
        for (int w = 0; w < kAhead; ++w)     // (a piece behind the last row's reads columns that nobody uses)
          if (u + w < kUnits) tmem_load_8_nowait(at + (2 * (u + w) + half) * 8, v[w]);
        tmem_load_wait();
#pragma unroll
        for (int w = 0; w < kAhead; ++w)
          if (u + w < kUnits) {
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[u + w][e] += v[w][e];
          }
      }
      tmem_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sum_empty[buffer]);
    }
    const int n_in = (warp & 3) * 32 + lane;
    if (splits == 1) {
      if (ok && n0 + n_in < p.N) {
        float* out = p.C + (size_t)m0 * p.ldc + n0 + n_in;
#pragma unroll
        for (int u = 0; u < kUnits; ++u) {
          const int c0 = (2 * u + half) * 8;
#pragma unroll
          for (int e = 0; e < 8; ++e)
            if (c0 + e < tn && m0 + c0 + e < p.M) {
              out[(size_t)(c0 + e) * p.ldc] = acc[u][e];
              fine = fine && as_it_is(acc[u][e]);
            }
        }
      }
    } else {
      // (all MMAs of this block have finished and every piece of the ring has been read: the room is free)
      float* mine = reinterpret_cast<float*>(smem);
#pragma unroll
      for (int u = 0; u < kUnits; ++u) {
        const int c0 = (2 * u + half) * 8;
        if (ok && c0 < tn) {
#pragma unroll
          for (int e = 0; e < 8; ++e) mine[(c0 + e) * kRows + n_in] = acc[u][e];
        }
      }
    }
  } else if (warp == 16) {
    if (lane == 0) {
      // ---------------- W, 32 k at a time (zeros behind the last row and the last k)
      bool ok = true;
      int i = 0, piece = 0;
      unsigned turn = 1;
      for (; i < 2 * stages; ++i) {
        if (!(ok = mbar_wait(&empty[piece], turn, p.error_flag, 56))) break;
        mbar_expect_tx(&full[piece], kPieceBytes);
        tma_load_2d(ring + piece * kPieceBytes, &map_w, &full[piece], first * kStage + i * kPiece, n0);
        if (++piece == pieces) piece = 0, turn ^= 1;
      }
      if (!ok || *reinterpret_cast<volatile int*>(p.error_flag) != 0) let_copies_land(full, pieces, i, p.error_flag);
    }
  } else if (warp < 19) {
    if (lane == 0) {
      // ---------------- MMA issue, every other stage
      const unsigned idesc = umma_idesc(kRows, tn);
      const unsigned part = tn * 4;          // of A in shared memory, in units of sixteen bytes
      const int stage = warp - 17;
      bool ok = true;
      int piece = 2 * stage;
      unsigned turn = 0;
      const unsigned sum = tmem_base + stage * sum_columns(tn), w = tmem_base + operand_column + stage * kOperandColumns;
      for (int s = stage; s < stages; s += 2) {
        const unsigned parity = (s >> 1) & 1;
        // (W first: its cutting warps have waited for the MMAs of every stage up to the one before last, so that the parities below mean
        // this stage's phases; the sums last: theirs is the longest way round, and each wait takes a hundred clocks of its own)
        ok = mbar_wait(&cut_full[stage], parity, p.error_flag, 59);
        int two = piece + 1;
        unsigned two_turn = turn;
        if (two == row_pieces) two = 0, two_turn ^= 1;
        ok = ok && mbar_wait(&rows_full[piece], turn, p.error_flag, 58) && mbar_wait(&rows_full[two], two_turn, p.error_flag, 58) &&
             mbar_wait(&sum_empty[stage], parity ^ 1, p.error_flag, 57);
        if (!ok) break;
        const int one = piece;
        if ((piece += 4) >= row_pieces) piece -= row_pieces, turn ^= 1;
        tmem_fence_after();
        const uint64_t a[2] = {rows_desc(smem + one * rows_bytes(tn)), rows_desc(smem + two * rows_bytes(tn))};
        const int w_part[6] = {2, 0, 1, 1, 0, 0}, a_part[6] = {0, 2, 1, 0, 1, 0};        // smallest products first
#pragma unroll
        for (int q = 0; q < 6; ++q)
#pragma unroll
          for (int k = 0; k < kStage / 16; ++k)
            umma_bf16_a_tmem(sum, w + w_part[q] * 32 + k * 8, a[k >> 1] + (uint64_t)(a_part[q] * part + 2 * (k & 1)), idesc, (q | k) != 0 ? 1u : 0u);
        umma_commit(&cut_empty[stage]);
        umma_commit(&rows_empty[one]);
        umma_commit(&rows_empty[two]);
        umma_commit(&sum_full[stage]);
      }
    }
  } else if (lane == 0) {
    // ---------------- parts of A (rows behind the last are those of the next part, or zeros: what they give is not stored)
    bool ok = true;
    int i = 0, piece = 0;
    unsigned turn = 1;
    for (; i < 2 * stages; ++i) {
      if (!(ok = mbar_wait(&rows_empty[piece], turn, p.error_flag, 60))) break;
      mbar_expect_tx(&rows_full[piece], rows_bytes(tn));
#pragma unroll
      for (int part = 0; part < 3; ++part)
        tma_load_2d(smem + piece * rows_bytes(tn) + part * tn * 64, &map_a, &rows_full[piece], first * kStage + i * kPiece, part * p.M + m0);
      if (++piece == row_pieces) piece = 0, turn ^= 1;
    }
    if (!ok || *reinterpret_cast<volatile int*>(p.error_flag) != 0) let_copies_land(rows_full, row_pieces, i, p.error_flag);
  }

  tmem_fence_before();
  const bool again = __syncthreads_or(!fine);
  if (warp == 17) {
    tmem_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(columns) : "memory");
  }
  if (splits == 1) {
    if (again) plain_sums(p, reinterpret_cast<float*>(smem), n0, m0, 0, tn);
    return;
  }
  cluster_sync_all();                        // every rank's sums are there
  const int c_first = tn * rank / splits, c_last = tn * (rank + 1) / splits;
  const bool wide = (p.ldc & 3) == 0 && (reinterpret_cast<size_t>(p.C) & 15) == 0;
  for (int i = threadIdx.x; i < (c_last - c_first) * (kRows / 4); i += kThreads) {
    const int c = c_first + i / (kRows / 4), n = i % (kRows / 4) * 4;
    if (m0 + c >= p.M || n0 + n >= p.N) continue;
    const unsigned at = smem_u32(smem) + (unsigned)(c * kRows + n) * 4;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    for (int r = 0; r < splits; ++r) {
      const float4 part = load_shared_of(address_in_rank(at, r));
      v[0] += part.x, v[1] += part.y, v[2] += part.z, v[3] += part.w;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) fine = fine && (n0 + n + e >= p.N || as_it_is(v[e]));
    float* out = p.C + (size_t)(m0 + c) * p.ldc + n0 + n;
    if (wide && n0 + n + 4 <= p.N) {
      *reinterpret_cast<float4*>(out) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (n0 + n + e < p.N) out[e] = v[e];
    }
  }
  cluster_sync_all();                        // nobody reads this block's sums any more
  if (__syncthreads_or(!fine)) plain_sums(p, reinterpret_cast<float*>(smem), n0, m0, c_first, c_last);
}

// Rows of 32 numbers a box: float32 ones 128 bytes wide, parts 64, either with the swizzle of that width.
static bool encode_rows(CUtensorMap* map, bool parts, const void* at, long long rows, int k, int ld, int box_rows) {
  EncodeTiled encode = encode_tiled();
  const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * (parts ? 2 : 4)};
  const cuuint32_t box[2] = {(cuuint32_t)kPiece, (cuuint32_t)box_rows}, elem[2] = {1, 1};
  return encode != nullptr && encode(map, parts ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(at), dims,
                                     strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, parts ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace t5f
}  // namespace ms

using namespace ms;
using namespace ms::t5f;

// Whether ms_gemm_f32_tcgen05 takes these sizes and is the faster way: a question of N and K alone, so that a row's bits do not depend on
// how many rows there are.  Two launches and a block's fixed costs make it 15 us for a single row of short sums, where the plain kernel's time goes
// with K: 1,024 x 1,024 14 against 15, 2,048 x 1,024 13 against 17, 8,192 x 1,024 23 against 22, 16 x 2,048 20 against 15, 2,048 x 2,048
// 23 against 19, 6,144 x 1,536 27 against 25; with 389 rows all of these are two to four times as fast here.
MS_EXPORT int ms_gemm_f32_tcgen05_takes(int N, int K) { return K % 4 == 0 && (K >= 1536 || (K >= 1024 && N >= 8192)); }

// Rows of A that are cut and multiplied at a time.  More are a loop of launches, so that no number of rows is too large and the scratch stays that of
// these (1.5 times their size).  They fill the processors well: 114 tiles of 144 rows, with 2,048 rows of W 12.3 rounds.
static int rows_at_a_time(int K) { return (int)std::min(16384LL, ((1LL << 31) - 1) / (K / 4)); }

// Bytes of scratch (on a 16-byte boundary) for the parts of M rows of K.
MS_EXPORT long long ms_gemm_f32_tcgen05_scratch(int M, int K) { return 6LL * std::min(M, rows_at_a_time(K)) * (((long long)K + 7) / 8 * 8); }

static int multiply(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, void* scratch, int* error_flag,
                    cudaStream_t stream) {
  // Clusters of c blocks, a block a multiprocessor, that run at a time (cudaOccupancyMaxActiveClusters): the largest c that lets all tiles of
  // W run at once, with 256 k a block at least.
  constexpr int kActive[8] = {148, 74, 45, 33, 26, 22, 15, 15};
  const int tiles_n = (N + kRows - 1) / kRows, all_stages = (K + kStage - 1) / kStage;
  int splits = 1;
  for (int c = 2; c <= 8; ++c)
    if (kActive[c - 1] >= tiles_n && K / c >= 256) splits = c;
  // Rows of A a block: the number of tiles whose rounds take least.  In clocks a stage takes about 1,500 and 5 more a row (measured: 1,800
  // for 16 rows, 2,245 for 144, where the MMAs alone are 1,560 and 1,730), a tile about 12,000 before its first stage and behind its last.
  const int fewest = (M + kMost - 1) / kMost;
  int tn = 0;
  double least = 0.0;
  for (int t = fewest; t <= fewest + 8; ++t) {
    const int rows = ((M + t - 1) / t + 15) / 16 * 16;
    const long long tiles = (long long)tiles_n * ((M + rows - 1) / rows);
    const double cost = (double)((tiles + kActive[splits - 1] - 1) / kActive[splits - 1]) *
                        ((double)((all_stages + splits - 1) / splits) * (1500 + 5 * rows) + 12000);
    if (tn == 0 || cost < least) tn = rows, least = cost;
    if (rows == 16) break;
  }
  const int tiles_m = (M + tn - 1) / tn;
  // The rings: two and a half stages of A and four pieces of W in the largest tiles.
  constexpr int kShared = 226 * 1024 - 1024;
  const int row_pieces = tn > 128 ? 5 : 6;
  int pieces = (kShared - row_pieces * (int)rows_bytes(tn)) / (int)kPieceBytes;
  pieces = pieces > kMaxPieces ? kMaxPieces : pieces & ~1;       // (even: a place in the ring is always the same half's)
  const size_t smem = 1024 + (size_t)row_pieces * rows_bytes(tn) + (size_t)pieces * kPieceBytes;
  const int ld = (K + 7) / 8 * 8;
  CUtensorMap map_w, map_a;
  MS_REQUIRE(encode_rows(&map_w, false, W, N, K, ldw, kRows) &&
                 encode_rows(&map_a, true, scratch, 3LL * M, K, ld, tn),
             "gemm_f32_tcgen05: cuTensorMapEncodeTiled failed (%d x %d x %d)", M, N, K);
  if (allow_shared(gemm_f32_tcgen05_kernel, smem) != cudaSuccess) MS_FAIL("gemm_f32_tcgen05: %zu bytes of shared memory refused", smem);
  const unsigned threads = (unsigned)M * (K / 4);
  ms::launch(cut_rows_kernel, dim3((threads + 255) / 256), dim3(256), 0, stream, A, lda, M, K, ld, reinterpret_cast<uint2*>(scratch));
  MS_CHECK_LAUNCH("gemm_f32_tcgen05: rows cut");
  const Args args{A, W, C, M, N, K, lda, ldw, ldc, tn, pieces, row_pieces, splits, error_flag};
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(tiles_n * splits, tiles_m), config.blockDim = dim3(kThreads), config.dynamicSmemBytes = smem, config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = splits, attributes[0].val.clusterDim.y = 1, attributes[0].val.clusterDim.z = 1;
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attributes, config.numAttrs = dependent_launch_enabled() ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&config, gemm_f32_tcgen05_kernel, map_w, map_a, args);
  if (e != cudaSuccess) MS_FAIL("gemm_f32_tcgen05: launch failed: %s", cudaGetErrorString(e));
  return 0;
}

// C[M, N] = A[M, K] * W[N, K]^T in float32; bases on 16-byte boundaries, rows of a multiple of four numbers apart.
MS_EXPORT int ms_gemm_f32_tcgen05(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, void* scratch,
                                  int* error_flag, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  MS_REQUIRE(K > 0 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && lda >= K && ldw >= K && ldc >= N, "gemm_f32_tcgen05: %d x %d x %d, rows of %d %d %d",
             M, N, K, lda, ldw, ldc);
  MS_REQUIRE(((reinterpret_cast<size_t>(A) | reinterpret_cast<size_t>(W) | reinterpret_cast<size_t>(scratch)) & 15) == 0,
             "gemm_f32_tcgen05: operands must be 16-byte aligned");
  MS_REQUIRE(error_flag != nullptr && scratch != nullptr, "gemm_f32_tcgen05: an error flag and scratch on the device are required");
  const int rows = rows_at_a_time(K);
  for (long long m = 0; m < M; m += rows)
    if (multiply(A + m * lda, W, C + m * ldc, (int)std::min((long long)rows, M - m), N, K, lda, ldw, ldc, scratch, error_flag, stream)) return 1;
  return 0;
}
