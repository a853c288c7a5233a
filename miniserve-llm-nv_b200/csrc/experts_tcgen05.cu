// The experts' products on the fifth-generation tensor cores: C[i, :] = act(A[src(i), :] W_e^T) for every place i of expert e's segment
// of the sorted (token, choice) pairs, W [experts, N, K], bfloat16 operands, float32 accumulation in tensor memory.  src(i) = order[i] /
// top (rows gathered from the tokens), or i.
//
// One thread block per multiprocessor walks over BM x BN tiles (an expert's row tiles before its next columns, so that neighbours
// share a tile of W); how many tiles there are is read from the device's segment offsets, so no launch waits for the host:
//   warp 0       one thread fetches W tiles by TMA (128-byte swizzle) into a ring of shared-memory stages;
//   warps 6..9   fetch the rows of A by cp.async into the same stages, 128 contiguous bytes of a row for eight lanes, placed as the swizzle
//                wants them; their arrival is counted by the copies themselves (cp.async.mbarrier.arrive), so that the loaders run on
//                as far as the ring is free (waiting for a stage's copies before announcing it kept them one stage ahead of the
//                multiplication: 145 us for both products of the prompt below).  Rows behind a segment's end are not
//                fetched: a row of the result depends on its own row of A alone, and theirs is not stored;
//   warp 1       one thread issues tcgen05.mma into one of two accumulators (the copies' writes are of the generic proxy: it orders them
//                before its reads by a proxy fence);
//   warps 2..5   read an accumulator out (a row a thread), apply the activation and store, while the next tile is multiplied.
//
// Bound by the tensor cores where segments are long, by the weights' way from memory in decode steps, where a tile holds a row or
// two: there the ring is what counts (160 KB of W a multiprocessor on their way), and 64 rows of multiplication cost nothing that
// the memory would not.
// Two products of 2,048 tokens, four of 16 experts of 1,024, width 2,048: 382 us on mma.sync, 110 here (103 GFLOP, 940 TFLOP/s); of 8
// tokens, six of 60 experts of 1,408: 168 -> 107 us (571 MB of weights, 5.3 TB/s).
//
// Every wait on an mbarrier is bounded: a wait that does not finish sets the error flag that the host checks, all roles drain and
// tensor memory is freed on every path.
#include "expert_activation.cuh"
#include "tcgen05.cuh"

namespace ms {
namespace t5e {
using namespace t5;

constexpr int BK = 64, UMMA_K = 16;
constexpr int THREADS = 320;                 // warps 0..9
constexpr int LOADERS = 128;                 // threads that fetch A

template <int BM, int BN, int STAGES>
struct Layout {
  static constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr size_t RING = (size_t)STAGES * STAGE_BYTES + 1024;      // + room to align to 1024 bytes
};

// A tile of the walk: its expert's segment, its first row and column.  `expert` moves forward with `tile` from call to call.
template <int BM>
struct Walk {
  const int *first_tile, *offsets;           // [experts + 1]: tiles before an expert's first; segment borders
  int tiles_n, bn, expert;
  __device__ __forceinline__ void at(int tile, int& row0, int& end, int& column0) {
    while (tile >= first_tile[expert + 1]) ++expert;
    const int first = offsets[expert], local = tile - first_tile[expert];
    end = offsets[expert + 1];
    const int tiles_m = (end - first + BM - 1) / BM;
    row0 = first + local % tiles_m * BM;
    column0 = local / tiles_m * bn;
  }
};

// 32 neighbouring results of a row, from column `col` of the product on: the activation, and the row of C that they become.
__device__ __forceinline__ void store_row(float (&v)[32], __nv_bfloat16* row, int col, int columns, int activation, float limit, float scale,
                                          bool wide) {
  int count = 32;
  if (activation >= kActClampedGlu) {                  // columns alternate (gate, up): two of them give one result
    count = 16, col >>= 1;
#pragma unroll
    for (int i = 0; i < 16; ++i)
      v[i] = activation == kActSiluGlu ? silu_glu(v[2 * i], v[2 * i + 1], scale) : clamped_glu(v[2 * i], v[2 * i + 1], limit);
  } else if (activation == kActReluSquare) {
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const float z = fmaxf(v[i], 0.f);
      v[i] = z * z;
    }
  }
  __nv_bfloat16* dst = row + col;
  if (wide && col + count <= columns) {
#pragma unroll
    for (int i = 0; i < 32; i += 8) {
      if (i >= count) break;
      uint4 packed;
      __nv_bfloat162* pairs = reinterpret_cast<__nv_bfloat162*>(&packed);
#pragma unroll
      for (int j = 0; j < 4; ++j) pairs[j] = __floats2bfloat162_rn(v[i + 2 * j], v[i + 2 * j + 1]);
      *reinterpret_cast<uint4*>(dst + i) = packed;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (i < count && col + i < columns) dst[i] = __float2bfloat16_rn(v[i]);
  }
}

template <int BM, int BN, int STAGES>
__global__ void __launch_bounds__(THREADS, 1)
expert_tcgen05_kernel(const __nv_bfloat16* __restrict__ A, int lda, const int* __restrict__ order, int top,
                      const __grid_constant__ CUtensorMap map_w, __nv_bfloat16* __restrict__ C, int ldc,
                      const int* __restrict__ offsets, int experts, int N, int K, int activation, float limit,
                      const float* __restrict__ pair_scale, int* __restrict__ error_flag) {
  using L = Layout<BM, BN, STAGES>;
  constexpr int ACCUMULATORS = 2;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  int* first_tile = reinterpret_cast<int*>(smem + (size_t)STAGES * L::STAGE_BYTES);        // [experts + 1]
  int* borders = first_tile + experts + 1;                                                 // [experts + 1]
  __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[ACCUMULATORS], acc_empty[ACCUMULATORS];
  __shared__ unsigned tmem_base_s;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_n = (N + BN - 1) / BN, num_k = (K + BK - 1) / BK;

  if (warp == 0 && lane == 0) {
#pragma unroll
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1 + LOADERS);
      mbar_init(&empty_bar[s], 1);
    }
#pragma unroll
    for (int b = 0; b < ACCUMULATORS; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 4);         // one arrival per epilogue warp
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(ACCUMULATORS * BN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  grid_dependency_wait();
  grid_dependency_launch();
  for (int e = threadIdx.x; e <= experts; e += THREADS) borders[e] = offsets[e];
  __syncthreads();
  if (warp == 0) {                          // tiles before each expert's first: a running sum over 32 experts at a time
    int before = 0;
    for (int e0 = 0; e0 < experts; e0 += 32) {
      const int e = e0 + lane;
      int sum = e < experts ? (borders[e + 1] - borders[e] + BM - 1) / BM * tiles_n : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int other = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += other;
      }
      if (e < experts) first_tile[e + 1] = before + sum;
      before += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) first_tile[0] = 0;
  }
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  const unsigned tmem_base = tmem_base_s;
  const int n_tiles = first_tile[experts];
  Walk<BM> walk{first_tile, borders, tiles_n, BN, 0};
  int row0, end, column0;

  if (warp == 0) {
    if (lane == 0) {
      // ---------------- W tiles, one running count of k-blocks over all tiles of this block
      int it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
        walk.at(tile, row0, end, column0);
        const int w_row = walk.expert * N + column0;
        for (int kb = 0; kb < num_k; ++kb, ++it) {
          const int stage = it % STAGES;
          if (!(ok = mbar_wait(&empty_bar[stage], ((it / STAGES) & 1) ^ 1, error_flag, 1))) break;
          mbar_expect_tx(&full_bar[stage], L::B_BYTES);
          tma_load_2d(smem + (size_t)stage * L::STAGE_BYTES + L::A_BYTES, &map_w, &full_bar[stage], kb * BK, w_row);
        }
      }
      if (!ok || *reinterpret_cast<volatile int*>(error_flag) != 0) let_copies_land(full_bar, STAGES, it, error_flag);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ---------------- MMA issue
      constexpr unsigned idesc = umma_idesc(BM, BN);
      int it = 0, done = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x, ++done) {
        const int buf = done % ACCUMULATORS;
        if (!(ok = mbar_wait(&acc_empty[buf], ((done / ACCUMULATORS) & 1) ^ 1, error_flag, 4))) break;
        const unsigned accumulator = tmem_base + buf * BN;
        for (int kb = 0; kb < num_k; ++kb, ++it) {
          const int stage = it % STAGES;
          if (!(ok = mbar_wait(&full_bar[stage], (it / STAGES) & 1, error_flag, 2))) break;
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          tmem_fence_after();
          unsigned char* a_s = smem + (size_t)stage * L::STAGE_BYTES;
          const uint64_t a_desc = umma_desc(a_s), b_desc = umma_desc(a_s + L::A_BYTES);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)      // 16 elements (32 bytes) along K inside the swizzled row: +2 in 16-byte units
            umma_bf16(accumulator, a_desc + 2 * k, b_desc + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
          umma_commit(&empty_bar[stage]);            // the stage is free once these MMAs have read it
        }
        if (ok) umma_commit(&acc_full[buf]);
      }
    }
  } else if (warp >= 6) {
    // ---------------- rows of A: thread l has piece l % 8 (sixteen bytes) of rows l / 8, l / 8 + 16, ... of the tile
    const int l = threadIdx.x - (THREADS - LOADERS), piece = l & 7;
    const unsigned smem_base = smem_u32(smem);
    int it = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
      walk.at(tile, row0, end, column0);
      const __nv_bfloat16* source[BM / 16];
#pragma unroll
      for (int i = 0; i < BM / 16; ++i) {
        const int m = row0 + (l >> 3) + 16 * i;
        source[i] = m < end ? A + (size_t)(order ? order[m] / top : m) * lda + piece * 8 : nullptr;
      }
      for (int kb = 0; kb < num_k; ++kb, ++it) {
        const int stage = it % STAGES;
        if (!(ok = mbar_wait(&empty_bar[stage], ((it / STAGES) & 1) ^ 1, error_flag, 1))) break;
        const unsigned a_s = smem_base + stage * L::STAGE_BYTES;
        const unsigned bytes = kb * BK + piece * 8 < K ? 16u : 0u;          // (zeros behind the inner size)
#pragma unroll
        for (int i = 0; i < BM / 16; ++i) {
          const int r = (l >> 3) + 16 * i;
          if (source[i] != nullptr)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a_s + r * 128 + ((piece ^ (r & 7)) << 4)),
                         "l"(bytes ? source[i] + kb * BK : source[i]), "r"(bytes) : "memory");
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full_bar[stage])) : "memory");
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    // ---------------- epilogue: warps 2..5 own the tensor-memory lane quarters 2, 3, 0, 1; with 64 rows a quarter holds
    // sixteen of them in its first sixteen lanes
    const int quarter = warp & 3, quarter_row = quarter * (BM / 4);
    const bool gated = activation >= kActClampedGlu;
    const int columns = gated ? N / 2 : N;             // of C
    const bool wide = (ldc & 7) == 0 && (columns & 7) == 0 && (reinterpret_cast<size_t>(C) & 15) == 0;
    int done = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++done) {
      walk.at(tile, row0, end, column0);
      const int buf = done % ACCUMULATORS, row = row0 + quarter_row + lane;
      const bool mine = lane < BM / 4 && row < end;
      const float scale = activation == kActSiluGlu && pair_scale && mine ? pair_scale[order[row]] : 1.f;
      ok = ok && mbar_wait(&acc_full[buf], (done / ACCUMULATORS) & 1, error_flag, 3);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tmem_fence_after();
      if (row0 + quarter_row < end) {                            // (a warp without rows reads nothing)
#pragma unroll 1
        for (int c = 0; c < BN; c += 32) {
          if (column0 + c >= N) break;
          float v[32];
          tmem_load_32(tmem_base + ((unsigned)(quarter * 32) << 16) + (unsigned)(buf * BN + c), v);
          if (mine) store_row(v, C + (size_t)row * ldc, column0 + c, columns, activation, limit, scale, wide);
          __syncwarp();                              // (the next read of tensor memory is the whole warp's)
        }
      }
      tmem_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);      // the accumulator may be overwritten
    }
  }

  tmem_fence_before();
  __syncthreads();
  if (warp == 1) {
    tmem_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(ACCUMULATORS * BN) : "memory");
  }
}

template <int BM, int BN, int STAGES>
static int launch(const void* A, int lda, const int* order, int top, const void* W, void* C, int ldc, const int* offsets, int experts,
                  int pairs, int N, int K, int activation, float limit, const float* pair_scale, int* error_flag, cudaStream_t stream) {
  EncodeTiled encode = encode_tiled();
  CUtensorMap map_w;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)experts * N};
  const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
  const cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)BN}, elem[2] = {1, 1};
  MS_REQUIRE(encode != nullptr && encode(&map_w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(W), dims, strides, box, elem,
                                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS,
             "expert_linear: cuTensorMapEncodeTiled failed (%d experts of %d x %d)", experts, N, K);
  auto kernel = expert_tcgen05_kernel<BM, BN, STAGES>;
  const size_t smem = Layout<BM, BN, STAGES>::RING + sizeof(int) * 2 * ((size_t)experts + 1);
  const cudaError_t allowed = allow_shared(kernel, smem);
  if (allowed != cudaSuccess) MS_FAIL("expert_linear: %zu bytes of shared memory refused: %s", smem, cudaGetErrorString(allowed));
  static int sms = 0;
  if (sms == 0) {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms <= 0)
      sms = 148;
  }
  // (every segment may end in a partial tile)
  const long long most = ((long long)pairs / BM + (experts < pairs ? experts : pairs)) * ((N + BN - 1) / BN);
  const cudaError_t e = ms::launch(kernel, dim3((unsigned)(most < sms ? most : sms)), dim3(THREADS), smem, stream, (const __nv_bfloat16*)A, lda,
                                   order, top, map_w, (__nv_bfloat16*)C, ldc, offsets, experts, N, K, activation, limit, pair_scale, error_flag);
  if (e != cudaSuccess) MS_FAIL("expert_linear: launch failed: %s", cudaGetErrorString(e));
  return 0;
}

}  // namespace t5e
}  // namespace ms

using namespace ms;

// Whether ms_expert_linear_tcgen05 takes these sizes (bfloat16): rows of 16-byte pieces, a table of the experts beside the ring.
MS_EXPORT int ms_expert_tcgen05_supports(int experts, int N, int K) {
  return experts >= 1 && experts <= 2048 && K >= 8 && K % 8 == 0 && N >= 8 && N % 8 == 0 && (long long)experts * N < 2147483647LL;
}

// Arguments as ms_expert_linear in bfloat16; A, W and their rows on 16-byte boundaries.  error_flag: one int on the device that a kernel
// which gave up waiting sets.
MS_EXPORT int ms_expert_linear_tcgen05(const void* A, int lda, const int* order, int top, const void* W, void* C, int ldc,
                                       const int* offsets, int experts, int pairs, int N, int K, int activation, float limit,
                                       const float* pair_scale, int* error_flag, cudaStream_t stream) {
  if (pairs == 0 || N == 0 || experts == 0) return 0;
  MS_REQUIRE(ms_expert_tcgen05_supports(experts, N, K) && top > 0 && lda % 8 == 0 && lda >= K, "expert_linear: %d experts of %d x %d, rows of %d",
             experts, N, K, lda);
  MS_REQUIRE(reinterpret_cast<size_t>(A) % 16 == 0 && reinterpret_cast<size_t>(W) % 16 == 0, "expert_linear: operands must be 16-byte aligned");
  MS_REQUIRE(activation >= kActNone && activation <= kActSiluGlu, "expert_linear: activation %d", activation);
  MS_REQUIRE(pair_scale == nullptr || (activation == kActSiluGlu && order != nullptr),
             "expert_linear: a scale per pair goes with the silu-gated activation and gathered rows");
  MS_REQUIRE(error_flag != nullptr, "expert_linear: an error flag on the device is required");
  // Tiles of 128 rows where segments fill them; of 64 where they do not (a deeper ring of W in the room that the rows leave), and of 128
  // columns instead of 256 where even every expert's would leave multiprocessors idle.  Measured (us, first / second product; 128 x
  // 256, 64 x 256, 64 x 128): 2,048 tokens, four of 16 experts of 1,024: 69 / 42, 112 / 65, 187 / 101; 500 tokens: 46 / 30, 38 / 24, 58
  // / 34; 8 tokens, six of 60 experts of 1,408: 71 / 38, 69 / 38, 69 / 42; one token: 26, 26, 24.
  const long long column_tiles = (long long)(experts < pairs ? experts : pairs) * ((N + 255) / 256);
#define MS_EXPERT_TILE(BM, BN, STAGES) \
  return t5e::launch<BM, BN, STAGES>(A, lda, order, top, W, C, ldc, offsets, experts, pairs, N, K, activation, limit, pair_scale, error_flag, stream)
  if (pairs >= 128LL * experts) MS_EXPERT_TILE(128, 256, 4);
  if (column_tiles >= 148) MS_EXPERT_TILE(64, 256, 5);
  MS_EXPERT_TILE(64, 128, 8);
#undef MS_EXPERT_TILE
}
