// Latent attention of prompt portions on the fifth-generation tensor cores.
//
// All heads of a token attend to the same cached rows [c ; k_r], whose first RANK numbers are also the values, so a request's
// query rows (token-major, head-minor) are one matrix Q [tokens * H, RANK + rot] against one key matrix.  A thread block has 128 of
// those rows and walks over the keys in tiles of 64, which lie in shared memory once and serve both products: as K-major
// operand of S = Q K^T (RANK + rot deep) and, their first RANK columns, as MN-major operand of O += P V.  The block is that of
// attention_tcgen05_turns.cu, whose comments on waits by parity hold here too:
//   warp 0       TMA loads, one box of 64 columns per cache page and column block (the last block's columns behind the row are filled with
//                zeros): the query rows once, then the key tiles, a ring of three, free again after a tile's output;
//   warps 1, 3   one thread each issues tcgen05.mma: warp 1 the scores, as far ahead as three score buffers in tensor memory allow, warp 3
//                the outputs, with P read from tensor memory;
//   warps 4..7   softmax of the even tiles, warps 8..11 of the odd ones, a thread a row: mask, running maximum (passed from group to
//                group through shared memory), P over the scores it came from, as two bfloat16 numbers (its rounding and what that
//                leaves); the output is rescaled only when a row's maximum has grown by more than 2^8.
// Bound by the tensor cores: a tile is (RANK + rot) / 16 products of 128 x 64 x 16 (48 clocks each) and four of 128 x RANK x 16 (128
// clocks for 256) for either part of P, 1,888 clocks for a latent of 256 + 32, where the softmax takes two groups about 1,200.  The second part
// costs a third of the time, and is there because the largest probability of a row, relative to a maximum that lags behind, is not
// 1: rounded, it put the layer further from float64 than tiles with the exact maximum do (0.00490 against 0.00488 for the prompt below; with both parts
// 0.00476).  Tiles of 64 keys
// because three of them fit beside the queries: of 128 keys two would, and a tile would be waited for.
// 2,048 tokens of 16 heads, 256 + 32: 225 us on mma.sync (attention_latent_mma.cu), 63 here, 58 with one part of P (36.5 GFLOP of scores and
// one part); the layer, whose eager pass waits for the host, takes 135 to 140 us either way.
// All mbarrier waits are bounded; a wait that runs out sets the error flag and every role drains and returns.
#include "tcgen05.cuh"

namespace ms {
namespace t5l {

using namespace ms::t5;

constexpr int ROWS = 128, BN = 64, THREADS = 384, S_BUFFERS = 3, STAGES = 3;

__device__ __forceinline__ float fast_exp2(float x) {          // ex2.approx: relative error about 2^-22, -inf gives 0
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int RANK>
struct Layout {
  static constexpr int VBLOCKS = RANK / 64, BLOCKS = VBLOCKS + 1;     // column blocks of 64: the values, and the rotated part
  static constexpr int Q_BYTES = ROWS * BLOCKS * 128, TILE_BYTES = BN * BLOCKS * 128;
  static constexpr size_t TOTAL = (size_t)Q_BYTES + (size_t)STAGES * TILE_BYTES + 1024;
  static constexpr int TMEM_COLUMNS = S_BUFFERS * BN + RANK <= 256 ? 256 : 512;
};

template <int RANK>
__global__ void __launch_bounds__(THREADS, 1)
latent_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                      const __grid_constant__ CUtensorMap map_out, const int* __restrict__ block_tables, int table_stride,
                      const int* __restrict__ query_start, const int* __restrict__ context_lens, int page_size, int heads, int dk,
                      float scale_log2, int window, __nv_bfloat16* __restrict__ out, int* __restrict__ error_flag) {
  using L = Layout<RANK>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* q_s = smem;
  auto key_stage = [&](int s) { return smem + L::Q_BYTES + (size_t)s * L::TILE_BYTES; };
  __shared__ uint64_t q_full, k_full[STAGES], k_empty[STAGES];
  __shared__ uint64_t s_full[S_BUFFERS], p_full[S_BUFFERS], s_free[S_BUFFERS];
  // (three score buffers: tile j's scores come behind tile j - 3's output, which the wait by parity for tile j - 1's relies on)
  __shared__ uint64_t pv_done[2], all_done;
  __shared__ uint64_t m_ready[2];
  __shared__ float m_shared[ROWS];
  __shared__ float sums[2][ROWS];
  __shared__ unsigned tmem_base_s;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int request = blockIdx.y;
  const int q0 = query_start[request];
  const int q_len = query_start[request + 1] - q0;
  const int ctx = context_lens[request];
  const int rows_total = q_len * heads;
  const int row0 = ((rows_total + ROWS - 1) / ROWS - 1 - (int)blockIdx.x) * ROWS;   // last tiles, which have the most keys, first
  const bool active = row0 >= 0;
  const int first_pos = ctx - q_len;
  const int t_lo = active ? row0 / heads : 0;
  const int t_hi = active ? (min(rows_total, row0 + ROWS) - 1) / heads : 0;
  int key_begin = 0;
  if (window > 0) key_begin = max(0, first_pos + t_lo - window + 1);
  const int key_end = first_pos + t_hi + 1;
  const int tile_begin = (key_begin / BN) * BN;
  const int n_tiles = active ? (key_end - tile_begin + BN - 1) / BN : 0;
  const int* table = block_tables + (size_t)request * table_stride;

  if (warp == 0 && lane == 0) {
    mbar_init(&q_full, 1);
#pragma unroll
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
    }
#pragma unroll
    for (int b = 0; b < S_BUFFERS; ++b) {
      mbar_init(&s_full[b], 1);
      mbar_init(&p_full[b], ROWS);
      mbar_init(&s_free[b], 1);
    }
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      mbar_init(&pv_done[b], 1);
      mbar_init(&m_ready[b], ROWS);
    }
    mbar_init(&all_done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(L::TMEM_COLUMNS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  const unsigned tmem_base = tmem_base_s;
  auto s_column = [&](int b) { return (unsigned)(b * BN); };
  const unsigned o_column = S_BUFFERS * BN;

  grid_dependency_wait();
  grid_dependency_launch();

  if (warp == 0) {
    if (active) {
      // ---------------- loads: lane 0 announces the bytes, all lanes issue the page loads
      if (lane == 0) {
        mbar_expect_tx(&q_full, L::Q_BYTES);
#pragma unroll
        for (int db = 0; db < L::BLOCKS; ++db)
          tma_load_3d(q_s + db * (ROWS * 128), &map_q, &q_full, db * 64, 0, q0 + t_lo);
      }
      const int box = min(page_size, BN), boxes = BN / box;         // keys of a box, boxes of a tile and column block
      bool ok = true;
      int j = 0;
      for (; j < n_tiles; ++j) {
        const int stage = j % STAGES;
        if (lane == 0) {
          ok = mbar_wait(&k_empty[stage], ((j / STAGES) & 1) ^ 1, error_flag, 31);
          if (ok) mbar_expect_tx(&k_full[stage], L::TILE_BYTES);
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (!ok) break;
        const int key0 = tile_begin + j * BN;
        for (int i = lane; i < boxes * L::BLOCKS; i += 32) {
          const int p = i / L::BLOCKS, db = i % L::BLOCKS, key = key0 + p * box;
          // pages past the context are replaced by the request's first page: finite numbers that the mask removes
          const int row = key < key_end ? table[key / page_size] * page_size + key % page_size : table[0] * page_size;
          tma_load_2d(key_stage(stage) + (size_t)db * (BN * 128) + (size_t)(p * box) * 128, &map_k, &k_full[stage], db * 64, row);
        }
      }
      if (lane == 0 && (!ok || *reinterpret_cast<volatile int*>(error_flag) != 0)) {
        let_copies_land(&q_full, 1, 1, error_flag);
        let_copies_land(k_full, STAGES, j, error_flag);
      }
    }
  } else if (warp == 1) {
    if (active) {
      // ---------------- MMA issue, scores: one thread; the warp clears what the last tile holds behind the context (a page's stale
      // rows, whose probability is zero, but zero times an infinity is not)
      constexpr unsigned idesc_s = umma_idesc(ROWS, BN, false);
      constexpr uint64_t TILE_UNITS = L::TILE_BYTES / 16, Q_BLOCK = (ROWS * 128) / 16, K_BLOCK = (BN * 128) / 16;
      const uint64_t q_desc = umma_desc(q_s), k_desc = umma_desc(key_stage(0));
      const int steps = dk / 16;
      bool ok = true;
      if (lane == 0) ok = mbar_wait(&q_full, 0, error_flag, 32);
      for (int j = 0; j < n_tiles; ++j) {
        const int stage = j % STAGES, b = j % S_BUFFERS;
        if (lane == 0) {
          if (ok && j >= S_BUFFERS) ok = mbar_wait(&s_free[b], (unsigned)(j / S_BUFFERS - 1) & 1u, error_flag, 33);
          ok = ok && mbar_wait(&k_full[stage], (j / STAGES) & 1, error_flag, 34);
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (!ok) break;
        const int behind = key_end - (tile_begin + j * BN);        // rows of this tile from here on are no keys
        if (behind < BN) {
          for (int i = lane; i < (BN - behind) * L::BLOCKS * 8; i += 32) {
            const int row = behind + i / (L::BLOCKS * 8), piece = i % (L::BLOCKS * 8);
            *reinterpret_cast<uint4*>(key_stage(stage) + (size_t)(piece / 8) * (BN * 128) + row * 128 + piece % 8 * 16) = make_uint4(0u, 0u, 0u, 0u);
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
        }
        if (lane == 0) {
          tmem_fence_after();
          const uint64_t keys = k_desc + (uint64_t)stage * TILE_UNITS;
          const unsigned scores = tmem_base + s_column(b);
#pragma unroll 4
          for (int kk = 0; kk < steps; ++kk)
            umma_bf16(scores, q_desc + (kk / 4) * Q_BLOCK + 2 * (kk % 4), keys + (kk / 4) * K_BLOCK + 2 * (kk % 4), idesc_s, kk != 0 ? 1u : 0u);
          umma_commit(&s_full[b]);
        }
        __syncwarp();
      }
    }
  } else if (warp == 3) {
    if (active && lane == 0) {
      // ---------------- MMA issue, outputs
      constexpr unsigned idesc_pv = umma_idesc(ROWS, RANK, true);
      constexpr uint64_t TILE_UNITS = L::TILE_BYTES / 16;
      const uint64_t v_desc = umma_desc_mn_major(key_stage(0), BN * 128);
      bool ok = true;
      for (int j = 0; j < n_tiles && ok; ++j) {
        const int stage = j % STAGES, b = j % S_BUFFERS;
        ok = mbar_wait(&p_full[b], (j / S_BUFFERS) & 1, error_flag, 35) &&
             mbar_wait(&k_full[stage], (j / STAGES) & 1, error_flag, 36);      // (long there: the scores came from it)
        if (!ok) break;
        tmem_fence_after();
        const uint64_t values = v_desc + (uint64_t)stage * TILE_UNITS;
        const unsigned p = tmem_base + s_column(b);
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk)      // sixteen keys further: 16 rows of 128 bytes, 8 columns of packed P
          umma_bf16_a_tmem(tmem_base + o_column, p + kk * 8, values + kk * (16 * 128 / 16), idesc_pv, (j | kk) != 0 ? 1u : 0u);
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk)      // and what rounding has left of P
          umma_bf16_a_tmem(tmem_base + o_column, p + BN / 2 + kk * 8, values + kk * (16 * 128 / 16), idesc_pv, 1u);
        umma_commit(&pv_done[j & 1]);
        umma_commit(&s_free[b]);
        umma_commit(&k_empty[stage]);
        if (j == n_tiles - 1) umma_commit(&all_done);
      }
    }
  } else if (warp >= 4) {
    if (active) {
      // ---------------- softmax and output: one thread per query row, the two groups take the key tiles in turn
      const int quarter = warp & 3, turn = warp >= 8 ? 1 : 0;
      const int local_row = quarter * 32 + lane;
      const int row = row0 + local_row;
      const int pos = first_pos + row / heads;
      const unsigned lane_field = (unsigned)(quarter * 32) << 16;
      const unsigned o_addr = tmem_base + lane_field + o_column;
      float m_mine = -INFINITY;      // the maximum this thread's sum is relative to
      float l = 0.f;                 // the sum over this group's tiles
      bool ok = true;
      for (int j = turn; j < n_tiles; j += 2) {
        const int b = j % S_BUFFERS;
        const unsigned s_addr = tmem_base + lane_field + s_column(b);
        const int key0 = tile_begin + j * BN;
        const bool full = (key0 + BN - 1 <= first_pos + t_lo) && (window <= 0 || key0 >= first_pos + t_hi - window + 1);
        ok = ok && mbar_wait(&s_full[b], (j / S_BUFFERS) & 1, error_flag, 38);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tmem_fence_after();
        float v[BN];
#pragma unroll
        for (int c = 0; c < BN; c += 32) tmem_load_32_nowait(s_addr + c, *reinterpret_cast<float(*)[32]>(&v[c]));
        tmem_load_wait();
        // eight independent partial maxima (and sums below): a single running value would chain 128 operations
        float part_max[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) part_max[e] = -INFINITY;
        if (full) {
#pragma unroll
          for (int i = 0; i < BN; ++i) part_max[i & 7] = fmaxf(part_max[i & 7], v[i]);
        } else {
          // key key0 + i is visible to this row if first <= i <= last (causal: last = pos - key0; a window cuts
          // below): one subtraction and one unsigned comparison per score
          const int last = pos - key0;
          const int first = window > 0 ? max(0, pos - window + 1 - key0) : 0;
          const int below = last >= first ? -first : -(1 << 20);           // (nothing visible: no i passes)
          const unsigned span = last >= first ? (unsigned)(last - first) : 0u;
#pragma unroll
          for (int i = 0; i < BN; ++i) {
            if ((unsigned)(i + below) > span) v[i] = -INFINITY;
            part_max[i & 7] = fmaxf(part_max[i & 7], v[i]);
          }
        }
        const float tile_max = fmaxf(fmaxf(fmaxf(part_max[0], part_max[1]), fmaxf(part_max[2], part_max[3])),
                                     fmaxf(fmaxf(part_max[4], part_max[5]), fmaxf(part_max[6], part_max[7])));
        // the maximum in use after the tile before (which the other group has worked on, or is still working on)
        float m_used = -INFINITY;
        if (j > 0) {
          ok = mbar_wait(&m_ready[turn ^ 1], ((j - 1) / 2) & 1, error_flag, 41);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          m_used = m_shared[local_row];
        }
        const float candidate = fmaxf(m_used, tile_max);
        // the output is rescaled when the maximum has grown by more than 8 in the exponent (or was still -inf)
        const bool grow = candidate != -INFINITY && (m_used == -INFINITY || (candidate - m_used) * scale_log2 > 8.f);
        if (__any_sync(0xffffffffu, grow)) {
          const float factor = grow ? (m_used == -INFINITY ? 0.f : exp2f((m_used - candidate) * scale_log2)) : 1.f;
          if (j > 0) {
            // the output must be complete up to tile j - 1 (tile j - 3's is: this tile's scores came behind it)
            ok = mbar_wait(&pv_done[(j - 1) & 1], ((j - 1) / 2) & 1, error_flag, 39);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tmem_fence_after();
#pragma unroll 1
            for (int c = 0; c < RANK; c += 32) {
              float o[32];
              tmem_load_32(o_addr + c, o);
              unsigned scaled[32];
#pragma unroll
              for (int i = 0; i < 32; ++i) scaled[i] = __float_as_uint(o[i] * factor);
              tmem_store_32(o_addr + c, scaled);
            }
            tmem_store_wait();
          }
          if (grow) m_used = candidate;
        }
        m_shared[local_row] = m_used;
        mbar_arrive(&m_ready[turn]);               // (the group of tile j + 1 may go on)
        // this group's sum follows the maximum in use
        if (m_used != m_mine) {
          l *= m_mine == -INFINITY ? 0.f : exp2f((m_mine - m_used) * scale_log2);
          m_mine = m_used;
        }
        const float base = m_used == -INFINITY ? 0.f : m_used * scale_log2;
        float part_sum[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) part_sum[e] = 0.f;
#pragma unroll
        for (int c = 0; c < BN; c += 32) {
          unsigned packed[16], rest[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float p0 = fast_exp2(v[c + i] * scale_log2 - base);
            const float p1 = fast_exp2(v[c + i + 1] * scale_log2 - base);
            const __nv_bfloat162 two = __floats2bfloat162_rn(p0, p1);
            packed[i / 2] = *reinterpret_cast<const unsigned*>(&two);
            part_sum[(i >> 1) & 7] += p0 + p1;
            const __nv_bfloat162 left = __floats2bfloat162_rn(p0 - __uint_as_float(packed[i / 2] << 16),
                                                              p1 - __uint_as_float(packed[i / 2] & 0xffff0000u));
            rest[i / 2] = *reinterpret_cast<const unsigned*>(&left);
          }
          tmem_store_16(s_addr + c / 2, packed);
          tmem_store_16(s_addr + BN / 2 + c / 2, rest);
        }
        tmem_store_wait();
        tmem_fence_before();
        mbar_arrive(&p_full[b]);
        l += ((part_sum[0] + part_sum[1]) + (part_sum[2] + part_sum[3])) + ((part_sum[4] + part_sum[5]) + (part_sum[6] + part_sum[7]));
      }
      // All 256 threads pass these barriers together; they also tell everyone whether anyone gave up a wait.
      auto all_ok = [](bool mine) {
        unsigned result;
        asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbar.red.and.pred q, 1, 256, p;\nselp.u32 %0, 1, 0, q;\n}"
                     : "=r"(result) : "r"((unsigned)mine) : "memory");
        return result != 0;
      };
      // every output is complete (a barrier that completes once: nothing to tell apart)
      if (ok) ok = mbar_wait(&all_done, 0u, error_flag, 40);
      ok = __all_sync(0xffffffffu, ok);
      ok = all_ok(ok);                  // every maximum is final
      const float m_final = m_shared[local_row];
      if (m_mine != m_final) l *= m_mine == -INFINITY ? 0.f : exp2f((m_mine - m_final) * scale_log2);
      sums[turn][local_row] = l;
      if (all_ok(ok)) {
        tmem_fence_after();
        l = sums[0][local_row] + sums[1][local_row];                  // the same sum in either thread of the row
        const float inv = l > 0.f ? 1.f / l : 0.f;
        // Each of the row's two threads takes half of its columns.  A whole tile goes through the shared memory of
        // the queries (no longer needed; the same layout) and leaves by TMA in whole lines: a thread storing its
        // own row touches 32 lines per instruction, 1,700 cycles for the tile.  A tile that the request's rows do not
        // fill is stored by its threads (what lies behind the rows belongs to the next request).
        const bool whole = row0 + ROWS <= rows_total;
        __nv_bfloat16* dst = out + ((size_t)q0 * heads + row) * RANK + turn * (RANK / 2);
#pragma unroll 1
        for (int c = 0; c < RANK / 2; c += 32) {
          float o[32];
          tmem_load_32(o_addr + turn * (RANK / 2) + c, o);
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint4 packed;
            __nv_bfloat162* pairs = reinterpret_cast<__nv_bfloat162*>(&packed);
#pragma unroll
            for (int e = 0; e < 4; ++e) pairs[e] = __floats2bfloat162_rn(o[i + 2 * e] * inv, o[i + 2 * e + 1] * inv);
            if (whole) {
              const int column = turn * (RANK / 2) + c + i;          // of the row: 128-byte block column / 64, 16-byte piece within
              *reinterpret_cast<uint4*>(q_s + (column / 64) * (ROWS * 128) + local_row * 128 + ((((column % 64) / 8) ^ (local_row & 7)) << 4)) = packed;
            } else if (row < rows_total) {
              *reinterpret_cast<uint4*>(dst + c + i) = packed;
            }
          }
        }
        if (whole) {
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          all_ok(true);                                   // the tile is in shared memory
          if (warp == 4 && lane == 0) {
#pragma unroll
            for (int db = 0; db < L::VBLOCKS; ++db)
              asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
                           ::"l"(reinterpret_cast<uint64_t>(&map_out)), "r"(smem_u32(q_s + db * (ROWS * 128))), "r"(db * 64),
                             "r"(0), "r"(q0 + t_lo) : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");      // shared memory has been read before the block ends
          }
        }
      }
    }
  }

  tmem_fence_before();
  __syncthreads();
  if (warp == 1) {
    tmem_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(L::TMEM_COLUMNS) : "memory");
  }
}

static bool encode(CUtensorMap* map, int rank, const void* base, const cuuint64_t* dims, const cuuint64_t* strides,
                   const cuuint32_t* box) {
  EncodeTiled fn = encode_tiled();
  if (fn == nullptr) return false;
  const cuuint32_t elem[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(base), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int RANK>
int launch(const void* q, const void* cache, int n_pages, const int* block_tables, int table_stride, const int* query_start,
           const int* context_lens, int page_size, int heads, int rot, float scale, int window, void* out, int n_requests,
           int max_query_len, int n_tokens, int* error_flag, cudaStream_t stream) {
  const int dk = RANK + rot;
  CUtensorMap map_q, map_k, map_out;
  {
    const cuuint64_t dims[3] = {(cuuint64_t)dk, (cuuint64_t)heads, (cuuint64_t)n_tokens}, out_dims[3] = {RANK, dims[1], dims[2]};
    const cuuint64_t strides[2] = {(cuuint64_t)dk * 2, (cuuint64_t)heads * dk * 2}, out_strides[2] = {RANK * 2, (cuuint64_t)heads * RANK * 2};
    const cuuint32_t box[3] = {64, (cuuint32_t)heads, (cuuint32_t)(ROWS / heads)};
    MS_REQUIRE(encode(&map_q, 3, q, dims, strides, box) && encode(&map_out, 3, out, out_dims, out_strides, box),
               "latent_attention: tensor map of the queries or of the output failed");
  }
  {
    const cuuint64_t dims[2] = {(cuuint64_t)dk, (cuuint64_t)n_pages * page_size};
    const cuuint64_t strides[1] = {(cuuint64_t)dk * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)(page_size < BN ? page_size : BN)};
    MS_REQUIRE(encode(&map_k, 2, cache, dims, strides, box), "latent_attention: tensor map of the cache failed");
  }
  auto kernel = latent_tcgen05_kernel<RANK>;
  const cudaError_t allowed = allow_shared(kernel, Layout<RANK>::TOTAL);
  if (allowed != cudaSuccess) MS_FAIL("latent_attention: %zu bytes of shared memory refused: %s", Layout<RANK>::TOTAL, cudaGetErrorString(allowed));
  const long long tiles = ((long long)max_query_len * heads + ROWS - 1) / ROWS;
  MS_REQUIRE(tiles <= 2147483647LL && n_requests <= 65535, "latent_attention: grid exceeds the launch limits");
  const cudaError_t e = ms::launch(kernel, dim3((unsigned)tiles, n_requests), dim3(THREADS), Layout<RANK>::TOTAL, stream, map_q, map_k, map_out,
                                   block_tables, table_stride, query_start, context_lens, page_size, heads, dk, scale * 1.4426950408889634f,
                                   window, (__nv_bfloat16*)out, error_flag);
  if (e != cudaSuccess) MS_FAIL("latent_attention: launch failed: %s", cudaGetErrorString(e));
  return 0;
}

}  // namespace t5l
}  // namespace ms

using namespace ms;

// Whether ms_latent_attention_tcgen05 takes these sizes: a latent of 64, 128 or 256 numbers, a rotated part of at most 64 that is a
// multiple of 16, heads that fill rows of 128 evenly, pages that fill tiles of 64 keys or are filled by them.
MS_EXPORT int ms_latent_attention_tcgen05_supports(int rank, int rot, int heads, int page_size) {
  return (rank == 64 || rank == 128 || rank == 256) && rot >= 0 && rot <= 64 && rot % 16 == 0 && heads >= 1 && heads <= 128 && 128 % heads == 0 &&
         page_size >= 8 && (page_size <= 64 ? 64 % page_size == 0 : page_size % 64 == 0);
}

// q_full [n_tokens, heads, rank + rot] and out [n_tokens, heads, rank] bfloat16; cache [n_pages, page_size, rank + rot]; all on 16-byte
// boundaries.  error_flag: one int on the device that a kernel which gave up waiting sets.
MS_EXPORT int ms_latent_attention_tcgen05(const void* q_full, const void* cache, int n_pages, const int* block_tables, int table_stride,
                                          const int* query_start, const int* context_lens, int page_size, int heads, int rank, int rot,
                                          float scale, int window, void* out, int n_requests, int max_query_len, int n_tokens,
                                          int* error_flag, cudaStream_t stream) {
  if (n_tokens == 0 || n_requests == 0) return 0;
  MS_REQUIRE(ms_latent_attention_tcgen05_supports(rank, rot, heads, page_size), "latent_attention: %d + %d, %d heads, pages of %d are not taken",
             rank, rot, heads, page_size);
  MS_REQUIRE(max_query_len > 0 && error_flag != nullptr, "latent_attention: longest portion %d, an error flag on the device is required", max_query_len);
  MS_REQUIRE(((reinterpret_cast<size_t>(q_full) | reinterpret_cast<size_t>(cache) | reinterpret_cast<size_t>(out)) & 15) == 0,
             "latent_attention: operands must be 16-byte aligned");
  auto launch = rank == 64 ? t5l::launch<64> : rank == 128 ? t5l::launch<128> : t5l::launch<256>;
  return launch(q_full, cache, n_pages, block_tables, table_stride, query_start, context_lens, page_size, heads, rot, scale, window, out,
                n_requests, max_query_len, n_tokens, error_flag, stream);
}
