// Latent attention of decode steps (one token a request) for a latent of 256 numbers: bfloat16, mma.sync.m16n8k16, float32 scores and
// sums.  A request brings H query rows, at most sixteen to a block, against all its cached rows [c ; k_r], whose first 256 numbers are
// also the values: 36 products of 16 x 8 x 16 for sixteen keys of 9 KB, so what a step costs is the cache's way from memory, if
// nothing stands in it.
//
// A block has four warps that share nothing on the way: each takes every fourth piece of sixteen keys of the block's range, with the
// queries' fragments (72 registers for 256 + 32) and its own output of 16 x 256 (128 registers) in registers, and a ring of three
// pieces of its own (two for 256 + 64), the others on their way while one is multiplied.  A piece comes by one bulk copy a row (cp.async.bulk, sixteen
// instructions; rows lie sixteen bytes apart from one another's banks), counted by a barrier.  The probabilities go from the
// scores' registers to the second product's operand without leaving the warp; the output is rescaled only when a row's maximum has
// grown by more than 2^8.  At the end the four outputs meet in shared memory.  (No row is asked for before the wait for the kernel before: a
// caller may have written all of them just now.)
// (Four warps that share each piece of 32 keys meet three times for it, and fetch the queries' fragments again each time: a piece's
// chain of some 2,900 clocks, not the memory, set the pace.)
// 32 requests of 16 heads and some 7,200 keys (147 MB): 49 us that way, 35.5 here.
#include "attention_latent_tiles.cuh"
#include "tcgen05.cuh"

namespace ms {
namespace latent_decode {

constexpr int DV = 256, WARPS = 4, KEYS = 16, UNIT = WARPS * KEYS, OLD = DV + 4;
constexpr int TILE_BUFFERS = 4;        // of attention_latent_tiles.cuh

// Pieces of a warp's ring: as many as let two blocks share a multiprocessor (three with a rotated part of 64 would not).
__host__ __device__ constexpr int stages_of(int nkc) { return nkc <= 18 ? 3 : 2; }
constexpr size_t smem_bytes(int nkc) {
  const size_t rings = (size_t)WARPS * stages_of(nkc) * KEYS * (nkc * 32 + 16), tiles = latent_tiles_smem(WARPS, TILE_BUFFERS, nkc * 16);
  return rings > tiles ? rings : tiles;
}

// NKC: steps of 16 along a row of (256 + rot) numbers.
template <int NKC>
__global__ void __launch_bounds__(32 * WARPS, 2)
latent_decode_kernel(const __nv_bfloat16* __restrict__ q_full, const __nv_bfloat16* __restrict__ cache,
                     const int* __restrict__ block_tables, int table_stride, const int* __restrict__ query_start,
                     const int* __restrict__ context_lens, int page_size, int heads, float scale_log2, int window,
                     __nv_bfloat16* __restrict__ out, float* __restrict__ part_o, float* __restrict__ part_lse, int splits,
                     int ranges, int least, int tile_ranges, int* __restrict__ error_flag) {
  constexpr int DK = NKC * 16, ROW = NKC * 32 + 16, STAGE = KEYS * ROW, STAGES = stages_of(NKC);
  extern __shared__ __align__(128) unsigned char decode_smem[];
  __shared__ uint64_t full[WARPS][STAGES];
  __shared__ float peaks[WARPS][16], sums[WARPS][16];
  grid_dependency_wait();
  grid_dependency_launch();
  const int req = blockIdx.y, split = blockIdx.z;
  const int q0 = query_start[req], q_len = query_start[req + 1] - q0, ctx = context_lens[req];
  const int rows = q_len * heads, m0 = blockIdx.x * 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (m0 >= rows) return;
  if ((window > 0 ? min(ctx, window) : ctx) < least) {
    latent_decode_tiles<DV, WARPS, TILE_BUFFERS>(q_full, cache, block_tables, table_stride, query_start, context_lens, page_size, heads, DK,
                                                 scale_log2, window, out, part_o, part_lse, splits, tile_ranges, decode_smem);
    return;
  }
  const int* table = block_tables + (size_t)req * table_stride;
  const int pos_last = ctx - q_len + (min(m0 + 16, rows) - 1) / heads, pos_first = ctx - q_len + m0 / heads;
  const int key_begin = window > 0 ? max(0, pos_first - window + 1) : 0;
  const int unit_begin = key_begin / UNIT, unit_end = pos_last / UNIT + 1;
  const int per_split = (unit_end - unit_begin + ranges - 1) / ranges;
  const int first_unit = unit_begin + split * per_split, units = min(unit_end, first_unit + per_split) - first_unit;
  if (units <= 0 && splits > 1) {                // a range behind the request's keys: the merge reads no more of it than this
    if (threadIdx.x < 16 && m0 + threadIdx.x < rows) part_lse[((size_t)q0 * heads + m0 + threadIdx.x) * splits + split] = -INFINITY;
    return;
  }
  const int first_key = first_unit * UNIT + warp * KEYS;
  // this warp's pieces: first_key, first_key + 64, ...
  const int pieces = units <= 0 ? 0 : units - (first_key + (units - 1) * UNIT > pos_last ? 1 : 0);
  unsigned char* ring = decode_smem + (size_t)warp * STAGES * STAGE;
  if (lane == 0) {
#pragma unroll
    for (int s = 0; s < STAGES; ++s) t5::mbar_init(&full[warp][s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  auto request = [&](int i) {
    const int key0 = first_key + i * UNIT, count = min(KEYS, pos_last + 1 - key0);
    unsigned char* stage = ring + (i % STAGES) * STAGE;
    uint64_t* bar = &full[warp][i % STAGES];
    if (lane == 0) t5::mbar_expect_tx(bar, (unsigned)(count * DK * 2));
    __syncwarp();
    if (lane < count) {
      const int key = key0 + lane;
      const __nv_bfloat16* row = cache + ((size_t)table[key / page_size] * page_size + key % page_size) * DK;
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                   ::"r"(t5::smem_u32(stage + lane * ROW)), "l"(row), "r"(DK * 2), "r"(t5::smem_u32(bar)) : "memory");
    }
    if (count < KEYS) {                                                          // behind the context: zeros
      for (int j = count * (ROW / 16) + lane; j < KEYS * (ROW / 16); j += 32) *reinterpret_cast<uint4*>(stage + j * 16) = make_uint4(0u, 0u, 0u, 0u);
      __syncwarp();                                                              // (other lanes read them; the copies' barrier does not order them)
    }
  };
#pragma unroll
  for (int i = 0; i < STAGES - 1; ++i)
    if (i < pieces) request(i);

  const int row_a = m0 + (lane >> 2), row_b = row_a + 8;
  unsigned q[NKC][4];
  {
    const __nv_bfloat16* at = q_full + (size_t)q0 * heads * DK + (lane & 3) * 2;
#pragma unroll
    for (int kc = 0; kc < NKC; ++kc) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = e & 1 ? row_b : row_a;
        q[kc][e] = row < rows && pieces > 0 ? *reinterpret_cast<const unsigned*>(at + (size_t)row * DK + kc * 16 + (e >> 1) * 8) : 0u;
      }
    }
  }
  const int pos_a = row_a < rows ? ctx - q_len + row_a / heads : -1;     // -1: no key is visible (a row beyond the request's)
  const int pos_b = row_b < rows ? ctx - q_len + row_b / heads : -1;
  const int low_a = window > 0 ? pos_a - window : -2147483647, low_b = window > 0 ? pos_b - window : -2147483647;
  float m_a = -INFINITY, m_b = -INFINITY, l_a = 0.f, l_b = 0.f;
  float o[DV / 8][4];
#pragma unroll
  for (int i = 0; i < DV / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;

  for (int i = 0; i < pieces; ++i) {
    const bool ok = t5::mbar_wait(&full[warp][i % STAGES], (i / STAGES) & 1, error_flag, 51);
    if (!__all_sync(0xffffffffu, ok)) {
      t5::let_copies_land(full[warp], STAGES, min(pieces, i + STAGES - 1), error_flag);
      break;
    }
    if (i + STAGES - 1 < pieces) request(i + STAGES - 1);                // (its stage's last reads lie before this wait)
    const unsigned char* kt = ring + (i % STAGES) * STAGE;
    float s[2][4], s_odd[2][4];                                          // two chains of products, added at the end
#pragma unroll
    for (int n = 0; n < 2; ++n) s[n][0] = s[n][1] = s[n][2] = s[n][3] = s_odd[n][0] = s_odd[n][1] = s_odd[n][2] = s_odd[n][3] = 0.f;
#pragma unroll
    for (int kc = 0; kc < NKC; ++kc) {
      unsigned b[4];
      ldmatrix_x4(b, kt + ((lane & 7) + (lane >> 4) * 8) * ROW + kc * 32 + ((lane >> 3) & 1) * 16);
      mma_bf16(kc & 1 ? s_odd[0] : s[0], q[kc], b[0], b[1]);
      mma_bf16(kc & 1 ? s_odd[1] : s[1], q[kc], b[2], b[3]);
    }
    const int key0 = first_key + i * UNIT;
    float max_a = -INFINITY, max_b = -INFINITY;
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int key = key0 + n * 8 + (lane & 3) * 2 + e;
        s[n][e] = (key <= pos_a && key > low_a) ? (s[n][e] + s_odd[n][e]) * scale_log2 : -INFINITY;
        s[n][2 + e] = (key <= pos_b && key > low_b) ? (s[n][2 + e] + s_odd[n][2 + e]) * scale_log2 : -INFINITY;
        max_a = fmaxf(max_a, s[n][e]);
        max_b = fmaxf(max_b, s[n][2 + e]);
      }
    max_a = fmaxf(max_a, __shfl_xor_sync(0xffffffffu, max_a, 1));
    max_a = fmaxf(max_a, __shfl_xor_sync(0xffffffffu, max_a, 2));
    max_b = fmaxf(max_b, __shfl_xor_sync(0xffffffffu, max_b, 1));
    max_b = fmaxf(max_b, __shfl_xor_sync(0xffffffffu, max_b, 2));
    const bool grow_a = max_a > m_a + 8.f, grow_b = max_b > m_b + 8.f;   // (anything above minus infinity + 8)
    if (__any_sync(0xffffffffu, grow_a || grow_b)) {
      const float factor_a = grow_a ? exp2f(m_a - max_a) : 1.f, factor_b = grow_b ? exp2f(m_b - max_b) : 1.f;
      if (grow_a) m_a = max_a;
      if (grow_b) m_b = max_b;
      l_a *= factor_a, l_b *= factor_b;
#pragma unroll
      for (int n = 0; n < DV / 8; ++n) o[n][0] *= factor_a, o[n][1] *= factor_a, o[n][2] *= factor_b, o[n][3] *= factor_b;
    }
    const float use_a = m_a == -INFINITY ? 0.f : m_a, use_b = m_b == -INFINITY ? 0.f : m_b;      // (nothing seen yet: all p are 0)
    unsigned p[4];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const float p0 = exp2f(s[n][0] - use_a), p1 = exp2f(s[n][1] - use_a), p2 = exp2f(s[n][2] - use_b), p3 = exp2f(s[n][3] - use_b);
      p[2 * n] = pack_bf16(p0, p1);
      p[2 * n + 1] = pack_bf16(p2, p3);
      // (the sum is that of the rounded ones: relative to a maximum that may lag behind, the largest is not 1, and its rounding would
      // scale the whole output)
      l_a += __uint_as_float(p[2 * n] << 16) + __uint_as_float(p[2 * n] & 0xffff0000u);
      l_b += __uint_as_float(p[2 * n + 1] << 16) + __uint_as_float(p[2 * n + 1] & 0xffff0000u);
    }
#pragma unroll
    for (int np = 0; np < DV / 16; ++np) {
      unsigned b[4];
      ldmatrix_x4_trans(b, kt + ((lane & 7) + ((lane >> 3) & 1) * 8) * ROW + np * 32 + (lane >> 4) * 16);
      mma_bf16(o[2 * np], p, b[0], b[1]);
      mma_bf16(o[2 * np + 1], p, b[2], b[3]);
    }
    __syncwarp();                                                        // every lane has read this stage
  }

  // the four warps' outputs meet: relative to the largest maximum, added in warp order
  l_a += __shfl_xor_sync(0xffffffffu, l_a, 1);
  l_a += __shfl_xor_sync(0xffffffffu, l_a, 2);
  l_b += __shfl_xor_sync(0xffffffffu, l_b, 1);
  l_b += __shfl_xor_sync(0xffffffffu, l_b, 2);
  if ((lane & 3) == 0) {
    peaks[warp][lane >> 2] = m_a, peaks[warp][(lane >> 2) + 8] = m_b;
    sums[warp][lane >> 2] = l_a, sums[warp][(lane >> 2) + 8] = l_b;
  }
  __syncthreads();                                                       // (and every warp is done with its ring)
  auto together = [&](int row, float& top) {                             // the row's sum relative to its largest maximum
    top = fmaxf(fmaxf(peaks[0][row], peaks[1][row]), fmaxf(peaks[2][row], peaks[3][row]));
    float l = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) l += top == -INFINITY ? 0.f : sums[w][row] * exp2f(peaks[w][row] - top);
    return l;
  };
  float top_a, top_b;
  const float total_a = together(lane >> 2, top_a), total_b = together((lane >> 2) + 8, top_b);
  const float factor_a = total_a > 0.f ? exp2f(m_a - top_a) / total_a : 0.f, factor_b = total_b > 0.f ? exp2f(m_b - top_b) / total_b : 0.f;
  float* meet = reinterpret_cast<float*>(decode_smem);                   // [WARPS][16][OLD]
#pragma unroll
  for (int n = 0; n < DV / 8; ++n) {
    float* at = meet + (warp * 16 + (lane >> 2)) * OLD + n * 8 + (lane & 3) * 2;
    *reinterpret_cast<float2*>(at) = make_float2(o[n][0] * factor_a, o[n][1] * factor_a);
    *reinterpret_cast<float2*>(at + 8 * OLD) = make_float2(o[n][2] * factor_b, o[n][3] * factor_b);
  }
  __syncthreads();
  for (int j = threadIdx.x; j < 16 * (DV / 4); j += 32 * WARPS) {
    const int row = j / (DV / 4), c = j % (DV / 4) * 4;
    if (m0 + row >= rows) break;
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float4 part = *reinterpret_cast<const float4*>(meet + (w * 16 + row) * OLD + c);
      sum.x += part.x, sum.y += part.y, sum.z += part.z, sum.w += part.w;
    }
    const size_t item = (size_t)q0 * heads + m0 + row;
    if (splits == 1) {
      uint2 packed;
      packed.x = pack_bf16(sum.x, sum.y), packed.y = pack_bf16(sum.z, sum.w);
      *reinterpret_cast<uint2*>(out + item * DV + c) = packed;
    } else {
      *reinterpret_cast<float4*>(part_o + (item * splits + split) * DV + c) = sum;
      if (c == 0) {
        float top;
        const float total = together(row, top);
        part_lse[item * splits + split] = total > 0.f ? top + log2f(total) : -INFINITY;
      }
    }
  }
}

template <int NKC>
static int launch(const void* q_full, const void* cache, const int* block_tables, int table_stride, const int* query_start,
                  const int* context_lens, int page_size, int heads, float scale, int window, void* out, float* part_o, float* part_lse,
                  int splits, int ranges, int least, int tile_ranges, int n_requests, int* error_flag, cudaStream_t stream) {
  static_assert(2 * (smem_bytes(NKC) + 2048) <= 228 * 1024, "the ranges are chosen for two blocks a multiprocessor");
  auto kernel = latent_decode_kernel<NKC>;
  const cudaError_t e = allow_shared(kernel, smem_bytes(NKC));
  if (e != cudaSuccess) MS_FAIL("latent_decode: %zu bytes of shared memory refused: %s", smem_bytes(NKC), cudaGetErrorString(e));
  ms::launch(kernel, dim3((heads + 15) / 16, n_requests, splits), 32 * WARPS, smem_bytes(NKC), stream, (const __nv_bfloat16*)q_full,
             (const __nv_bfloat16*)cache, block_tables, table_stride, query_start, context_lens, page_size, heads,
             scale * 1.4426950408889634f, window, (__nv_bfloat16*)out, part_o, part_lse, splits, ranges, least, tile_ranges, error_flag);
  MS_CHECK_LAUNCH("latent_decode");
  return 0;
}

}  // namespace latent_decode
}  // namespace ms

using namespace ms;

// Whether ms_latent_decode takes these sizes: a latent of 256 numbers and a rotated part of 0, 32 or 64 (the queries' fragments lie in
// registers, whose number is fixed when the kernel is built).
MS_EXPORT int ms_latent_decode_supports(int rank, int rot, int heads) {
  return rank == 256 && (rot == 0 || rot == 32 || rot == 64) && heads >= 1 && heads <= 65535;
}

// How many ranges the keys are cut into: the number whose blocks, in rounds of two a multiprocessor, take the fewest units of 64 keys,
// what a block costs beside them (about four units) and what a range more costs the merge included; at least two units a range, at most
// 32 ranges.
MS_EXPORT int ms_latent_decode_splits(int heads, int n_requests, int max_context_len) {
  constexpr int kUnit = latent_decode::UNIT;
  const long long rows = (long long)n_requests * ((heads + 15) / 16), slots = 2 * 148;
  const int units = max_context_len / kUnit + 1, by_keys = (max_context_len + 2 * kUnit - 1) / (2 * kUnit);
  const int most = by_keys < 32 ? by_keys : 32;
  int best = 1;
  long long least = -1;
  for (int splits = 1; splits <= most; ++splits) {
    const long long cost = 8 * ((rows * splits + slots - 1) / slots) * ((units + splits - 1) / splits + 4) + splits;
    if (least < 0 || cost < least) best = splits, least = cost;
  }
  return best;
}

// Arguments as ms_latent_attention_mma for steps of single tokens.  A request's keys are cut into `ranges`; one that sees fewer than `least`
// keys is attended to in tiles that its blocks' warps share (attention_latent_tiles.cuh), cut into tile_ranges.  Partial results are for
// max(ranges, tile_ranges).  error_flag: one int on the device that a kernel which gave up waiting sets.  Cache rows on 16-byte boundaries.
MS_EXPORT int ms_latent_decode(const void* q_full, const void* cache, const int* block_tables, int table_stride, const int* query_start,
                               const int* context_lens, int page_size, int heads, int rank, int rot, float scale, int window, void* out,
                               float* part_o, float* part_lse, int ranges, int least, int tile_ranges, int n_requests, int n_tokens, int* error_flag,
                               cudaStream_t stream) {
  if (n_tokens == 0 || n_requests == 0) return 0;
  MS_REQUIRE(ms_latent_decode_supports(rank, rot, heads) && page_size > 0, "latent_decode: %d + %d, %d heads, pages of %d", rank, rot, heads, page_size);
  const int splits = ranges > tile_ranges ? ranges : tile_ranges;
  MS_REQUIRE(ranges >= 1 && tile_ranges >= 1 && splits <= 32 && (splits == 1 || (part_o && part_lse)), "latent_decode: %d ranges, or %d",
             ranges, tile_ranges);
  MS_REQUIRE(n_requests <= 65535 && error_flag != nullptr, "latent_decode: %d requests, an error flag on the device is required", n_requests);
  MS_REQUIRE(((reinterpret_cast<size_t>(q_full) | reinterpret_cast<size_t>(cache) | reinterpret_cast<size_t>(out)) & 15) == 0,
             "latent_decode: operands must be 16-byte aligned");
  auto launch = rot == 0 ? latent_decode::launch<16> : rot == 32 ? latent_decode::launch<18> : latent_decode::launch<20>;
  if (launch(q_full, cache, block_tables, table_stride, query_start, context_lens, page_size, heads, scale, window, out, part_o, part_lse,
             splits, ranges, least, tile_ranges, n_requests, error_flag, stream))
    return 1;
  if (splits > 1) {
    launch_attention_combine<256>(part_o, part_lse, (__nv_bfloat16*)out, splits, n_tokens * heads, stream);
    MS_CHECK_LAUNCH("latent_decode: merge of the key ranges");
  }
  return 0;
}
