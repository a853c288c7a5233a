// The products of the scans in chunks (chunk_scan.cu says what they are) on the fifth-generation tensor cores, chunks of 128 tokens:
//   gates_kernel   a chunk's products of decays
//   local_kernel   every chunk's own matrix, sum over s of D(end, s) w_s v_s k_s^T
//   join_long_kernel  what each chunk starts from, and the request's new state
//   read_kernel    y
//
// Float32 operands are cut into three bfloat16 parts that add up to them exactly (from 2^-110 on; the parts of smaller ones end at 2^-133), and the six
// products of parts that reach a float32's last bit are summed, smallest first; what comes in bfloat16 already (queries, keys and values straight from a projection) is one part, and its
// products with three parts are three.  An addition in tensor memory drops the bits behind its last instead of rounding, so a sum
// lives there for 64 numbers only (16 or 32 where it is a score, whose error a row's values share, or a state's) and sums of those are added in
// float32 registers; what such sums drop on average is in the decays (gates_kernel).  Relative errors against 64 bits (2-norm), the float32 pipe's and these,
// portions of 33 to 2,048 tokens: memory form, 8 heads of 128 x 256, bfloat16, y 1.05e-7 and 0.74e-7, states 0.72e-7 to 0.79e-7 and 0.41e-7 to 0.47e-7; positive operands y
// 0.68e-7 and 0.49e-7; decays near one y 1.2e-7 to 2.0e-7 and 0.74e-7 to 0.92e-7; selective, 64 channels, states of 128, y 1.6e-7 and 0.9e-7, states 0.7e-7 to 0.8e-7 both.
//
// Who comes here: the memory form with bfloat16 or float32 inputs, the selective form and the delta form's read with float32 ones.  The constant decay
// comes only from a caller that has nothing done to the inputs (the engine's layer asks for SiLU, which the float32 pipe's kernels apply), the
// delta form's bfloat16 queries with float32 values only from one whose inputs are bfloat16 (the engine's are not).
//
// In the read kernel the scores pass from tensor memory through registers, where they get their decays, back to tensor memory as the parts of the
// next product's operand: they are never in memory.
//
// A product runs over all tokens of a chunk at once.  What a token must not see has a score of zero, and a value that is not finite is a
// zero to the product (zero times an infinity is not); rows from such a value's token on, and those whose result is not finite, are
// summed again by plain multiply-adds.
//
// Every wait on an mbarrier is bounded: after one that gave up (it sets the error flag that the host checks) the roles run through without
// waiting, and tensor memory is freed on every path.
#include "chunk_scan.cuh"
#include "mma_common.cuh"
#include "tcgen05.cuh"

namespace ms {
namespace chunk_scan {
using namespace t5;

constexpr int kTile = 64;                    // value columns of a unit
// Warps 0..7: operands (read_kernel: and results); 8..15 (local_kernel) results, 16 and 17 the MMAs; (read_kernel) scores and the MMAs: sixteen
// warps, for 128 registers a thread.  What is spilled here comes back from the L2, since shared memory takes nearly all of the L1 cache.
constexpr int kFetchers = 256, kThreads = 576, kFirstIssuer = 16, kReadThreads = 512;
constexpr unsigned kRowsBlock = kChunk * 128, kTileBlock = kTile * 128;        // bytes of 64 bfloat16 columns of 128 rows, of 64

// ------------------------------------------------------------------------------------------------------------- decays
// grid (heads, chunks), a token a thread.  Products of decays are formed in double precision and rounded once (a pair of floats where they
// are a factor of one more product): their errors would be the same for a whole row of scores, where the walk's fall on each number of S alone.
__device__ __forceinline__ float2 pair_of(double v) {
  const float hi = (float)v;
  return make_float2(hi, is_finite(hi) ? (float)(v - (double)hi) : 0.f);
}

// An addition in tensor memory drops the bits behind its last, towards zero: half a unit of the last place on average, 4.3e-8 of a result.  Half a unit
// added to what is summed makes of dropping bits the rounding of them, so a decay that a summed number is multiplied with is larger by a `share` of
// itself.  How much: 4.3e-8 for the last step of a row's sums, as much again for a score's own sum of 16 key entries (half of that where products of
// bfloat16 numbers meet, which have 16 bits: their sums drop less), a quarter to a half more where such a sum takes two steps; S_0's sums of up to four
// steps find a part of the sum at each.  Measured, on operands of either sign and on positive ones: rows of exact scores 6.3e-8 and 8.2e-8 (key entries in
// one block 5.1e-8, 6.1e-8), of scores of three parts 8.3e-8 and 9.5e-8 (7.6e-8, 8.5e-8); S_0 of 64 entries and more 5.9e-8 and 7.8e-8, of 32 4.0e-8
// and 4.5e-8; matrices 3.8e-8, 4.7e-8.  The shares are the means of the two.
//
// A decay of at most eight bits (one, powers of two) gets none: products with it may be exact, and small whole numbers' sums are.  Other rows with
// such decays keep what their sums drop.  A score that is exact (bfloat16 queries and keys of a few entries, whole numbers) under another decay gets
// up to 4e-8 too much: its own sum has dropped nothing.  Those are the two ends: rows of positive numbers are off by 0.5e-7 with the shares, 1.1e-7 without.
// What is summed outside of tensor memory (plain_row, plain_entry) takes the share off again.
__device__ __forceinline__ double rows_share(const Problem& p) { return p.qk_dtype == MS_BF16 ? (p.dim > 64 ? 7.2e-8 : 5.6e-8) : p.dim > 64 ? 8.9e-8 : 8.0e-8; }
__device__ __forceinline__ double start_share(const Problem& p) { return 1.7e-8 + 1.25e-8 * min(4, (p.dim + 15) / 16); }
constexpr double kMatrixShare = 4.2e-8;
__device__ __forceinline__ bool few_bits(float v) { return (__float_as_uint(v) & 0xffffu) == 0u; }
__device__ __forceinline__ double with_share(double v, double share) {
  return (__double2loint(v) | (__double2hiint(v) & 0x1fff)) == 0 ? v : fma(v, share, v);
}
// (of a factor out of a record, in float32: a factor with its share has few bits only by chance)
__device__ __forceinline__ float without_share(float v, double share) { return few_bits(v) ? v : (float)((double)v * (1.0 - share)); }

template <int FORM>
__global__ void __launch_bounds__(kChunk)
gates_kernel(const __grid_constant__ Problem p) {
  grid_dependency_wait();
  grid_dependency_launch();
  int count;
  const Where w = chunk_of<kChunk>(p, blockIdx.y, count);
  if (w.len <= 0) return;
  __shared__ double blocks[4];
  const int t = threadIdx.x, lane = t & 31, block = t >> 5, head = blockIdx.x;
  float2 gate = make_float2(1.f, 0.f);
  if (t < w.len) {
    gate = gate_of<FORM>(p, w.first + t, head);
    if (FORM == kDelta) gate.y = 1.f;        // (what reads take for w v is u)
  }
  const double g = gate.x, weight = gate.y, scaled = weight * (double)p.q_scale, share = rows_share(p);
  double upto = g, behind = g;               // products of the block's decays up to and with t, from t on
#pragma unroll
  for (int d = 1; d < 32; d *= 2) {
    const double before = __shfl_up_sync(0xffffffffu, upto, d), after = __shfl_down_sync(0xffffffffu, behind, d);
    if (lane >= d) upto *= before;
    if (lane + d < 32) behind *= after;
  }
  behind = __shfl_down_sync(0xffffffffu, behind, 1);
  if (lane == 31) {
    behind = 1.0;
    blocks[block] = upto;
  }
  __syncthreads();
  float* record = p.records + (w.place * p.heads + head) * (size_t)kRecord;
  reinterpret_cast<float2*>(record + kRecordA)[t] = pair_of(upto);
  double product = behind;                   // from behind t to the start of block b
#pragma unroll
  for (int b = 1; b < 4; ++b) {
    reinterpret_cast<float2*>(record + kRecordF)[(b - 1) * kChunk + t] = block < b ? pair_of(with_share(product * scaled, share)) : make_float2(0.f, 0.f);
    if (block < b) product *= blocks[b];
  }
  reinterpret_cast<float2*>(record + kRecordEnd)[t] = t < w.len ? pair_of(with_share(product * weight, kMatrixShare)) : make_float2(0.f, 0.f);
  double from_start = upto;
  for (int b = 0; b < block; ++b) from_start *= blocks[b];
  record[kRecordG + t] = (float)with_share(from_start * (double)p.q_scale, start_share(p));
  if (t == kChunk - 1) record[kRecordAll] = (float)from_start;
  double d = 1.0;
  for (int j = 31; j >= 0; --j) {            // D(t, block's token j), t's own block
    const double next = __shfl_sync(0xffffffffu, g, (j + 1) & 31), w_j = __shfl_sync(0xffffffffu, scaled, j);
    if (j < lane) d *= next;
    record[kRecordDiag + (block * 32 + j) * 32 + lane] = j <= lane ? (float)with_share(d * w_j, share) : 0.f;
  }
}

// ------------------------------------------------------------------------------------------------------------ operands
struct Raw { uint4 a, b; };                  // eight numbers of a row: all of it in float32, `a` in bfloat16

// Rows of whole 16-byte pieces: `valid` numbers of eight are there (no branches, so that several fetches are on their way together).
__device__ __forceinline__ Raw fetch_eight(const void* at, int dtype, size_t index, int valid) {
  const uint4* from = reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(at) + index * (dtype == MS_F32 ? 4 : 2));
  const uint4 none = make_uint4(0u, 0u, 0u, 0u);
  Raw r;
  r.a = valid > 0 ? from[0] : none;
  r.b = dtype == MS_F32 && valid > 4 ? from[1] : none;
  return r;
}
// (numbers of other types than the pieces are read as)
__device__ __forceinline__ void put_shared(const void* at, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(smem_u32(at)), "f"(v) : "memory"); }
__device__ __forceinline__ void put_shared(const void* at, unsigned short v) { asm volatile("st.shared.u16 [%0], %1;" ::"r"(smem_u32(at)), "h"(v) : "memory"); }
// The same into this thread's own places of shared memory (of pieces of kFetchers threads each): by asynchronous copies, or number by
// number where rows are not made of whole pieces.  Nothing here or below is a call: around one the compiler keeps what lives in
// local memory, and with this much shared memory that comes back from the L2 (700 clocks).
__device__ __forceinline__ void stage_eight(uint4* to, const void* at, int dtype, size_t index, int valid, bool wide) {
  const char* from = reinterpret_cast<const char*>(at) + index * (dtype == MS_F32 ? 4 : 2);
  if (wide) {
    cp_async_16(to, valid > 0 ? from : at, valid > 0);
    if (dtype == MS_F32) cp_async_16(to + kFetchers, valid > 4 ? from + 16 : at, valid > 4);
  } else if (dtype == MS_F32) {
#pragma unroll 1
    for (int e = 0; e < 8; ++e) put_shared(reinterpret_cast<char*>(to + (e >> 2) * kFetchers) + 4 * (e & 3), e < valid ? reinterpret_cast<const float*>(from)[e] : 0.f);
  } else {
#pragma unroll 1
    for (int e = 0; e < 8; ++e) put_shared(reinterpret_cast<char*>(to) + 2 * e, e < valid ? reinterpret_cast<const unsigned short*>(from)[e] : (unsigned short)0);
  }
}
// ... and back.
__device__ __forceinline__ Raw staged_eight(const uint4* from, int dtype) {
  return Raw{from[0], dtype == MS_F32 ? from[kFetchers] : make_uint4(0u, 0u, 0u, 0u)};
}
__device__ __forceinline__ void floats_of(const Raw& r, int dtype, float (&v)[8]) {
  const unsigned w[8] = {r.a.x, r.a.y, r.a.z, r.a.w, r.b.x, r.b.y, r.b.z, r.b.w};
#pragma unroll
  for (int e = 0; e < 8; ++e)
    v[e] = __uint_as_float(dtype == MS_F32 ? w[e] : e % 2 == 0 ? w[e / 2] << 16 : w[e / 2] & 0xffff0000u);
}
__device__ __forceinline__ void cut_eight(const float (&v)[8], uint4 (&part)[3]) {
  cut(v[0], v[1], part[0].x, part[1].x, part[2].x);
  cut(v[2], v[3], part[0].y, part[1].y, part[2].y);
  cut(v[4], v[5], part[0].z, part[1].z, part[2].z);
  cut(v[6], v[7], part[0].w, part[1].w, part[2].w);
}
__device__ __forceinline__ void cut_eight(const float (&v)[8], const float (&more)[8], uint4 (&part)[3]) {
  cut(v[0], v[1], more[0], more[1], part[0].x, part[1].x, part[2].x);
  cut(v[2], v[3], more[2], more[3], part[0].y, part[1].y, part[2].y);
  cut(v[4], v[5], more[4], more[5], part[0].z, part[1].z, part[2].z);
  cut(v[6], v[7], more[6], more[7], part[0].w, part[1].w, part[2].w);
}
// Whether any of eight leading parts is an infinity or a NaN: zero times it is not zero.
__device__ __forceinline__ bool any_endless(const uint4& v) {
  unsigned sum = 0;
  const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) asm("fma.rn.bf16x2 %0, %1, %2, %0;" : "+r"(sum) : "r"(w[i]), "r"(0u));
  return (sum & 0x7fff7fffu) != 0;
}
// Where eight numbers from column 8 c of a 128-byte row lie, rows 128 bytes apart with the 128-byte swizzle.
__device__ __forceinline__ unsigned place_of(int row, int c) { return (unsigned)row * 128u + (unsigned)((c ^ (row & 7)) << 4); }

// The products of parts (i of PA, j of PB) in the order in which they are summed: smallest first.
template <int PA, int PB, typename F>
__device__ __forceinline__ void products(F&& product) {
  bool first = true;
#pragma unroll
  for (int sum = 2; sum >= 0; --sum)
#pragma unroll
    for (int i = 2; i >= 0; --i) {
      const int j = sum - i;
      if (i < PA && j >= 0 && j < PB) {
        product(i, j, first);
        first = false;
      }
    }
}

// A descriptor that the compiler does not know across iterations (it would keep every sum with an offset in registers, and spill them).
__device__ __forceinline__ uint64_t afresh(uint64_t desc) {
  asm volatile("" : "+l"(desc));
  return desc;
}

// A unit of the work, 64 value columns of a head and a chunk.  Units that share their queries and keys (a head's tiles, a group's heads) are neighbours.
struct Unit { int tile, head, first, len, place; bool new_keys, new_head; };
struct Run { int unit, last, tiles, per_group; };                // a block's units: `unit` is where it begins
__device__ __forceinline__ Run run_of(const Problem& p) {
  Run run;
  int count = 0;
  chunk_of<kChunk>(p, 0x7fffffff, count);
  run.tiles = (p.columns + kTile - 1) / kTile, run.per_group = p.heads / p.kv_heads;
  const long long units = (long long)count * p.heads * run.tiles;
  run.unit = (int)(units * blockIdx.x / gridDim.x), run.last = (int)(units * (blockIdx.x + 1) / gridDim.x);
  return run;
}
__device__ __forceinline__ void enter_chunk(const Problem& p, int chunk, Unit& u) {
  u.place = chunk, u.len = 0;
  if (p.requests == 1) {
    const int first = p.query_start[0], tokens = p.query_start[1] - first;
    u.first = first + chunk * kChunk, u.len = min(tokens - chunk * kChunk, kChunk);
    return;
  }
  int count = 0;
#pragma unroll 1
  for (int r0 = 0; r0 < p.requests; r0 += 32) {
    const Lane l = portions_from<kChunk>(p.query_start, p.requests, p.least, r0);
    const unsigned found = __ballot_sync(0xffffffffu, count + l.upto > chunk);
    if (found) {
      const int at = __ffs(found) - 1, mine = chunk - count - __shfl_sync(0xffffffffu, l.upto - l.chunks, at);
      u.first = __shfl_sync(0xffffffffu, l.first, at) + mine * kChunk;
      u.len = min(__shfl_sync(0xffffffffu, l.tokens, at) - mine * kChunk, kChunk);
      return;
    }
    count += __shfl_sync(0xffffffffu, l.upto, 31);
  }
}
__device__ __forceinline__ Unit first_unit(const Problem& p, const Run& run) {
  Unit u;
  const unsigned rest = (unsigned)run.unit / run.tiles, chunk = rest / p.heads;
  u.tile = run.unit - rest * run.tiles, u.head = rest - chunk * p.heads;
  enter_chunk(p, (int)chunk, u);
  u.new_head = u.new_keys = true;
  return u;
}
__device__ __forceinline__ void next_unit(const Problem& p, const Run& run, Unit& u) {
  u.new_head = u.new_keys = false;
  if (++u.tile < run.tiles) return;
  u.tile = 0, u.new_head = true;
  if (++u.head == p.heads) {
    u.head = 0;
    enter_chunk(p, u.place + 1, u);
  }
  u.new_keys = run.per_group == 1 || u.head % run.per_group == 0;
}
__device__ __forceinline__ int columns_at(const Problem& p, const Unit& u) { return min(kTile, p.columns - u.tile * kTile); }
__device__ __forceinline__ float* record_at(const Problem& p, const Unit& u) { return p.records + ((size_t)u.place * p.heads + u.head) * kRecord; }
__device__ __forceinline__ float* start_at(const Problem& p, const Unit& u) {
  return p.chunk_states + (((size_t)u.place * p.heads + u.head) * p.columns + u.tile * kTile) * p.dim;
}

// A unit's keys (and queries: MATRICES 2, the first) into shared memory: 64-entry blocks of 128 rows, `PARTS` parts, a matrix behind `apart`
// bytes.  `own`: eight floats of this thread.
template <int PARTS, int NB, int MATRICES>
__device__ __forceinline__ void place_rows(const Problem& p, const Unit& u, int kv_head, unsigned char* to, unsigned apart, float* own) {
  const int dtype = PARTS == 1 ? (int)MS_BF16 : p.qk_dtype;
  auto put = [&](const Raw& raw, int type, int matrix, int row, int c) {
    unsigned char* at = to + matrix * apart + (c >> 3) * kRowsBlock + place_of(row, c & 7);
    if (PARTS == 1 && type == MS_BF16) {
      *reinterpret_cast<uint4*>(at) = raw.a;
    } else {
      float v[8];
      uint4 part[3];
      floats_of(raw, type, v);
      cut_eight(v, part);
#pragma unroll
      for (int q = 0; q < PARTS; ++q) *reinterpret_cast<uint4*>(at + q * NB * kRowsBlock) = part[q];
    }
  };
  auto rows_of = [&](int matrix) -> const Rows& { return MATRICES == 2 && matrix == 0 ? p.q : p.k; };
  auto index_of = [&](int matrix, int row, int c) {
    const Rows& rows = rows_of(matrix);
    return (size_t)(u.first + row) * rows.ld + rows.col + (size_t)kv_head * p.dim + 8 * c;
  };
  const int tid = threadIdx.x, c = tid % (8 * NB), row0 = tid / (8 * NB);
  constexpr int STEP = kFetchers / (8 * NB);
  constexpr int AHEAD = PARTS == 1 ? 4 : 4 / MATRICES;       // rows of a matrix on their way together: what there are registers for
  if (p.wide) {
#pragma unroll 1
    for (int i0 = 0; i0 < kChunk / STEP; i0 += AHEAD) {
      Raw raw[MATRICES][AHEAD];
#pragma unroll
      for (int m = 0; m < MATRICES; ++m)
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
          const int row = row0 + (i0 + i) * STEP;
          raw[m][i] = fetch_eight(rows_of(m).at, dtype, index_of(m, row, c), row < u.len ? p.dim - 8 * c : 0);
        }
#pragma unroll
      for (int m = 0; m < MATRICES; ++m)
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) put(raw[m][i], dtype, m, row0 + (i0 + i) * STEP, c);
    }
  } else {                                   // any rows, number by number
#pragma unroll 1
    for (int i = 0; i < MATRICES * kChunk; i += STEP) {
      const int matrix = i / kChunk, row = row0 + i % kChunk;
#pragma unroll 1
      for (int e = 0; e < 8; ++e)
        put_shared(own + e, row < u.len && 8 * c + e < p.dim ? load_as_float(rows_of(matrix).at, dtype, index_of(matrix, row, c) + e) : 0.f);
      put(Raw{*reinterpret_cast<const uint4*>(own), *reinterpret_cast<const uint4*>(own + 4)}, MS_F32, matrix, row, c);
    }
  }
}
// A unit's values: a row, and the eight columns of this thread.
__device__ __forceinline__ size_t value_index(const Problem& p, const Unit& u, int row) {
  return (size_t)(u.first + row) * p.v.ld + p.v.col + (size_t)u.head * p.vdim + u.tile * kTile + 8 * (threadIdx.x & 7);
}
__device__ __forceinline__ int values_valid(const Problem& p, const Unit& u, int row) {
  return row < u.len ? p.vdim - u.tile * kTile - 8 * (int)(threadIdx.x & 7) : 0;
}

template <int ID, int THREADS> __device__ __forceinline__ void named_barrier() { asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(THREADS) : "memory"); }
__device__ __forceinline__ void named_barrier(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// The waits of a role: after one that gave up none waits any more, and the role runs through (it takes part in the block's barriers).
struct Waits {
  int* error_flag;
  bool ok;
  __device__ __forceinline__ void wait(uint64_t* bar, unsigned parity, int code) {
    if (ok) ok = mbar_wait(bar, parity, error_flag, code);
    ok = __all_sync(0xffffffffu, ok);
  }
};

// A number of q, k or v; a column of the values behind the last is the memory form's one.
__device__ __forceinline__ float number_at(const Problem& p, const Rows& rows, int dtype, int token, int column) {
  return load_as_float(rows.at, dtype, (size_t)token * rows.ld + rows.col + column);
}
__device__ __forceinline__ float value_at(const Problem& p, int token, int head, int column) {
  return column < p.vdim ? number_at(p, p.v, p.v_dtype, token, head * p.vdim + column) : 1.f;
}

// (a NaN of the products is kept where the last column, the memory form's divisor, would hide it, until the row is summed again)
__device__ __forceinline__ void store_result(const Problem& p, size_t token, int column, float v, bool keep) {
  if (column < p.vdim) p.y[token * p.vdim + column] = v;
  else p.bottom[token] = keep && v != v ? v : fmaxf(fabsf(v), p.gates[token * 3 + 2]) + 1e-6f;
}
// Whether anything holds for a thread of the operand warps (a barrier of theirs).
__device__ __forceinline__ bool any_fetcher(bool what) {
  unsigned any;
  asm volatile("{ .reg .pred p, q; setp.ne.u32 p, %1, 0; bar.red.or.pred q, 6, %2, p; selp.u32 %0, 1, 0, q; }"
               : "=r"(any) : "r"((unsigned)what), "n"(kFetchers) : "memory");
  return any != 0;
}
// Rows of a unit by plain multiply-adds and to memory: see the top of this file.  Of row t, columns 32 h to 32 h + 31 of the tile if bit t of
// rows[h] is set.  All operand warps take part, with the keys, S_0 and 32 rows' queries and scores at a time in shared memory (`room`).  A prompt of 2,048 tokens with a NaN
// among its first keys, 8 heads of 128 x 256, whose every later row is summed again: 1.3 ms (0.12 without it); a thread for each row and half a tile, 189 ms.
template <int NB> struct PlainRoom {
  static constexpr int LD = 64 * NB + 1, KEYS = 0, START = KEYS + kChunk * LD, QUERIES = START + kTile * LD, SCORES = QUERIES + 32 * LD;
  static constexpr int FLOATS = SCORES + 32 * (kChunk + 1);
};
template <int NB>
__device__ __noinline__ void plain_rows(const Problem& p, const Unit u, const unsigned (&rows)[2][4], float* room) {
  using R = PlainRoom<NB>;
  float *ks = room + R::KEYS, *start = room + R::START, *qs = room + R::QUERIES, *scores = room + R::SCORES;
  const int tid = threadIdx.x, columns = columns_at(p, u), kv = u.head / (p.heads / p.kv_heads) * p.dim;
  const float* record = record_at(p, u);
  const double share = rows_share(p);
#pragma unroll 8
  for (int i = tid; i < u.len * p.dim; i += kFetchers) ks[i / p.dim * R::LD + i % p.dim] = number_at(p, p.k, p.qk_dtype, u.first + i / p.dim, kv + i % p.dim);
#pragma unroll 8
  for (int i = tid; i < columns * p.dim; i += kFetchers) start[i / p.dim * R::LD + i % p.dim] = start_at(p, u)[i];
#pragma unroll 1
  for (int block = 0; block < 4; ++block) {
    const unsigned mine = rows[0][block] | rows[1][block];
    const int t0 = 32 * block;
    if (mine == 0u) continue;
    any_fetcher(false);                      // (the block before has been read)
#pragma unroll 8
    for (int i = tid; i < min(32, u.len - t0) * p.dim; i += kFetchers)
      qs[i / p.dim * R::LD + i % p.dim] = number_at(p, p.q, p.qk_dtype, u.first + t0 + i / p.dim, kv + i % p.dim);
    any_fetcher(false);
    {
      const int r = tid >> 3, t = t0 + r;
      if (mine >> r & 1u) {
        const float2 a = reinterpret_cast<const float2*>(record + kRecordA)[t];
        for (int s0 = tid & 7; s0 <= t; s0 += 32) {              // (four at a time)
          float dot[4] = {0.f, 0.f, 0.f, 0.f};
          for (int n = 0; n < p.dim; ++n) {
            const float query = qs[r * R::LD + n];
#pragma unroll
            for (int j = 0; j < 4; ++j) dot[j] = fmaf(query, ks[min(s0 + 8 * j, t) * R::LD + n], dot[j]);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int s = s0 + 8 * j;
            if (s > t) continue;
            float score = s < t0 ? dot[j] * (a.x * without_share(record[kRecordF + 2 * ((block - 1) * kChunk + s)], share))
                                 : dot[j] * without_share(record[kRecordDiag + s * 32 + r], share);
            if (s == t && p.skip != nullptr) score += p.skip[u.head];
            scores[r * (kChunk + 1) + s] = score;
          }
        }
      }
    }
    any_fetcher(false);
    const int c = tid & 63, r0 = 8 * (tid >> 6), column = u.tile * kTile + c;
    if (c < columns) {
      float sum[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) sum[r] = 0.f;
      for (int n = 0; n < p.dim; ++n) {
        const float from = start[c * R::LD + n];
#pragma unroll
        for (int r = 0; r < 8; ++r) sum[r] = fmaf(qs[(r0 + r) * R::LD + n], from, sum[r]);
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) sum[r] *= without_share(record[kRecordG + t0 + r0 + r], start_share(p));
      const int last = min(t0 + r0 + 8, u.len);
      for (int s0 = 0; s0 < last; s0 += 8) {
        float value[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) value[j] = value_at(p, u.first + min(s0 + j, last - 1), u.head, column);
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int r = 0; r < 8; ++r)
            if (s0 + j <= t0 + r0 + r) sum[r] = fmaf(scores[(r0 + r) * (kChunk + 1) + s0 + j], value[j], sum[r]);
      }
#pragma unroll
      for (int r = 0; r < 8; ++r)
        if (rows[c >> 5][block] >> (r0 + r) & 1u) store_result(p, (size_t)(u.first + t0 + r0 + r) * p.heads + u.head, column, sum[r], false);
    }
  }
}
// A warp's numbers of a chunk's own matrix (an entry a lane, `here` columns from `column` on) by plain multiply-adds, where `to` has one that is not finite.
__device__ __noinline__ void plain_entries(const Problem& p, const Unit u, int column, int here, int entry, float* to) {
  const float2* weights = reinterpret_cast<const float2*>(record_at(p, u) + kRecordEnd);
  const int lane = threadIdx.x & 31, kv = u.head / (p.heads / p.kv_heads) * p.dim;
  float sum[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) sum[i] = 0.f;
#pragma unroll 4
  for (int s = 0; s < u.len; ++s) {
    const float key = entry < p.dim ? number_at(p, p.k, p.qk_dtype, u.first + s, kv + entry) : 0.f;
    const float value = lane < here ? without_share(weights[s].x, kMatrixShare) * value_at(p, u.first + s, u.head, column + lane) : 0.f;
#pragma unroll
    for (int i = 0; i < 32; ++i) sum[i] = fmaf(__shfl_sync(0xffffffffu, value, i), key, sum[i]);
  }
#pragma unroll
  for (int i = 0; i < 32; ++i)
    if (entry < p.dim && i < here && !is_finite(to[(size_t)i * p.dim])) to[(size_t)i * p.dim] = sum[i];
}

// ------------------------------------------------------------------------------------------------------- the rows of y
// A block a multiprocessor, each with a run of units.
//   warps 0..7     operands and results.  Queries and keys when they change; a unit's S_0, then its values, half of each sum's 64 numbers in
//                  a place of its own (slot), cut from raw copies that were requested a unit earlier; the results of either product, a row a
//                  thread (two for each), and their way to memory while the next product runs;
//   warps 8..15    scores: a row a thread (two for each), times their decays, cut, into tensor memory.  A thread of the two warps with the first
//                  rows issues the MMAs of the first and the second 64 numbers of every sum.
// Tensor memory: q k^T (128 columns), the parts of the scores (192), two results of 64; before those q k^T as four sums of a quarter of the entries each.
// A slot's next operand is announced only after its last results have been read, so that one barrier says both.  (Every unit takes the
// same steps whatever its tokens: waits by parity must not be overtaken.)
//
// What binds it is the chain between the roles (keys cut, scores into registers and back, results out), not a unit: on 2,048 tokens the tensor pipe is busy
// for 11 % of the cycles (memory form) and 22 % (selective), the memory system for 23 to 28 %, and warps wait for loads and for barriers.
// The float32 pipe's kernel, which its multiply-adds bound, and this: memory form, 8 heads of 128 x 256 in bfloat16,
// 74.1 and 36.9 us; selective, 64 of 128 x 64, 121.5 and 73.3; delta, 16 of 128 x 128, 75.8 and 51.4.
template <int QP, int VP, int NB>
struct ReadLayout {
  static constexpr unsigned QUERIES = QP * NB * kRowsBlock, SLOT = 3 * kTileBlock;
  static constexpr unsigned RAW_START = NB * 4 * kFetchers * 16, RAW_VALUES = 8 * kFetchers * 16;
  static constexpr unsigned USED = 2 * SLOT + RAW_START + RAW_VALUES, SECOND = QUERIES > USED ? QUERIES : USED;        // keys, or these
  static constexpr unsigned FACTORS = 2 * 192 * 8;                                               // two heads' F
  static constexpr unsigned ROOM = 8 * 32 * 12 * 4;                                              // a warp's 32 rows of eight results
  static constexpr size_t BYTES = 1024 + QUERIES + SECOND + FACTORS + ROOM;
};
constexpr unsigned kScores = 0, kParts = 128, kResult = 320;
static_assert(PlainRoom<1>::FLOATS * 4 <= ReadLayout<1, 1, 1>::QUERIES + ReadLayout<1, 1, 1>::SECOND &&
                  PlainRoom<2>::FLOATS * 4 <= ReadLayout<1, 1, 2>::QUERIES + ReadLayout<1, 1, 2>::SECOND,
              "rows that are summed again have no room");

template <int QP, int VP, int NB>
__global__ void __launch_bounds__(kReadThreads, 1)
read_kernel(const __grid_constant__ Problem p) {
  using L = ReadLayout<QP, VP, NB>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* q_s = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char *k_s = q_s + L::QUERIES, *slots = k_s;
  float2* factors = reinterpret_cast<float2*>(q_s + L::QUERIES + L::SECOND);         // [2][192]: 32, 64 and 96 tokens' for the blocks 1, 2, 3
  __shared__ uint64_t keys_full, scores_full, scores_read, slot_full[2], result_full[2], parts_full, parts_free;
  __shared__ unsigned again[2][4];           // rows that are summed again
  __shared__ int endless[4];                 // first token whose value is not finite, of the last units
  __shared__ unsigned tmem_base_s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(&keys_full, 8);
    mbar_init(&scores_full, NB);
    mbar_init(&scores_read, 8);
    mbar_init(&parts_full, 8);
    mbar_init(&parts_free, 2);
    for (int h = 0; h < 2; ++h) {
      mbar_init(&slot_full[h], 8);
      mbar_init(&result_full[h], 1);
    }
    for (int i = 0; i < 4; ++i) endless[i] = kChunk;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_base_s)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  const unsigned tmem = tmem_base_s;
  grid_dependency_wait();
  grid_dependency_launch();
  const Run run = run_of(p);
  Waits waits{p.error_flag, true};
  unsigned n = 0;                            // units so far
  Unit u = first_unit(p, run);

  if (warp < 8) {
    // ---------------- operands and results.  Of a slot's 64 x 64 numbers a thread has eight of the rows row0 and row0 + 32; of the results 32
    // columns of row t
    const int tid = threadIdx.x, c = tid & 7, row0 = tid >> 3, quarter = warp & 3, half = warp >> 2, t = quarter * 32 + lane;
    const unsigned row = tmem + ((unsigned)(quarter * 32) << 16) + kResult + 32 * half;
    const bool start_wide = p.dim % 4 == 0, one_column = p.columns > p.vdim, rows_wide = p.vdim % 4 == 0 && (reinterpret_cast<size_t>(p.y) & 15) == 0;
    const int v_dtype = VP == 1 ? (int)MS_BF16 : p.v_dtype;
    uint4* raw_start = reinterpret_cast<uint4*>(slots + 2 * L::SLOT) + tid;
    uint4* raw_values = raw_start + L::RAW_START / 16;
    float* room = reinterpret_cast<float*>(factors + 384) + warp * 32 * 12;
    auto request_start = [&](const Unit& u) {
      const float* from = start_at(p, u);
      const int rows = columns_at(p, u);
#pragma unroll
        for (int i = 0; i < 2 * NB; ++i) {
          const int row = row0 + 32 * (i & 1), entry = 64 * (i >> 1) + 8 * c;
          stage_eight(raw_start + 2 * i * kFetchers, from, MS_F32, (size_t)(row * p.dim + entry), row < rows ? p.dim - entry : 0, start_wide);
        }
      cp_async_commit();
    };
    auto request_values = [&](const Unit& u) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int token = row0 + 32 * i;
        stage_eight(raw_values + 2 * i * kFetchers, p.v.at, v_dtype, value_index(p, u, token), values_valid(p, u, token), p.v_wide);
      }
      cp_async_commit();
    };
    auto announce = [&](uint64_t* bar) {
      tmem_fence_before();                   // (results that these threads have read may be overwritten from here on)
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    float sum[32];
    unsigned results[2] = {0, 0};
    auto add_results = [&](int halves, float scale) {          // (of what there is)
#pragma unroll 1
      for (int h = 0; h < halves; ++h) {
        waits.wait(&result_full[h], (h == 0 ? results[0]++ : results[1]++) & 1, 77);
        tmem_fence_after();
#pragma unroll
        for (int i0 = 0; i0 < 32; i0 += 16) {
          float v[16];
          tmem_load_16_nowait(row + 64 * h + i0, v);
          tmem_load_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) sum[i0 + i] = fmaf(sum[i0 + i], scale, v[i]);
        }
        scale = 1.f;
      }
    };
    // a unit's results to memory: eight columns at a time by way of shared memory, so that a store takes whole sectors.  Rows from a value on
    // that is not finite become NaNs, which are looked for at the end
    bool finite = true;
    auto store_rows = [&](const Unit& u, unsigned n) {
      const int column = u.tile * kTile + 32 * half, here = min(32, p.columns - column), left = u.len - quarter * 32;
      const size_t token = (size_t)(u.first + quarter * 32) * p.heads + u.head;
      float* to = p.y + (token + (size_t)(lane >> 1) * p.heads) * p.vdim + column + (lane & 1) * 4;
      const size_t half_way = (size_t)16 * p.heads * p.vdim;
      float zero = t >= endless[n & 3] ? __int_as_float(0x7fc00000) : 0.f;
#pragma unroll
      for (int i = 0; i < 32; ++i) sum[i] += zero;
#pragma unroll
      for (int i0 = 0; i0 < 32; i0 += 8) {
        if (i0 >= here) break;
#pragma unroll
        for (int i = 0; i < 8; i += 4)
          *reinterpret_cast<float4*>(room + lane * 12 + i) = make_float4(sum[i0 + i], sum[i0 + i + 1], sum[i0 + i + 2], sum[i0 + i + 3]);
#pragma unroll
        for (int i = 0; i < 8; ++i) zero = fmaf(sum[i0 + i], 0.f, zero);
        __syncwarp();
        if (rows_wide && column + i0 + 8 <= p.vdim) {
          const float* from = room + (lane >> 1) * 12 + (lane & 1) * 4;
          if ((lane >> 1) < left) *reinterpret_cast<float4*>(to) = *reinterpret_cast<const float4*>(from);
          if ((lane >> 1) + 16 < left) *reinterpret_cast<float4*>(to + half_way) = *reinterpret_cast<const float4*>(from + 16 * 12);
        } else if (lane < left) {
#pragma unroll 1
          for (int i = 0; i < 8 && i0 + i < here; ++i) store_result(p, token + (size_t)lane * p.heads, column + i0 + i, room[lane * 12 + i], true);
        }
        to += 8;
        __syncwarp();
      }
      if (lane < left && (zero != 0.f || zero != zero)) finite = false;        // (at worst of a column behind the last: looked at for nothing)
    };
    unsigned groups = 0;
    Unit before = u;
    for (int at = run.unit;; ++at, ++n) {
      Unit next = u;
      next_unit(p, run, next);
      const bool more = at + 1 < run.last && !next.new_keys, store_first = at >= run.last || u.new_keys;
      // the last unit's results go to memory while this one's first product runs, or before the keys change (they need the registers)
#pragma unroll 1
      for (int step = 0; step < 2; ++step) {
        if ((step == 0) == store_first) {
          if (n > 0) store_rows(before, n - 1);
          continue;
        }
        if (at >= run.last) break;
        if (u.new_keys) {
          // (everything that reads shared memory or writes results has finished: the last unit's results have been read)
          place_rows<QP, NB, 2>(p, u, u.head / run.per_group, q_s, L::QUERIES, room + lane * 12);
          announce(&keys_full);
          waits.wait(&scores_full, groups++ & 1, 73);    // (what follows takes the keys' place)
          request_start(u);
          request_values(u);
        }
        cp_async_wait<1>();
#pragma unroll 1
        for (int h = 0; h < NB; ++h) {
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int row = row0 + 32 * i;
            float v[8];
            uint4 part[3];
            floats_of(staged_eight(raw_start + 2 * (2 * h + i) * kFetchers, MS_F32), MS_F32, v);
            cut_eight(v, part);
#pragma unroll
            for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(slots + h * L::SLOT + q * kTileBlock + place_of(row, c)) = part[q];
          }
          announce(&slot_full[h]);
        }
        if (more) request_start(next);
        else cp_async_commit();
      }
      if (at >= run.last) break;
      const float decayed = record_at(p, u)[kRecordG + t];
#pragma unroll
      for (int i = 0; i < 32; ++i) sum[i] = 0.f;
      add_results(NB, 1.f);
      cp_async_wait<1>();
      if (tid == 0) endless[(n + 2) & 3] = kChunk;       // (every warp is done with the results of the unit before the last)
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int token = 64 * h + row0 + 32 * i;
          const Raw raw = staged_eight(raw_values + 2 * (2 * h + i) * kFetchers, v_dtype);
          const int one = one_column && token < u.len ? p.vdim - u.tile * kTile - 8 * c : -1;        // (the memory form's column of ones)
          uint4 part[3];
          if constexpr (VP == 1) {
            part[0] = raw.a;
            const unsigned bits = one % 2 ? 0x3f800000u : 0x3f80u;
            if (one >> 1 == 0) part[0].x |= bits;
            if (one >> 1 == 1) part[0].y |= bits;
            if (one >> 1 == 2) part[0].z |= bits;
            if (one >> 1 == 3) part[0].w |= bits;
          } else {
            float v[8];
            floats_of(raw, v_dtype, v);
            if (one_column) {
#pragma unroll
              for (int e = 0; e < 8; ++e)
                if (e == one) v[e] = 1.f;
            }
            cut_eight(v, part);
          }
          if (any_endless(part[0])) {
            part[0] = part[1] = part[2] = make_uint4(0u, 0u, 0u, 0u);
            atomicMin(&endless[n & 3], token);
          }
#pragma unroll
          for (int q = 0; q < VP; ++q)
            *reinterpret_cast<uint4*>(slots + h * L::SLOT + q * kTileBlock + place_of(row0 + 32 * i, c)) = part[q];
        }
        announce(&slot_full[h]);
      }
      if (more) request_values(next);
      else cp_async_commit();
      add_results(2, decayed);
      before = u, u = next;
    }
    cp_async_wait<0>();
    if (any_fetcher(!finite)) {              // the rows with a result that is not finite, again (shared memory is free by now)
      Unit one = first_unit(p, run);
      for (int at = run.unit; at < run.last; ++at, next_unit(p, run, one)) {
        const int column = one.tile * kTile + 32 * half, here = min(32, p.columns - column);
        bool bad = false;
        for (int i = 0; i < here && t < one.len; ++i) {
          const size_t token = (size_t)(one.first + t) * p.heads + one.head;
          bad = bad || !is_finite(column + i < p.vdim ? p.y[token * p.vdim + column + i] : p.bottom[token]);
        }
        const unsigned mask = __ballot_sync(0xffffffffu, bad);
        if (lane == 0) again[half][quarter] = mask;
        if (any_fetcher(mask != 0u)) plain_rows<NB>(p, one, again, reinterpret_cast<float*>(q_s));
        any_fetcher(false);                  // (read, all of it)
      }
    }
  } else {
    // ---------------- scores: row t, every other 16 columns; MMAs
    const int tid = threadIdx.x - kFetchers, quarter = warp & 3, half = (warp - 8) >> 2, t = quarter * 32 + lane;
    const unsigned row = tmem + ((unsigned)(quarter * 32) << 16);
    // a head's factors into shared memory, its rows' own decays into registers: while the head before is at work
    float own[16];                           // decays within the row's own 32 tokens
    float2 a;
    auto fetch_record = [&](const float* record, int buffer) {
      if (tid < 96) {                        // two tokens' factors a thread
        const int block = tid < 16 ? 0 : tid < 48 ? 1 : 2, s = 2 * (tid - (tid < 16 ? 0 : tid < 48 ? 16 : 48));
        cp_async_16(factors + buffer * 192 + 2 * tid, record + kRecordF + 2 * (block * kChunk + s), true);
      }
      cp_async_commit();
      a = reinterpret_cast<const float2*>(record + kRecordA)[t];
#pragma unroll
      for (int i = 0; i < 16; ++i) own[i] = record[kRecordDiag + (quarter * 32 + half * 16 + i) * 32 + lane];
    };
    // the two warps of the first rows, which have the fewest scores, issue the MMAs of numbers 64 h .. 64 h + 63 of every sum
    const bool issues = quarter == 0;
    const int h = half;
    const uint64_t q_desc = umma_desc(q_s + h * kRowsBlock), k_desc = umma_desc(k_s + h * kRowsBlock);
    const uint64_t start_desc = umma_desc(slots + h * L::SLOT), v_desc = umma_desc_mn_major(slots + h * L::SLOT, kTileBlock);
    const unsigned result = tmem + kResult + 64 * h, parts = tmem + kParts + 32 * h;
    unsigned operands = 0;
    auto multiply_start = [&](unsigned width) {
      waits.wait(&slot_full[h], operands++ & 1, 79);
      if (lane == 0 && waits.ok) {
        tmem_fence_after();
        const uint64_t a = afresh(q_desc), b = afresh(start_desc);
        products<QP, 3>([&](int i, int j, bool first) {
#pragma unroll 1
          for (int k = 0; k < 4; ++k)
            umma_bf16(result, a + (uint64_t)(i * NB * (kRowsBlock / 16) + 2 * k), b + (uint64_t)(j * (kTileBlock / 16) + 2 * k),
                      umma_idesc(kChunk, width), !first || k != 0);
        });
        umma_commit(&result_full[h]);
      }
      __syncwarp();
    };
    unsigned heads = 0, groups = 0;
    const float* record = record_at(p, u);
    if (run.unit < run.last) fetch_record(record, 0);
    for (int at = run.unit; at < run.last; ++at, ++n, next_unit(p, run, u)) {
      const unsigned width = (unsigned)(columns_at(p, u) + 15) / 16 * 16;
      if (u.new_head) {
        cp_async_wait<0>();
        named_barrier<1, kFetchers>();       // this head's factors are there, those before the last head's have been read
      }
      if (issues && h < NB) {
        if (u.new_keys) {
          waits.wait(&keys_full, groups & 1, 78);
          if (lane == 0 && waits.ok) {
            tmem_fence_after();
            const uint64_t a = afresh(q_desc), b = afresh(k_desc);
            products<QP, QP>([&](int i, int j, bool first) {
#pragma unroll 1
              for (int k = 0; k < 4; ++k)
                umma_bf16(tmem + kScores + (NB == 2 ? 256 * h + 128 * (k >> 1) : 128 * k), a + (uint64_t)(i * NB * (kRowsBlock / 16) + 2 * k),
                          b + (uint64_t)(j * NB * (kRowsBlock / 16) + 2 * k), umma_idesc(kChunk, kChunk), !first || (NB == 2 && (k & 1) != 0));
            });
            umma_commit(&scores_full);
          }
          __syncwarp();
        } else {
          multiply_start(width);
        }
      }
      // (Once a head, not once a unit: within a head the two warps that issue the MMAs need nothing of the other six, and could take the barrier
      // two phases on while one of those has not looked at it yet.  From head to head they need every warp's parts.)
      if (u.new_head && heads > 0) waits.wait(&parts_free, (heads - 1) & 1, 72);
      if (u.new_head) {
        const float skip = p.skip != nullptr ? p.skip[u.head] : 0.f;
        const float2* factor = factors + (heads & 1) * 192 + (quarter == 2 ? 32 : quarter == 3 ? 96 : 0);
        ++heads;
        if (u.new_keys) {
          waits.wait(&scores_full, groups++ & 1, 76);
          tmem_fence_after();
          for (int b = half; b < 2 * (quarter + 1); b += 2) {
            float x[16], y[16];
            unsigned both[16];
            tmem_load_16_nowait(row + kScores + 16 * b, x);
#pragma unroll 1
            for (int part = 1; part < 4; ++part) {
              tmem_load_16_nowait(row + kScores + 128 * part + 16 * b, y);
              tmem_load_wait();
#pragma unroll
              for (int i = 0; i < 16; ++i) x[i] += y[i];
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) both[i] = __float_as_uint(x[i]);
            tmem_store_16(row + kScores + 16 * b, both);
          }
          tmem_store_wait();
          tmem_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&scores_read);        // (results may take the partial sums' place)
          named_barrier(2 + quarter, 64);      // both warps have read the partial sums of these rows
          const unsigned none[8] = {0, 0, 0, 0, 0, 0, 0, 0};
          for (int b = 2 * (quarter + 1) + half; b < 8; b += 2) {          // tokens that no row of these sees
#pragma unroll
            for (int q = 0; q < 3; ++q) tmem_store_8(row + kParts + 64 * q + 8 * b, none);
          }
          if (issues && h < NB) {
            waits.wait(&scores_read, (groups - 1) & 1, 80);
            multiply_start(width);
          }
        }
        tmem_fence_after();
        for (int b = half; b < 2 * (quarter + 1); b += 2) {
          float score[16];
          tmem_load_16_nowait(row + kScores + 16 * b, score);
          tmem_load_wait();
          if (b < 2 * quarter) {
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
              const float4 two = *reinterpret_cast<const float4*>(factor + 16 * b + i);
              score[i] *= fmaf(a.x, two.x, fmaf(a.x, two.y, a.y * two.x));
              score[i + 1] *= fmaf(a.x, two.z, fmaf(a.x, two.w, a.y * two.z));
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int j = 16 * half + i;
              score[i] = j <= lane ? score[i] * own[i] : 0.f;
              if (j == lane) score[i] += skip;
            }
          }
          unsigned hi[8], mid[8], lo[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) cut(score[2 * i], score[2 * i + 1], hi[i], mid[i], lo[i]);
          tmem_store_8(row + kParts + 8 * b, hi);
          tmem_store_8(row + kParts + 64 + 8 * b, mid);
          tmem_store_8(row + kParts + 128 + 8 * b, lo);
        }
        tmem_store_wait();
        tmem_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&parts_full);
        record += kRecord;                     // (the next head's, or the next chunk's first)
        if (at + run.tiles - u.tile < run.last) fetch_record(record, heads & 1);         // (its factors lie in the other buffer)
      }
      if (issues) {
        if (u.new_head) waits.wait(&parts_full, (heads - 1) & 1, 82);
        waits.wait(&slot_full[h], operands++ & 1, 81);
        if (lane == 0 && waits.ok) {
          tmem_fence_after();
          const uint64_t b = afresh(v_desc);
          products<3, VP>([&](int i, int j, bool first) {
#pragma unroll 1
            for (int k = 0; k < 4; ++k)
              umma_bf16_a_tmem(result, parts + 64 * i + 8 * k, b + (uint64_t)(j * (kTileBlock / 16) + 128 * k), umma_idesc(kChunk, width, true),
                               !first || k != 0);
          });
          umma_commit(&result_full[h]);
          if (u.tile + 1 == run.tiles && at + 1 < run.last) umma_commit(&parts_free);        // (and somebody waits for it)
        }
        __syncwarp();
      }
    }
    cp_async_wait<0>();
  }
  tmem_fence_before();
  __syncthreads();
  if (warp == 8) {
    tmem_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

// ------------------------------------------------------------------------------------------------- a chunk's own matrix
// The same roles; a unit is the product of the keys (their 64-entry blocks are the MMA's rows, read transposed) and the 64 weighted value
// columns over the chunk's tokens, each quarter of them a sum.  Values and results have two buffers each.  Bound by the cutting of keys and
// values and, in the memory form, by what it writes: the float32 pipe's kernel and this, 2,048 tokens: memory, 8 heads of 128 x 256, 28.9 and 15.8 us;
// selective, 64 of 128 x 64, 57.9 and 28.2.  The join has half as many matrices: 14.2 and 10.1, 43.8 and 16.2 us.
template <int KP, int NB>
struct LocalLayout {
  static constexpr unsigned KEYS = KP * NB * kRowsBlock, VALUES = 3 * kRowsBlock;
  static constexpr size_t BYTES = 1024 + KEYS + 2 * VALUES + 8 * kFetchers * 16;                   // and the next unit's values as they are
};

template <int KP, int NB>
__global__ void __launch_bounds__(kThreads, 1)
local_kernel(const __grid_constant__ Problem p) {
  using L = LocalLayout<KP, NB>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* k_s = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* v_s = k_s + L::KEYS;
  __shared__ uint64_t keys_full, values_full[2], values_free[2], result_full[2], result_empty[2];
  __shared__ unsigned tmem_base_s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(&keys_full, 8);
    for (int b = 0; b < 2; ++b) {
      mbar_init(&values_full[b], 8);
      mbar_init(&values_free[b], 2);
      mbar_init(&result_full[b], 2);
      mbar_init(&result_empty[b], 8);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kFirstIssuer) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_base_s)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  const unsigned tmem = tmem_base_s;
  grid_dependency_wait();
  grid_dependency_launch();
  const Run run = run_of(p);
  Waits waits{p.error_flag, true};

  if (warp < 8) {
    const int c = threadIdx.x & 7, row0 = threadIdx.x >> 3;
    const bool one_column = p.columns > p.vdim;
    uint4* raw_values = reinterpret_cast<uint4*>(v_s + 2 * L::VALUES) + threadIdx.x;
    float2 weight[4];
    auto request_values = [&](const Unit& u) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        stage_eight(raw_values + 2 * i * kFetchers, p.v.at, p.v_dtype, value_index(p, u, row0 + 32 * i), values_valid(p, u, row0 + 32 * i), p.v_wide);
      cp_async_commit();
      const float2* weights = reinterpret_cast<const float2*>(record_at(p, u) + kRecordEnd) + row0;
#pragma unroll
      for (int i = 0; i < 4; ++i) weight[i] = weights[32 * i];
    };
    unsigned n = 0;
    Unit u = first_unit(p, run);
    if (run.unit < run.last) request_values(u);
    for (int at = run.unit; at < run.last; ++at, ++n) {
      const int buffer = n & 1;
      if (u.new_keys) {
        if (n > 0) waits.wait(&values_free[buffer ^ 1], ((n - 1) >> 1) & 1, 84);      // the unit before has read its keys
        place_rows<KP, NB, 1>(p, u, u.head / run.per_group, k_s, 0, reinterpret_cast<float*>(v_s) + threadIdx.x * 8);
        if (!p.wide) named_barrier<1, kFetchers>();         // (number by number by way of the values' room: before any is put there)
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&keys_full);
      }
      waits.wait(&values_free[buffer], ((n >> 1) & 1) ^ 1, 85);
      cp_async_wait<0>();
      const int one = one_column ? p.vdim - u.tile * kTile - 8 * c : -1;          // (the memory form's column of ones)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int token = row0 + 32 * i;
        float v[8], more[8];
        uint4 part[3];
        floats_of(staged_eight(raw_values + 2 * i * kFetchers, p.v_dtype), p.v_dtype, v);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float value = e == one ? 1.f : v[e];
          v[e] = weight[i].x * value;
          more[e] = fmaf(weight[i].y, value, fmaf(weight[i].x, value, -v[e]));
        }
        cut_eight(v, more, part);
#pragma unroll
        for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(v_s + buffer * L::VALUES + q * kRowsBlock + place_of(token, c)) = part[q];
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&values_full[buffer]);
      next_unit(p, run, u);
      if (at + 1 < run.last) request_values(u);
    }
    cp_async_wait<0>();
  } else if (warp < kFirstIssuer) {
    const int quarter = warp & 3, half = (warp - 8) >> 2, entry = quarter * 32 + lane;
    const unsigned row = tmem + ((unsigned)(quarter * 32) << 16);
    unsigned n = 0;
    Unit u = first_unit(p, run);
    for (int at = run.unit; at < run.last; ++at, ++n, next_unit(p, run, u)) {
      const int buffer = n & 1;
      waits.wait(&result_full[buffer], (n >> 1) & 1, 86);
      tmem_fence_after();
      float sum[32];
      tmem_load_32(row + 256 * buffer + 32 * half, sum);
#pragma unroll 1
      for (int part = 1; part * 32 < u.len; ++part) {
        float v[32];
        tmem_load_32(row + 256 * buffer + 64 * part + 32 * half, v);
#pragma unroll
        for (int i = 0; i < 32; ++i) sum[i] += v[i];
      }
      tmem_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&result_empty[buffer]);
      const int column = u.tile * kTile + 32 * half;
      float* to = p.chunk_states + ((u.place * p.heads + u.head) * (size_t)p.columns + column) * p.dim + entry;
      const int here = min(32, p.columns - column);
      float zero = 0.f;                      // a sum of zeros unless one of them is not finite
      if (entry < p.dim) {
        float* at_column = to;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          if (i < here) {
            *at_column = sum[i];
            zero = fmaf(sum[i], 0.f, zero);
          }
          at_column += p.dim;
        }
      }
      if (__any_sync(0xffffffffu, zero != zero)) plain_entries(p, u, column, here, entry, to);
      __syncwarp();
    }
  } else {
    const int h = warp - kFirstIssuer;
    // (keys of at most 64 entries: both blocks of the MMA's 128 rows are the same)
    const uint64_t k_desc = umma_desc_mn_major(k_s, NB == 2 ? kRowsBlock : 0) + (uint64_t)(h * 64 * 128 / 16);
    const uint64_t v_desc = umma_desc_mn_major(v_s, kRowsBlock) + (uint64_t)(h * 64 * 128 / 16);
    unsigned n = 0, groups = 0;
    Unit u = first_unit(p, run);
    for (int at = run.unit; at < run.last; ++at, ++n, next_unit(p, run, u)) {
      const int buffer = n & 1;
      const unsigned width = (unsigned)(columns_at(p, u) + 15) / 16 * 16;
      if (u.new_keys) waits.wait(&keys_full, groups++ & 1, 87);
      waits.wait(&values_full[buffer], (n >> 1) & 1, 88);
      waits.wait(&result_empty[buffer], ((n >> 1) & 1) ^ 1, 89);
      if (lane == 0 && waits.ok) {
        tmem_fence_after();
        const uint64_t a = afresh(k_desc), b = afresh(v_desc) + (uint64_t)(buffer * (L::VALUES / 16));
        if (h == 0 || u.len > 64)
          products<KP, 3>([&](int i, int j, bool first) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_bf16(tmem + 256 * buffer + 128 * h + 64 * (k >> 1), a + (uint64_t)(i * NB * (kRowsBlock / 16) + 128 * k), b + (uint64_t)(j * (kRowsBlock / 16) + 128 * k),
                        umma_idesc(kChunk, width, true) | 1u << 15, !first || k % 2 != 0);        // (bit 15: A transposed as well)
          });
        umma_commit(&values_free[buffer]);
        umma_commit(&result_full[buffer]);
      }
      __syncwarp();
    }
  }
  tmem_fence_before();
  __syncthreads();
  if (warp == kFirstIssuer) {
    tmem_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

// --------------------------------------------------------------------------------------------------- chunks joined
// grid (pieces of the heads' states, portions), PER numbers a thread: bound by memory (each chunk's matrix read and written once), four
// chunks' matrices requested at a time.
template <int PER> struct alignas(4 * PER) Numbers { float v[PER]; };

template <int PER>
__global__ void __launch_bounds__(256)
join_long_kernel(const __grid_constant__ Problem p) {
  grid_dependency_wait();
  grid_dependency_launch();
  const Portion portion = portion_of<kChunk>(p, blockIdx.y);
  const int count = (portion.tokens + kChunk - 1) / kChunk;
  const size_t all = (size_t)p.heads * p.columns * p.dim, at = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * PER;
  if (count <= 0 || at >= all) return;
  const int head = (int)(at / ((size_t)p.columns * p.dim));
  const size_t place = portion.place;
  float* kept = p.states + (long long)p.state_slots[portion.request] * p.state_stride + p.state_offset + at;
  Numbers<PER> s;
#pragma unroll
  for (int e = 0; e < PER; ++e) s.v[e] = kept[e];
  for (int c0 = 0; c0 < count; c0 += 4) {
    Numbers<PER> wrote[4];
    float decay[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (c0 + u >= count) continue;
      wrote[u] = *reinterpret_cast<const Numbers<PER>*>(p.chunk_states + (place + c0 + u) * all + at);
      decay[u] = p.records[((place + c0 + u) * p.heads + head) * (size_t)kRecord + kRecordAll];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (c0 + u >= count) break;
      *reinterpret_cast<Numbers<PER>*>(p.chunk_states + (place + c0 + u) * all + at) = s;
#pragma unroll
      for (int e = 0; e < PER; ++e) s.v[e] = decay[u] * s.v[e] + wrote[u].v[e];
    }
  }
#pragma unroll
  for (int e = 0; e < PER; ++e) kept[e] = s.v[e];
}

// ------------------------------------------------------------------------------------------------------------ launches
static int processors() {
  int device = 0, sms = 148;
  if (cudaGetDevice(&device) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  return sms;
}
static long long units_of(const Problem& p, const Bounds& most) { return (long long)((p.columns + kTile - 1) / kTile) * p.heads * most.chunks; }

int launch_gates(int form, const Problem& p, const Bounds& most, cudaStream_t stream) {
  auto kernel = form == kMemory ? gates_kernel<kMemory> : form == kDelta ? gates_kernel<kDelta> : form == kDecay ? gates_kernel<kDecay> : gates_kernel<kSelective>;
  ms::launch(kernel, dim3(p.heads, most.chunks), dim3(kChunk), 0, stream, p);
  MS_CHECK_LAUNCH("chunk_scan: decays");
  return 0;
}

int launch_local(const Problem& p, const Bounds& most, cudaStream_t stream) {
  const bool exact = p.qk_dtype == MS_BF16, two = p.dim > 64;
  auto kernel = exact ? (two ? local_kernel<1, 2> : local_kernel<1, 1>) : (two ? local_kernel<3, 2> : local_kernel<3, 1>);
  const size_t bytes = exact ? (two ? LocalLayout<1, 2>::BYTES : LocalLayout<1, 1>::BYTES) : (two ? LocalLayout<3, 2>::BYTES : LocalLayout<3, 1>::BYTES);
  if (allow_shared(kernel, bytes) != cudaSuccess) MS_FAIL("chunk_scan: shared memory refused");
  const long long units = units_of(p, most), sms = processors();
  ms::launch(kernel, dim3((unsigned)(units < sms ? units : sms)), dim3(kThreads), bytes, stream, p);
  MS_CHECK_LAUNCH("chunk_scan: chunks alone");
  const bool four = p.dim % 4 == 0;
  const size_t threads = (size_t)p.heads * p.columns * p.dim / (four ? 4 : 1);
  ms::launch(four ? join_long_kernel<4> : join_long_kernel<1>, dim3((unsigned)((threads + 255) / 256), most.portions), dim3(256), 0, stream, p);
  MS_CHECK_LAUNCH("chunk_scan: chunks joined");
  return 0;
}

template <int QP, int VP>
static int launch_read_parts(const Problem& p, const Bounds& most, cudaStream_t stream) {
  const bool two = p.dim > 64;
  auto kernel = two ? read_kernel<QP, VP, 2> : read_kernel<QP, VP, 1>;
  const size_t bytes = two ? ReadLayout<QP, VP, 2>::BYTES : ReadLayout<QP, VP, 1>::BYTES;
  if (allow_shared(kernel, bytes) != cudaSuccess) MS_FAIL("chunk_scan: shared memory refused");
  const long long units = units_of(p, most), sms = processors();
  ms::launch(kernel, dim3((unsigned)(units < sms ? units : sms)), dim3(kReadThreads), bytes, stream, p);
  MS_CHECK_LAUNCH("chunk_scan: rows");
  return 0;
}

int launch_read(const Problem& p, const Bounds& most, cudaStream_t stream) {
  const bool exact = p.qk_dtype == MS_BF16;
  if (!exact) return launch_read_parts<3, 3>(p, most, stream);
  return p.v_dtype == MS_BF16 ? launch_read_parts<1, 1>(p, most, stream) : launch_read_parts<1, 3>(p, most, stream);
}

}  // namespace chunk_scan
}  // namespace ms
