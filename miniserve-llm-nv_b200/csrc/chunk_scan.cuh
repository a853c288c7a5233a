// What the kernels of the scans in chunks share: the problem, where its chunks lie, a token's gates.
#pragma once

#include "common.cuh"

namespace ms {
namespace chunk_scan {

constexpr int kChunk = 128;                              // tokens of a chunk on the tensor cores
constexpr int kSolved = 64;                              // on the float32 pipe, and of what the delta form solves at a time
enum Form : int { kMemory = 0, kDelta = 1, kDecay = 2, kSelective = 3 };

struct Rows { const void* at; int ld, col; };            // a head's rows: column col + head * size

struct Problem {
  Rows q, k, v;
  int qk_dtype, v_dtype;
  int heads, kv_heads, dim, vdim, columns;               // columns of a head's state: vdim, and one more in the memory form
  int input_act, wide, v_wide;                           // SiLU on q, k, v; rows on 16-byte boundaries in whole 16-byte pieces (q and k, v)
  float q_scale;
  const float* gates;                                    // memory [N, H, 3], delta [N, H, 2], decay [H]
  const void* step;                                      // selective: step sizes' logits, type, rows, first column
  int step_dtype, step_ld, step_col;
  const float *step_bias, *a_log, *skip;
  float* states;
  long long state_stride;
  int state_offset;
  const int *state_slots, *query_start;
  int requests, least;                                   // least: tokens from which on a portion is scanned here
  float *chunk_states, *chunk_decays, *records;          // [places][heads][columns][dim], [places][heads], [places][heads][kRecord] or null
  float *y, *bottom;
  int* error_flag;
};

// A block's chunk (its first token, its tokens, those of its portion from it on), or its portion and that one's first chunk.  Chunks are
// numbered through the step's portions of at least `least` tokens, which is where their matrices lie in the scratch.
struct Where { int request, first, len, left; size_t place; };
struct Portion { int request, first, tokens; size_t place; };

// The portions of 32 requests from r0 on, one a lane: its first token, its tokens (0: none, or too few for a chunk), and the chunks up to and
// with it.
struct Lane { int first, tokens, chunks, upto; };
template <int C>
__device__ __forceinline__ Lane portions_from(const int* query_start, int requests, int least, int r0) {
  const int lane = threadIdx.x & 31;
  Lane l = {};
  if (r0 + lane < requests) l.first = query_start[r0 + lane], l.tokens = query_start[r0 + lane + 1] - l.first;
  if (l.tokens < least) l.tokens = 0;
  l.chunks = (l.tokens + C - 1) / C, l.upto = l.chunks;
#pragma unroll
  for (int d = 1; d < 32; d *= 2) {
    const int before = __shfl_up_sync(0xffffffffu, l.upto, d);
    if (lane >= d) l.upto += before;
  }
  return l;
}

// The c-th chunk, looked up by a whole warp; `count` is how many there are (c beyond them: only that, and no tokens).  Several requests are
// searched out of line: a single one's kernels then need no more registers than without a search.
template <int C>
__device__ __noinline__ Where search_chunk(const int* query_start, int requests, int least, int c, int* all) {
  Where w = {};
  int count = 0;
  for (int r0 = 0; r0 < requests; r0 += 32) {
    const Lane l = portions_from<C>(query_start, requests, least, r0);
    const unsigned found = __ballot_sync(0xffffffffu, count + l.upto > c);
    if (found) {
      const int at = __ffs(found) - 1, first = __shfl_sync(0xffffffffu, l.first, at), tokens = __shfl_sync(0xffffffffu, l.tokens, at);
      const int mine = c - count - __shfl_sync(0xffffffffu, l.upto - l.chunks, at);
      w.request = r0 + at, w.left = tokens - mine * C, w.len = min(w.left, C), w.first = first + mine * C;
      w.place = (size_t)c;
      return w;
    }
    count += __shfl_sync(0xffffffffu, l.upto, 31);
  }
  *all = count;
  return w;
}
template <int C>
__device__ __forceinline__ Where chunk_of(const Problem& p, int c, int& count) {
  if (p.requests > 1) return search_chunk<C>(p.query_start, p.requests, p.least, c, &count);
  Where w = {};
  const int first = p.query_start[0], tokens = p.query_start[1] - first;
  count = (tokens + C - 1) / C;
  if (c < count) w.left = tokens - c * C, w.len = min(w.left, C), w.first = first + c * C, w.place = (size_t)c;
  return w;
}

// The k-th portion, looked up by a whole warp (no tokens: there are not as many).
template <int C>
__device__ __noinline__ Portion search_portion(const int* query_start, int requests, int least, int k) {
  int count = 0;
  for (int r0 = 0; r0 < requests; r0 += 32) {
    const Lane l = portions_from<C>(query_start, requests, least, r0);
    const unsigned scanned = __ballot_sync(0xffffffffu, l.tokens > 0);
    const unsigned found = __ballot_sync(0xffffffffu, l.tokens > 0 && __popc(scanned & ((1u << (threadIdx.x & 31)) - 1u)) == k);
    if (found) {
      const int at = __ffs(found) - 1;
      return Portion{r0 + at, __shfl_sync(0xffffffffu, l.first, at), __shfl_sync(0xffffffffu, l.tokens, at),
                     (size_t)(count + __shfl_sync(0xffffffffu, l.upto - l.chunks, at))};
    }
    k -= __popc(scanned), count += __shfl_sync(0xffffffffu, l.upto, 31);
  }
  return Portion{};
}
template <int C>
__device__ __forceinline__ Portion portion_of(const Problem& p, int k) {
  if (p.requests > 1) return search_portion<C>(p.query_start, p.requests, p.least, k);
  return Portion{0, p.query_start[0], p.query_start[1] - p.query_start[0], 0};
}

__device__ __forceinline__ float silu_of(float v) { return v * (1.f / (1.f + expf(-v))); }

// (g_t, w_t) of a token (delta: w is beta).
template <int FORM>
__device__ __forceinline__ float2 gate_of(const Problem& p, int token, int head) {
  const size_t at = (size_t)token * p.heads + head;
  if (FORM == kMemory) return make_float2(p.gates[at * 3], p.gates[at * 3 + 1]);
  if (FORM == kDelta) return make_float2(p.gates[at * 2], p.gates[at * 2 + 1]);
  if (FORM == kDecay) return make_float2(p.gates[head], 1.f);
  const float raw = load_as_float(p.step, p.step_dtype, (size_t)token * p.step_ld + p.step_col + head) + p.step_bias[head];
  const float step = raw > 20.f ? raw : log1pf(expf(raw));           // softplus; above 20 the two agree in float32
  return make_float2(expf(-expf(p.a_log[head]) * step), step);
}

// What a chunk's decays come to, one record per chunk and head (floats; see gates_kernel):
//   A      [128] pairs      product of the decays of token t's block of 32 up to t, as a float and what it lacks
//   F      [3][128] pairs   for the rows of block w + 1 (of 32): decays from s to the block's start, times w_s and the scale of the queries
//   diag   [4][32][32]      within block w: the same from token j (row) to token t (column)
//   G      [128]            decays from the chunk's start to t, times the scale
//   end    [128] pairs      decays from behind s to the chunk's end, times w_s
//   all    [1]              the product of all
constexpr int kRecordA = 0, kRecordF = 256, kRecordDiag = 1024, kRecordG = 5120, kRecordEnd = 5248, kRecordAll = 5504, kRecord = 5508;

// The portions and chunks of C tokens that a step of n tokens brings at most.
struct Bounds { int portions, chunks; };
template <int C>
static Bounds bounds_of(int n_tokens, int n_requests, int least) {
  const int portions = n_tokens / least < n_requests ? n_tokens / least : n_requests;
  return Bounds{portions, n_tokens / C + portions};
}

int launch_gates(int form, const Problem& p, const Bounds& most, cudaStream_t stream);         // every chunk's record
int launch_local(const Problem& p, const Bounds& most, cudaStream_t stream);                   // every chunk's own matrix, joined
int launch_read(const Problem& p, const Bounds& most, cudaStream_t stream);                    // the rows of y

}  // namespace chunk_scan
}  // namespace ms
