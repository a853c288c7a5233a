// Recurrences with one decay per token and head, S_t = g_t S_(t-1) + w_t v_t k_t^T, y_t = S_t q_t, for portions of many tokens: what
// ms_matrix_scan (memory, delta and constant-decay forms) and ms_selective_scan do token after token, as matrix products over chunks
// of 64 tokens, on the float32 pipe.  Where there is more work the products run on the tensor cores, over chunks of 128 (chunk_scan_tcgen05.cu;
// which of the two is the caller's rule): of the delta form, whose chunks follow one another, what is read then, and the rest here.  Walked, a portion is a chain of as many steps as it has tokens, whose every step waits for shared memory and for a
// butterfly of shuffles; in chunks nearly all of it is products whose operands a thread uses several times.
//
// With D(t, s) = g_(s+1) .. g_t (products of the factors themselves, not differences of their logarithms: a difference of two large
// sums would cost the digits that the products keep) and G_t = g_0 .. g_t within a chunk that starts from S_0,
//
//   y_t = G_t S_0 q_t + sum_(s <= t) D(t, s) w_s (q_t . k_s) v_s,      S_end = G_end S_0 + sum_s D(end, s) w_s v_s k_s^T.
//
//   memory, constant decay, selective:
//     local_kernel   every chunk's sum D(end, s) w_s v_s k_s^T and its G_end
//     join_kernel    S <- G_end S + sum over a portion's chunks: what each starts from, and the request's new state
//     read_kernel    y
//   delta (u_t = beta_t (v_t - S k_t) takes the place of w_t v_t, and depends on S):
//     solve_kernel   within a chunk, u = U - W S_0 with (I + A) [U | W] = [beta v | beta G k], A(t, s) = beta_t D(t, s) k_t . k_s below
//                    the diagonal: forward substitution, a thread per column
//     carry_kernel   the chunks in order, sixteen columns of S a block: u, S_end; S_0 of every chunk
//     read_kernel    y, with u for v
//
// Measured (one request in bfloat16, the scan's launches together; us walked, here, on the tensor cores): memory form, 8 heads of 128 x 256,
// 2,048 tokens 658, 119, 65; selective, 64 heads of 128 x 64, 2,048 tokens 496, 210, 124; delta, 16 heads of 128 x 128, 2,048 tokens 566, 234, 212;
// 512 tokens of the same (here, tensor cores): 43, 34; 69, 58; 71, 76.
//
// All arithmetic is float32 on float32 copies of the projections, products of decays in double.  A token's result uses nothing of the tokens behind it (what is
// masked is not multiplied: a zero would turn an infinity behind it into a NaN before it).
#include "chunk_scan.cuh"
#include "mma_common.cuh"

namespace ms {
namespace chunk_scan {

constexpr int kC = kSolved, kThreads = 256, kTile = 64;  // tokens of a chunk; value columns of a block
constexpr int kLd = kTile + 4;

// 64 rows of WIDTH numbers into shared memory as float32, zeros beyond `len` rows and `width` numbers.
template <typename T, int WIDTH>
__device__ __forceinline__ void load_rows(float* to, int to_ld, const T* from, size_t ld, int len, int width, int wide, int act) {
  constexpr int E = 16 / sizeof(T), PER_ROW = WIDTH / E, TIMES = kC * PER_ROW / kThreads;
  if (wide) {
    uint4 raw[TIMES];
#pragma unroll
    for (int i = 0; i < TIMES; ++i) {
      const int piece = threadIdx.x + i * kThreads, t = piece / PER_ROW, c = piece % PER_ROW * E;
      raw[i] = t < len && c < width ? *reinterpret_cast<const uint4*>(from + (size_t)t * ld + c) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int i = 0; i < TIMES; ++i) {
      const int piece = threadIdx.x + i * kThreads, t = piece / PER_ROW, c = piece % PER_ROW * E;
      const T* v = reinterpret_cast<const T*>(&raw[i]);
#pragma unroll
      for (int e = 0; e < E; e += 4) {
        float4 four = make_float4(to_float(v[e]), to_float(v[e + 1]), to_float(v[e + 2]), to_float(v[e + 3]));
        if (act) four = make_float4(silu_of(four.x), silu_of(four.y), silu_of(four.z), silu_of(four.w));
        *reinterpret_cast<float4*>(to + t * to_ld + c + e) = four;
      }
    }
  } else {
    for (int i = threadIdx.x; i < kC * WIDTH; i += kThreads) {
      const int t = i / WIDTH, c = i % WIDTH;
      float v = t < len && c < width ? to_float(from[(size_t)t * ld + c]) : 0.f;
      if (act) v = silu_of(v);
      to[t * to_ld + c] = v;
    }
  }
}

// a_t . b_s for a warp's tile of 16 rows and 32 columns: rows row0 + ty + 4 i, columns column0 + tx + 8 j for the first `blocks` of four
// (ty 0..3, tx 0..7; pairs of entries apart).  Eight reads of shared memory, each of at most eight different rows (one pass of its
// banks), for 32 packed multiply-adds: tiles of 8 x 64 take half as many passes again and were bound by them (72 % busy).
template <int NP>
__device__ __forceinline__ void dot_tile(const float* a, const float* b, int row0, int column0, int blocks, int tx, int ty,
                                         unsigned long long (&acc)[4][4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
  const float* a_at = a + (row0 + ty) * (NP + 4);
  const float* b_at = b + (column0 + tx) * (NP + 4);
#pragma unroll 4
  for (int n = 0; n < NP; n += 4) {
    ulonglong2 x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const ulonglong2*>(a_at + 4 * i * (NP + 4) + n);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (j >= blocks) continue;
      const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(b_at + 8 * j * (NP + 4) + n);
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i][j] = fma2(x[i].y, w.y, fma2(x[i].x, w.x, acc[i][j]));
    }
  }
}

// The warps' tiles of a chunk's scores: (16 rows, 32 columns) where any column is at or below the diagonal, six of eight, dealt so
// that the two warps of a scheduler (w and w + 4) have few blocks of eight columns together.  blocks: those that a tile needs.
struct Tile { int row0, column0, blocks; };
__device__ __forceinline__ Tile score_tile(int warp) {
  if (warp < 2) return Tile{48, 32 * warp, 4};
  if (warp == 2) return Tile{32, 0, 4};
  if (warp == 3) return Tile{16, 0, 4};
  if (warp == 4) return Tile{32, 32, 2};
  if (warp == 5) return Tile{0, 0, 2};
  return Tile{kC, 0, 0};
}
__device__ __forceinline__ float both(unsigned long long two) {
  float a, b;
  unpack2(two, a, b);
  return a + b;
}

// The product of a chunk's decays of tokens first <= r < end, as four chains of sixteen.  Products of decays are formed in double
// precision and rounded once: their errors would be the same for a whole row of scores, where the walk's fall on each number of S
// alone (float32 products left the delta form's state 1.6 times as far from the definition as the walk's).
__device__ __forceinline__ double decay_between(const double* keep, int first, int end) {
  double p[4] = {1.0, 1.0, 1.0, 1.0};
#pragma unroll
  for (int r = 0; r < 16; ++r)
#pragma unroll
    for (int b = 0; b < 4; ++b)
      if (16 * b + r >= first && 16 * b + r < end) p[b] *= keep[16 * b + r];
  return (p[0] * p[1]) * (p[2] * p[3]);
}

// ------------------------------------------------------------------------------------------------- a chunk's own matrix
// grid (value tiles, heads, chunks).  Bound by its multiply-adds, 64 x 64 x dim a block: a thread has four or eight value columns and
// four key entries, a token costs it a read of keys and one or two of values for eight or sixteen packed multiply-adds.
template <typename T, int FORM, int NP>
__global__ void __launch_bounds__(kThreads, NP == 128 ? 4 : 1)              // (as many as the shared memory has room for)
local_kernel(const Problem p) {
  grid_dependency_wait();
  grid_dependency_launch();
  int count;
  const Where w = chunk_of<kC>(p, blockIdx.z, count);
  if (w.len <= 0) return;
  extern __shared__ __align__(16) float chunk_smem[];
  float* ks = chunk_smem;                     // [64][NP + 4]
  float* vs = ks + kC * (NP + 4);             // [64][kLd]
  double* keep = reinterpret_cast<double*>(vs + kC * kLd);
  float* weight = reinterpret_cast<float*>(keep + kC);
  const int tid = threadIdx.x, head = blockIdx.y, kv_head = head / (p.heads / p.kv_heads), first_column = blockIdx.x * kTile;
  const T* k = reinterpret_cast<const T*>(p.k.at) + (size_t)w.first * p.k.ld + p.k.col + kv_head * p.dim;
  const T* v = reinterpret_cast<const T*>(p.v.at) + (size_t)w.first * p.v.ld + p.v.col + (size_t)head * p.vdim + first_column;
  float2 gate = make_float2(1.f, 0.f);
  if (tid < w.len) gate = gate_of<FORM>(p, w.first + tid, head);
  load_rows<T, NP>(ks, NP + 4, k, p.k.ld, w.len, p.dim, p.wide, p.input_act);
  load_rows<T, kTile>(vs, kLd, v, p.v.ld, w.len, p.vdim - first_column, p.wide, p.input_act);
  if (tid < kC) keep[tid] = gate.x;
  __syncthreads();
  if (tid < kC) {
    const double after = decay_between(keep, tid + 1, kC);         // the decays behind the token
    weight[tid] = tid < w.len ? gate.y * (float)after : 0.f;
    if (tid == 0 && blockIdx.x == 0) p.chunk_decays[w.place * p.heads + head] = (float)(after * keep[0]);
  }
  __syncthreads();
  for (int i = tid; i < kC * (kTile / 4); i += kThreads) {       // the values times their weights
    const int t = i / (kTile / 4);
    float4* at = reinterpret_cast<float4*>(vs + t * kLd + i % (kTile / 4) * 4);
    const float f = weight[t];
    *at = make_float4(f * at->x, f * at->y, f * at->z, f * at->w);
  }
  __syncthreads();
  constexpr int GROUPS = NP / 64;               // of four value columns a thread has
  const int warp = tid >> 5, lane = tid & 31, tx = lane & 7, ty = lane >> 3;
  const int value0 = NP == 128 ? 32 * (warp & 1) + 4 * ty : 16 * (warp >> 1) + 4 * ty;
  const int n = 32 * (NP == 128 ? warp >> 1 : warp & 1) + 4 * tx;
  unsigned long long acc[GROUPS][4][2];
#pragma unroll
  for (int g = 0; g < GROUPS; ++g)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[g][i][0] = acc[g][i][1] = 0ull;
#pragma unroll 4
  for (int s = 0; s < w.len; ++s) {
    const ulonglong2 key = *reinterpret_cast<const ulonglong2*>(ks + s * (NP + 4) + n);
#pragma unroll
    for (int g = 0; g < GROUPS; ++g) {
      const float4 four = *reinterpret_cast<const float4*>(vs + s * kLd + value0 + 16 * g);
      const unsigned long long value[4] = {pack2(four.x, four.x), pack2(four.y, four.y), pack2(four.z, four.z), pack2(four.w, four.w)};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc[g][i][0] = fma2(value[i], key.x, acc[g][i][0]);
        acc[g][i][1] = fma2(value[i], key.y, acc[g][i][1]);
      }
    }
  }
  float* out = p.chunk_states + (w.place * p.heads + head) * (size_t)p.columns * p.dim;
  const bool four_wide = p.dim % 4 == 0;
#pragma unroll
  for (int g = 0; g < GROUPS; ++g)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int column = first_column + value0 + 16 * g + i;
      if (column >= p.vdim) continue;
      float* at = out + (size_t)column * p.dim + n;
      float e[4];
      unpack2(acc[g][i][0], e[0], e[1]);
      unpack2(acc[g][i][1], e[2], e[3]);
      if (four_wide) {
        if (n < p.dim) *reinterpret_cast<float4*>(at) = make_float4(e[0], e[1], e[2], e[3]);
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (n + u < p.dim) at[u] = e[u];
      }
    }
  if (FORM == kMemory && blockIdx.x == 0 && tid < p.dim) {       // the column n: its "value" is 1
    float sum = 0.f;
    for (int s = 0; s < w.len; ++s) sum += weight[s] * ks[s * (NP + 4) + tid];
    out[(size_t)p.vdim * p.dim + tid] = sum;
  }
}

// --------------------------------------------------------------------------------------------------- chunks joined
// grid (pieces of the heads' states, requests), PER numbers a thread: bound by memory (each chunk's matrix read and written once), four
// chunks' matrices requested at a time.
template <int PER> struct alignas(4 * PER) Piece { float v[PER]; };

template <int PER>
__global__ void __launch_bounds__(256)
join_kernel(const Problem p) {
  grid_dependency_wait();
  grid_dependency_launch();
  const Portion portion = portion_of<kC>(p, blockIdx.y);
  const int count = (portion.tokens + kC - 1) / kC;
  const size_t all = (size_t)p.heads * p.columns * p.dim, at = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * PER;
  if (count <= 0 || at >= all) return;
  const int head = (int)(at / ((size_t)p.columns * p.dim));
  const size_t place = portion.place;
  float* kept = p.states + (long long)p.state_slots[portion.request] * p.state_stride + p.state_offset + at;
  Piece<PER> s;
#pragma unroll
  for (int e = 0; e < PER; ++e) s.v[e] = kept[e];
  for (int c0 = 0; c0 < count; c0 += 4) {
    Piece<PER> wrote[4];
    float decay[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (c0 + u >= count) continue;
      wrote[u] = *reinterpret_cast<const Piece<PER>*>(p.chunk_states + (place + c0 + u) * all + at);
      decay[u] = p.chunk_decays[(place + c0 + u) * p.heads + head];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (c0 + u >= count) break;
      *reinterpret_cast<Piece<PER>*>(p.chunk_states + (place + c0 + u) * all + at) = s;
#pragma unroll
      for (int e = 0; e < PER; ++e) s.v[e] = decay[u] * s.v[e] + wrote[u].v[e];
    }
  }
#pragma unroll
  for (int e = 0; e < PER; ++e) kept[e] = s.v[e];
}

// ------------------------------------------------------------------------------------------------------- the rows of y
// Two blocks a multiprocessor, each with a run of the work's units: 64 value columns of a head and a chunk.  Units that share their
// queries and keys (a head's value tiles, the heads of a group) are neighbours, so that a block loads those and forms q k^T, which it
// keeps in registers, once for several units, and the next unit's values and gates are on their way during the last product.  Bound by
// its multiply-adds: q k^T below the diagonal, scores times values, q S_0, which arrives in the keys' place while the values are summed.
// (A block per unit took 151, 79 and 80 us for the selective, memory and delta workloads at the top of this file, this 122, 72 and 77.)
// (neighbouring threads have every fourth column of S_0: those lie in neighbouring rows)
__device__ __forceinline__ int place_of_column(int c) { return (c & 32) + (c & 3) * 8 + ((c >> 2) & 7); }

template <typename T, typename V, int FORM, int NP>
__global__ void __launch_bounds__(kThreads, 2)
read_kernel(const Problem p) {
  grid_dependency_wait();
  grid_dependency_launch();
  extern __shared__ __align__(16) float chunk_smem[];
  float* qs = chunk_smem;                     // [64][NP + 4]
  float* ks = qs + kC * (NP + 4);             // [64][NP + 4], then S_0, value column c in row place_of_column(c)
  float* vs = ks + kC * (NP + 4);             // [64][kLd]
  float* scores = vs + kC * kLd;              // [64][kLd]
  double* keep = reinterpret_cast<double*>(scores + kC * kLd);
  float* weight = reinterpret_cast<float*>(keep + kC);
  float* decayed = weight + kC;               // G_t
  float* n0 = decayed + kC;                   // [NP] (memory form)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, tx = lane & 7, ty = lane >> 3;
  const int tiles = (p.vdim + kTile - 1) / kTile, per_group = p.heads / p.kv_heads;
  const bool four_wide = p.dim % 4 == 0;
  int count;
  chunk_of<kC>(p, 0x7fffffff, count);
  const long long units = (long long)count * p.heads * tiles;
  const long long last = units * (blockIdx.x + 1) / gridDim.x;
  long long unit = units * blockIdx.x / gridDim.x;
  if (unit >= last) return;
  // the unit's place: value tile, head, chunk
  int tile, head, chunk;
  {
    const long long rest = unit / tiles;
    tile = (int)(unit % tiles), head = (int)(rest % p.heads), chunk = (int)(rest / p.heads);
  }
  Where w = chunk_of<kC>(p, chunk, count);
  // values: float32 ones that nothing is done to by asynchronous copies, 16-bit ones through registers, others when their unit begins
  constexpr bool kCopied = sizeof(V) == 4;
  constexpr int kPieces = kC * kTile * (int)sizeof(V) / 16 / kThreads, kEach = 16 / (int)sizeof(V), kPerRow = kTile / kEach;
  uint4 ahead[kCopied ? 1 : kPieces];
  auto request_values = [&]() {
    const int first_column = tile * kTile;
    const V* v = reinterpret_cast<const V*>(p.v.at) + (size_t)w.first * p.v.ld + p.v.col + (size_t)head * p.vdim + first_column;
    if (p.wide && !(kCopied && p.input_act)) {
#pragma unroll
      for (int i = 0; i < kPieces; ++i) {
        const int t = (tid + i * kThreads) / kPerRow, c = (tid + i * kThreads) % kPerRow * kEach;
        const bool real = t < w.len && first_column + c < p.vdim;
        if constexpr (kCopied) cp_async_16(vs + t * kLd + c, v + (real ? (size_t)t * p.v.ld + c : 0), real);
        else ahead[i] = real ? *reinterpret_cast<const uint4*>(v + (size_t)t * p.v.ld + c) : make_uint4(0u, 0u, 0u, 0u);
      }
    }
    cp_async_commit();
  };
  auto place_values = [&]() {
    if (!p.wide || (kCopied && p.input_act)) {
      const int first_column = tile * kTile;
      const V* v = reinterpret_cast<const V*>(p.v.at) + (size_t)w.first * p.v.ld + p.v.col + (size_t)head * p.vdim + first_column;
      load_rows<V, kTile>(vs, kLd, v, p.v.ld, w.len, p.vdim - first_column, p.wide, p.input_act);
    } else if constexpr (!kCopied) {
#pragma unroll
      for (int i = 0; i < kPieces; ++i) {
        const int t = (tid + i * kThreads) / kPerRow, c = (tid + i * kThreads) % kPerRow * kEach;
        const V* from = reinterpret_cast<const V*>(&ahead[i]);
#pragma unroll
        for (int e = 0; e < kEach; e += 4) {
          float4 four = make_float4(to_float(from[e]), to_float(from[e + 1]), to_float(from[e + 2]), to_float(from[e + 3]));
          if (p.input_act) four = make_float4(silu_of(four.x), silu_of(four.y), silu_of(four.z), silu_of(four.w));
          *reinterpret_cast<float4*>(vs + t * kLd + c + e) = four;
        }
      }
    }
  };
  auto gates_of = [&]() { return tid < w.len ? gate_of<FORM>(p, w.first + tid, head) : make_float2(1.f, 0.f); };
  request_values();
  float2 gate = gates_of();
  float raw[4][4];                            // q k^T of the warp's tile
  const Tile own = score_tile(warp);
  const int half = warp >> 2, row0 = 16 * (half ? 3 - (warp & 3) : warp & 3);
  bool new_keys = true, new_head = true;
  for (;; ++unit) {
    __syncthreads();                          // the unit before has been read
    if (new_keys) {
      const int kv_head = head / per_group;
      const T* q = reinterpret_cast<const T*>(p.q.at) + (size_t)w.first * p.q.ld + p.q.col + kv_head * p.dim;
      const T* k = reinterpret_cast<const T*>(p.k.at) + (size_t)w.first * p.k.ld + p.k.col + kv_head * p.dim;
      load_rows<T, NP>(qs, NP + 4, q, p.q.ld, w.len, p.dim, p.wide, p.input_act);
      load_rows<T, NP>(ks, NP + 4, k, p.k.ld, w.len, p.dim, p.wide, p.input_act);
      __syncthreads();
      if (own.row0 < w.len) {
        unsigned long long acc[4][4];
        dot_tile<NP>(qs, ks, own.row0, own.column0, own.blocks, tx, ty, acc);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) raw[i][j] = p.q_scale * both(acc[i][j]);
      }
      __syncthreads();                        // the keys have been read
    }
    const int first_column = tile * kTile;
    const float* start = p.chunk_states + (w.place * p.heads + head) * (size_t)p.columns * p.dim;
    place_values();
    if (four_wide) {
      for (int i = tid; i < kTile * (NP / 4); i += kThreads) {
        const int c = i / (NP / 4), n = i % (NP / 4) * 4;
        const bool real = first_column + c < p.vdim && n < p.dim;
        cp_async_16(ks + place_of_column(c) * (NP + 4) + n, start + (real ? (size_t)(first_column + c) * p.dim + n : 0), real);
      }
    } else {
      for (int i = tid; i < kTile * NP; i += kThreads) {
        const int c = i / NP, n = i % NP;
        ks[place_of_column(c) * (NP + 4) + n] = first_column + c < p.vdim && n < p.dim ? start[(size_t)(first_column + c) * p.dim + n] : 0.f;
      }
    }
    cp_async_commit();
    if (FORM == kMemory && tile == 0 && tid < NP) n0[tid] = tid < p.dim ? start[(size_t)p.vdim * p.dim + tid] : 0.f;
    if (new_head) {
      if (tid < kC) {
        keep[tid] = gate.x;
        weight[tid] = FORM == kDelta ? 1.f : gate.y;
      }
      __syncthreads();
      // scores[t][s] = D(t, s) w_s: a thread has column s and sixteen rows
      const int s = tid & (kC - 1), t0 = (tid >> 6) * 16;
      double product = decay_between(keep, s + 1, t0);
      const float mine = weight[s];
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        if (t0 + r > s) product *= keep[t0 + r];
        scores[(t0 + r) * kLd + s] = (float)product * mine;
      }
      if (tid < kC) decayed[tid] = (float)decay_between(keep, 0, tid + 1);
      __syncthreads();
      if (own.row0 < w.len) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (j < own.blocks) scores[(own.row0 + ty + 4 * i) * kLd + own.column0 + tx + 8 * j] *= raw[i][j];        // (s > t is never read)
      }
    }
    cp_async_wait<1>();
    __syncthreads();                          // values and scores are there
    // results: 16 tokens and 32 value columns a warp, four neighbouring columns a thread; the two warps of a scheduler have 80 tokens' scores
    const bool busy = row0 < w.len;
    unsigned long long out[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i) out[i][0] = out[i][1] = 0ull;
    const float* my_scores = scores + (row0 + ty) * kLd;
    const float* my_values = vs + 32 * half + 4 * tx;
    if (busy) {
      for (int s = 0; s < row0; s += 4) {
        float4 row[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) row[i] = *reinterpret_cast<const float4*>(my_scores + 4 * i * kLd + s);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const ulonglong2 value = *reinterpret_cast<const ulonglong2*>(my_values + (s + u) * kLd);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float f = u == 0 ? row[i].x : u == 1 ? row[i].y : u == 2 ? row[i].z : row[i].w;
            out[i][0] = fma2(pack2(f, f), value.x, out[i][0]);
            out[i][1] = fma2(pack2(f, f), value.y, out[i][1]);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < 16; ++u) {            // the tile's own tokens: each row up to itself
        const ulonglong2 value = *reinterpret_cast<const ulonglong2*>(my_values + (row0 + u) * kLd);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (u <= ty + 4 * i) {
            const float f = my_scores[4 * i * kLd + row0 + u];
            out[i][0] = fma2(pack2(f, f), value.x, out[i][0]);
            out[i][1] = fma2(pack2(f, f), value.y, out[i][1]);
          }
      }
      if (FORM == kSelective) {
        const float skip = p.skip[head];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const ulonglong2 value = *reinterpret_cast<const ulonglong2*>(my_values + (row0 + ty + 4 * i) * kLd);
          out[i][0] = fma2(pack2(skip, skip), value.x, out[i][0]);
          out[i][1] = fma2(pack2(skip, skip), value.y, out[i][1]);
        }
      }
    }
    if (FORM == kMemory && tile == 0) {
      for (int t = 8 * warp; t < min(8 * warp + 8, w.len); ++t) {
        float sum = 0.f, read = 0.f;
#pragma unroll
        for (int s = lane; s < kC; s += 32)
          if (s <= t) sum += scores[t * kLd + s];
#pragma unroll
        for (int n = lane; n < NP; n += 32) read += qs[t * (NP + 4) + n] * n0[n];
        const float total = warp_sum(sum + decayed[t] * p.q_scale * read);
        const size_t at = (size_t)(w.first + t) * p.heads + head;
        if (lane == 0) p.bottom[at] = fmaxf(fabsf(total), p.gates[at * 3 + 2]) + 1e-6f;
      }
    }
    cp_async_wait<0>();
    __syncthreads();                          // S_0 is there, values and scores have been read
    const int my_head = head, my_len = w.len, column = first_column + 32 * half + 4 * tx;
    float* at = p.y + ((size_t)(w.first + row0 + ty) * p.heads + my_head) * p.vdim + column;
    const bool more = unit + 1 < last;
    if (more) {                               // the next unit
      new_keys = new_head = false;
      if (++tile == tiles) {
        tile = 0;
        new_head = true;
        if (++head == p.heads) {
          head = 0;
          w = chunk_of<kC>(p, ++chunk, count);
        }
        new_keys = head % per_group == 0;
      }
      request_values();
      if (new_head) gate = gates_of();
    }
    if (busy) {
      unsigned long long acc[4][4];
      dot_tile<NP>(qs, ks, row0, 32 * half, 4, tx, ty, acc);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = row0 + ty + 4 * i;
        if (t >= my_len) continue;
        const float factor = p.q_scale * decayed[t];
        float e[4];
        unpack2(out[i][0], e[0], e[1]);
        unpack2(out[i][1], e[2], e[3]);
#pragma unroll
        for (int j = 0; j < 4; ++j) e[j] += factor * both(acc[i][j]);
        float* row = at + (size_t)(4 * i) * p.heads * p.vdim;
        if (p.vdim % 4 == 0) {
          if (column < p.vdim) *reinterpret_cast<float4*>(row) = make_float4(e[0], e[1], e[2], e[3]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (column + j < p.vdim) row[j] = e[j];
        }
      }
    }
    if (!more) return;
  }
}

// ------------------------------------------------------------------------------------------- delta: within the chunks
// grid (256 columns of [W | U], heads, chunks).  Forward substitution by sixteen rows: what the rows before them contribute, a read of
// the column's own earlier result and four broadcast reads of A for sixteen multiply-adds, then the sixteen among themselves.
struct Solved { float *w, *u, *ke; };         // [N][heads][dim], [N][heads][vdim], [N][heads][dim]: W, U, D(end, t) k_t

template <typename T, int NP>
__global__ void __launch_bounds__(kThreads, 2)
solve_kernel(const Problem p, const Solved out) {
  grid_dependency_wait();
  grid_dependency_launch();
  int count;
  const Where w = chunk_of<kC>(p, blockIdx.z, count);
  if (w.len <= 0) return;
  extern __shared__ __align__(16) float chunk_smem[];
  float* ks = chunk_smem;                     // [64][NP + 4]
  float* a = ks + kC * (NP + 4);              // [s][t], rows of kLd
  float* x = a + kC * kLd;                    // [48][256]
  double* keep = reinterpret_cast<double*>(x + 48 * kThreads);
  float* beta = reinterpret_cast<float*>(keep + kC);
  float* factor = beta + kC;                  // beta_t G_t
  float* after = factor + kC;                 // D(end, t)
  const int tid = threadIdx.x, head = blockIdx.y, kv_head = head / (p.heads / p.kv_heads);
  const T* k = reinterpret_cast<const T*>(p.k.at) + (size_t)w.first * p.k.ld + p.k.col + kv_head * p.dim;
  const T* v = reinterpret_cast<const T*>(p.v.at) + (size_t)w.first * p.v.ld + p.v.col + (size_t)head * p.vdim;
  float2 gate = make_float2(1.f, 0.f);
  if (tid < w.len) gate = gate_of<kDelta>(p, w.first + tid, head);
  load_rows<T, NP>(ks, NP + 4, k, p.k.ld, w.len, p.dim, p.wide, 0);
  if (tid < kC) {
    keep[tid] = gate.x;
    beta[tid] = gate.y;
  }
  __syncthreads();
  {
    // a[s][t] = beta_t D(t, s): a thread has row t and sixteen s, the latest first
    const int t = tid & (kC - 1), s0 = (tid >> 6) * 16;
    double product = decay_between(keep, s0 + 16, t + 1);
    const float mine = beta[t];
#pragma unroll
    for (int r = 15; r >= 0; --r) {
      a[(s0 + r) * kLd + t] = mine * (float)product;
      if (s0 + r <= t) product *= keep[s0 + r];
    }
    if (tid < kC) {
      factor[tid] = beta[tid] * (float)decay_between(keep, 0, tid + 1);
      const double behind = decay_between(keep, tid + 1, kC);
      after[tid] = (float)behind;
      if (tid == 0 && blockIdx.x == 0) p.chunk_decays[w.place * p.heads + head] = (float)(behind * keep[0]);
    }
  }
  __syncthreads();
  {
    const int lane = tid & 31, tx = lane & 7, ty = lane >> 3;
    const Tile tile = score_tile(tid >> 5);
    if (tile.row0 < w.len) {
      unsigned long long acc[4][4];
      dot_tile<NP>(ks, ks, tile.row0, tile.column0, tile.blocks, tx, ty, acc);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j < tile.blocks) a[(tile.column0 + tx + 8 * j) * kLd + tile.row0 + ty + 4 * i] *= both(acc[i][j]);
    }
    if (blockIdx.x == 0) {                    // the keys as the chunk's end sees them
      float* ke = out.ke + ((size_t)w.first * p.heads + head) * p.dim;
      if (p.dim % 4 == 0) {
        for (int i = tid; i < w.len * (NP / 4); i += kThreads) {
          const int t = i / (NP / 4), n = i % (NP / 4) * 4;
          if (n >= p.dim) continue;
          const float4 key = *reinterpret_cast<const float4*>(ks + t * (NP + 4) + n);
          const float f = after[t];
          *reinterpret_cast<float4*>(ke + (size_t)t * p.heads * p.dim + n) = make_float4(f * key.x, f * key.y, f * key.z, f * key.w);
        }
      } else {
        for (int i = tid; i < w.len * NP; i += kThreads) {
          const int t = i / NP, n = i % NP;
          if (n < p.dim) ke[(size_t)t * p.heads * p.dim + n] = after[t] * ks[t * (NP + 4) + n];
        }
      }
    }
  }
  __syncthreads();
  const int column = blockIdx.x * kThreads + tid;
  const bool of_w = column < p.dim, real = column < p.dim + p.vdim;
  if (!real) return;
  float* result = of_w ? out.w + ((size_t)w.first * p.heads + head) * p.dim + column
                       : out.u + ((size_t)w.first * p.heads + head) * p.vdim + column - p.dim;
  const int result_ld = p.heads * (of_w ? p.dim : p.vdim);
  const T* value = v + (of_w ? 0 : column - p.dim);
  for (int t0 = 0; t0 < w.len; t0 += 16) {
    const int here = min(16, w.len - t0);
    unsigned long long sum[8];                // rows t0 + 2 r, t0 + 2 r + 1
    {
      float right[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        if (of_w) {
          right[r] = factor[t0 + r] * ks[(t0 + r) * (NP + 4) + column];
        } else {
          right[r] = r < here ? to_float(*value) : 0.f;
          if (r < here) value += p.v.ld;
        }
      }
      if (!of_w) {
#pragma unroll
        for (int r = 0; r < 16; ++r) right[r] *= beta[t0 + r];
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) sum[r] = pack2(right[2 * r], right[2 * r + 1]);
    }
#pragma unroll 4
    for (int s = 0; s < t0; ++s) {
      const float before = -x[s * kThreads + tid];
      const unsigned long long two = pack2(before, before);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const ulonglong2 four = *reinterpret_cast<const ulonglong2*>(a + s * kLd + t0 + 4 * r);
        sum[2 * r] = fma2(four.x, two, sum[2 * r]);
        sum[2 * r + 1] = fma2(four.y, two, sum[2 * r + 1]);
      }
    }
    float row[16];
#pragma unroll
    for (int r = 0; r < 8; ++r) unpack2(sum[r], row[2 * r], row[2 * r + 1]);
#pragma unroll
    for (int s = 0; s < 15; ++s)
#pragma unroll
      for (int q = (s + 1) / 4; q < 4; ++q) {
        const float4 four = *reinterpret_cast<const float4*>(a + (t0 + s) * kLd + t0 + 4 * q);
        if (4 * q > s) row[4 * q] = fmaf(-four.x, row[s], row[4 * q]);
        if (4 * q + 1 > s) row[4 * q + 1] = fmaf(-four.y, row[s], row[4 * q + 1]);
        if (4 * q + 2 > s) row[4 * q + 2] = fmaf(-four.z, row[s], row[4 * q + 2]);
        if (4 * q + 3 > s) row[4 * q + 3] = fmaf(-four.w, row[s], row[4 * q + 3]);
      }
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      if (t0 < 48) x[(t0 + r) * kThreads + tid] = row[r];
      if (r < here) {
        *result = row[r];
        result += result_ld;
      }
    }
  }
}

// --------------------------------------------------------------------------------------- delta: from chunk to chunk
// grid (16 value columns, heads, requests): the only part that is a chain, of chunks instead of tokens.  S is in registers, and in shared
// memory for W S_0; beside it lie two chunks of W, D(end, t) k_t and U (the next one on its way).  Both products are cut along the
// sum (key entries by four, tokens by two or four) so that a thread has sixteen results of either, not two or four: the reads of
// shared memory bound them otherwise (a chunk took 4.5 us).
constexpr int kCarry = 16, kPartLd = 20;

template <int NP>
__global__ void __launch_bounds__(kThreads)
carry_kernel(const Problem p, const Solved in) {
  grid_dependency_wait();
  grid_dependency_launch();
  constexpr int LD = NP + 4, NWARPS = NP / 32, TOKENS = 8 / NWARPS;
  extern __shared__ __align__(16) float chunk_smem[];
  float* ws = chunk_smem;                     // [2][64][LD]
  float* es = ws + 2 * kC * LD;               // [2][64][LD]
  float* us = es + 2 * kC * LD;               // [2][64][16]
  float* s_at = us + 2 * kC * kCarry;         // [16][LD]
  float* u_now = s_at + kCarry * LD;          // [64][16]
  float* parts = u_now + kC * kCarry;         // [4][64][kPartLd]: quarters of W S_0; [1 or 3][16][LD]: sums over other threads' tokens
  const int tid = threadIdx.x, head = blockIdx.y, first_column = blockIdx.x * kCarry;
  const Portion portion = portion_of<kC>(p, blockIdx.z);
  // (what is read on the tensor cores starts from every second chunk's S_0)
  const int every = p.records != nullptr ? kChunk / kC : 1;
  const size_t kept_place = p.records != nullptr ? portion_of<kChunk>(p, blockIdx.z).place : portion.place;
  const int request = portion.request, first = portion.first, q_len = portion.tokens, count = (q_len + kC - 1) / kC;
  if (count <= 0) return;
  const size_t place = portion.place;
  const int columns_here = min(kCarry, p.vdim - first_column);
  const bool four_wide = p.dim % 4 == 0, four_values = p.vdim % 4 == 0;
  auto fetch = [&](int c, int stage) {
    const int len = min(kC, q_len - c * kC);
    const size_t token = (size_t)(first + c * kC) * p.heads + head;
    float* to_w = ws + stage * kC * LD;
    float* to_e = es + stage * kC * LD;
    float* to_u = us + stage * kC * kCarry;
    if (four_wide) {
      for (int i = tid; i < kC * (NP / 4); i += kThreads) {
        const int t = i / (NP / 4), n = i % (NP / 4) * 4;
        const bool real = t < len && n < p.dim;
        const size_t at = real ? (token + (size_t)t * p.heads) * p.dim + n : 0;
        cp_async_16(to_w + t * LD + n, in.w + at, real);
        cp_async_16(to_e + t * LD + n, in.ke + at, real);
      }
    } else {
      for (int i = tid; i < kC * NP; i += kThreads) {
        const int t = i / NP, n = i % NP;
        const bool real = t < len && n < p.dim;
        const size_t at = (token + (size_t)t * p.heads) * p.dim + n;
        to_w[t * LD + n] = real ? in.w[at] : 0.f;
        to_e[t * LD + n] = real ? in.ke[at] : 0.f;
      }
    }
    if (four_values) {
      const int t = tid >> 2, c4 = (tid & 3) * 4;
      const bool real = t < len && c4 < columns_here;
      cp_async_16(to_u + t * kCarry + c4, in.u + (real ? (token + (size_t)t * p.heads) * p.vdim + first_column + c4 : 0), real);
    } else {
      for (int i = tid; i < kC * kCarry; i += kThreads) {
        const int t = i / kCarry, c16 = i % kCarry;
        to_u[i] = t < len && c16 < columns_here ? in.u[(token + (size_t)t * p.heads) * p.vdim + first_column + c16] : 0.f;
      }
    }
    cp_async_commit();
  };
  // this thread's part of S: four value columns and four key entries, summed over every TOKENS-th token of a chunk; the threads of the
  // first tokens keep S
  const int warp = tid >> 5, lane = tid & 31, turn = warp / NWARPS;
  const int n = 32 * (warp % NWARPS) + 4 * (lane & 7), column = 4 * (lane >> 3);
  const bool keeps = turn == 0;
  float* kept = p.states + (long long)p.state_slots[request] * p.state_stride + p.state_offset + ((size_t)head * p.vdim + first_column) * p.dim;
  float s[4][4];
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      s[m][e] = keeps && column + m < columns_here && n + e < p.dim ? kept[(size_t)(column + m) * p.dim + n + e] : 0.f;
  auto store = [&](float* to, bool wide) {
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      if (column + m >= columns_here) continue;
      float* at = to + (size_t)(column + m) * p.dim + n;
      if (wide) {
        if (n < p.dim) *reinterpret_cast<float4*>(at) = make_float4(s[m][0], s[m][1], s[m][2], s[m][3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (n + e < p.dim) at[e] = s[m][e];
      }
    }
  };
  fetch(0, 0);
  for (int c = 0; c < count; ++c) {
    const int stage = c & 1, len = min(kC, q_len - c * kC);
    const float decay = p.chunk_decays[(place + c) * p.heads + head];
    if (keeps) {
#pragma unroll
      for (int m = 0; m < 4; ++m) *reinterpret_cast<float4*>(s_at + (column + m) * LD + n) = make_float4(s[m][0], s[m][1], s[m][2], s[m][3]);
    }
    cp_async_wait<0>();
    __syncthreads();                          // this chunk is there, S is there, the chunk before has been read
    if (c + 1 < count) fetch(c + 1, stage ^ 1);
    if (keeps && c % every == 0) store(p.chunk_states + ((kept_place + c / every) * p.heads + head) * (size_t)p.vdim * p.dim + (size_t)first_column * p.dim, four_wide);
    {
      // W S_0 over a quarter of the key entries: tokens t0 + 8 i, columns c0 + 4 j
      const int quarter = warp >> 1, t0 = 32 * (warp & 1) + (lane >> 2), c0 = lane & 3;
      const float* w_at = ws + stage * kC * LD + t0 * LD + quarter * (NP / 4);
      const float* s_row = s_at + c0 * LD + quarter * (NP / 4);
      unsigned long long acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
#pragma unroll
      for (int k = 0; k < NP / 4; k += 4) {
        ulonglong2 four[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) four[i] = *reinterpret_cast<const ulonglong2*>(w_at + 8 * i * LD + k);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const ulonglong2 state = *reinterpret_cast<const ulonglong2*>(s_row + 4 * j * LD + k);
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[i][j] = fma2(four[i].y, state.y, fma2(four[i].x, state.x, acc[i][j]));
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) parts[(quarter * kC + t0 + 8 * i) * kPartLd + c0 + 4 * j] = both(acc[i][j]);
    }
    __syncthreads();
    {
      const int t = tid >> 2, c4 = 4 * (tid & 3);
      float4 u = *reinterpret_cast<const float4*>(us + stage * kC * kCarry + t * kCarry + c4);
      float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 part = *reinterpret_cast<const float4*>(parts + (q * kC + t) * kPartLd + c4);
        sum = make_float4(sum.x + part.x, sum.y + part.y, sum.z + part.z, sum.w + part.w);
      }
      u = make_float4(u.x - sum.x, u.y - sum.y, u.z - sum.z, u.w - sum.w);
      *reinterpret_cast<float4*>(u_now + t * kCarry + c4) = u;
      if (t < len) {
        float* at = in.u + ((size_t)(first + c * kC + t) * p.heads + head) * p.vdim + first_column + c4;
        if (four_values) {
          if (c4 < columns_here) *reinterpret_cast<float4*>(at) = u;
        } else {
          if (c4 < columns_here) at[0] = u.x;
          if (c4 + 1 < columns_here) at[1] = u.y;
          if (c4 + 2 < columns_here) at[2] = u.z;
          if (c4 + 3 < columns_here) at[3] = u.w;
        }
      }
    }
    __syncthreads();
    unsigned long long sum[4][2];
#pragma unroll
    for (int m = 0; m < 4; ++m) sum[m][0] = pack2(decay * s[m][0], decay * s[m][1]), sum[m][1] = pack2(decay * s[m][2], decay * s[m][3]);
    const float* e_at = es + stage * kC * LD + n;
#pragma unroll 8
    for (int t = turn; t < len; t += TOKENS) {
      const ulonglong2 key = *reinterpret_cast<const ulonglong2*>(e_at + t * LD);
      const float4 u = *reinterpret_cast<const float4*>(u_now + t * kCarry + column);
      const unsigned long long value[4] = {pack2(u.x, u.x), pack2(u.y, u.y), pack2(u.z, u.z), pack2(u.w, u.w)};
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        sum[m][0] = fma2(value[m], key.x, sum[m][0]);
        sum[m][1] = fma2(value[m], key.y, sum[m][1]);
      }
    }
    if (!keeps) {
#pragma unroll
      for (int m = 0; m < 4; ++m)
        *reinterpret_cast<ulonglong2*>(parts + ((turn - 1) * kCarry + column + m) * LD + n) = make_ulonglong2(sum[m][0], sum[m][1]);
    }
    __syncthreads();
    if (keeps) {
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        unpack2(sum[m][0], s[m][0], s[m][1]);
        unpack2(sum[m][1], s[m][2], s[m][3]);
#pragma unroll
        for (int t = 1; t < TOKENS; ++t) {
          const float4 part = *reinterpret_cast<const float4*>(parts + ((t - 1) * kCarry + column + m) * LD + n);
          s[m][0] += part.x, s[m][1] += part.y, s[m][2] += part.z, s[m][3] += part.w;
        }
      }
    }
  }
  if (keeps) store(kept, false);
}

// ------------------------------------------------------------------------------------------------------------ launches
constexpr size_t local_bytes(int np) { return sizeof(float) * (size_t)(kC * (np + 4) + kC * kLd + 3 * kC); }
constexpr size_t read_bytes(int np) { return sizeof(float) * (size_t)(2 * kC * (np + 4) + 2 * kC * kLd + 4 * kC + np); }
constexpr size_t solve_bytes(int np) { return sizeof(float) * (size_t)(kC * (np + 4) + kC * kLd + 48 * kThreads + 5 * kC); }
constexpr size_t carry_bytes(int np) { return sizeof(float) * (size_t)(4 * kC * (np + 4) + 3 * kC * kCarry + kCarry * (np + 4) + 4 * kC * kPartLd); }

template <typename T, int FORM, int NP>
static int scan(const Problem& p, const Bounds& most, const Bounds& kept, const Solved& solved, cudaStream_t stream) {
  const int tiles = (p.vdim + kTile - 1) / kTile;
  const dim3 grid(tiles, p.heads, most.chunks);
  const long long units = (long long)tiles * p.heads * most.chunks;                    // at most
  int device = 0, sms = 148;
  if (cudaGetDevice(&device) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  const dim3 readers((unsigned)min(units, 2ll * sms));
  if constexpr (FORM == kDelta) {
    auto solve = solve_kernel<T, NP>;
    auto carry = carry_kernel<NP>;
    auto read = read_kernel<T, float, kDelta, NP>;
    if (allow_shared(solve, solve_bytes(NP)) != cudaSuccess || allow_shared(carry, carry_bytes(NP)) != cudaSuccess ||
        allow_shared(read, read_bytes(NP)) != cudaSuccess)
      MS_FAIL("chunk_scan: shared memory refused");
    ms::launch(solve, dim3((p.dim + p.vdim + kThreads - 1) / kThreads, p.heads, most.chunks), kThreads, solve_bytes(NP), stream, p,
               solved);
    MS_CHECK_LAUNCH("chunk_scan: within the chunks");
    ms::launch(carry, dim3((p.vdim + kCarry - 1) / kCarry, p.heads, most.portions), kThreads, carry_bytes(NP), stream, p, solved);
    MS_CHECK_LAUNCH("chunk_scan: from chunk to chunk");
    Problem reading = p;
    reading.v = Rows{solved.u, p.heads * p.vdim, 0};
    if (p.records != nullptr) {
      reading.v_dtype = MS_F32, reading.v_wide = p.vdim % 4 == 0;
      return launch_read(reading, kept, stream);
    }
    if (p.vdim % 4) reading.wide = 0;
    ms::launch(read, readers, kThreads, read_bytes(NP), stream, reading);
  } else {
    auto local = local_kernel<T, FORM, NP>;
    auto read = read_kernel<T, T, FORM, NP>;
    if (allow_shared(local, local_bytes(NP)) != cudaSuccess || allow_shared(read, read_bytes(NP)) != cudaSuccess)
      MS_FAIL("chunk_scan: shared memory refused");
    ms::launch(local, grid, kThreads, local_bytes(NP), stream, p);
    MS_CHECK_LAUNCH("chunk_scan: chunks alone");
    const bool four = p.dim % 4 == 0;
    const size_t threads = (size_t)p.heads * p.columns * p.dim / (four ? 4 : 1);
    ms::launch(four ? join_kernel<4> : join_kernel<1>, dim3((unsigned)((threads + 255) / 256), most.portions), 256, 0, stream, p);
    MS_CHECK_LAUNCH("chunk_scan: chunks joined");
    ms::launch(read, readers, kThreads, read_bytes(NP), stream, p);
  }
  MS_CHECK_LAUNCH("chunk_scan: rows");
  return 0;
}

template <typename T, int FORM>
static int scan_keys(const Problem& p, const Bounds& most, const Bounds& kept, const Solved& solved, cudaStream_t stream) {
  return p.dim <= 64 ? scan<T, FORM, 64>(p, most, kept, solved, stream) : scan<T, FORM, 128>(p, most, kept, solved, stream);
}

template <typename T>
static int scan_form(int form, const Problem& p, const Bounds& most, const Bounds& kept, const Solved& solved, cudaStream_t stream) {
  if (form == kMemory) return scan_keys<T, kMemory>(p, most, kept, solved, stream);
  if (form == kDelta) return scan_keys<T, kDelta>(p, most, kept, solved, stream);
  return scan_keys<T, kDecay>(p, most, kept, solved, stream);
}

// All of a scan: on the tensor cores where there are records (the decays first, which nothing else waits for long).
static int scan_any(int form, const Problem& p, int n_tokens, const Solved& solved, cudaStream_t stream) {
  const Bounds most = bounds_of<kC>(n_tokens, p.requests, p.least), kept = bounds_of<kChunk>(n_tokens, p.requests, p.least);
  if (p.records != nullptr) {
    if (launch_gates(form, p, kept, stream)) return 1;
    if (form != kDelta) return launch_local(p, kept, stream) || launch_read(p, kept, stream);
  }
  if (form == kSelective) return scan_keys<float, kSelective>(p, most, kept, solved, stream);
  return p.qk_dtype == MS_F32 ? scan_form<float>(form, p, most, kept, solved, stream) : scan_form<__nv_bfloat16>(form, p, most, kept, solved, stream);
}

}  // namespace chunk_scan
}  // namespace ms

using namespace ms;
using namespace ms::chunk_scan;

// The tokens of a chunk (64) if portions of max_query_len tokens can be scanned in chunks, 0 if the walk, token after token, is the only
// way: keys of more than 128 entries, or nothing to scan.  (From which sizes on the scans are ahead is the caller's rule.)
MS_EXPORT int ms_chunk_scan_chunk(int n_requests, int max_query_len, int heads, int dim) {
  return n_requests > 0 && max_query_len > 0 && heads > 0 && heads <= 65535 && dim > 0 && dim <= 128 ? kC : 0;
}

// Tokens of a chunk on the tensor cores, and the floats of such a chunk's record (per head).
MS_EXPORT int ms_chunk_scan_tokens() { return kChunk; }
MS_EXPORT int ms_chunk_scan_record() { return kRecord; }

// Arguments as ms_matrix_scan's forms 0 (memory), 1 (delta) and 2 (constant decay); portions of fewer than `least` tokens are left
// alone.  chunk_states float32 [places, heads, columns, dim] and chunk_decays float32 [places, heads], places = n_tokens / 64 +
// min(n_requests, n_tokens / least), at most 65,535; delta: w, ke float32 [n_tokens, heads, dim], u float32 [n_tokens, heads, vdim].
// records not null: on the tensor cores.  chunk_states has places = n_tokens / 128 + min(n_requests, n_tokens / least) then, and records are
// float32 [those places, heads, ms_chunk_scan_record()]; only the delta form needs chunk_decays; not with input_act.  All on 16-byte
// boundaries.  error_flag: one int on the device that a kernel which gave up waiting sets.
MS_EXPORT int ms_chunk_scan(int form, const void* q, int q_ld, int q_col, const void* k, int k_ld, int k_col, const void* v, int v_ld,
                            int v_col, int dtype, float q_scale, const float* gates, float* states, long long state_stride,
                            int state_offset, const int* state_slots, const int* query_start, int n_requests, int n_tokens, int least,
                            int heads, int kv_heads, int dim, int vdim, float* y, float* bottom, int input_act, float* chunk_states,
                            float* chunk_decays, float* w, float* u, float* ke, float* records, int* error_flag, cudaStream_t stream) {
  if (n_requests == 0 || n_tokens == 0 || heads == 0) return 0;
  MS_REQUIRE(form >= kMemory && form <= kDecay, "chunk_scan: form %d", form);
  MS_REQUIRE(kv_heads > 0 && heads % kv_heads == 0 && dim >= 1 && dim <= 128 && vdim >= 1, "chunk_scan: %d/%d heads of %d/%d", heads,
             kv_heads, dim, vdim);
  MS_REQUIRE(form != kDelta || !input_act, "chunk_scan: the delta form takes its inputs as they are");
  MS_REQUIRE(form != kMemory || bottom != nullptr, "chunk_scan: the memory form writes the tokens' divisors");
  MS_REQUIRE(chunk_states && (chunk_decays || (records && form != kDelta)) && (form != kDelta || (w && u && ke)) && (!records || error_flag),
             "chunk_scan: scratch is missing");
  MS_REQUIRE(!records || !input_act, "chunk_scan: the tensor cores take inputs as they are");
  MS_REQUIRE(dtype == MS_F32 || dtype == MS_BF16, "unknown element type code %d", dtype);
  MS_REQUIRE(least >= 1, "chunk_scan: portions of %d tokens and more", least);
  const Bounds most = bounds_of<kC>(n_tokens, n_requests, least);
  if (most.portions == 0) return 0;
  MS_REQUIRE(heads <= 65535 && most.chunks <= 65535, "chunk_scan: %d heads, %d chunks exceed the launch limits", heads, most.chunks);
  const int per = dtype == MS_F32 ? 4 : 8;
  auto aligned = [](const void* at) { return reinterpret_cast<size_t>(at) % 16 == 0; };
  const int wide = aligned(q) && aligned(k) && aligned(v) && q_ld % per == 0 && k_ld % per == 0 && v_ld % per == 0 && q_col % per == 0 &&
                   k_col % per == 0 && v_col % per == 0 && dim % per == 0 && vdim % per == 0;
  Problem p = {};
  p.q = Rows{q, q_ld, q_col}, p.k = Rows{k, k_ld, k_col}, p.v = Rows{v, v_ld, v_col};
  p.heads = heads, p.kv_heads = kv_heads, p.dim = dim, p.vdim = vdim, p.columns = form == kMemory ? vdim + 1 : vdim;
  p.qk_dtype = p.v_dtype = dtype, p.input_act = input_act, p.wide = p.v_wide = wide, p.q_scale = q_scale, p.gates = gates;
  p.states = states, p.state_stride = state_stride, p.state_offset = state_offset, p.state_slots = state_slots, p.query_start = query_start;
  p.requests = n_requests, p.least = least, p.chunk_states = chunk_states, p.chunk_decays = chunk_decays, p.y = y, p.bottom = bottom;
  p.records = records, p.error_flag = error_flag;
  return scan_any(form, p, n_tokens, Solved{w, u, ke}, stream);
}

// Arguments as ms_selective_scan; `least` and scratch as above with columns = p (a head's channels) and dim = n_state.
MS_EXPORT int ms_selective_chunk_scan(const float* conv, int conv_ld, const void* proj, int dtype, int ld, int dt_col, const float* dt_bias,
                                      const float* a_log, const float* d, float* states, long long state_stride, int state_offset,
                                      const int* state_slots, const int* query_start, int n_requests, int n_tokens, int least, int heads,
                                      int channels, int n_state, int groups, float* y, float* chunk_states, float* chunk_decays,
                                      float* records, int* error_flag, cudaStream_t stream) {
  if (n_requests == 0 || n_tokens == 0) return 0;
  MS_REQUIRE(heads > 0 && groups > 0 && heads % groups == 0, "selective_chunk_scan: %d heads in %d groups", heads, groups);
  MS_REQUIRE(n_state >= 1 && n_state <= 128 && channels >= 1, "selective_chunk_scan: a state of %d numbers for %d channels", n_state, channels);
  MS_REQUIRE(dtype == MS_F32 || dtype == MS_BF16, "unknown element type code %d", dtype);
  MS_REQUIRE(chunk_states && (chunk_decays || (records && error_flag)), "selective_chunk_scan: scratch is missing");
  MS_REQUIRE(least >= 1, "selective_chunk_scan: portions of %d tokens and more", least);
  const Bounds most = bounds_of<kC>(n_tokens, n_requests, least);
  if (most.portions == 0) return 0;
  MS_REQUIRE(heads <= 65535 && most.chunks <= 65535, "selective_chunk_scan: %d heads, %d chunks exceed the launch limits", heads, most.chunks);
  const int inner = heads * channels;
  Problem p = {};
  p.v = Rows{conv, conv_ld, 0}, p.k = Rows{conv, conv_ld, inner}, p.q = Rows{conv, conv_ld, inner + groups * n_state};
  p.heads = heads, p.kv_heads = groups, p.dim = n_state, p.vdim = channels, p.columns = channels;
  p.qk_dtype = p.v_dtype = MS_F32;
  p.wide = p.v_wide = conv_ld % 4 == 0 && inner % 4 == 0 && n_state % 4 == 0 && channels % 4 == 0 && reinterpret_cast<size_t>(conv) % 16 == 0;
  p.q_scale = 1.f;
  p.step = proj, p.step_dtype = dtype, p.step_ld = ld, p.step_col = dt_col, p.step_bias = dt_bias, p.a_log = a_log, p.skip = d;
  p.states = states, p.state_stride = state_stride, p.state_offset = state_offset, p.state_slots = state_slots, p.query_start = query_start;
  p.requests = n_requests, p.least = least, p.chunk_states = chunk_states, p.chunk_decays = chunk_decays, p.y = y;
  p.records = records, p.error_flag = error_flag;
  return scan_any(kSelective, p, n_tokens, Solved{}, stream);
}
