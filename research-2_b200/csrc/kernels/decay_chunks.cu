// Linear attention with one fixed decay per head over prompts, in chunks of 64 rows instead of row by row:
//
//     S_t = decay S_(t-1) + k_t v_t^T,  o_t = S_t^T q_t          (S: [dim x vdim] per head, from the request's slot or zero)
//
// For a chunk that starts with the state S and rows i, j = 0, 1, .. of it:
//
//     o_i = decay^(i + 1) S^T q_i + sum over j <= i of decay^(i - j) (q_i . k_j) v_j
//     state after n rows = decay^n S + U,   U = sum over j of decay^(n - 1 - j) k_j v_j^T
//
// Three launches, the first and the last over all chunks of all entries and heads at once:
//   decay_chunk_sums     U of every chunk (a product over the chunk's rows)
//   decay_chunk_states   entry by entry: every chunk's state at its start (written over U) and the request's new state; elementwise
//   decay_chunk_outputs  o of every chunk: two products with a triangle of decays between them, and one with the chunk's first state
//
// and one for decode steps, in which (nearly) every entry is one row:
//   decay_step           S and o of a row as they are written above, every load of the state in flight at once
//
// The products run on the warp-level tensor cores (mma.sync, bfloat16 with float sums). Everything that enters them is float: silu of
// queries, keys and values (where asked for), powers of the decay, states, weighted scores; each operand is the sum of two bfloat16
// terms (16 bits of mantissa), of whose four products three are taken. States and sums stay float.
//
// Queries and keys that are rotated by position on their way in (retention; in float, so that what enters the recurrence is never
// rounded to 16 bits) take three terms (24 bits, a float's) and the six products above 2^-24 of them; values are then bfloat16
// already and one term. What bounded the walk row by row was its chain, 160 to 270 us for portions of up to 1,000 rows, 12 heads of
// 32 x 64, whatever their number of heads; in chunks the three launches take 32 (700 and 324 rows; 235 row by row on the same GPU).
#include <math.h>

#include "common.cuh"
#include "mma_sync.cuh"

namespace {

constexpr int CHUNK = 64, THREADS = 128, COLS = 64;   // rows of a chunk; four warps; value columns a CTA takes
constexpr int MAX_DIM = 256;

struct ChunkArgs {
  const bf16* q; int q_stride;
  const bf16* k; int k_stride;
  const bf16* v; int v_stride;     // [T, heads * vdim]
  const float* decay;              // [heads]
  float k_scale; int silu_in;
  float* sums;                     // [tiles][heads][dim][vdim]: U, then the states at the chunks' starts
  float* state; long long slot_stride;
  const int32_t* q_start; const int32_t* state_slot; const int32_t* fresh;
  int n_entries;
  float* out; int out_stride;
  int n_heads, dim, vdim, dim16;   // dim16: dim to a multiple of 16
  int vec;                         // rows, heads and slices start on 16-byte boundaries and hold multiples of eight numbers
  const float* inv_freq; int rot_half;   // of q and k the first 2 * rot_half dimensions turn, dimension i with i + rot_half, by the
  const int32_t* positions;              // angle positions[row] * inv_freq[i] (rot_half 0: none do)
};

struct Tile { int entry, row0, rows; };   // entry -1: no such chunk

// Chunks are numbered entry by entry. One warp finds a chunk's entry.
__device__ __forceinline__ Tile find_tile(const int32_t* q_start, int n_entries, int tile) {
  const int lane = threadIdx.x & 31;
  int left = tile;
  for (int base = 0; base < n_entries; base += 32) {
    const int e = base + lane;
    const int first = e < n_entries ? q_start[e] : 0, rows = e < n_entries ? q_start[e + 1] - first : 0;
    const int own = (rows + CHUNK - 1) / CHUNK;
    int upto = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int other = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += other;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, upto > left);
    if (hit != 0) {
      const int at = __ffs(hit) - 1;
      const int within = left - (__shfl_sync(0xffffffffu, upto, at) - __shfl_sync(0xffffffffu, own, at));
      const int row0 = __shfl_sync(0xffffffffu, first, at) + within * CHUNK;
      return {base + at, row0, min(CHUNK, __shfl_sync(0xffffffffu, first + rows, at) - row0)};
    }
    left -= __shfl_sync(0xffffffffu, upto, 31);
  }
  return {-1, 0, 0};
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ float silu(float x) { return __fdividef(x, 1.f + __expf(-x)); }   // (a few units of the last place)
__device__ __forceinline__ uint32_t pack_pair(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// decay^n by squaring (decay^0 is one, also for a decay of zero)
__device__ __forceinline__ float power(float decay, int n) {
  float out = 1.f, square = decay;
  for (; n > 0; n >>= 1, square *= square)
    if (n & 1) out *= square;
  return out;
}

// The same to 48 bits: a float's rounding and what it leaves. (A factor's own error is the same at every chunk, so it adds up over a
// state's memory where roundings cancel: by squaring in float, 900 rows of a decay of 1 - 2^-8 were off by four times the walk's error.)
__device__ __forceinline__ float2 exact_power(float decay, int n) {
  double out = 1.0, square = decay;
  for (; n > 0; n >>= 1, square *= square)
    if (n & 1) out *= square;
  const float head = float(out);
  return make_float2(head, float(out - double(head)));
}
template <int N>
__device__ __forceinline__ float power_for(float decay, int n) { return N > 2 ? exact_power(decay, n).x : power(decay, n); }

// A matrix in shared memory as N bfloat16 terms, rows `stride` numbers apart.
template <int N>
struct Split { bf16* term[N]; int stride; };

template <int N>
__device__ __forceinline__ void put2(const Split<N>& m, int r, int c, float x, float y) {
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint32_t head = pack_pair(x, y);
    *reinterpret_cast<uint32_t*>(m.term[i] + r * m.stride + c) = head;
    if (i + 1 < N) {
      const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&head));
      x -= f.x;
      y -= f.y;
    }
  }
}

// cos and sin of a chunk's rows: [CHUNK][rot_half] each
struct Turns { const float* cos; const float* sin; int half; };
__device__ __forceinline__ Turns make_turns(const ChunkArgs& a, int row0, int rows, float* at) {
  const int half = a.rot_half;
  for (int i = threadIdx.x; i < rows * half; i += THREADS) {
    const int r = i / half, d = i - r * half;
    sincosf(float(a.positions[row0 + r]) * a.inv_freq[d], at + CHUNK * half + i, at + i);
  }
  return {at, at + CHUNK * half, half};
}

// `rows` rows of `cols` numbers (zeros up to CHUNK rows and `padded` columns), turned or silu, times `scale` and, with `powers`, times
// powers[rows - 1 - row].
template <int N>
__device__ __forceinline__ void stage(const Split<N>& m, const bf16* src, long long stride, int rows, int cols, int padded, bool silu_in, float scale,
                                      const float* powers, bool vec, Turns turns = {nullptr, nullptr, 0}) {
  const int pieces = padded / 8;
  for (int i = threadIdx.x; i < CHUNK * pieces; i += THREADS) {
    const int r = i / pieces, c = (i - r * pieces) * 8;
    float x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = 0.f;
    if (r < rows && c < cols) {
      const bf16* p = src + r * stride + c;
      if (vec) {
        const uint4 w = *reinterpret_cast<const uint4*>(p);
        const __nv_bfloat162* w2 = reinterpret_cast<const __nv_bfloat162*>(&w);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float2 f = __bfloat1622float2(w2[u]);
          x[2 * u] = f.x;
          x[2 * u + 1] = f.y;
        }
      } else {
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (c + u < cols) x[u] = to_float(p[u]);
      }
      if (turns.half > 0) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int d = c + u;
          if (d < 2 * turns.half && d < cols) {   // the pair (u, v) becomes (u cos - v sin, v cos + u sin)
            const bool low = d < turns.half;
            const int pair = low ? d : d - turns.half, at = r * turns.half + pair;
            const float other = to_float(src[r * stride + (low ? d + turns.half : pair)]);
            x[u] = fmaf(x[u], turns.cos[at], other * (low ? -turns.sin[at] : turns.sin[at]));
          }
        }
      }
      const float factor = powers != nullptr ? scale * powers[rows - 1 - r] : scale;
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = (silu_in ? silu(x[u]) : x[u]) * factor;
    }
#pragma unroll
    for (int u = 0; u < 8; u += 2) put2(m, r, c + u, x[u], x[u + 1]);
  }
}

// Operand fragments of mma.sync m16n8k16 (lane addresses for ldmatrix).
// a: 16 x 16 of a matrix stored by rows, from (r, c) on
__device__ __forceinline__ void load_a(const bf16* m, int stride, int r, int c, uint32_t (&f)[4]) {
  const int lane = threadIdx.x & 31;
  ldmatrix_x4(smem_u32(m + (r + (lane & 15)) * stride + c + (lane >> 4) * 8), f[0], f[1], f[2], f[3]);
}
// a: 16 x 16 of the transpose of a matrix stored by rows: rows of the operand are the stored columns from c on, its k the stored rows
__device__ __forceinline__ void load_a_transposed(const bf16* m, int stride, int k, int c, uint32_t (&f)[4]) {
  const int lane = threadIdx.x & 31;
  ldmatrix_x4_trans(smem_u32(m + (k + (lane & 7) + (lane >> 4) * 8) * stride + c + ((lane >> 3) & 1) * 8), f[0], f[1], f[2], f[3]);
}
// b: k 16 x n 16 (two tiles of 8 columns: f[0..1], f[2..3]) of a matrix stored by rows of n
__device__ __forceinline__ void load_b(const bf16* m, int stride, int n, int k, uint32_t (&f)[4]) {
  const int lane = threadIdx.x & 31;
  ldmatrix_x4(smem_u32(m + (n + (lane & 7) + (lane >> 4) * 8) * stride + k + ((lane >> 3) & 1) * 8), f[0], f[1], f[2], f[3]);
}
// b: k 16 x n 16 of a matrix stored by rows of k
__device__ __forceinline__ void load_b_transposed(const bf16* m, int stride, int k, int n, uint32_t (&f)[4]) {
  const int lane = threadIdx.x & 31;
  ldmatrix_x4_trans(smem_u32(m + (k + (lane & 15)) * stride + n + (lane >> 4) * 8), f[0], f[1], f[2], f[3]);
}
// (the sum of a's terms)(the sum of b's terms) for one tile of 8 columns, smallest products first; those below the last term of the longer
// operand are left out. The tensor core cuts its sums off instead of rounding them, a bias that grows with every step along K. Three
// terms are there for a float's accuracy, so theirs keeps the large products' sums of 16 apart, added by rounding additions, and the
// small products (2^-8 of them) in an accumulator of their own, `low`. (A prompt of 900 rows, 12 heads of 32 x 64, against 64 bits: the walk
// row by row 2.3e-7, one accumulator for all and powers by squaring in float 6.1e-7, now 1.1e-7.)
template <int N, int M>
__device__ __forceinline__ void mma_split(float (&c)[4], float (&low)[4], const uint32_t (&a)[N][4], const uint32_t (&b)[M][4], int half) {
#pragma unroll
  for (int order = (N > M ? N : M) - 1; order >= 0; --order)
#pragma unroll
    for (int i = N - 1; i >= 0; --i) {
      const int j = order - i;
      if (j < 0 || j >= M) continue;
      const int at = j < 0 || j >= M ? 0 : j;
      if (N == 2) {
        mma_bf16(c, a[i][0], a[i][1], a[i][2], a[i][3], b[at][2 * half], b[at][2 * half + 1]);
      } else if (order > 0) {
        mma_bf16(low, a[i][0], a[i][1], a[i][2], a[i][3], b[at][2 * half], b[at][2 * half + 1]);
      } else {
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
        mma_bf16(sum, a[i][0], a[i][1], a[i][2], a[i][3], b[at][2 * half], b[at][2 * half + 1]);
#pragma unroll
        for (int u = 0; u < 4; ++u) c[u] += sum[u];
      }
    }
}
// the small products' sums join the large ones'
template <int N, int TILES>
__device__ __forceinline__ void join(float (&c)[TILES][4], float (&low)[TILES][4]) {
  if (N == 2) return;
#pragma unroll
  for (int t = 0; t < TILES; ++t)
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      c[t][u] += low[t][u];
      low[t][u] = 0.f;
    }
}

template <int N>
__device__ __forceinline__ Split<N> carve(uint8_t*& at, int rows, int stride) {
  Split<N> m;
#pragma unroll
  for (int i = 0; i < N; ++i) m.term[i] = reinterpret_cast<bf16*>(at) + size_t(i) * rows * stride;
  m.stride = stride;
  at += size_t(rows) * stride * N * sizeof(bf16);
  return m;
}

// N: terms of queries, keys, states and weighted scores; M: of values.
// U of a chunk: [dim x COLS of the value columns]. Grid: chunks, heads, slices of the columns.
template <int N, int M, bool FIXED>
__global__ void __launch_bounds__(THREADS)
decay_chunk_sums_kernel(const ChunkArgs a) {
  pdl_launch_dependents();
  pdl_wait_before_operands<FIXED>();
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ float powers[CHUNK];
  const Tile tile = find_tile(a.q_start, a.n_entries, blockIdx.x);
  const int h = blockIdx.y, col0 = blockIdx.z * COLS, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < CHUNK; i += THREADS) powers[i] = power_for<N>(a.decay[h], i);
  __syncthreads();
  pdl_wait_after_operands<FIXED>();
  if (tile.entry < 0) return;
  uint8_t* at = smem;
  const Split<N> k = carve<N>(at, CHUNK, a.dim16 + 8);
  const Split<M> v = carve<M>(at, CHUNK, COLS + 8);
  Turns turns = {nullptr, nullptr, 0};
  if (a.rot_half > 0) {
    turns = make_turns(a, tile.row0, tile.rows, reinterpret_cast<float*>(at));
    __syncthreads();
  }
  const int cols = min(COLS, a.vdim - col0);
  stage(k, a.k + size_t(tile.row0) * a.k_stride + size_t(h) * a.dim, a.k_stride, tile.rows, a.dim, a.dim16, a.silu_in, a.k_scale, powers, a.vec, turns);
  stage(v, a.v + size_t(tile.row0) * a.v_stride + size_t(h) * a.vdim + col0, a.v_stride, tile.rows, cols, COLS, a.silu_in, 1.f, nullptr, a.vec);
  __syncthreads();
  float* sums = a.sums + (size_t(blockIdx.x) * a.n_heads + h) * a.dim * a.vdim + col0;
  for (int m0 = warp * 16; m0 < a.dim16; m0 += (THREADS / 32) * 16) {
    float acc[COLS / 8][4] = {}, acc_low[COLS / 8][4] = {};
    for (int j = 0; j < tile.rows; j += 16) {
      uint32_t kf[N][4];
#pragma unroll
      for (int i = 0; i < N; ++i) load_a_transposed(k.term[i], k.stride, j, m0, kf[i]);
#pragma unroll
      for (int n = 0; n < COLS; n += 16) {
        uint32_t vf[M][4];
#pragma unroll
        for (int i = 0; i < M; ++i) load_b_transposed(v.term[i], v.stride, j, n, vf[i]);
        mma_split(acc[n / 8], acc_low[n / 8], kf, vf, 0);
        mma_split(acc[n / 8 + 1], acc_low[n / 8 + 1], kf, vf, 1);
      }
    }
    join<N>(acc, acc_low);
#pragma unroll
    for (int t = 0; t < COLS / 8; ++t) {
      const int c = t * 8 + (lane & 3) * 2;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int r = m0 + (lane >> 2) + half * 8;
        if (r < a.dim) {
          float* dst = sums + size_t(r) * a.vdim + c;
          if (c + 1 < cols && (a.vdim & 1) == 0) {
            *reinterpret_cast<float2*>(dst) = make_float2(acc[t][2 * half], acc[t][2 * half + 1]);
          } else {
            if (c < cols) dst[0] = acc[t][2 * half];
            if (c + 1 < cols) dst[1] = acc[t][2 * half + 1];
          }
        }
      }
    }
  }
}

// The states at the chunks' starts, and the request's new one. Grid: entries, heads, pieces of the state.
template <int N, bool FIXED>
__global__ void __launch_bounds__(256)
decay_chunk_states_kernel(const ChunkArgs a) {
  pdl_launch_dependents();
  pdl_wait_before_operands<FIXED>();
  __shared__ float scratch[33];
  const int e = blockIdx.x, h = blockIdx.y;
  const int row0 = a.q_start[e], rows = a.q_start[e + 1] - row0;
  int before = 0;   // chunks of the entries before this one
  for (int i = threadIdx.x; i < e; i += blockDim.x) before += (a.q_start[i + 1] - a.q_start[i] + CHUNK - 1) / CHUNK;
  const int first = int(block_sum(float(before), scratch));   // (small whole numbers: exact)
  const bool is_fresh = a.fresh[e] != 0;
  const int size = a.dim * a.vdim, i = blockIdx.z * blockDim.x + threadIdx.x;
  const float decay = a.decay[h];
  const int last_rows = rows - (rows - 1) / CHUNK * CHUNK;
  const float2 whole = N > 2 ? exact_power(decay, CHUNK) : make_float2(power(decay, CHUNK), 0.f);
  const float2 last = N > 2 ? exact_power(decay, last_rows) : make_float2(power(decay, last_rows), 0.f);
  pdl_wait_after_operands<FIXED>();
  if (rows <= 0 || i >= size) return;   // an entry without rows touches no slot
  float* slot = a.state + size_t(a.state_slot[e]) * a.slot_stride + size_t(h) * size + i;
  float s = is_fresh ? 0.f : *slot;
  float* sums = a.sums + (size_t(first) * a.n_heads + h) * size + i;
  const size_t step = size_t(a.n_heads) * size;
  const int n = (rows + CHUNK - 1) / CHUNK;
  for (int base = 0; base < n; base += 8) {   // eight chunks' sums in flight
    float u[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) u[c] = base + c < n ? sums[(base + c) * step] : 0.f;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      if (base + c < n) {
        sums[(base + c) * step] = s;
        const float2 keep = base + c == n - 1 ? last : whole;
        s = fmaf(keep.x, s, N > 2 ? fmaf(keep.y, s, u[c]) : u[c]);
      }
    }
  }
  *slot = s;
}

// Outputs of a chunk. Grid: chunks, heads, slices of the columns. A warp has 16 of the chunk's rows.
template <int N, int M, bool FIXED>
__global__ void __launch_bounds__(THREADS)
decay_chunk_outputs_kernel(const ChunkArgs a) {
  pdl_launch_dependents();
  pdl_wait_before_operands<FIXED>();
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ float powers[CHUNK + 1];
  const Tile tile = find_tile(a.q_start, a.n_entries, blockIdx.x);
  const int h = blockIdx.y, col0 = blockIdx.z * COLS, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i <= CHUNK; i += THREADS) powers[i] = power_for<N>(a.decay[h], i);
  __syncthreads();
  pdl_wait_after_operands<FIXED>();
  if (tile.entry < 0) return;
  uint8_t* at = smem;
  const Split<N> q = carve<N>(at, CHUNK, a.dim16 + 8), k = carve<N>(at, CHUNK, a.dim16 + 8);
  const Split<M> v = carve<M>(at, CHUNK, COLS + 8);
  const Split<N> s = carve<N>(at, a.dim16, COLS + 8);
  Turns turns = {nullptr, nullptr, 0};
  if (a.rot_half > 0) {
    turns = make_turns(a, tile.row0, tile.rows, reinterpret_cast<float*>(at));
    __syncthreads();
  }
  const int cols = min(COLS, a.vdim - col0);
  stage(q, a.q + size_t(tile.row0) * a.q_stride + size_t(h) * a.dim, a.q_stride, tile.rows, a.dim, a.dim16, a.silu_in, 1.f, nullptr, a.vec, turns);
  stage(k, a.k + size_t(tile.row0) * a.k_stride + size_t(h) * a.dim, a.k_stride, tile.rows, a.dim, a.dim16, a.silu_in, a.k_scale, nullptr, a.vec, turns);
  stage(v, a.v + size_t(tile.row0) * a.v_stride + size_t(h) * a.vdim + col0, a.v_stride, tile.rows, cols, COLS, a.silu_in, 1.f, nullptr, a.vec);
  const float* start = a.sums + (size_t(blockIdx.x) * a.n_heads + h) * a.dim * a.vdim + col0;
  for (int i = threadIdx.x; i < a.dim16 * (COLS / 2); i += THREADS) {
    const int r = i / (COLS / 2), c = (i - r * (COLS / 2)) * 2;
    const float* p = start + size_t(r) * a.vdim + c;
    put2(s, r, c, r < a.dim && c < cols ? p[0] : 0.f, r < a.dim && c + 1 < cols ? p[1] : 0.f);
  }
  __syncthreads();
  const int i0 = warp * 16;
  if (i0 >= tile.rows) return;   // (no barrier follows)
  // what the chunk's first state gives, and the scores of the rows up to each row
  float acc[COLS / 8][4] = {}, acc_low[COLS / 8][4] = {}, p[CHUNK / 8][4] = {}, p_low[CHUNK / 8][4] = {};
  for (int d = 0; d < a.dim16; d += 16) {
    uint32_t qf[N][4];
#pragma unroll
    for (int i = 0; i < N; ++i) load_a(q.term[i], q.stride, i0, d, qf[i]);
#pragma unroll
    for (int n = 0; n < COLS; n += 16) {
      uint32_t sf[N][4];
#pragma unroll
      for (int i = 0; i < N; ++i) load_b_transposed(s.term[i], s.stride, d, n, sf[i]);
      mma_split(acc[n / 8], acc_low[n / 8], qf, sf, 0);
      mma_split(acc[n / 8 + 1], acc_low[n / 8 + 1], qf, sf, 1);
    }
#pragma unroll
    for (int j = 0; j < CHUNK; j += 16) {
      if (j <= i0) {   // (later rows are seen by none of the warp's)
        uint32_t kf[N][4];
#pragma unroll
        for (int i = 0; i < N; ++i) load_b(k.term[i], k.stride, j, d, kf[i]);
        mma_split(p[j / 8], p_low[j / 8], qf, kf, 0);
        mma_split(p[j / 8 + 1], p_low[j / 8 + 1], qf, kf, 1);
      }
    }
  }
  join<N>(acc, acc_low);
  join<N>(p, p_low);
  const int r = i0 + (lane >> 2);   // this lane's rows: r and r + 8
  const float lead0 = powers[r + 1], lead1 = powers[r + 9];
#pragma unroll
  for (int t = 0; t < COLS / 8; ++t) {
    acc[t][0] *= lead0;
    acc[t][1] *= lead0;
    acc[t][2] *= lead1;
    acc[t][3] *= lead1;
  }
#pragma unroll
  for (int j = 0; j < CHUNK; j += 16) {
    if (j > i0) break;
    uint32_t wf[N][4];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float* w = p[j / 8 + half];
      const int c = j + half * 8 + (lane & 3) * 2;
      float w0 = c <= r ? w[0] * powers[r - c] : 0.f, w1 = c + 1 <= r ? w[1] * powers[r - c - 1] : 0.f;
      float w2 = c <= r + 8 ? w[2] * powers[r + 8 - c] : 0.f, w3 = c + 1 <= r + 8 ? w[3] * powers[r + 7 - c] : 0.f;
#pragma unroll
      for (int i = 0; i < N; ++i) {
        wf[i][2 * half] = pack_pair(w0, w1);
        wf[i][2 * half + 1] = pack_pair(w2, w3);
        const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&wf[i][2 * half]));
        const float2 g = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&wf[i][2 * half + 1]));
        w0 -= f.x;
        w1 -= f.y;
        w2 -= g.x;
        w3 -= g.y;
      }
    }
#pragma unroll
    for (int n = 0; n < COLS; n += 16) {
      uint32_t vf[M][4];
#pragma unroll
      for (int i = 0; i < M; ++i) load_b_transposed(v.term[i], v.stride, j, n, vf[i]);
      mma_split(acc[n / 8], acc_low[n / 8], wf, vf, 0);
      mma_split(acc[n / 8 + 1], acc_low[n / 8 + 1], wf, vf, 1);
    }
  }
  join<N>(acc, acc_low);
  float* out = a.out + size_t(h) * a.vdim + col0;
  const bool pairs = (a.vdim & 1) == 0 && (a.out_stride & 1) == 0;
#pragma unroll
  for (int t = 0; t < COLS / 8; ++t) {
    const int c = t * 8 + (lane & 3) * 2;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      if (r + half * 8 < tile.rows) {
        float* dst = out + size_t(tile.row0 + r + half * 8) * a.out_stride + c;
        if (c + 1 < cols && pairs) {
          *reinterpret_cast<float2*>(dst) = make_float2(acc[t][2 * half], acc[t][2 * half + 1]);
        } else {
          if (c < cols) dst[0] = acc[t][2 * half];
          if (c + 1 < cols) dst[1] = acc[t][2 * half + 1];
        }
      }
    }
  }
}

// Decode steps. A CTA has one (entry, head, slice of the columns); a thread has V neighbouring columns of every row_groups-th row, and
// the row groups' sums meet in shared memory, in order.
constexpr int STEP_THREADS = 128, STEP_ROWS = 8;
template <int V, bool FIXED>
__global__ void __launch_bounds__(STEP_THREADS)
decay_step_kernel(const ChunkArgs a, int slice) {
  pdl_launch_dependents();
  pdl_wait_before_operands<FIXED>();
  __shared__ float qs[MAX_DIM], ks[MAX_DIM], sums[STEP_THREADS][V];
  const int e = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * slice;
  const int row0 = a.q_start[e], row1 = a.q_start[e + 1];
  const bool is_fresh = a.fresh[e] != 0;
  const float decay = a.decay[h];
  const int groups = slice / V, row_groups = STEP_THREADS / groups;   // (groups divides the threads)
  const int g = threadIdx.x % groups, rg = threadIdx.x / groups, j = col0 + g * V;
  const bool mine = j < a.vdim;
  float* head_state = a.state + size_t(a.state_slot[e]) * a.slot_stride + size_t(h) * a.dim * a.vdim;
  pdl_wait_after_operands<FIXED>();
  for (int t = row0; t < row1; ++t) {
    const bool zero = is_fresh && t == row0;
    float s[STEP_ROWS][V], v[V], acc[V] = {};
#pragma unroll
    for (int i = 0; i < STEP_ROWS; ++i) {   // the first rows' states, asked for before anything is waited for
      const int r = rg + i * row_groups;
#pragma unroll
      for (int u = 0; u < V; ++u) s[i][u] = 0.f;
      if (mine && r < a.dim && !zero) {
        const float* p = head_state + size_t(r) * a.vdim + j;
        if (V == 4) {
          const float4 f = *reinterpret_cast<const float4*>(p);
          s[i][0] = f.x;
          s[i][V > 1 ? 1 : 0] = f.y;
          s[i][V > 2 ? 2 : 0] = f.z;
          s[i][V > 3 ? 3 : 0] = f.w;
        } else {
          s[i][0] = *p;
        }
      }
    }
    const bf16* q = a.q + size_t(t) * a.q_stride + size_t(h) * a.dim;
    const bf16* k = a.k + size_t(t) * a.k_stride + size_t(h) * a.dim;
    for (int i = threadIdx.x; i < a.dim; i += STEP_THREADS) {
      float x = to_float(q[i]), y = to_float(k[i]);
      if (i < 2 * a.rot_half) {
        const bool low = i < a.rot_half;
        const int other = low ? i + a.rot_half : i - a.rot_half;
        float sn, cs;
        sincosf(float(a.positions[t]) * a.inv_freq[low ? i : other], &sn, &cs);
        if (low) sn = -sn;
        x = fmaf(x, cs, to_float(q[other]) * sn);
        y = fmaf(y, cs, to_float(k[other]) * sn);
      }
      qs[i] = a.silu_in ? silu(x) : x;
      ks[i] = (a.silu_in ? silu(y) : y) * a.k_scale;
    }
#pragma unroll
    for (int u = 0; u < V; ++u) {
      const float x = mine ? to_float(a.v[size_t(t) * a.v_stride + size_t(h) * a.vdim + j + u]) : 0.f;
      v[u] = a.silu_in ? silu(x) : x;
    }
    __syncthreads();
    auto row = [&](int r, float (&state)[V]) {
#pragma unroll
      for (int u = 0; u < V; ++u) {
        state[u] = fmaf(decay, state[u], ks[r] * v[u]);
        acc[u] = fmaf(state[u], qs[r], acc[u]);
      }
      float* p = head_state + size_t(r) * a.vdim + j;
      if (V == 4) *reinterpret_cast<float4*>(p) = make_float4(state[0], state[V > 1 ? 1 : 0], state[V > 2 ? 2 : 0], state[V > 3 ? 3 : 0]);
      else *p = state[0];
    };
    if (mine) {
#pragma unroll
      for (int i = 0; i < STEP_ROWS; ++i)
        if (rg + i * row_groups < a.dim) row(rg + i * row_groups, s[i]);
      for (int r = rg + STEP_ROWS * row_groups; r < a.dim; r += row_groups) {
        const float* p = head_state + size_t(r) * a.vdim + j;
        float state[V];
#pragma unroll
        for (int u = 0; u < V; ++u) state[u] = zero ? 0.f : p[u];
        row(r, state);
      }
    }
#pragma unroll
    for (int u = 0; u < V; ++u) sums[threadIdx.x][u] = acc[u];
    __syncthreads();
    if (rg == 0 && mine) {
#pragma unroll
      for (int u = 0; u < V; ++u) {
        float o = 0.f;
        for (int i = 0; i < row_groups; ++i) o += sums[i * groups + g][u];
        a.out[size_t(t) * a.out_stride + size_t(h) * a.vdim + j + u] = o;
      }
    }
    __syncthreads();   // (the vectors and sums of the next row)
  }
}

size_t split_bytes(int rows, int stride, int terms) { return size_t(rows) * stride * terms * sizeof(bf16); }

template <int N, int M, bool FIXED>
int launch_chunks(const ChunkArgs& a, int n_tiles, cudaStream_t stream) {
  const size_t rows_q = split_bytes(CHUNK, a.dim16 + 8, N), rows_v = split_bytes(CHUNK, COLS + 8, M), turns = size_t(2) * CHUNK * a.rot_half * sizeof(float);
  const size_t smem_sums = rows_q + rows_v + turns, smem_out = 2 * rows_q + rows_v + split_bytes(a.dim16, COLS + 8, N) + turns;
  constexpr size_t MOST = 226 * 1024;   // (beside the kernels' own few hundred bytes)
  if (smem_out > MOST) return R2_UNSUPPORTED;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(decay_chunk_outputs_kernel<N, M, FIXED>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(MOST));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(decay_chunk_sums_kernel<N, M, FIXED>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(MOST));
    if (e != cudaSuccess) {
      cudaGetLastError();
      return R2_UNSUPPORTED;
    }
    configured = true;
  }
  const dim3 grid(n_tiles, a.n_heads, (a.vdim + COLS - 1) / COLS);
  r2_launch(decay_chunk_sums_kernel<N, M, FIXED>, grid, dim3(THREADS), smem_sums, stream, a);
  r2_launch(decay_chunk_states_kernel<N, FIXED>, dim3(a.n_entries, a.n_heads, (a.dim * a.vdim + 255) / 256), dim3(256), size_t(0), stream, a);
  r2_launch(decay_chunk_outputs_kernel<N, M, FIXED>, grid, dim3(THREADS), smem_out, stream, a);
  return launch_status();
}

}  // namespace

// Floats of scratch for a batch whose entries have n_tiles chunks in all (each entry's last chunk may be short).
extern "C" long long r2_decay_chunks_floats(int n_tiles, int n_heads, int dim, int vdim) { return (long long)n_tiles * n_heads * dim * vdim; }

// q, k [T, heads * dim], v [T, heads * vdim] bfloat16 (slices of a projection); decay float [heads]; silu_in: silu of all three on their
// way in, k then times k_scale; state float [slots][heads][dim][vdim]; n_tiles at least the sum over entries of ceil(rows / 64); scratch
// float (r2_decay_chunks_floats); out float [T, heads * vdim]. inv_freq float [rot_half] and positions [T] where q and k turn (then without
// silu). `fixed` (here and below): no launch shortly before writes the decays or the batch's arrays, which are then read ahead of the wait
// for it. Three launches. R2_UNSUPPORTED: heads of more than 256 rows (fewer, where they turn: what an SM's shared memory holds).
extern "C" int r2_decay_chunks(const void* q, int q_stride, const void* k, int k_stride, const void* v, int v_stride, const float* decay, float k_scale,
                               int silu_in, float* state, long long slot_stride, const int32_t* q_start, const int32_t* state_slot, const int32_t* fresh,
                               int n_entries, int n_tiles, float* scratch, long long scratch_floats, float* out, int out_stride, int n_heads, int dim,
                               int vdim, const float* inv_freq, int rot_half, const int32_t* positions, int fixed, cudaStream_t stream) {
  if (n_entries <= 0 || n_tiles <= 0) return R2_OK;
  if (rot_half < 0 || 2 * rot_half > dim || (rot_half > 0 && (inv_freq == nullptr || positions == nullptr || silu_in))) return R2_BAD_SHAPE;
  if (n_heads < 1 || dim < 1 || vdim < 1 || scratch == nullptr || scratch_floats < r2_decay_chunks_floats(n_tiles, n_heads, dim, vdim)) return R2_BAD_SHAPE;
  if (dim > MAX_DIM || n_heads > 65535 || n_tiles > (1 << 20)) return R2_UNSUPPORTED;
  ChunkArgs a = {};
  a.q = (const bf16*)q; a.q_stride = q_stride; a.k = (const bf16*)k; a.k_stride = k_stride; a.v = (const bf16*)v; a.v_stride = v_stride;
  a.decay = decay; a.k_scale = k_scale; a.silu_in = silu_in; a.sums = scratch; a.state = state; a.slot_stride = slot_stride;
  a.q_start = q_start; a.state_slot = state_slot; a.fresh = fresh; a.n_entries = n_entries; a.out = out; a.out_stride = out_stride;
  a.n_heads = n_heads; a.dim = dim; a.vdim = vdim; a.dim16 = (dim + 15) / 16 * 16;
  a.vec = dim % 8 == 0 && vdim % 8 == 0 && q_stride % 8 == 0 && k_stride % 8 == 0 && v_stride % 8 == 0 &&
          !((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) & 15);
  a.inv_freq = inv_freq; a.rot_half = rot_half; a.positions = positions;
  if (rot_half > 0) return fixed ? launch_chunks<3, 1, true>(a, n_tiles, stream) : launch_chunks<3, 1, false>(a, n_tiles, stream);
  return fixed ? launch_chunks<2, 2, true>(a, n_tiles, stream) : launch_chunks<2, 2, false>(a, n_tiles, stream);
}

// The same for batches in which (nearly) every entry is one row: one launch, no scratch.
extern "C" int r2_decay_step(const void* q, int q_stride, const void* k, int k_stride, const void* v, int v_stride, const float* decay, float k_scale,
                             int silu_in, float* state, long long slot_stride, const int32_t* q_start, const int32_t* state_slot, const int32_t* fresh,
                             int n_entries, float* out, int out_stride, int n_heads, int dim, int vdim, int n_sms, const float* inv_freq, int rot_half,
                             const int32_t* positions, int fixed, cudaStream_t stream) {
  if (n_entries <= 0) return R2_OK;
  if (rot_half < 0 || 2 * rot_half > dim || (rot_half > 0 && (inv_freq == nullptr || positions == nullptr || silu_in))) return R2_BAD_SHAPE;
  if (n_heads < 1 || dim < 1 || vdim < 1 || n_sms < 1) return R2_BAD_SHAPE;
  if (dim > MAX_DIM || n_heads > 65535) return R2_UNSUPPORTED;
  ChunkArgs a = {};
  a.q = (const bf16*)q; a.q_stride = q_stride; a.k = (const bf16*)k; a.k_stride = k_stride; a.v = (const bf16*)v; a.v_stride = v_stride;
  a.decay = decay; a.k_scale = k_scale; a.silu_in = silu_in; a.state = state; a.slot_stride = slot_stride;
  a.q_start = q_start; a.state_slot = state_slot; a.fresh = fresh; a.n_entries = n_entries; a.out = out; a.out_stride = out_stride;
  a.n_heads = n_heads; a.dim = dim; a.vdim = vdim;
  a.inv_freq = inv_freq; a.rot_half = rot_half; a.positions = positions;
  // as many columns a CTA as leave twice as many CTAs as the GPU has SMs
  int slice = 64;
  while (slice > 16 && (long long)n_entries * n_heads * ((vdim + slice - 1) / slice) < 2ll * n_sms) slice /= 2;
  const dim3 grid(n_entries, n_heads, (vdim + slice - 1) / slice);
  const bool quads = vdim % 4 == 0 && slot_stride % 4 == 0 && !(reinterpret_cast<uintptr_t>(state) & 15);
  auto go = [&](auto kernel) { r2_launch(kernel, grid, dim3(STEP_THREADS), size_t(0), stream, a, slice); };
  if (quads) fixed ? go(decay_step_kernel<4, true>) : go(decay_step_kernel<4, false>);
  else fixed ? go(decay_step_kernel<1, true>) : go(decay_step_kernel<1, false>);
  return launch_status();
}
