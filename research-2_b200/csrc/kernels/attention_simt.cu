// Paged causal attention on the CUDA cores, all arithmetic in float: the true 32-bit path, and
// the general path of the bfloat16 engine for head sizes or batches the tensor-core kernels refuse.
//
// A CTA computes one (row, head): the row's visible keys are cut into tiles of 32 in position order, tile i is warp i % 8's. A warp
// keeps a running maximum and sum (online softmax) over its tiles (lane = key for the scores, lanes over the head dimension for
// P.V), and the eight warps' parts are merged in warp order at the end. The walk depends only on the row's position, its window and
// the head size, never on how the step was cut or batched, so a row's output is the same bits
// whichever batch it came in. What bounds it is the latency of its loads: a key row is read in 16-byte pieces, eight of them in flight
// (sixteen, a whole row, for float heads of up to 64), a tile's value rows sixteen at a time for heads of up to 64, eight for up
// to 128 and one after the other beyond, where a lane's share of a row is eight numbers and more; and eight warps share a row's
// keys (3 rows x 12 heads of 64, float, 200 keys: 148 us with one warp a (row, head) and one number a load, 14 us now; 332 rows: 242
// and 71 us). It also takes what the fast kernels leave out: a value head size that
// differs from the key's, a window that keeps a sequence's first keys, a sink in the softmax's
// denominator, an output gate, chunks, a bias by distance, and values that are the first numbers of the key rows themselves (a
// cache of latents: the value pointer is the key pointer and a value row is as long as a key row).
//
// Reference formulas: kelpie-models/kelpie_models/kernels/ops/paged_attention.py:160-240
// (scores * scale 179, visibility 186-212, softmax 215-240, PV 182-183, pad rows zero 140).
#include <math.h>

#include "common.cuh"

namespace {

constexpr int WARPS = 8;
constexpr int WIDE_HEAD_DIM = 1024;   // an instance takes rows of up to this many numbers (a cache of long latents)

__device__ __forceinline__ void widen(const uint4& w, float (&x)[4]) {
  x[0] = __uint_as_float(w.x);
  x[1] = __uint_as_float(w.y);
  x[2] = __uint_as_float(w.z);
  x[3] = __uint_as_float(w.w);
}
__device__ __forceinline__ void widen(const uint4& w, float (&x)[8]) {
  const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    x[2 * i] = __uint_as_float(u[i] << 16);
    x[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
  }
}

// q . k over head_dim numbers; VEC: in 16-byte pieces, AT_ONCE of them in flight, the sums of every fourth column apart.
template <typename T, bool VEC, int AT_ONCE>
__device__ __forceinline__ float dot_row(const float* q, const T* k, int head_dim) {
  if (!VEC) {
    float dot = 0.f;
#pragma unroll 8
    for (int d = 0; d < head_dim; ++d) dot = fmaf(q[d], to_float(k[d]), dot);
    return dot;
  }
  constexpr int N = 16 / sizeof(T);
  const uint4* row = reinterpret_cast<const uint4*>(k);
  float part[4] = {0.f, 0.f, 0.f, 0.f};
  const int pieces = head_dim / N;
  int i = 0;
  for (; i + AT_ONCE <= pieces; i += AT_ONCE) {
    uint4 w[AT_ONCE];
#pragma unroll
    for (int u = 0; u < AT_ONCE; ++u) w[u] = row[i + u];
#pragma unroll
    for (int u = 0; u < AT_ONCE; ++u) {
      float x[N];
      widen(w[u], x);
#pragma unroll
      for (int c = 0; c < N; ++c) part[c % 4] = fmaf(q[(i + u) * N + c], x[c], part[c % 4]);
    }
  }
  for (; i < pieces; ++i) {
    float x[N];
    widen(row[i], x);
#pragma unroll
    for (int c = 0; c < N; ++c) part[c % 4] = fmaf(q[i * N + c], x[c], part[c % 4]);
  }
  return (part[0] + part[1]) + (part[2] + part[3]);
}

template <typename T, int MAX_HEAD_DIM, bool VEC>
__global__ void __launch_bounds__(WARPS * 32)
attention_simt_kernel(const T* __restrict__ q, int q_row_stride, T* __restrict__ out, int out_row_stride,
                      const T* __restrict__ k_cache, const T* __restrict__ v_cache, long long page_stride,
                      int page_size, int page_shift, const int32_t* __restrict__ block_tables, int table_width,
                      const int32_t* __restrict__ row_entry, const int32_t* __restrict__ positions,
                      const int32_t* __restrict__ seq_lens, int n_heads, int n_kv_heads, int head_dim, int v_head_dim,
                      float scale, int window, int keep_first, int sink, const T* __restrict__ gate, int gate_row_stride,
                      int n_pages, float softcap, const float* __restrict__ sinks, const float* __restrict__ head_gate,
                      int head_gate_stride, int v_row_stride, int chunk, const float* __restrict__ dist_bias, int bias_len,
                      float out_scale) {
  constexpr int PER_LANE = MAX_HEAD_DIM / 32;
  pdl_launch_dependents();  // the next kernel may begin its prologue
  __shared__ __align__(16) float q_s[MAX_HEAD_DIM];
  __shared__ float part_s[WARPS][MAX_HEAD_DIM];
  __shared__ float max_s[WARPS], sum_s[WARPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x, h = blockIdx.y;
  pdl_wait();               // the previous kernel's writes are visible from here on (the index arrays may be among them)
  const int e = row_entry[t];
  const int pos = e < 0 ? 0 : positions[t], seq_len = e < 0 ? 0 : seq_lens[e];
  T* o = out + size_t(t) * out_row_stride + size_t(h) * v_head_dim;
  if (e < 0) {  // a pad row
    for (int d = threadIdx.x; d < v_head_dim; d += WARPS * 32) o[d] = from_float<T>(0.f);
    return;
  }
  const int kvh = h / (n_heads / n_kv_heads);
  const int32_t* table = block_tables + size_t(e) * table_width;
  const T* qr = q + size_t(t) * q_row_stride + size_t(h) * head_dim;
  for (int d = threadIdx.x; d < head_dim; d += WARPS * 32) q_s[d] = to_float(qr[d]);
  __syncthreads();

  const int last = pos < seq_len - 1 ? pos : seq_len - 1;       // newest visible key
  const int first = chunk > 0 ? pos / chunk * chunk : (window > 0 ? (pos - window + 1 > 0 ? pos - window + 1 : 0) : 0);
  const float* bias = dist_bias != nullptr ? dist_bias + size_t(h) * bias_len : nullptr;
  // With a window, the sequence's first `keep_first` keys stay visible: they are walked first, as a
  // range of their own, so that the walk depends on the row's position alone.
  const int kept = window > 0 ? (keep_first < first ? keep_first : first) : 0;
  const int kept_tiles = (kept + 31) / 32, n_tiles = kept_tiles + (last >= first ? (last - first) / 32 + 1 : 0);
  float m = -INFINITY, l = 0.f;
  float acc[PER_LANE];
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) acc[i] = 0.f;
  const size_t k_head_off = size_t(kvh) * page_size * head_dim;
  const size_t v_head_off = size_t(kvh) * page_size * v_row_stride;

  for (int tile = warp; tile < n_tiles; tile += WARPS) {
    const int j0 = tile < kept_tiles ? tile * 32 : first + (tile - kept_tiles) * 32;
    const int hi = tile < kept_tiles ? kept - 1 : last;
    const int j = j0 + lane;
    const bool valid = j <= hi;
    const int n_valid = hi - j0 + 1 < 32 ? hi - j0 + 1 : 32;
    constexpr int AHEAD = PER_LANE <= 2 ? 16 : PER_LANE <= 4 ? 8 : 1;   // value rows whose loads are in flight together
    float s = -INFINITY;
    long long v_off = 0;
    const T* kr = k_cache;
    if (valid) {
      int page = table[page_index(j, page_size, page_shift)];
      page = (page < 0 || page >= n_pages) ? 0 : page;
      const int within = page_offset(j, page_size, page_shift);
      v_off = (long long)page * page_stride + (long long)(v_head_off + size_t(within) * v_row_stride);
      kr += size_t(page) * page_stride + k_head_off + size_t(within) * head_dim;
    }
    float v[AHEAD][PER_LANE];
    auto load_values = [&](int jj) {
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        const T* vr = v_cache + __shfl_sync(0xffffffffu, v_off, jj + u);
#pragma unroll
        for (int i = 0; i < PER_LANE; ++i) v[u][i] = lane + 32 * i < v_head_dim ? to_float(vr[lane + 32 * i]) : 0.f;
      }
    };
    const bool first_ahead = AHEAD > 1 && n_valid >= AHEAD;
    if (first_ahead) load_values(0);   // (they do not wait for the scores)
    if (valid) {
      s = dot_row<T, VEC, (MAX_HEAD_DIM <= 64 && sizeof(T) == 4 ? 16 : 8)>(q_s, kr, head_dim) * scale;
      if (softcap > 0.f) s = softcap * tanhf(s / softcap);   // scores are capped before the softmax
      if (bias != nullptr) s += bias[pos - j < bias_len ? pos - j : bias_len - 1];
    }
    const float m_new = fmaxf(m, warp_max(s));
    // (a warp whose keys so far all score -inf, a bias that forbids their distance, has nothing to measure by: its weights are 0, not NaN)
    const float base = m_new == -INFINITY ? 0.f : m_new;
    const float corr = expf(m - base);  // exp(-inf) = 0 on the first tile
    const float p = valid ? expf(s - base) : 0.f;
    l = l * corr + warp_sum(p);
    m = m_new;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) acc[i] *= corr;
    int jj = 0;
    for (; jj + AHEAD <= n_valid; jj += AHEAD) {
      if (jj > 0 || !first_ahead) load_values(jj);
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        const float pj = __shfl_sync(0xffffffffu, p, jj + u);
#pragma unroll
        for (int i = 0; i < PER_LANE; ++i) acc[i] = fmaf(pj, v[u][i], acc[i]);
      }
    }
    for (; jj < n_valid; ++jj) {
      const float pj = __shfl_sync(0xffffffffu, p, jj);
      const T* vr = v_cache + __shfl_sync(0xffffffffu, v_off, jj);
#pragma unroll
      for (int i = 0; i < PER_LANE; ++i)
        if (lane + 32 * i < v_head_dim) acc[i] = fmaf(pj, to_float(vr[lane + 32 * i]), acc[i]);
    }
  }

  // the warps' parts, merged in warp order
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i)
    if (lane + 32 * i < v_head_dim) part_s[warp][lane + 32 * i] = acc[i];
  if (lane == 0) {
    max_s[warp] = m;
    sum_s[warp] = l;
  }
  __syncthreads();
  // a sink: an extra term in the sum and nothing in the output; exp(0), or exp(sinks[h]) where heads have learned ones
  const bool has_sink = sink || sinks != nullptr;
  const float sink_at = sinks != nullptr ? sinks[h] : 0.f;
  const int used = n_tiles < WARPS ? n_tiles : WARPS;
  float top = has_sink ? sink_at : -INFINITY;
  for (int w = 0; w < used; ++w) top = fmaxf(top, max_s[w]);
  if (top == -INFINITY) top = 0.f;   // no key and no sink: every share is 0
  float share[WARPS], total = has_sink ? expf(sink_at - top) : 0.f;
#pragma unroll
  for (int w = 0; w < WARPS; ++w) {
    share[w] = w < used ? expf(max_s[w] - top) : 0.f;
    if (w < used) total = fmaf(sum_s[w], share[w], total);
  }
  float inv = total > 0.f ? out_scale / total : 0.f;
  const T* gr = gate != nullptr ? gate + size_t(t) * gate_row_stride + size_t(h) * v_head_dim : nullptr;
  // one gate per head: sigmoid of a float logit
  if (head_gate != nullptr) inv *= 1.f / (1.f + expf(-head_gate[size_t(t) * head_gate_stride + h]));
  for (int d = threadIdx.x; d < v_head_dim; d += WARPS * 32) {
    float y = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w)
      if (w < used) y = fmaf(part_s[w][d], share[w], y);
    y *= inv;
    if (gr != nullptr) y *= 1.f / (1.f + expf(-to_float(gr[d])));   // the output gate: sigmoid of the gate's column
    o[d] = from_float<T>(y);
  }
}

}  // namespace

// q [T, n_heads * head_dim] with row stride q_row_stride (it may be a slice of a fused projection),
// out [T, n_heads * v_head_dim]; the cache of this layer as in r2_kv_write. `window` > 0 limits a row
// at position p to the keys (p - window, p] and, with `keep_first`, the sequence's first keep_first keys;
// `sink` adds one to the softmax's denominator; `gate` (may be null; [T, n_heads * v_head_dim] with its
// own row stride) multiplies the output by its sigmoid. `softcap` > 0 caps the scaled scores (cap * tanh(s / cap));
// `sinks` (may be null; float [n_heads]) puts exp(sinks[h]) into head h's denominator; `head_gate` (may be null; float
// [T, n_heads] with its own row stride) multiplies head h's output by the sigmoid of its entry. `v_row_stride` (0: v_head_dim)
// is the length of a value row in the cache: with v_cache = k_cache and v_row_stride = head_dim the values are the first
// v_head_dim numbers of the keys. `chunk` > 0 (without a window) limits a row at position p to the keys of its own chunk,
// [p / chunk * chunk, p]. `dist_bias` (may be null; float [n_heads][bias_len]) is added to head h's score of a key n positions
// back: its entry n, the last entry for every larger n. `out_scale` multiplies the output.
extern "C" int r2_attention_simt(const void* q, int q_row_stride, void* out, int out_row_stride, const void* k_cache,
                                 const void* v_cache, long long page_stride, int page_size,
                                 const int32_t* block_tables, int table_width, const int32_t* row_entry,
                                 const int32_t* positions, const int32_t* seq_lens, int n_rows, int n_heads,
                                 int n_kv_heads, int head_dim, int v_head_dim, float scale, int window, int keep_first,
                                 int sink, const void* gate, int gate_row_stride, int n_pages, int dtype,
                                 float softcap, const float* sinks, const float* head_gate, int head_gate_stride,
                                 int v_row_stride, int chunk, const float* dist_bias, int bias_len, float out_scale,
                                 cudaStream_t stream) {
  if (n_rows <= 0) return R2_OK;
  if (head_dim < 1 || head_dim > WIDE_HEAD_DIM || v_head_dim < 1 || v_head_dim > WIDE_HEAD_DIM) return R2_UNSUPPORTED;
  if (n_heads < 1 || n_kv_heads < 1 || n_heads % n_kv_heads != 0 || page_size < 1 || window < 0 || keep_first < 0 || chunk < 0) return R2_BAD_SHAPE;
  if ((chunk > 0 && window > 0) || (dist_bias != nullptr && bias_len < 1)) return R2_BAD_SHAPE;
  if (v_row_stride <= 0) v_row_stride = v_head_dim;   // values in rows of their own
  if (v_row_stride < v_head_dim) return R2_BAD_SHAPE;
  if (dtype != R2_F32 && dtype != R2_BF16) return R2_BAD_DTYPE;
  const int most = head_dim > v_head_dim ? head_dim : v_head_dim, shift = page_shift_of(page_size);
  const int piece = dtype == R2_F32 ? 4 : 8;   // numbers in 16 bytes
  const bool vec = reinterpret_cast<uintptr_t>(k_cache) % 16 == 0 && page_stride % piece == 0 && head_dim % piece == 0;
  auto go = [&](auto kernel, auto zero) {
    using T = decltype(zero);
    r2_launch(kernel, dim3(n_rows, n_heads), dim3(WARPS * 32), size_t(0), stream, (const T*)q, q_row_stride, (T*)out, out_row_stride, (const T*)k_cache,
              (const T*)v_cache, page_stride, page_size, shift, block_tables, table_width, row_entry, positions, seq_lens, n_heads, n_kv_heads, head_dim,
              v_head_dim, scale, window, keep_first, sink, (const T*)gate, gate_row_stride, n_pages, softcap, sinks, head_gate, head_gate_stride,
              v_row_stride, chunk, dist_bias, bias_len, out_scale);
  };
  auto pick = [&](auto zero) {
    using T = decltype(zero);
    if (most <= 64) vec ? go(attention_simt_kernel<T, 64, true>, zero) : go(attention_simt_kernel<T, 64, false>, zero);
    else if (most <= 128) vec ? go(attention_simt_kernel<T, 128, true>, zero) : go(attention_simt_kernel<T, 128, false>, zero);
    else if (most <= 256) vec ? go(attention_simt_kernel<T, 256, true>, zero) : go(attention_simt_kernel<T, 256, false>, zero);
    else vec ? go(attention_simt_kernel<T, WIDE_HEAD_DIM, true>, zero) : go(attention_simt_kernel<T, WIDE_HEAD_DIM, false>, zero);
  };
  if (dtype == R2_F32) pick(0.f);
  else pick(bf16());
  return launch_status();
}
