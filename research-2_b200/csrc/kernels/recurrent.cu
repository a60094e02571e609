// Mixers that carry a state of fixed size from token to token instead of a cache that grows: a matrix
// memory with exponential gates (mLSTM), a state-space layer (Mamba-2's recurrence) and retention (linear attention
// with one fixed decay per head, keep_t = decay and take_t = 1; its queries and keys are rotated by position on their way
// into shared memory, in float, so what enters the recurrence is never rounded to 16 bits), all of the form
//
//     S_t = keep_t * S_(t-1) + take_t * w_t v_t^T        S: [rows x columns] per head, float
//     y_t = S_t^T r_t  (+ what the layer adds)
//
// with a write vector w (keys; B), a read vector r (queries; C) and values v. One kernel serves both and
// serves prompts, portions and single decoded tokens alike: a CTA owns one (entry, head, slice of the
// value columns), takes the state from the request's slot (or zeros for a sequence's first rows), walks the
// entry's rows in order and puts the state back. A thread keeps RPT rows of one column in registers; the
// rows of a column are spread over G neighbouring lanes, so the sum over rows is a shuffle and the walk
// needs no barrier but the one that stages the next rows' vectors in shared memory. All arithmetic that
// enters the recurrence is float: gates, decays, their logarithms and exponentials, step sizes, the state.
// The order of operations depends on the row's position alone, so a row's result is the same bits however
// its prompt was cut into steps.
//
// Beside it: the short causal convolution in front of the state-space recurrence (its last inputs are
// state too), and the norm over groups of columns with a gate that follows both mixers.
#include <math.h>

#include <type_traits>

#include "common.cuh"
#include "scan_pieces.cuh"

namespace {

// Rows whose vectors are staged at a time: 32 (16 where a thread has 32 rows of a column in registers); 4 for launches in
// which every entry is a single decoded row (less shared memory: more CTAs to an SM).
constexpr int MAX_TILE = 32, SMALL_TILE = 4;
constexpr int SCAN_THREADS = 64;  // of a CTA that walks a prompt's rows, while there are slices (scan_shape)
constexpr int NORM_COPIES = 8;  // copies of a matrix memory's normaliser and maximum: one per slice of the columns at most

constexpr int MODE_MLSTM = 0, MODE_SSD = 1, MODE_DECAY = 2;

__device__ __forceinline__ float soft_cap(float x, float cap) { return cap > 0.f ? cap * tanhf(x / cap) : x; }
__device__ __forceinline__ float log_sigmoid(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }
__device__ __forceinline__ float silu(float x) { return __fdividef(x, 1.f + expf(-x)); }
__device__ __forceinline__ float softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }

struct ScanArgs {
  const void* read; int read_stride;     // r: [T, groups * rows] (queries: a group per head)
  const void* write; int write_stride;   // w: [T, groups * rows]
  const void* value; int value_stride;   // v: [T, heads * cols]
  const float* gates; int gates_stride;  // mLSTM: [T, 2 heads] input gates then forget gates, before the cap
                                         // state space: [T, heads] step sizes before bias and softplus
  const float* step_bias;                // state space, per head
  const float* log_rate;                 // state space, per head: the decay is exp(-exp(log_rate) * step)
  const float* skip;                     // state space, per head: y += skip * v
  float cap;                             // mLSTM: gates are cap * tanh(x / cap); 0 = no cap
  float read_scale;                      // r is multiplied by it
  float write_scale;                     // retention: w is multiplied by it (after the rotation)
  const float* decay;                    // retention, per head: keep
  const float* inv_freq; int rot_half;   // retention: of r and w the first 2 * rot_half dimensions turn, dimension i with
  const int32_t* positions;              // i + rot_half, by the angle positions[row] * inv_freq[i] (rot_half 0: no rotation)
  int silu_in;                           // retention: r, w and v pass silu on their way in
  float* state; long long slot_stride;   // per request slot; per head: S [rows][cols] (+ mLSTM: NORM_COPIES times n [rows], m)
  int head_stride;
  const int32_t* q_start; const int32_t* state_slot; const int32_t* fresh;
  float* out; int out_stride;            // [T, heads * cols] float
  int heads_per_group, rows, cols, G, cv;
  int single_rows;                       // a hint: no entry has more than one row (a decode step)
  int pieces;                            // every row of every operand starts on a 16-byte boundary: tiles are copied ahead
  // state space: the convolution's last inputs, renewed by the entry's CTAs together
  const void* conv_in; int conv_in_stride; int conv_channels, conv_taps; long long conv_state_off;
};

template <typename T, int RPT, int MODE, int TILE>
__global__ void __launch_bounds__(256, 1)
outer_scan_kernel(const ScanArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float smem[];
  const int e = blockIdx.x, h = blockIdx.y;
  const int row0 = a.q_start[e], row1 = a.q_start[e + 1];
  if (row1 <= row0) return;  // an entry without rows touches no slot
  const int G = a.G, cv = a.cv, rows = a.rows, cols = a.cols;
  const int padded = RPT * G;
  float* rs = smem;                       // [TILE][padded]
  float* ws = rs + TILE * padded;         // [TILE][padded]
  float* vs = ws + TILE * padded;         // [TILE][cv]
  float* g0 = vs + TILE * cv;             // [TILE] log input gate, then take | step
  float* g1 = g0 + TILE;                  // [TILE] log forget gate, then keep | decay
  float* g2 = g1 + TILE;                  // [TILE] running maximum after the row
  // a thread has the rows g * RPT .. g * RPT + RPT - 1 of column j; the G threads of a column are neighbouring lanes
  const int tid = threadIdx.x, g = tid % G, jl = tid / G;
  const int j = blockIdx.z * cv + jl;
  const bool is_fresh = a.fresh[e] != 0;
  float* head_state = a.state + size_t(a.state_slot[e]) * a.slot_stride + size_t(h) * a.head_stride;
  // the normaliser and the running maximum are kept NORM_COPIES times: the CTA of slice z reads copy z and renews the
  // copies z, z + slices, z + 2 slices, ..., so that every copy is current whatever the number of slices of a launch
  float* norm_state = head_state + size_t(rows) * cols;

  if (MODE == MODE_SSD && a.conv_in != nullptr) {
    // the inputs of the convolution's last taps - 1 positions: this step's newest rows, and before them what the
    // slot held (each channel is one thread's: it reads a place before it writes over it), spread over the entry's CTAs
    const int part = h * gridDim.z + blockIdx.z, n_parts = gridDim.y * gridDim.z;
    const T* in = static_cast<const T*>(a.conv_in);
    float* cs = a.state + size_t(a.state_slot[e]) * a.slot_stride + a.conv_state_off;
    const int keep = a.conv_taps - 1, n = row1 - row0;
    for (int c = part * blockDim.x + tid; c < a.conv_channels; c += n_parts * blockDim.x)
      for (int s = 0; s < keep; ++s) {
        const int l = n - keep + s;
        float val = 0.f;
        if (l >= 0) val = to_float(in[size_t(row0 + l) * a.conv_in_stride + c]);
        else if (!is_fresh) val = cs[size_t(s + n) * a.conv_channels + c];
        cs[size_t(s) * a.conv_channels + c] = val;
      }
  }

  uint64_t S[RPT / 2], nrm[RPT / 2];   // in twos: rows g * RPT + 2 r and the one after it
  float m = 0.f;
#pragma unroll
  for (int r = 0; r < RPT / 2; ++r) {
    float s2[2], n2[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = g * RPT + 2 * r + u;
      s2[u] = (!is_fresh && i < rows && j < cols) ? head_state[size_t(i) * cols + j] : 0.f;
      n2[u] = (MODE == MODE_MLSTM && !is_fresh && i < rows) ? norm_state[size_t(blockIdx.z) * (rows + 1) + i] : 0.f;
    }
    S[r] = pair_of(s2[0], s2[1]);
    nrm[r] = pair_of(n2[0], n2[1]);
  }
  if (MODE == MODE_MLSTM && !is_fresh) m = norm_state[size_t(blockIdx.z) * (rows + 1) + rows];

  const T* read = static_cast<const T*>(a.read) + size_t(h / a.heads_per_group) * rows;
  const T* write = static_cast<const T*>(a.write) + size_t(h / a.heads_per_group) * rows;
  const T* value = static_cast<const T*>(a.value) + size_t(h) * cols + size_t(blockIdx.z) * cv;
  const float skip = MODE == MODE_SSD ? a.skip[h] : 0.f;

  // A prompt's rows come a tile ahead: as they are stored, by asynchronous copies, next to the float vectors of the tile in use; the
  // gates in a register of the thread that turns them into factors. (Fetched when their tile began, every tile of 32 rows first
  // waited for memory: see the figures at the launch.)
  constexpr bool AHEAD = TILE > SMALL_TILE && MODE != MODE_DECAY;
  constexpr int PER = 16 / int(sizeof(T));
  const bool ahead = AHEAD && a.pieces != 0;
  const int copy_cols = max(0, min(cv, cols - int(blockIdx.z) * cv)), raw_stage = TILE * (2 * rows + cv);
  T* raw = reinterpret_cast<T*>(g2 + TILE);   // two stages of [TILE][rows] r, [TILE][rows] w, [TILE][cv] v
  const PieceWalk of_vectors(rows / PER), of_values(copy_cols / PER);
  float gate_a = 0.f, gate_b = 0.f;
  auto gates_of = [&](int t) {
    if (tid < TILE && t + tid < row1) {
      const float* gr = a.gates + size_t(t + tid) * a.gates_stride;
      gate_a = gr[h];
      if (MODE == MODE_MLSTM) gate_b = gr[gridDim.y + h];
    }
  };
  auto issue = [&](int t, int stage) {
    T* to = raw + stage * raw_stage;
    const int n = min(TILE, row1 - t);
    stage_rows<T>(to, rows, read + size_t(t) * a.read_stride, a.read_stride, of_vectors, n, true);
    stage_rows<T>(to + TILE * rows, rows, write + size_t(t) * a.write_stride, a.write_stride, of_vectors, n, true);
    if (copy_cols > 0) stage_rows<T>(to + 2 * TILE * rows, cv, value + size_t(t) * a.value_stride, a.value_stride, of_values, n, true);
  };
  if (ahead) {
    for (int i = tid; i < TILE * (2 * padded + cv); i += blockDim.x) smem[i] = 0.f;   // (dimensions and columns beyond the head's)
    issue(row0, 0);
    gates_of(row0);
  }
  int stage = 0;
  for (int t0 = row0; t0 < row1; t0 += TILE, stage ^= 1) {
    const int nt = row1 - t0 < TILE ? row1 - t0 : TILE;
    if (ahead) asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();  // the last rows' vectors have been used (and the copies of this tile's are there)
    float now_a = gate_a, now_b = gate_b;
    if (ahead) {
      if (t0 + TILE < row1) {
        issue(t0 + TILE, stage ^ 1);
        gates_of(t0 + TILE);
      }
      const T* from = raw + stage * raw_stage;
      spread_rows<T>(rs, padded, from, rows, of_vectors, nt, a.read_scale);
      spread_rows<T>(ws, padded, from + TILE * rows, rows, of_vectors, nt, 1.f);
      if (copy_cols > 0) spread_rows<T>(vs, cv, from + 2 * TILE * rows, cv, of_values, nt, 1.f);
    } else {
      // (loads in batches of eight before their stores: a loop of load-then-store would wait for every load in turn)
      for (int base = 0; base < nt * padded; base += 8 * blockDim.x) {
        float tr[8], tw[8];
  #pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int idx = base + u * blockDim.x + tid;
          const int tt = idx / padded, i = idx - tt * padded;
          const bool live = idx < nt * padded && i < rows;
          const size_t row = size_t(t0 + tt);
          tr[u] = live ? to_float(read[row * a.read_stride + i]) : 0.f;
          tw[u] = live ? to_float(write[row * a.write_stride + i]) : 0.f;
          if (MODE == MODE_DECAY && live && i < 2 * a.rot_half) {
            // the pair (u, v) = (x[i], x[i + half]) becomes (u cos - v sin, v cos + u sin); position and angle are float
            const bool low = i < a.rot_half;
            const int other = low ? i + a.rot_half : i - a.rot_half;
            float sn, cs;
            sincosf(float(a.positions[row]) * a.inv_freq[low ? i : other], &sn, &cs);
            if (low) sn = -sn;
            tr[u] = fmaf(tr[u], cs, to_float(read[row * a.read_stride + other]) * sn);
            tw[u] = fmaf(tw[u], cs, to_float(write[row * a.write_stride + other]) * sn);
          }
          if (MODE == MODE_DECAY && a.silu_in) {
            tr[u] = silu(tr[u]);
            tw[u] = silu(tw[u]);
          }
        }
  #pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int idx = base + u * blockDim.x + tid;
          if (idx < nt * padded) {
            rs[idx] = tr[u] * a.read_scale;
            ws[idx] = MODE == MODE_DECAY ? tw[u] * a.write_scale : tw[u];
          }
        }
      }
      for (int base = 0; base < nt * cv; base += 4 * blockDim.x) {
        float tv[4];
  #pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int idx = base + u * blockDim.x + tid;
          const int tt = idx / cv, c = idx - tt * cv;
          tv[u] = (idx < nt * cv && blockIdx.z * cv + c < cols) ? to_float(value[size_t(t0 + tt) * a.value_stride + c]) : 0.f;
        }
  #pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int idx = base + u * blockDim.x + tid;
          if (idx < nt * cv) vs[idx] = (MODE == MODE_DECAY && a.silu_in) ? silu(tv[u]) : tv[u];
        }
      }
      if (MODE != MODE_DECAY && tid < nt) {
        const float* gr = a.gates + size_t(t0 + tid) * a.gates_stride;
        now_a = gr[h];
        if (MODE == MODE_MLSTM) now_b = gr[gridDim.y + h];
      }
    }
    if (MODE == MODE_DECAY) {
      if (tid < nt) {
        g0[tid] = 1.f;
        g1[tid] = a.decay[h];
      }
    } else if (tid < nt) {
      if (MODE == MODE_MLSTM) {
        g0[tid] = soft_cap(now_a, a.cap);
        g1[tid] = log_sigmoid(soft_cap(now_b, a.cap));
      } else {
        const float step = softplus(now_a + a.step_bias[h]);
        g0[tid] = step;
        g1[tid] = expf(-expf(a.log_rate[h]) * step);
      }
    }
    __syncthreads();
    if (MODE == MODE_MLSTM) {
      // the running maximum is a chain of an addition and a maximum per row: every one of the first nt threads walks
      // it up to its own row (in the rows' order, so the result does not depend on where a tile begins); the
      // exponentials, which are what costs, are then one per thread
      float keep = 0.f, take = 0.f, top = 0.f;
      if (tid < nt) {
        float li[TILE], lf[TILE];   // (all loads first: the chain is then an addition and a maximum a row)
#pragma unroll
        for (int tt = 0; tt < TILE; ++tt) {
          li[tt] = g0[tt];
          lf[tt] = g1[tt];
        }
        float before = m;
        top = m;
#pragma unroll
        for (int tt = 0; tt < TILE; ++tt) {
          if (tt <= tid) {
            before = top;
            top = fmaxf(lf[tt] + before, li[tt]);
          }
        }
        keep = expf(g1[tid] + before - top);
        take = expf(g0[tid] - top);
      }
      __syncthreads();
      if (tid < nt) {
        g0[tid] = take;
        g1[tid] = keep;
        g2[tid] = top;
      }
      __syncthreads();
      m = g2[nt - 1];
    }
    // a row: this lane's shares of S^T r and, with a normaliser, of n . r
    auto walk = [&](int tt, float& acc_n) {
      const float take = g0[tt], keep = g1[tt];
      const float tv = take * vs[tt * cv + jl];
      const uint64_t keep2 = pair_of(keep, keep), tv2 = pair_of(tv, tv), take2 = pair_of(take, take);
      const float4* wr = reinterpret_cast<const float4*>(ws + tt * padded + g * RPT);
      const float4* rr = reinterpret_cast<const float4*>(rs + tt * padded + g * RPT);
      float acc = 0.f;
      acc_n = 0.f;
#pragma unroll
      for (int r4 = 0; r4 < RPT / 4; ++r4) {
        const float4 w4 = wr[r4], q4 = rr[r4];
        const uint64_t w[2] = {pair_of(w4.x, w4.y), pair_of(w4.z, w4.w)};
        const float q[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int r = r4 * 2 + u;
          S[r] = fma_pair(keep2, S[r], mul_pair(w[u], tv2));
          const float2 s2 = both(S[r]);
          acc = fmaf(s2.y, q[2 * u + 1], fmaf(s2.x, q[2 * u], acc));
          if (MODE == MODE_MLSTM) {
            nrm[r] = fma_pair(keep2, nrm[r], mul_pair(take2, w[u]));
            const float2 n2 = both(nrm[r]);
            acc_n = fmaf(n2.y, q[2 * u + 1], fmaf(n2.x, q[2 * u], acc_n));
          }
        }
      }
      return acc;
    };
    auto store = [&](int tt, float num, float nq) {
      float y;
      if (MODE == MODE_MLSTM) y = num / (fmaxf(fabsf(nq), expf(-g2[tt])) + 1e-6f);
      else y = fmaf(skip, vs[tt * cv + jl], num);
      a.out[size_t(t0 + tt) * a.out_stride + size_t(h) * cols + j] = y;
    };
    // four rows at a time: their sums are independent of each other, and their shuffles overlap
    int tt = 0;
    for (; TILE > SMALL_TILE && tt + 4 <= nt; tt += 4) {
      float num[4], nq[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) num[i] = walk(tt + i, nq[i]);
      if (G >= 4) {
        const float y = sums_of_four(num[0], num[1], num[2], num[3], g, G);
        const float z = MODE == MODE_MLSTM ? sums_of_four(nq[0], nq[1], nq[2], nq[3], g, G) : 0.f;
        if ((g & ((G >> 2) - 1)) == 0 && j < cols) store(tt + ((g & (G >> 1)) ? 2 : 0) + ((g & (G >> 2)) ? 1 : 0), y, z);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (G == 2) {
            num[i] += __shfl_xor_sync(0xffffffffu, num[i], 1);
            if (MODE == MODE_MLSTM) nq[i] += __shfl_xor_sync(0xffffffffu, nq[i], 1);
          }
          if (g == 0 && j < cols) store(tt + i, num[i], nq[i]);
        }
      }
    }
    for (; tt < nt; ++tt) {
      float nq, num = walk(tt, nq);
      for (int o = G >> 1; o > 0; o >>= 1) {
        num += __shfl_xor_sync(0xffffffffu, num, o);
        if (MODE == MODE_MLSTM) nq += __shfl_xor_sync(0xffffffffu, nq, o);
      }
      if (g == 0 && j < cols) store(tt, num, nq);
    }
  }
#pragma unroll
  for (int r = 0; r < RPT; ++r) {
    const int i = g * RPT + r;
    const float2 s2 = both(S[r / 2]);
    if (i < rows && j < cols) head_state[size_t(i) * cols + j] = (r & 1) ? s2.y : s2.x;
  }
  if (MODE == MODE_MLSTM && jl == 0) {
    for (int copy = blockIdx.z; copy < NORM_COPIES; copy += gridDim.z) {
#pragma unroll
      for (int r = 0; r < RPT; ++r) {
        const int i = g * RPT + r;
        const float2 n2 = both(nrm[r / 2]);
        if (i < rows) norm_state[size_t(copy) * (rows + 1) + i] = (r & 1) ? n2.y : n2.x;
      }
      if (tid == 0) norm_state[size_t(copy) * (rows + 1) + rows] = m;
    }
  }
}

// How a head's state is spread over threads: RPT rows of a column in a thread's registers, a column's rows over G
// neighbouring lanes (a power of two up to 32), cv columns a CTA and the columns over 1, 2, 4 or 8 CTAs: as few as the
// threads of a CTA allow, and more while the launch has fewer CTAs than the GPU has SMs. `wide`: 256 threads instead of SCAN_THREADS.
struct ScanShape { int rpt, G, threads, cv, splits; };

ScanShape scan_shape(int rows, int cols, int pairs, bool wide, int per_piece) {
  ScanShape s;
  s.rpt = 4;
  while (s.rpt < 32 && (rows + s.rpt - 1) / s.rpt > 4) s.rpt *= 2;
  s.G = 1;
  while (s.G * s.rpt < rows) s.G *= 2;
  const int G = s.G > 32 ? 32 : s.G;
  const int granule = !wide && per_piece > 32 / G ? per_piece : 32 / G;   // columns: whole warps and, where rows are copied, whole pieces
  s.splits = 1;
  for (;;) {
    s.cv = ((cols + s.splits - 1) / s.splits + granule - 1) / granule * granule;
    s.threads = s.cv * G;
    if (s.splits == NORM_COPIES) break;
    const bool fits = s.threads <= (wide ? 256 : SCAN_THREADS), enough = pairs * s.splits >= 120 || s.threads <= 64;
    if (fits && enough) break;
    s.splits *= 2;
  }
  return s;
}

// A walk's launch. Tiles are copied ahead (`pieces`) where whole 16-byte pieces can be (`aligned`: the operands' addresses and strides) and
// two stages fit beside the floats. With the rows' sums four at a time: 900 rows beside 7 decoded ones, 12 heads, state space of 32 x 64
// 245 to 103 us, matrix memory of 64 x 64 477 to 242; what is left is a warp's issue and latencies (some 90 instructions a row, one
// warp to a scheduler).
// Such prompts take 64 threads: of a batch's entries few are long, and those then have their columns over as many SMs as there are
// slices (that matrix memory: 311 us with 256 threads, 242; 16 entries of 64 rows 59 and 55). A walk that stages a tile when it begins
// takes 256, since every slice stages the vectors again (16 entries of 64 rows, the fixed decay: 57 us, 87 with 64 threads; matrix
// memory of 64 x 64 in unaligned rows 59 and 75, state space 78 and 97), and so do decode steps.
// The room for the copies is what two CTAs to an SM leave: in 48 KB only bfloat16 heads of up to 64 rows and 65 to 150, and float32
// heads of up to 32, had it (900 rows beside 7 decoded ones, matrix memory: float32 64 x 64 391 us without copies, 250 with; bfloat16 200 x 64
// 2,189 and 1,441).
struct ScanPlan { ScanShape shape; int tile, pieces; size_t smem; };

constexpr size_t SCAN_SMEM = 48 * 1024, AHEAD_SMEM = 100 * 1024;   // without and with tiles copied ahead (two such CTAs to an SM)

ScanPlan scan_plan(int rows, int cols, int pairs, bool single_rows, bool fixed_decay, int elem, bool aligned) {
  const int per_piece = 16 / elem;
  ScanPlan p = {};
  auto take = [&](bool wide) {
    p.shape = scan_shape(rows, cols, pairs, wide, per_piece);
    p.tile = single_rows ? SMALL_TILE : (p.shape.rpt <= 16 ? MAX_TILE : 16);
    p.smem = sizeof(float) * (size_t(p.tile) * (2 * p.shape.rpt * p.shape.G + p.shape.cv) + 3 * p.tile);
  };
  if (!single_rows && !fixed_decay) {
    take(false);
    const size_t raw = 2 * size_t(p.tile) * (2 * rows + p.shape.cv) * elem;
    p.pieces = aligned && p.smem <= SCAN_SMEM && p.smem + raw <= AHEAD_SMEM && rows % per_piece == 0 && cols % per_piece == 0 && p.shape.cv % per_piece == 0;
    if (p.pieces) {
      p.smem += raw;
      return p;
    }
  }
  take(true);
  if (p.smem > SCAN_SMEM && !single_rows && !fixed_decay) take(false);   // (narrower slices may still fit)
  return p;
}

template <typename T, int MODE>
int launch_scan(const ScanArgs& in, int n_entries, int n_heads, cudaStream_t stream) {
  ScanArgs a = in;
  const bool single_rows = a.single_rows != 0;
  auto on_pieces = [](const void* p, int stride) { return reinterpret_cast<uintptr_t>(p) % 16 == 0 && stride * sizeof(T) % 16 == 0; };
  const bool aligned = on_pieces(a.read, a.read_stride) && on_pieces(a.write, a.write_stride) && on_pieces(a.value, a.value_stride);
  const ScanPlan plan = scan_plan(a.rows, a.cols, n_entries * n_heads, single_rows, MODE == MODE_DECAY, int(sizeof(T)), aligned);
  const int rpt = plan.shape.rpt, threads = plan.shape.threads, splits = plan.shape.splits;
  const size_t smem = plan.smem;
  if (plan.shape.G > 32 || threads > 256 || smem > (plan.pieces ? AHEAD_SMEM : SCAN_SMEM)) return R2_UNSUPPORTED;
  a.G = plan.shape.G;
  a.cv = plan.shape.cv;
  a.pieces = plan.pieces;
  dim3 grid(n_entries, n_heads, splits);
#define R2_SCAN(RPT_, TILE_)                                                                        \
  do {                                                                                              \
    static std::atomic<bool> allowed[64];                                                           \
    if (smem > SCAN_SMEM)                                                                           \
      if (int status = allow_smem(outer_scan_kernel<T, RPT_, MODE, TILE_>, AHEAD_SMEM, allowed)) return status; \
    r2_launch(outer_scan_kernel<T, RPT_, MODE, TILE_>, grid, dim3(threads), smem, stream, a);       \
  } while (0)
  switch (rpt) {
    case 4: if (single_rows) R2_SCAN(4, SMALL_TILE); else R2_SCAN(4, MAX_TILE); break;
    case 8: if (single_rows) R2_SCAN(8, SMALL_TILE); else R2_SCAN(8, MAX_TILE); break;
    case 16: if (single_rows) R2_SCAN(16, SMALL_TILE); else R2_SCAN(16, MAX_TILE); break;
    default: if (single_rows) R2_SCAN(32, SMALL_TILE); else R2_SCAN(32, 16); break;
  }
#undef R2_SCAN
  return launch_status();
}

// ---- the short causal convolution --------------------------------------------------------------
// out[t][c] = silu(bias[c] + sum_d taps[c][d] * in[t - (n_taps - 1) + d][c]); inputs before this step's first row
// of an entry come from the request's slot (the inputs of its last n_taps - 1 positions), zeros before a sequence's
// start. The slot is only read here; the recurrence's kernel, which runs after this one, renews it.
template <typename T, bool FIXED>
__global__ void __launch_bounds__(256)
causal_conv_kernel(const T* __restrict__ in, int in_stride, T* __restrict__ out, int out_stride, const float* __restrict__ taps,
                   const float* __restrict__ bias, int n_taps, int channels, const float* __restrict__ state, long long slot_stride,
                   long long conv_state_off, const int32_t* __restrict__ row_entry, const int32_t* __restrict__ q_start,
                   const int32_t* __restrict__ state_slot, const int32_t* __restrict__ fresh) {
  pdl_launch_dependents();
  // (FIXED: the batch's arrays and the weights are no kernel's output, and what is looked up in them does not wait for the kernel before)
  pdl_wait_before_operands<FIXED>();
  const int t = blockIdx.x;
  const int e = row_entry[t];
  const int l = e < 0 ? 0 : t - q_start[e];
  const bool is_fresh = e < 0 || fresh[e] != 0;
  const float* cs = state + (e < 0 ? 0 : size_t(state_slot[e])) * slot_stride + conv_state_off;
  const int c_first = blockIdx.y * blockDim.x + threadIdx.x;
  float first_tap[4], first_bias = 0.f;   // of this thread's first channel
  const bool four = n_taps <= 4;
  if (four && c_first < channels) {
#pragma unroll
    for (int d = 0; d < 4; ++d) first_tap[d] = d < n_taps ? taps[size_t(c_first) * n_taps + d] : 0.f;
    first_bias = bias != nullptr ? bias[c_first] : 0.f;
  }
  pdl_wait_after_operands<FIXED>();
  T* o = out + size_t(t) * out_stride;
  if (e < 0) {  // a pad row
    for (int c = c_first; c < channels; c += gridDim.y * blockDim.x) o[c] = from_float<T>(0.f);
    return;
  }
  auto input = [&](int c, int d) {
    const int src = l - (n_taps - 1) + d;
    if (src >= 0) return to_float(in[size_t(t - (n_taps - 1) + d) * in_stride + c]);
    return is_fresh ? 0.f : cs[size_t(n_taps - 1 + src) * channels + c];
  };
  for (int c = c_first; c < channels; c += gridDim.y * blockDim.x) {
    float acc;
    if (four) {   // all inputs asked for at once
      float val[4];
#pragma unroll
      for (int d = 0; d < 4; ++d) val[d] = d < n_taps ? input(c, d) : 0.f;
      acc = c == c_first ? first_bias : bias != nullptr ? bias[c] : 0.f;
#pragma unroll
      for (int d = 0; d < 4; ++d)
        if (d < n_taps) acc = fmaf(c == c_first ? first_tap[d] : taps[size_t(c) * n_taps + d], val[d], acc);
    } else {
      acc = bias != nullptr ? bias[c] : 0.f;
      for (int d = 0; d < n_taps; ++d) acc = fmaf(taps[size_t(c) * n_taps + d], input(c, d), acc);
    }
    o[c] = from_float<T>(acc / (1.f + expf(-acc)));
  }
}

// ---- norm over groups of columns, with a gate ---------------------------------------------------
// One warp per (row, group). gate_first 1: y <- y * silu(gate), then the group's RMS norm, times weight.
// 0: the group's RMS norm, times weight, times sigmoid(gate). 2: the group's RMS norm, times weight, times silu(gate).
// weight may be null: a gain of one. A few rows' time is a chain of round trips, so a thread's first NORM_HELD columns stay in
// registers: gains before the wait on the kernel before this one (FIXED: they are no kernel's output), values and gates at once;
// what lies beyond is read twice.
constexpr int NORM_HELD = 4;

// what a column adds to the sum and what it is multiplied by besides the norm and the gain
template <typename T>
__device__ __forceinline__ void gated_value(float v, const T gate, int gate_first, float& value, float& factor) {
  const float z = to_float(gate);
  value = v;
  factor = 1.f;
  if (gate_first == 1) value = v * (z / (1.f + expf(-z)));
  else factor = (gate_first == 2 ? z : 1.f) / (1.f + expf(-z));
}

// A group's columns by `threads` threads, this one the `me`-th; `sum` adds their shares up.
template <bool FIXED, typename T, typename F>
__device__ __forceinline__ void norm_group(const float* yr, const T* gr, const float* wr, T* o, int group_size, float eps, int gate_first, int me, int threads, F sum) {
  pdl_wait_before_operands<FIXED>();
  float value[NORM_HELD], factor[NORM_HELD], gain[NORM_HELD];
#pragma unroll
  for (int i = 0; i < NORM_HELD; ++i) gain[i] = wr != nullptr && me + i * threads < group_size ? wr[me + i * threads] : 1.f;
  pdl_wait_after_operands<FIXED>();
  T gate[NORM_HELD];
#pragma unroll
  for (int i = 0; i < NORM_HELD; ++i) {
    const int d = me + i * threads;
    value[i] = d < group_size ? yr[d] : 0.f;
    gate[i] = d < group_size ? gr[d] : from_float<T>(0.f);
  }
  float sq = 0.f;
#pragma unroll
  for (int i = 0; i < NORM_HELD; ++i) {
    gated_value(value[i], gate[i], gate_first, value[i], factor[i]);
    if (me + i * threads < group_size) sq = fmaf(value[i], value[i], sq);
  }
  for (int d = me + NORM_HELD * threads; d < group_size; d += threads) {
    float v, f;
    gated_value(yr[d], gr[d], gate_first, v, f);
    sq = fmaf(v, v, sq);
  }
  const float inv = 1.f / sqrtf(sum(sq) / float(group_size) + eps);
  auto result = [&](float v, float f, float w) { return from_float<T>(gate_first == 1 ? v * inv * w : v * inv * w * f); };
#pragma unroll
  for (int i = 0; i < NORM_HELD; ++i)
    if (me + i * threads < group_size) o[me + i * threads] = result(value[i], factor[i], gain[i]);
  for (int d = me + NORM_HELD * threads; d < group_size; d += threads) {
    float v, f;
    gated_value(yr[d], gr[d], gate_first, v, f);
    o[d] = result(v, f, wr != nullptr ? wr[d] : 1.f);
  }
}

template <typename T, bool FIXED>
__global__ void __launch_bounds__(128)
group_norm_gated_kernel(const float* __restrict__ y, int y_stride, const T* __restrict__ gate, int gate_stride,
                        const float* __restrict__ weight, T* __restrict__ out, int out_stride, int n_rows, int n_groups,
                        int group_size, float eps, int gate_first) {
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31;
  const long long unit = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (unit >= (long long)n_rows * n_groups) {
    pdl_wait();
    return;
  }
  const int t = int(unit / n_groups), grp = int(unit % n_groups);
  norm_group<FIXED>(y + size_t(t) * y_stride + size_t(grp) * group_size, gate + size_t(t) * gate_stride + size_t(grp) * group_size,
             weight != nullptr ? weight + size_t(grp) * group_size : nullptr, out + size_t(t) * out_stride + size_t(grp) * group_size, group_size, eps,
             gate_first, lane, 32, [](float x) { return warp_sum(x); });
}

// The same with a CTA per (row, group), for groups of many columns.
template <typename T, bool FIXED>
__global__ void __launch_bounds__(256)
group_norm_gated_block_kernel(const float* __restrict__ y, int y_stride, const T* __restrict__ gate, int gate_stride,
                              const float* __restrict__ weight, T* __restrict__ out, int out_stride, int n_groups,
                              int group_size, float eps, int gate_first) {
  pdl_launch_dependents();
  __shared__ float scratch[33];
  const int t = blockIdx.x / n_groups, grp = blockIdx.x % n_groups;
  norm_group<FIXED>(y + size_t(t) * y_stride + size_t(grp) * group_size, gate + size_t(t) * gate_stride + size_t(grp) * group_size,
             weight != nullptr ? weight + size_t(grp) * group_size : nullptr, out + size_t(t) * out_stride + size_t(grp) * group_size, group_size, eps,
             gate_first, int(threadIdx.x), int(blockDim.x), [&](float x) { return block_sum(x, scratch); });
}

}  // namespace

// Floats of one head's state in a request slot: the matrix, and NORM_COPIES times the normaliser vector with the
// running maximum.
extern "C" long long r2_mlstm_state_floats(int dim, int vdim) {
  if (dim < 1 || vdim < 1) return 0;
  return (long long)dim * vdim + (long long)NORM_COPIES * (dim + 1);
}

// The matrix memory's recurrence over a batch of entries. q, k [T, heads * dim] and v [T, heads * vdim] (slices of a
// projection, each with its row stride); gates [T, 2 * heads] float (input gates, then forget gates, before the
// cap); state [slots][heads][r2_mlstm_state_floats(dim, vdim)] float; out [T, heads * vdim] float, before the heads' norm.
extern "C" int r2_mlstm_scan(const void* q, int q_stride, const void* k, int k_stride, const void* v, int v_stride,
                             const float* gates, int gates_stride, float cap, float q_scale, float* state,
                             long long slot_stride, const int32_t* q_start, const int32_t* state_slot, const int32_t* fresh,
                             int n_entries, float* out, int out_stride, int n_heads, int dim, int vdim, int single_rows,
                             int dtype, cudaStream_t stream) {
  if (n_entries <= 0) return R2_OK;
  if (n_heads < 1 || dim < 1 || vdim < 1) return R2_BAD_SHAPE;
  ScanArgs a = {};
  a.read = q; a.read_stride = q_stride; a.write = k; a.write_stride = k_stride; a.value = v; a.value_stride = v_stride;
  a.gates = gates; a.gates_stride = gates_stride; a.cap = cap; a.read_scale = q_scale;
  a.state = state; a.slot_stride = slot_stride; a.head_stride = int(r2_mlstm_state_floats(dim, vdim));
  a.q_start = q_start; a.state_slot = state_slot; a.fresh = fresh; a.out = out; a.out_stride = out_stride;
  a.heads_per_group = 1; a.rows = dim; a.cols = vdim; a.single_rows = single_rows;
  if (dtype == R2_F32) return launch_scan<float, MODE_MLSTM>(a, n_entries, n_heads, stream);
  if (dtype == R2_BF16) return launch_scan<bf16, MODE_MLSTM>(a, n_entries, n_heads, stream);
  return R2_BAD_DTYPE;
}

// The launch that a prompt's walk of the matrix memory or the state space takes (profiles, tests): threads of a CTA, slices of the columns,
// and whether its tiles are copied ahead.
extern "C" void r2_scan_plan(int rows, int cols, int n_entries, int n_heads, int dtype, int aligned, int* threads, int* splits, int* copied) {
  const ScanPlan p = scan_plan(rows, cols, n_entries * n_heads, false, false, dtype == R2_F32 ? 4 : 2, aligned != 0);
  *threads = p.shape.threads;
  *splits = p.shape.splits;
  *copied = p.pieces;
}

// Retention: S <- decay[h] S + k v^T, o = S^T q per head, with q and k rotated by position (the first rot_dims dimensions
// of a head, dimension i with i + rot_dims / 2, angle positions[t] * inv_freq[i]; rot_dims 0: none) and k multiplied by
// k_scale after the rotation. silu_in: q, k and v pass silu on their way in (then without a rotation). q, k [T, heads * dim], v [T, heads * vdim] (slices of a projection); decay float [heads];
// state float [slots][heads][dim][vdim]; out [T, heads * vdim] float, before the heads' norm.
extern "C" int r2_retention_scan(const void* q, int q_stride, const void* k, int k_stride, const void* v, int v_stride,
                                 const float* decay, float k_scale, const float* inv_freq, int rot_dims, const int32_t* positions,
                                 float* state, long long slot_stride, const int32_t* q_start, const int32_t* state_slot,
                                 const int32_t* fresh, int n_entries, float* out, int out_stride, int n_heads, int dim, int vdim,
                                 int single_rows, int silu_in, int dtype, cudaStream_t stream) {
  if (n_entries <= 0) return R2_OK;
  if (silu_in && rot_dims > 0) return R2_BAD_SHAPE;
  if (n_heads < 1 || dim < 1 || vdim < 1 || rot_dims < 0 || rot_dims % 2 != 0 || rot_dims > dim) return R2_BAD_SHAPE;
  if (rot_dims > 0 && (inv_freq == nullptr || positions == nullptr)) return R2_BAD_SHAPE;
  ScanArgs a = {};
  a.read = q; a.read_stride = q_stride; a.write = k; a.write_stride = k_stride; a.value = v; a.value_stride = v_stride;
  a.read_scale = 1.f; a.write_scale = k_scale; a.decay = decay; a.inv_freq = inv_freq; a.rot_half = rot_dims / 2; a.positions = positions; a.silu_in = silu_in;
  a.state = state; a.slot_stride = slot_stride; a.head_stride = dim * vdim;
  a.q_start = q_start; a.state_slot = state_slot; a.fresh = fresh; a.out = out; a.out_stride = out_stride;
  a.heads_per_group = 1; a.rows = dim; a.cols = vdim; a.single_rows = single_rows;
  if (dtype == R2_F32) return launch_scan<float, MODE_DECAY>(a, n_entries, n_heads, stream);
  if (dtype == R2_BF16) return launch_scan<bf16, MODE_DECAY>(a, n_entries, n_heads, stream);
  return R2_BAD_DTYPE;
}

// The state-space recurrence. x [T, heads * vdim], B and C [T, groups * n_state] (after convolution and silu), steps
// [T, heads] float before bias and softplus; per head step_bias, log_rate, skip. state per slot: S [heads][n_state][vdim]
// and, at conv_state_off, the convolution's last conv_taps - 1 inputs [conv_taps - 1][conv_channels], which this kernel
// renews from conv_in (the convolution's input rows of this step; null: no convolution state).
extern "C" int r2_ssd_scan(const void* x, int x_stride, const void* b, int b_stride, const void* c, int c_stride,
                           const float* steps, int steps_stride, const float* step_bias, const float* log_rate,
                           const float* skip, float* state, long long slot_stride, const int32_t* q_start,
                           const int32_t* state_slot, const int32_t* fresh, int n_entries, float* out, int out_stride,
                           int n_heads, int n_groups, int n_state, int vdim, const void* conv_in, int conv_in_stride,
                           int conv_channels, int conv_taps, long long conv_state_off, int single_rows, int dtype,
                           cudaStream_t stream) {
  if (n_entries <= 0) return R2_OK;
  if (n_heads < 1 || n_groups < 1 || n_heads % n_groups != 0 || n_state < 1 || vdim < 1) return R2_BAD_SHAPE;
  ScanArgs a = {};
  a.read = c; a.read_stride = c_stride; a.write = b; a.write_stride = b_stride; a.value = x; a.value_stride = x_stride;
  a.gates = steps; a.gates_stride = steps_stride; a.step_bias = step_bias; a.log_rate = log_rate; a.skip = skip;
  a.read_scale = 1.f; a.state = state; a.slot_stride = slot_stride; a.head_stride = n_state * vdim;
  a.q_start = q_start; a.state_slot = state_slot; a.fresh = fresh; a.out = out; a.out_stride = out_stride;
  a.heads_per_group = n_heads / n_groups; a.rows = n_state; a.cols = vdim; a.single_rows = single_rows;
  a.conv_in = conv_taps > 1 ? conv_in : nullptr; a.conv_in_stride = conv_in_stride; a.conv_channels = conv_channels;
  a.conv_taps = conv_taps; a.conv_state_off = conv_state_off;
  if (dtype == R2_F32) return launch_scan<float, MODE_SSD>(a, n_entries, n_heads, stream);
  if (dtype == R2_BF16) return launch_scan<bf16, MODE_SSD>(a, n_entries, n_heads, stream);
  return R2_BAD_DTYPE;
}

// `fixed` (here and in r2_group_norm_gated): no launch shortly before writes the weights or the batch's arrays, which are then read ahead
// of the wait for it.
extern "C" int r2_causal_conv(const void* in, int in_stride, void* out, int out_stride, const float* taps, const float* bias,
                              int n_taps, int channels, const float* state, long long slot_stride, long long conv_state_off,
                              const int32_t* row_entry, const int32_t* q_start, const int32_t* state_slot, const int32_t* fresh,
                              int n_rows, int dtype, int fixed, cudaStream_t stream) {
  if (n_rows <= 0) return R2_OK;
  if (n_taps < 1 || channels < 1) return R2_BAD_SHAPE;
  // a channel a thread for few rows, whose time is the chain of their loads; four for many
  const int per_cta = n_rows <= 64 ? 256 : 1024;
  if (dtype != R2_F32 && dtype != R2_BF16) return R2_BAD_DTYPE;
  auto go = [&](auto kernel, auto zero) {
    r2_launch(kernel, dim3(n_rows, (channels + per_cta - 1) / per_cta), dim3(256), size_t(0), stream, (const decltype(zero)*)in, in_stride, (decltype(zero)*)out, out_stride,
              taps, bias, n_taps, channels, state, slot_stride, conv_state_off, row_entry, q_start, state_slot, fresh);
  };
  if (dtype == R2_F32) fixed ? go(causal_conv_kernel<float, true>, 0.f) : go(causal_conv_kernel<float, false>, 0.f);
  else fixed ? go(causal_conv_kernel<bf16, true>, bf16()) : go(causal_conv_kernel<bf16, false>, bf16());
  return launch_status();
}

extern "C" int r2_group_norm_gated(const float* y, int y_stride, const void* gate, int gate_stride, const float* weight,
                                   void* out, int out_stride, int n_rows, int n_groups, int group_size, float eps,
                                   int gate_first, int dtype, int fixed, cudaStream_t stream) {
  if (n_rows <= 0) return R2_OK;
  if (n_groups < 1 || group_size < 1) return R2_BAD_SHAPE;
  const long long units = (long long)n_rows * n_groups;
  if (dtype != R2_F32 && dtype != R2_BF16) return R2_BAD_DTYPE;
  auto pick = [&](auto zero, auto is_fixed) {
    using T = decltype(zero);
    constexpr bool FIXED = decltype(is_fixed)::value;
    if (group_size > 256) {
      r2_launch(group_norm_gated_block_kernel<T, FIXED>, dim3((unsigned)units), dim3(256), size_t(0), stream, y, y_stride, (const T*)gate, gate_stride, weight, (T*)out,
                out_stride, n_groups, group_size, eps, gate_first);
      return;
    }
    r2_launch(group_norm_gated_kernel<T, FIXED>, dim3((unsigned)((units + 3) / 4)), dim3(128), size_t(0), stream, y, y_stride, (const T*)gate, gate_stride, weight, (T*)out,
              out_stride, n_rows, n_groups, group_size, eps, gate_first);
  };
  if (dtype == R2_F32) fixed ? pick(0.f, std::true_type()) : pick(0.f, std::false_type());
  else fixed ? pick(bf16(), std::true_type()) : pick(bf16(), std::false_type());
  return launch_status();
}
