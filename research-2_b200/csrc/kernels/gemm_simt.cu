// Matrix product on the CUDA cores with float accumulation: the true 32-bit path of every
// linear layer, and the fallback of the bfloat16 path for shapes the tensor-core kernel refuses.
//
//   out[m, n] = act(sum_k a[m, k] * w(k, n) + bias[n]) (+ residual[m, n])
//
// `w` is stored [K, N] (the Conv1D layout of GPT-2 checkpoints, x @ w:
// kelpie-models/kelpie_models/models/torch/gpt2.py:52-55) or [N, K] (a tied embedding used as
// the head, x @ wte^T: gpt2.py:101).
//
// The order of every sum is a matter of K alone: K is cut into slices of `slice_len(K)` neighbours (at most 32 slices), a
// slice is summed by fused multiply-adds in ascending order, the sums of up to eight neighbouring slices are added in ascending
// order to a group's sum, and the (up to four) groups' sums in ascending order to the total. Both kernels
// below keep to it, so a row's result is the same bits however many rows the call has and whichever kernel takes it.
//
//   gemm_rows_kernel   few rows. What bounds it is the stream of weights, so it is laid out for loads in flight: a warp has one slice
//                      of 32 columns, its lanes read 128-byte lines of 32 rows of it ahead of the multiply-adds (an [N, K] matrix
//                      passes through shared memory to be turned), and the groups of a column block are spread over a
//                      thread-block cluster whose first CTA adds them up.
//   gemm_tile_kernel   many rows: tiles in shared memory, the next stage's loads in flight under this one's multiply-adds; a
//                      thread keeps the current slice's sums, the group's and, where one CTA has them all, the total. With few
//                      tiles the groups go to the CTAs of a cluster: a lone CTA of four warps on an SM waits on its own latencies
//                      (0.31 instructions a cycle and scheduler).
//
// Measured inside GPT-2 124M's float32 step, one 64 x 64 tile form for everything before, these two now (us): 3 rows, K x N = 768 x 768
// 145 and 6, 3,072 x 768 580 and 10, 768 x 3,072 145 and 9, the head 288 and 44; 332 rows 155 and 40, 620 and 96, 223 and 78.
#include "common.cuh"

namespace {

constexpr int MAX_SLICES = 32, MAX_GROUPS = 4;

// Slices are multiples of 16 long, so that a stage of the tile kernel never straddles two.
__host__ __device__ constexpr int slice_len(int k_total) { return 16 * ((k_total + 16 * MAX_SLICES - 1) / (16 * MAX_SLICES)); }
constexpr int GROUP = MAX_SLICES / MAX_GROUPS;   // slices of a group

struct Product {
  const void* a;
  const void* w;
  int lda, ldw;
  const float* bias;
  const float* residual;
  int ldr;
  void* out;
  int ldo, m_total, n_total, k_total, act;
};

template <typename TO>
__device__ __forceinline__ void finish(const Product& p, int m, int n, float v) {
  if (p.bias != nullptr) v += p.bias[n];
  v = activate(v, p.act);
  if (p.residual != nullptr) v += p.residual[size_t(m) * p.ldr + n];
  static_cast<TO*>(p.out)[size_t(m) * p.ldo + n] = from_float<TO>(v);
}

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The float at the same shared-memory place of another CTA of the cluster.
__device__ __forceinline__ float remote_float(const float* mine, int rank) {
  uint32_t addr, there = uint32_t(__cvta_generic_to_shared(mine));
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(there), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

__device__ __forceinline__ float4 remote_float4(const float4* mine, int rank) {
  uint32_t addr, there = uint32_t(__cvta_generic_to_shared(mine));
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(there), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float4 plus(const float4& a, const float4& b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// Two floats in one register pair, and the two multiply-adds of such pairs as one instruction (each rounded as fmaf rounds).
__device__ __forceinline__ uint64_t pair(float lo, float hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ void unpair(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ void fma_pair(uint64_t& acc, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }

constexpr int ROW_WARPS = GROUP, ROW_COLS = 32;

// grid (cluster size, column blocks or fewer, blocks of MR rows), clusters along x. CTA r of a cluster of C has the groups
// [r * n_groups / C ..), one after the other, a slice a warp; a CTA without a cluster walks every gridDim.y-th column block. Shared
// memory: the slices' sums [slices of this CTA][MR][32], the rows of `a` [MR][K of this CTA] as floats, and for an [N, K] matrix a
// turning buffer of 32 x 33 floats a warp.
template <typename TA, typename TW, typename TO, bool W_IS_NK, int MR>
__global__ void __launch_bounds__(ROW_WARPS * 32)
gemm_rows_kernel(const Product p, int n_slices, int per_cta, int n_blocks) {
  constexpr int STEP = W_IS_NK || MR < 8 ? 32 : 16;   // lines in flight (with eight rows' sums beside 32 of them an SM holds one CTA)
  pdl_launch_dependents();  // the next kernel may begin its prologue
  extern __shared__ __align__(16) float smem[];
  const int len = slice_len(p.k_total);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x, n_ranks = gridDim.x;
  const int m0 = blockIdx.z * MR;
  const int first = rank * per_cta, mine = max(0, min(per_cta, n_slices - first));
  const int span = per_cta * len, k_first = first * len;
  float* sums = smem;                              // [per_cta][MR][32]
  float* rows = sums + per_cta * MR * ROW_COLS;    // [MR][span]
  float* turn = rows + MR * span + warp * 32 * 33; // [32][33] of this warp
  const TA* a = static_cast<const TA*>(p.a);
  const TW* w = static_cast<const TW*>(p.w);

  // the 32 rows (columns, for an [N, K] matrix) of a piece of a slice that lane's column (k) is read in
  float cur[STEP];
  auto load = [&](int n0, int s, int kc) {
    const int k0 = k_first + s * len + kc, here = min(STEP, len - kc);
    const TW* from = W_IS_NK ? w + size_t(n0) * p.ldw + k0 + lane : w + size_t(k0) * p.ldw + n0 + lane;
    // how many of the lines hold something for this lane
    int n_live = W_IS_NK ? ((lane < here && k0 + lane < p.k_total) ? p.n_total - n0 : 0) : (n0 + lane < p.n_total ? min(here, p.k_total - k0) : 0);
    if (s >= mine) n_live = 0;
#pragma unroll
    for (int u = 0; u < STEP; ++u, from += p.ldw) cur[u] = u < n_live ? to_float(*from) : 0.f;
  };

  pdl_wait();               // the previous kernel's writes are visible from here on (`w` may be one of them: any caller's tensor)
  load(blockIdx.y * ROW_COLS, warp, 0);
#pragma unroll
  for (int r = 0; r < MR; ++r)
    for (int k = threadIdx.x; k < mine * len; k += ROW_WARPS * 32)
      rows[r * span + k] = (m0 + r < p.m_total && k_first + k < p.k_total) ? to_float(a[size_t(m0 + r) * p.lda + k_first + k]) : 0.f;
  __syncthreads();

  for (int block = blockIdx.y; block < n_blocks; block += gridDim.y) {
    const int n0 = block * ROW_COLS;
    for (int s = warp; s < mine; s += ROW_WARPS) {
      const float* ar = rows + s * len;
      float acc[MR];
#pragma unroll
      for (int r = 0; r < MR; ++r) acc[r] = 0.f;
      for (int kc = 0; kc < len; kc += STEP) {
        float now[STEP];
        if (W_IS_NK) {
          __syncwarp();   // the piece before has been read
#pragma unroll
          for (int j = 0; j < STEP; ++j) turn[lane * 33 + j] = cur[j];
          __syncwarp();
#pragma unroll
          for (int u = 0; u < STEP; ++u) now[u] = turn[u * 33 + lane];
        } else {
#pragma unroll
          for (int u = 0; u < STEP; ++u) now[u] = cur[u];
        }
        // what this warp reads next: the slice's next piece, or the first one of its next slice or column block
        const bool in_slice = kc + STEP < len, in_block = s + ROW_WARPS < mine;
        load(in_slice || in_block ? n0 : n0 + int(gridDim.y) * ROW_COLS, in_slice ? s : in_block ? s + ROW_WARPS : warp, in_slice ? kc + STEP : 0);
#pragma unroll
        for (int u = 0; u < STEP; u += 4) {
          if (u == 16 && kc + 16 >= len) break;   // (a slice's last piece may be half as long)
#pragma unroll
          for (int r = 0; r < MR; ++r) {
            const float4 av = *reinterpret_cast<const float4*>(ar + r * span + kc + u);
            acc[r] = fmaf(av.x, now[u], acc[r]);
            acc[r] = fmaf(av.y, now[u + 1], acc[r]);
            acc[r] = fmaf(av.z, now[u + 2], acc[r]);
            acc[r] = fmaf(av.w, now[u + 3], acc[r]);
          }
        }
      }
#pragma unroll
      for (int r = 0; r < MR; ++r) sums[(s * MR + r) * ROW_COLS + lane] = acc[r];
    }
    __syncthreads();
    // groups first, each by the CTA that has it (over the group's first slice), then the groups
    const int own_groups = (mine + GROUP - 1) / GROUP;
    for (int i = threadIdx.x; i < own_groups * MR * ROW_COLS; i += ROW_WARPS * 32) {
      const int g = i / (MR * ROW_COLS), at = i % (MR * ROW_COLS);
      float* from = sums + g * GROUP * MR * ROW_COLS + at;
      const int n = min(GROUP, mine - g * GROUP);
      float t = from[0];
#pragma unroll
      for (int s = 1; s < GROUP; ++s)
        if (s < n) t += from[s * MR * ROW_COLS];
      from[0] = t;
    }
    __syncthreads();
    if (n_ranks > 1) cluster_barrier();
    if (rank == 0) {
      for (int i = threadIdx.x; i < MR * ROW_COLS; i += ROW_WARPS * 32) {
        const int gm = m0 + i / ROW_COLS, gn = n0 + i % ROW_COLS;
        if (gm >= p.m_total || gn >= p.n_total) continue;
        float total = sums[i];
        if (n_ranks > 1) {
          float part[MAX_GROUPS];   // (a cluster's CTA has one group)
#pragma unroll
          for (int q = 1; q < MAX_GROUPS; ++q) part[q] = q < n_ranks ? remote_float(sums + i, q) : 0.f;
#pragma unroll
          for (int q = 1; q < MAX_GROUPS; ++q)
            if (q < n_ranks) total += part[q];
        } else {
          for (int g = 1; g < own_groups; ++g) total += sums[g * GROUP * MR * ROW_COLS + i];
        }
        finish<TO>(p, gm, gn, total);
      }
    }
    if (n_ranks > 1) cluster_barrier();   // the first CTA reads the others' shared memory until here
    else __syncthreads();                 // the sums have been read
  }
}

// Tiles of BM x BN, stages of 16 along K in two buffers; a thread has 8 x 8 sums (four rows and four columns of either half of the
// tile): 64 independent multiply-adds per four 16-byte reads of shared memory keep a scheduler busy with a single warp. The current
// slice's sums are registers, the group's and the total lie in shared memory (a place a thread and four neighbouring columns, so that no
// barrier is needed), touched once a slice and once a group.
// VEC: float operands whose rows start on 16-byte
// boundaries and hold multiples of four along the contiguous axis. With a cluster along z its CTA r computes the groups from
// r * groups_per_cta on, and every CTA adds up and finishes a share of the tile's rows.
constexpr int BK = 16;

template <typename TA, typename TW, typename TO, bool W_IS_NK, int BM, int BN, bool VEC>
__global__ void __launch_bounds__(BM * BN / 64)
gemm_tile_kernel(const Product p, int groups_per_cta) {
  constexpr int THREADS = BM * BN / 64, TX = BN / 8;
  constexpr int A_PER = BM * BK / THREADS, W_PER = BN * BK / THREADS;   // numbers of a stage a thread brings
  static_assert(A_PER % 4 == 0 && W_PER % 4 == 0, "whole float4");
  pdl_launch_dependents();
  constexpr int A_FLOATS = 2 * BK * (BM + 4), W_FLOATS = 2 * BK * (BN + 4);
  extern __shared__ __align__(16) float smem[];   // the stages, the group's sums and the totals [16][THREADS] in fours
  float (*as)[BK][BM + 4] = reinterpret_cast<float (*)[BK][BM + 4]>(smem);
  float (*ws)[BK][BN + 4] = reinterpret_cast<float (*)[BK][BN + 4]>(smem + A_FLOATS);
  float4* sums = reinterpret_cast<float4*>(smem + A_FLOATS + W_FLOATS);
  float4* totals = sums + 16 * THREADS;
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  pdl_wait();
  const TA* a = static_cast<const TA*>(p.a);
  const TW* w = static_cast<const TW*>(p.w);
  const int len = slice_len(p.k_total);
  float av[A_PER], wv[W_PER];

  auto load = [&](int k0) {
    if (VEC) {
#pragma unroll
      for (int i = 0; i < A_PER / 4; ++i) {
        const int at = (i * THREADS + tid) * 4, mm = at / BK, kk = at % BK;
        const bool in = m0 + mm < p.m_total && k0 + kk < p.k_total;
        const float4 v = in ? *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(a) + size_t(m0 + mm) * p.lda + k0 + kk) : make_float4(0.f, 0.f, 0.f, 0.f);
        av[4 * i] = v.x; av[4 * i + 1] = v.y; av[4 * i + 2] = v.z; av[4 * i + 3] = v.w;
      }
#pragma unroll
      for (int i = 0; i < W_PER / 4; ++i) {
        const int at = (i * THREADS + tid) * 4;
        const int nn = W_IS_NK ? at / BK : at % BN, kk = W_IS_NK ? at % BK : at / BN;
        const bool in = n0 + nn < p.n_total && k0 + kk < p.k_total;
        const float* from = reinterpret_cast<const float*>(w) + (W_IS_NK ? size_t(n0 + nn) * p.ldw + k0 + kk : size_t(k0 + kk) * p.ldw + n0 + nn);
        const float4 v = in ? *reinterpret_cast<const float4*>(from) : make_float4(0.f, 0.f, 0.f, 0.f);
        wv[4 * i] = v.x; wv[4 * i + 1] = v.y; wv[4 * i + 2] = v.z; wv[4 * i + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < A_PER; ++i) {
        const int at = i * THREADS + tid, mm = at / BK, kk = at % BK;
        av[i] = (m0 + mm < p.m_total && k0 + kk < p.k_total) ? to_float(a[size_t(m0 + mm) * p.lda + k0 + kk]) : 0.f;
      }
#pragma unroll
      for (int i = 0; i < W_PER; ++i) {
        const int at = i * THREADS + tid, nn = W_IS_NK ? at / BK : at % BN, kk = W_IS_NK ? at % BK : at / BN;
        const bool in = n0 + nn < p.n_total && k0 + kk < p.k_total;
        wv[i] = in ? to_float(w[W_IS_NK ? size_t(n0 + nn) * p.ldw + k0 + kk : size_t(k0 + kk) * p.ldw + n0 + nn]) : 0.f;
      }
    }
  };
  auto store = [&](int b) {
    constexpr int RUN = VEC ? 4 : 1;
#pragma unroll
    for (int i = 0; i < A_PER; ++i) {
      const int at = (i / RUN * THREADS + tid) * RUN + i % RUN;
      as[b][at % BK][at / BK] = av[i];
    }
#pragma unroll
    for (int i = 0; i < W_PER; ++i) {
      const int at = (i / RUN * THREADS + tid) * RUN + i % RUN;
      ws[b][W_IS_NK ? at % BK : at / BN][W_IS_NK ? at / BK : at % BN] = wv[i];
    }
  };

  uint64_t acc[8][4];   // pairs of neighbouring columns
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0;

  const int rank = blockIdx.z, n_ranks = gridDim.z, group_len = GROUP * len;
  const int k_begin = rank * groups_per_cta * group_len, k_end = min(p.k_total, k_begin + groups_per_cta * group_len);
  bool first_slice = true, first_group = true;   // of the group; of this CTA
  load(k_begin);
  store(0);
  __syncthreads();
  int b = 0, left = len, slices_left = GROUP;
  for (int k0 = k_begin; k0 < k_end; k0 += BK, b ^= 1) {
    const bool more = k0 + BK < k_end;
    if (more) load(k0 + BK);
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float x[8];
      uint64_t y[4];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float4 v = *reinterpret_cast<const float4*>(&as[b][kk][u * (BM / 2) + ty * 4]);
        x[4 * u] = v.x; x[4 * u + 1] = v.y; x[4 * u + 2] = v.z; x[4 * u + 3] = v.w;
        const ulonglong2 z = *reinterpret_cast<const ulonglong2*>(&ws[b][kk][u * (BN / 2) + tx * 4]);
        y[2 * u] = z.x;
        y[2 * u + 1] = z.y;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint64_t xx = pair(x[i], x[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) fma_pair(acc[i][j], xx, y[j]);
      }
    }
    left -= BK;
    if (left == 0 || !more) {   // the slice's end
      left = len;
      const bool group_ends = --slices_left == 0 || !more;
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; j += 4) {
          const int at = (i * 2 + j / 4) * THREADS + tid;
          float4 v;
          unpair(acc[i][j / 2], v.x, v.y);
          unpair(acc[i][j / 2 + 1], v.z, v.w);
          if (!first_slice) v = plus(sums[at], v);
          if (!group_ends) sums[at] = v;
          else totals[at] = first_group ? v : plus(totals[at], v);
          acc[i][j / 2] = acc[i][j / 2 + 1] = 0;
        }
      first_slice = group_ends;
      if (group_ends) {
        slices_left = GROUP;
        first_group = false;
      }
    }
    if (more) store(b ^ 1);
    __syncthreads();
  }
  if (n_ranks > 1) cluster_barrier();
  for (int place = rank; place < 16; place += n_ranks) {   // the CTAs share a thread's 16 places
    const int at = place * THREADS + tid;
    const int gm = m0 + (place / 8) * (BM / 2) + ty * 4 + (place / 2) % 4, gn = n0 + (place % 2) * (BN / 2) + tx * 4;
    float4 v;
    if (n_ranks == 1) {
      v = totals[at];
    } else {
      float4 part[MAX_GROUPS];
#pragma unroll
      for (int q = 0; q < MAX_GROUPS; ++q) part[q] = q < n_ranks ? remote_float4(totals + at, q) : make_float4(0.f, 0.f, 0.f, 0.f);
      v = part[0];
#pragma unroll
      for (int q = 1; q < MAX_GROUPS; ++q)
        if (q < n_ranks) v = plus(v, part[q]);
    }
    if (gm >= p.m_total) continue;
    const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (gn + u < p.n_total) finish<TO>(p, gm, gn + u, x[u]);
  }
  if (n_ranks > 1) cluster_barrier();   // the others read this CTA's shared memory until here
}

int n_sms() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) {
    cudaGetLastError();
    return 1;
  }
  return n;
}

// `kernel` on a cluster of grid's extent along `axis` (0: x, 2: z), in programmatic stream order where that is on.
template <typename... KArgs, typename... Args>
int launch_clustered(void (*kernel)(KArgs...), dim3 grid, int threads, size_t smem, int axis, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = dim3(threads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attr[2];
  int n_attr = 0;
  if ((axis == 0 ? grid.x : grid.z) > 1) {
    attr[n_attr].id = cudaLaunchAttributeClusterDimension;
    attr[n_attr].val.clusterDim.x = axis == 0 ? grid.x : 1;
    attr[n_attr].val.clusterDim.y = 1;
    attr[n_attr].val.clusterDim.z = axis == 0 ? 1 : grid.z;
    ++n_attr;
  }
  if (g_r2_pdl && !t_r2_plain_order) {
    attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
    ++n_attr;
  }
  config.attrs = attr;
  config.numAttrs = n_attr;
  cudaLaunchKernelEx(&config, kernel, static_cast<Args&&>(args)...);   // a failure shows in launch_status()
  return launch_status();
}

constexpr size_t MOST_SMEM = 227 * 1024;

template <typename TA, typename TW, typename TO, bool W_IS_NK, int MR>
int launch_rows(const Product& p, cudaStream_t stream) {
  const int len = slice_len(p.k_total), n_slices = (p.k_total + len - 1) / len, n_groups = (n_slices + GROUP - 1) / GROUP;
  const int blocks = (p.n_total + ROW_COLS - 1) / ROW_COLS, row_blocks = (p.m_total + MR - 1) / MR, sms = n_sms();
  // a CTA walks all slices of its columns where the column blocks alone give every SM work (the head: 1,571 blocks); else a
  // cluster takes a slice a warp (an output product of 768 columns has 24 blocks)
  const int ranks = blocks * row_blocks >= sms / 2 ? 1 : n_groups;
  const int per_cta = ranks == 1 ? n_slices : GROUP;
  const size_t smem = sizeof(float) * (size_t(per_cta) * MR * ROW_COLS + size_t(MR) * per_cta * len + (W_IS_NK ? ROW_WARPS * 32 * 33 : 0));
  auto kernel = gemm_rows_kernel<TA, TW, TO, W_IS_NK, MR>;
  static std::atomic<bool> allowed[64];
  if (int status = allow_smem(kernel, MOST_SMEM, allowed)) return status;
  int grid_y = blocks;
  if (ranks == 1) {   // as many CTAs as are resident: the rows are staged once, and a warp's next lines are on their way over a block's end
    const int resident = int(size_t(220) * 1024 / (smem + 1024));
    const int most = sms * (resident < 1 ? 1 : resident > 3 ? 3 : resident) / row_blocks;
    if (grid_y > most) grid_y = most < 1 ? 1 : most;
  }
  return launch_clustered(kernel, dim3(ranks, grid_y, row_blocks), ROW_WARPS * 32, smem, 0, stream, p, n_slices, per_cta, blocks);
}

template <typename TA, typename TW, typename TO, bool W_IS_NK, int BM, int BN>
int launch_tiles(const Product& p, bool vec, int n_groups, int ranks, cudaStream_t stream) {
  const dim3 grid((p.n_total + BN - 1) / BN, (p.m_total + BM - 1) / BM, ranks);
  constexpr bool FLOATS = sizeof(TA) == 4 && sizeof(TW) == 4;
  const size_t smem = sizeof(float) * (2 * BK * (BM + 4) + 2 * BK * (BN + 4) + 2 * BM * BN);
  const bool pieces = vec && FLOATS;
  auto kernel = pieces ? gemm_tile_kernel<TA, TW, TO, W_IS_NK, BM, BN, FLOATS> : gemm_tile_kernel<TA, TW, TO, W_IS_NK, BM, BN, false>;
  static std::atomic<bool> allowed[2][64];
  if (int status = allow_smem(kernel, MOST_SMEM, allowed[pieces])) return status;
  return launch_clustered(kernel, grid, BM * BN / 64, smem, 2, stream, p, (n_groups + ranks - 1) / ranks);
}

// Up to this many rows the weights are streamed (a call's weights are then read once for every eight rows).
constexpr int FEW_ROWS = 32;
// ... as long as eight rows of `a` fit in shared memory as floats (beside the sums and the turning buffer)
constexpr int FEW_ROWS_MAX_K = 4096;

template <typename TA, typename TW, typename TO, bool W_IS_NK>
int launch(const Product& p, cudaStream_t stream) {
  if (p.m_total <= FEW_ROWS && p.k_total <= FEW_ROWS_MAX_K * 2) {
    if (p.m_total == 1) return launch_rows<TA, TW, TO, W_IS_NK, 1>(p, stream);
    if (p.m_total <= 4 || p.k_total > FEW_ROWS_MAX_K) return launch_rows<TA, TW, TO, W_IS_NK, 4>(p, stream);
    return launch_rows<TA, TW, TO, W_IS_NK, 8>(p, stream);
  }
  auto aligned = [](const void* q) { return reinterpret_cast<uintptr_t>(q) % 16 == 0; };
  const bool vec = aligned(p.a) && aligned(p.w) && p.lda % 4 == 0 && p.ldw % 4 == 0 && p.k_total % 4 == 0 && (W_IS_NK || p.n_total % 4 == 0);
  const int sms = n_sms(), len = slice_len(p.k_total), n_slices = (p.k_total + len - 1) / len, n_groups = (n_slices + GROUP - 1) / GROUP;
  auto tiles = [&](int bm, int bn) { return ((p.m_total + bm - 1) / bm) * ((p.n_total + bn - 1) / bn); };
  // fewer tiles than give every scheduler two warps: the groups of K in parallel
  if (p.m_total <= 64) return launch_tiles<TA, TW, TO, W_IS_NK, 64, 64>(p, vec, n_groups, tiles(64, 64) >= 4 * sms ? 1 : n_groups, stream);
  return launch_tiles<TA, TW, TO, W_IS_NK, 128, 64>(p, vec, n_groups, tiles(128, 64) >= 2 * sms ? 1 : n_groups, stream);
}

template <typename TA, typename TW, typename TO>
int launch(const Product& p, int w_is_nk, cudaStream_t stream) {
  return w_is_nk ? launch<TA, TW, TO, true>(p, stream) : launch<TA, TW, TO, false>(p, stream);
}

}  // namespace

// a [m, k] (leading dimension lda), w [k, n] or [n, k] (ldw), bias [n] float or null,
// residual [m, n] float or null (ldr), out [m, n] (ldo). Activations and weights share a dtype.
extern "C" int r2_gemm_simt(const void* a, int lda, const void* w, int ldw, int w_is_nk, const float* bias,
                            const float* residual, int ldr, void* out, int ldo, int m, int n, int k, int act,
                            int in_dtype, int out_dtype, cudaStream_t stream) {
  if (m <= 0 || n <= 0) return R2_OK;
  if (k < 1) return R2_BAD_SHAPE;
  if (act < R2_ACT_NONE || act > R2_ACT_GELU_ERF) return R2_UNSUPPORTED;
  const Product p = {a, w, lda, ldw, bias, residual, ldr, out, ldo, m, n, k, act};
  if (in_dtype == R2_F32 && out_dtype == R2_F32) return launch<float, float, float>(p, w_is_nk, stream);
  if (in_dtype == R2_BF16 && out_dtype == R2_F32) return launch<bf16, bf16, float>(p, w_is_nk, stream);
  if (in_dtype == R2_BF16 && out_dtype == R2_BF16) return launch<bf16, bf16, bf16>(p, w_is_nk, stream);
  return R2_BAD_DTYPE;
}
