// Products of few rows (decode steps): out = act(rows . w^T + bias) (+ residual) for up to 64 rows and w [N][K] bfloat16 stored [out, in];
// the rows are bfloat16, or a LayerNorm or RMS norm of float rows that is computed here (up to 16 rows of up to 1,024).
//
// What bounds it: inside a step such a product is a link of a chain. Its weights (1 to 8 MB) come while the kernels before it still run, so
// what is left is the hand-over from the kernel before (about 1.3 us from its last store to these threads), one round trip for the rows,
// the products, one exchange between warps and the stores. So everything is arranged for that path to be short:
//   * mma.sync m16n8k16 with the rows as the 16-row side: a CTA has 8, 16 or 32 features and all of K, its warps share K in blocks of 32,
//     and nothing leaves the SM but the result: no cluster, no tensor map, no barrier but the one before the warps' sums are added (in
//     warp order). The tcgen05 form's K split over a cluster, TMA and tensor-memory round trips cost 3.8 to 6 us.
//   * a lane's operands are 16 contiguous bytes of a feature's and of a row's values (which k a lane calls its first is free as long as
//     both sides agree), so rows go from L2 straight into the instruction's registers, weights through a private place in shared memory
//     that the lane itself fills with asynchronous copies ahead of the wait: no registers held meanwhile and no barrier.
//   * an RMS norm multiplies the sums at the end (its factor is a row's own), so the products do not wait for it; a LayerNorm's mean and
//     variance are joined from the warps' shares behind one barrier.
// Measured inside a graph of such products, 768 wide, us a launch, tcgen05 form and this one (one row / 8 / 16 / 32 rows): q/k/v of 2,304
// features 3.9 and 2.1 / 4.4 and 2.2 / 5.2 and 2.6 / 7.4 and 3.1; 768 x 768 3.8 and 1.9 / 4.0 and 2.1 / 4.5 and 2.2 / 6.2 and 2.7;
// 3,072 x 768 4.6 and 2.4 / 5.0 and 2.6 / 5.8 and 3.7 / 7.4 and 5.0. A decode step of GPT-2 124M with 200 keys a row: 348 us as the resident
// kernel, 406 as the chain with tcgen05 products, 222 as the chain with these (one row); 381, 445 and 251 (8 rows).
#include "common.cuh"
#include "mma_sync.cuh"

namespace {

struct FewRows {
  const bf16* a; int lda;                        // rows [m][k] (NORM: null)
  const float* x; int ldx;                       // NORM: rows [m][k] before the norm
  const float* gain; const float* shift;         // NORM: [k]; shift may be null
  float eps; int centred;                        // centred: LayerNorm, else RMS norm
  const bf16* w; int ldw;
  const float* bias; const float* residual; int ldr;
  void* out; int ldo; int out_bf16;
  int m, n, k, act;
  int group_n;                                   // > 0: features s * group_n .. read the rows' columns from s * k on
};

__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool there) {
  const int bytes = there ? 16 : 0;   // 0 source bytes: zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// MH: halves of eight rows (1, 2, 4 or 8), NT: tiles of eight features a CTA, KBN: NORM (more than 0), blocks of 32 k that a warp holds of
// every row, CENTRED: LayerNorm, else RMS norm
template <int MH, int NT, int WARPS, int KBN, bool CENTRED>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 8 && MH <= 2 ? 3 : 1) few_rows_kernel(const FewRows p) {
  constexpr bool NORM = KBN > 0;
  constexpr int MT = (MH + 1) / 2, CH = MH == 1 ? 2 : 4;   // row tiles of the matrix instruction; accumulators of one that rows use
  constexpr int THREADS = WARPS * 32, OUTS = MT * NT * CH * 32, PER = (OUTS + THREADS - 1) / THREADS;
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ float4 stats[NORM ? WARPS * 8 * MH : 1];   // NORM: the warps' shares of the rows' sums
  float* red = reinterpret_cast<float*>(smem);   // [WARPS][OUTS]
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3;
  const int f0 = blockIdx.x * (NT * 8);
  const int blocks = (p.k + 31) >> 5, kpad = blocks * 32;
  uint8_t* mine = smem + WARPS * OUTS * 4 + (NORM ? size_t(kpad) * 8 : 0) + threadIdx.x * 16;   // this thread's pieces of the weights, THREADS * 16 apart
  {
    const uint32_t dst = uint32_t(__cvta_generic_to_shared(mine));
    const bf16* src = p.w + size_t(f0 + gq) * p.ldw + tq * 8;
    int at = 0;
    for (int blk = warp; blk < blocks; blk += WARPS) {
      const int kk = blk * 32;
#pragma unroll
      for (int t = 0; t < NT; ++t, ++at) {
        const bool there = kk + tq * 8 < p.k && f0 + t * 8 + gq < p.n;
        copy16(dst + at * (THREADS * 16), there ? src + size_t(t) * 8 * p.ldw + kk : p.w, there);
      }
    }
  }
  pdl_wait();
  if constexpr (NORM) {
    const uint32_t dst = uint32_t(__cvta_generic_to_shared(smem + WARPS * OUTS * 4));
    for (int i = threadIdx.x * 4; i < kpad; i += THREADS * 4) {
      copy16(dst + i * 4, i < p.k ? p.gain + i : p.gain, i < p.k);
      copy16(dst + (kpad + i) * 4, i < p.k && p.shift != nullptr ? p.shift + i : p.gain, i < p.k && p.shift != nullptr);
    }
  }
  float acc[MT][NT][4];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int t = 0; t < NT; ++t) acc[i][t][0] = acc[i][t][1] = acc[i][t][2] = acc[i][t][3] = 0.f;
  // what this thread's outputs are added to: element i = threadIdx.x + j * THREADS of [MT][NT][CH][32 lanes]
  float add[PER], res[PER];
  auto place = [&](int j, int& row, int& col) {
    const int i = threadIdx.x + j * THREADS, l = i & 31, c = (i >> 5) % CH, t = (i >> 5) / CH % NT, mt = (i >> 5) / (CH * NT);
    row = mt * 16 + (l >> 2) + 8 * (c >> 1);
    col = f0 + t * 8 + 2 * (l & 3) + (c & 1);
    return i < OUTS && row < p.m && col < p.n;
  };
  auto ask = [&]() {
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      int row, col;
      const bool there = place(j, row, col);
      add[j] = there && p.bias != nullptr ? __ldcg(p.bias + col) : 0.f;
      res[j] = there && p.residual != nullptr ? __ldcg(p.residual + size_t(row) * p.ldr + col) : 0.f;
    }
  };
  if constexpr (NORM) {
    float4 v[KBN][MH][2];
#pragma unroll
    for (int b = 0; b < KBN; ++b) {
      const int kk = (warp + b * WARPS) * 32 + tq * 8;
#pragma unroll
      for (int h = 0; h < MH; ++h) {
        const bool there = gq + 8 * h < p.m && kk < p.k;
        const float4* at = reinterpret_cast<const float4*>(p.x + size_t(gq + 8 * h) * p.ldx + kk);
        v[b][h][0] = there ? __ldcg(at) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[b][h][1] = there ? __ldcg(at + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    ask();
    float mean[MH], rstd[MH];
    if constexpr (CENTRED) {
      // A warp's share of a row: its sum, then the squares about the share's own mean; the warps' shares join exactly as one set's would
      // (Chan, Golub and LeVeque's formula for the variance of joined samples).
      int count = 0;
#pragma unroll
      for (int b = 0; b < KBN; ++b) count += max(0, min(32, p.k - (warp + b * WARPS) * 32));
      const float inv = count > 0 ? 1.f / float(count) : 0.f;
#pragma unroll
      for (int h = 0; h < MH; ++h) {
        float s = 0.f, q = 0.f;
#pragma unroll
        for (int b = 0; b < KBN; ++b) {
          const float4 u = v[b][h][0], z = v[b][h][1];
          s += ((u.x + u.y) + (u.z + u.w)) + ((z.x + z.y) + (z.z + z.w));
        }
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        const float mu = s * inv;
#pragma unroll
        for (int b = 0; b < KBN; ++b) {
          const float4 u = v[b][h][0], z = v[b][h][1];
          const float e = (((u.x - mu) * (u.x - mu) + (u.y - mu) * (u.y - mu)) + ((u.z - mu) * (u.z - mu) + (u.w - mu) * (u.w - mu))) +
                          (((z.x - mu) * (z.x - mu) + (z.y - mu) * (z.y - mu)) + ((z.z - mu) * (z.z - mu) + (z.w - mu) * (z.w - mu)));
          if ((warp + b * WARPS) * 32 + tq * 8 < p.k) q += e;
        }
        q += __shfl_xor_sync(0xffffffffu, q, 1);
        q += __shfl_xor_sync(0xffffffffu, q, 2);
        if (tq == 0) stats[(warp * MH + h) * 8 + gq] = make_float4(s, q, mu, float(count));
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
      const float inv_k = 1.f / float(p.k);
#pragma unroll
      for (int h = 0; h < MH; ++h) {
        float s = 0.f, q = 0.f;
#pragma unroll
        for (int i = 0; i < WARPS; ++i) s += stats[(i * MH + h) * 8 + gq].x;
        mean[h] = s * inv_k;
#pragma unroll
        for (int i = 0; i < WARPS; ++i) {
          const float4 part = stats[(i * MH + h) * 8 + gq];
          const float d = part.z - mean[h];
          q += fmaf(part.w, d * d, part.y);
        }
        rstd[h] = 1.f / sqrtf(q * inv_k + p.eps);
      }
    } else {
      // an RMS norm's factor is a row's own: it multiplies the sums at the end, and the products need not wait for it
#pragma unroll
      for (int h = 0; h < MH; ++h) {
        float q = 0.f;
#pragma unroll
        for (int b = 0; b < KBN; ++b) {
          const float4 u = v[b][h][0], z = v[b][h][1];
          q += ((u.x * u.x + u.y * u.y) + (u.z * u.z + u.w * u.w)) + ((z.x * z.x + z.y * z.y) + (z.z * z.z + z.w * z.w));
        }
        q += __shfl_xor_sync(0xffffffffu, q, 1);
        q += __shfl_xor_sync(0xffffffffu, q, 2);
        if (tq == 0) stats[(warp * MH + h) * 8 + gq] = make_float4(0.f, q, 0.f, 0.f);
        mean[h] = 0.f;
        rstd[h] = 1.f;
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
    }
    const float* gs = reinterpret_cast<const float*>(smem + WARPS * OUTS * 4);
#pragma unroll
    for (int b = 0; b < KBN; ++b) {
      const int blk = warp + b * WARPS, kk = blk * 32 + tq * 8;
      if (blk < blocks) {   // (the same for a whole warp; past k gain, shift and weights are zeros)
        const float4 g0 = *reinterpret_cast<const float4*>(gs + kk), g1 = *reinterpret_cast<const float4*>(gs + kk + 4);
        float4 s0 = make_float4(0.f, 0.f, 0.f, 0.f), s1 = s0;
        if (CENTRED) s0 = *reinterpret_cast<const float4*>(gs + kpad + kk), s1 = *reinterpret_cast<const float4*>(gs + kpad + kk + 4);
        uint32_t f[2 * MT][4];
#pragma unroll
        for (int h = 0; h < 2 * MT; ++h) {
          if (h < MH) {
            const float4 u = v[b][h < MH ? h : 0][0], z = v[b][h < MH ? h : 0][1];
            const float mu = mean[h < MH ? h : 0], rs = rstd[h < MH ? h : 0];
            const __nv_bfloat162 t0 = __floats2bfloat162_rn((u.x - mu) * rs * g0.x + s0.x, (u.y - mu) * rs * g0.y + s0.y);
            const __nv_bfloat162 t1 = __floats2bfloat162_rn((u.z - mu) * rs * g0.z + s0.z, (u.w - mu) * rs * g0.w + s0.w);
            const __nv_bfloat162 t2 = __floats2bfloat162_rn((z.x - mu) * rs * g1.x + s1.x, (z.y - mu) * rs * g1.y + s1.y);
            const __nv_bfloat162 t3 = __floats2bfloat162_rn((z.z - mu) * rs * g1.z + s1.z, (z.w - mu) * rs * g1.w + s1.w);
            f[h][0] = *reinterpret_cast<const uint32_t*>(&t0); f[h][1] = *reinterpret_cast<const uint32_t*>(&t1);
            f[h][2] = *reinterpret_cast<const uint32_t*>(&t2); f[h][3] = *reinterpret_cast<const uint32_t*>(&t3);
          } else {
            f[h][0] = f[h][1] = f[h][2] = f[h][3] = 0u;
          }
        }
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const uint4 w = *reinterpret_cast<const uint4*>(mine + (b * NT + t) * (THREADS * 16));
#pragma unroll
          for (int i = 0; i < MT; ++i) {
            mma_bf16(acc[i][t], f[2 * i][0], f[2 * i + 1][0], f[2 * i][1], f[2 * i + 1][1], w.x, w.y);
            mma_bf16(acc[i][t], f[2 * i][2], f[2 * i + 1][2], f[2 * i][3], f[2 * i + 1][3], w.z, w.w);
          }
        }
      }
    }
    if constexpr (!CENTRED) {   // (the rows' factors, while the products run)
      float scale[MH];
#pragma unroll
      for (int h = 0; h < MH; ++h) {
        float q = 0.f;
#pragma unroll
        for (int i = 0; i < WARPS; ++i) q += stats[(i * MH + h) * 8 + gq].y;
        scale[h] = 1.f / sqrtf(q * (1.f / float(p.k)) + p.eps);
      }
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[i][t][c] *= 2 * i + (c >> 1) < MH ? scale[2 * i + (c >> 1) < MH ? 2 * i + (c >> 1) : 0] : 0.f;
    }
  } else {
    constexpr int AHEAD = MH == 1 ? 6 : MH == 2 ? 4 : MH == 4 ? 2 : 1;   // blocks of 32 k whose rows are asked for at a time
    const bf16* a = p.a + (p.group_n > 0 ? size_t(f0 / p.group_n) * p.k : 0) + size_t(gq) * p.lda + tq * 8;
    bool first = true;
    for (int b0 = 0; warp + b0 * WARPS < blocks; b0 += AHEAD) {
      uint4 v[AHEAD][2 * MT];
#pragma unroll
      for (int b = 0; b < AHEAD; ++b) {
        const int kk = (warp + (b0 + b) * WARPS) * 32;
#pragma unroll
        for (int h = 0; h < 2 * MT; ++h) {
          v[b][h] = h < MH && gq + 8 * h < p.m && kk + tq * 8 < p.k ? __ldcg(reinterpret_cast<const uint4*>(a + size_t(8 * h) * p.lda + kk)) : make_uint4(0u, 0u, 0u, 0u);
        }
      }
      if (first) {
        ask();
        asm volatile("cp.async.wait_all;" ::: "memory");   // (a thread reads only the pieces that it copied itself)
        first = false;
      }
#pragma unroll
      for (int b = 0; b < AHEAD; ++b) {
        if (warp + (b0 + b) * WARPS < blocks) {
#pragma unroll
          for (int t = 0; t < NT; ++t) {
            const uint4 w = *reinterpret_cast<const uint4*>(mine + ((b0 + b) * NT + t) * (THREADS * 16));
#pragma unroll
            for (int i = 0; i < MT; ++i) {
              mma_bf16(acc[i][t], v[b][2 * i].x, v[b][2 * i + 1].x, v[b][2 * i].y, v[b][2 * i + 1].y, w.x, w.y);
              mma_bf16(acc[i][t], v[b][2 * i].z, v[b][2 * i + 1].z, v[b][2 * i].w, v[b][2 * i + 1].w, w.z, w.w);
            }
          }
        }
      }
    }
    if (first) ask();   // (a warp without a share of k)
  }
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int c = 0; c < CH; ++c) red[warp * OUTS + ((i * NT + t) * CH + c) * 32 + lane] = acc[i][t][c];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    int row, col;
    if (place(j, row, col)) {
      float s = 0.f;
#pragma unroll
      for (int q = 0; q < WARPS; ++q) s += red[q * OUTS + threadIdx.x + j * THREADS];
      s += add[j];
      if (p.act == R2_ACT_GELU_TANH) s = p.out_bf16 ? gelu_tanh_hw(s) : gelu_tanh(s);
      else if (p.act == R2_ACT_GELU_ERF) s = p.out_bf16 ? gelu_erf_rounded(s) : gelu_erf(s);
      s += res[j];
      if (p.out_bf16) static_cast<bf16*>(p.out)[size_t(row) * p.ldo + col] = __float2bfloat16_rn(s);
      else static_cast<float*>(p.out)[size_t(row) * p.ldo + col] = s;
    }
  }
}

template <int MH, int NT, int WARPS, int KBN, bool CENTRED = false>
int launch(const FewRows& p, cudaStream_t stream) {
  constexpr int OUTS = (MH + 1) / 2 * NT * (MH == 1 ? 2 : 4) * 32;
  const int blocks = (p.k + 31) / 32;
  if (KBN > 0 && blocks > KBN * WARPS) return R2_UNSUPPORTED;
  const size_t smem = size_t(WARPS) * OUTS * 4 + (KBN > 0 ? size_t(blocks) * 256 : 0) + size_t((blocks + WARPS - 1) / WARPS) * NT * WARPS * 512;
  if (smem > 200 * 1024) return R2_UNSUPPORTED;
  static std::atomic<bool> allowed[64];
  if (smem > 40 * 1024) {
    const int status = allow_smem(few_rows_kernel<MH, NT, WARPS, KBN, CENTRED>, 200 * 1024, allowed);
    if (status != R2_OK) return status;
  }
  r2_launch(few_rows_kernel<MH, NT, WARPS, KBN, CENTRED>, dim3((p.n + NT * 8 - 1) / (NT * 8)), dim3(WARPS * 32), smem, stream, p);
  return launch_status();
}

// The split, by what measured best in whole decode steps (widths 768, 1,024 and 1,600; us a step): 16 warps to a CTA and a CTA to an SM, so the
// fewest features a CTA that leave one wave of 148: 16 up to 2,368 features, 32 up to 4,736 (K up to 1,024: the next kernel's CTAs find room
// beside them; 355M, 8 rows: 32 and 16 features 518 and 519, 24 rows 893 and 908). Beyond, 8 warps with 16 features and several CTAs to an SM
// (1.5B, one row: 1,619; 16 warps 1,870, 32 features 1,730). Long rows (K from 2,048) 8 features a CTA, so that the weights of a CTA stay
// below 100 KB (124M, 8 rows: 251, 16 features 259), of 8 warps where K is beyond 5,120 (1.5B, one row: 1,612 and 1,680). More than 16 rows
// make a CTA's rows the larger part: few features get 8 to a CTA (32 rows: 432 and 457).
template <int MH>
int by_form(const FewRows& p, cudaStream_t stream) {
  if (p.x != nullptr) {
    if constexpr (MH <= 2) return p.centred ? launch<MH, 4, 16, 2, true>(p, stream) : launch<MH, 4, 16, 2, false>(p, stream);
    return R2_UNSUPPORTED;
  }
  if (p.k >= 2048) {
    if constexpr (MH <= 2) {
      if (p.k > 5120) return launch<MH, 1, 8, 0>(p, stream);
    }
    return launch<MH, 1, 16, 0>(p, stream);
  }
  if (p.n <= 1184 && MH > 2) return launch<MH, 1, 16, 0>(p, stream);
  if (p.n <= 2368) return launch<MH, 2, 16, 0>(p, stream);
  if constexpr (MH <= 4) {
    if (p.n <= 4736 && p.k <= 1024) return launch<MH, 4, 16, 0>(p, stream);
    if constexpr (MH <= 2) {
      if (p.n > 7104 && p.k <= 1024) return launch<MH, 4, 8, 0>(p, stream);   // (9,216 x 768, 8 rows: 4.0 us, 16 features 4.5, tcgen05 6.4; 6,144: 3.4 and 3.3)
    }
    return launch<MH, 2, 8, 0>(p, stream);
  }
  return launch<MH, 2, 16, 0>(p, stream);
}

// The most features for which this kernel is no slower than the tcgen05 one, beside the bounds on all weights below. Both measured with 24
// launches one behind the other, and with a norm of the rows between them, over rows of 1 to 64, K of 64 to 12,288 and 8 to 12,288 features; the line
// lies where this kernel is more than about 1 us slower in both (an activation adds up to 3 us to the other one: 64 rows of 3,072 x 768
// take 8.0 / 7.4 us bare, and a step of GPT-2 124M, whose 12 have one, 0.722 / 0.737 ms). This kernel / the other one, us, one behind the other:
//   * every CTA reads all rows: with many features and a short K that is most of its work (64 rows of 64: 2,560 features 4.8 / 3.1, 6,144
//     7.0 / 3.2; 24 rows of 256: 8,192 features 5.0 / 4.4, 10,240 7.4 / 3.4). A LayerNorm inside is made anew by every CTA (8 rows of 768: 8,192 features
//     6.9 / 8.1, 10,240, a second wave, 10.2 / 7.3).
//   * long K: eight features to a CTA, so the CTAs are many (one row of 2,048: 3,072 features 6.0 / 6.5, 3,584 7.7 / 6.5; of 4,096: 2,560 8.6 / 7.7;
//     of 8,192: 1,280 9.9 / 8.2; 16 rows of 2,560: 2,560 9.4 / 7.4; 24 of 2,048: 2,560 9.0 / 7.8), and with more than 16 rows one to an SM:
//     160 of them are two waves (24 rows of 4,096: 1,280 features 9.0 / 7.5; 64 of 3,072: 1,280 12.3 / 9.0).
int most_features(int m, int k, int norm) {   // norm: 0 none, 1 RMS, 2 LayerNorm
  if (norm == 2) return 9472;
  if (m <= 8) return k < 2048 ? 12288 : k <= 3072 ? 3072 : k < 7000 ? 2368 : 1184;
  if (m <= 16) return k < 2048 ? 9472 : 2368;
  if (m <= 32) return k < 128 ? 4736 : k < 2048 ? 7104 : k <= 3072 ? 2368 : 1184;
  return k < 128 ? 2368 : k < 2048 ? 4608 : k <= 4608 ? 1184 : 0;
}

}  // namespace

// Whether the kernel is the choice for these sizes (`norm`: 0 none, 1 RMS norm, 2 LayerNorm). Bounds on all weights: many weights for many
// rows, where every CTA's reading of all rows outweighs the shorter path (K x N 6,400 x 1,600: 16 rows 9.4 us there and 9.7 here; 768 x 9,216, 24 rows: 7.3
// and 7.6; 1,600 x 4,800, 32 rows: 8.1 and 10.2; 64 rows of 4,608 x 768 8.9 and 8.9, of 6,144 x 768 9.9 and 10.9).
extern "C" int r2_few_rows_takes(int m, int n, int k, int norm) {
  const long long weights = (long long)n * k;
  const long long most = m > 32 ? (k >= 2048 ? 4000000LL : 2400000LL) : m > 16 ? (k >= 2048 ? 6500000LL : 4500000LL) : m > 8 ? (k > 4096 ? 5000000LL : 8000000LL) : 12000000LL;
  return m <= 64 && weights <= most && n <= most_features(m, k, norm);
}

// a [m, k] bfloat16 (row stride lda), or x [m, k] float with gain [k] and, centred, shift [k] (a is then ignored); w [n, k] bfloat16 (row
// stride ldw); bias [n] float or null; residual [m, n] float or null, added after the activation; out [m, n] bfloat16 or float. With
// group_n > 0 the rows are [m, n / group_n * k] wide and features s * group_n .. read the columns from s * k on.
// R2_UNSUPPORTED where the tcgen05 kernel must decide (more than 64 rows, norms beyond 16 rows or 1,024 numbers, rows that are no multiples of
// 16 bytes) or is the faster one (`most_features`).
extern "C" int r2_few_rows(const void* a, int lda, const float* x, int ldx, const float* gain, const float* shift, float eps, int centred,
                           const void* w, int ldw, const float* bias, const float* residual, int ldr, void* out, int ldo, int out_dtype,
                           int m, int n, int k, int act, int group_n, cudaStream_t stream) {
  if (m <= 0 || n <= 0) return R2_OK;
  if (act < R2_ACT_NONE || act > R2_ACT_GELU_ERF || k < 8 || k % 8 != 0 || ldw % 8 != 0 || (reinterpret_cast<uintptr_t>(w) & 15)) return R2_UNSUPPORTED;
  if (out_dtype != R2_F32 && out_dtype != R2_BF16) return R2_BAD_DTYPE;
  if (x != nullptr) {
    if (ldx % 4 != 0 || gain == nullptr || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(gain) & 15) || (reinterpret_cast<uintptr_t>(shift) & 15)) return R2_UNSUPPORTED;
    if (m > 16 || k > 1024 || (!centred && shift != nullptr)) return R2_UNSUPPORTED;
  } else if (lda % 8 != 0 || (reinterpret_cast<uintptr_t>(a) & 15)) {
    return R2_UNSUPPORTED;
  }
  if (!r2_few_rows_takes(m, n, k, x == nullptr ? 0 : centred ? 2 : 1)) return R2_UNSUPPORTED;
  if (group_n > 0 && (n % group_n != 0 || group_n % 32 != 0)) return R2_UNSUPPORTED;   // (a CTA's features lie in one group)
  const FewRows p{static_cast<const bf16*>(a), lda, x, ldx, gain, shift, eps, centred, static_cast<const bf16*>(w), ldw, bias, residual, ldr, out, ldo,
                  out_dtype == R2_BF16, m, n, k, act, group_n};
  if (m <= 8) return by_form<1>(p, stream);
  if (m <= 16) return by_form<2>(p, stream);
  if (m <= 32) return by_form<4>(p, stream);
  return by_form<8>(p, stream);
}
