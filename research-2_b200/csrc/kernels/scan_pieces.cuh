// What the walks over a recurrence's rows share: rows' vectors into shared memory ahead of their use, two floats an instruction, and the
// sums of several rows over a column's lanes.
#pragma once

#include <stdint.h>

namespace {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }

// How a CTA's threads go over the 16-byte pieces (or the elements) of some rows: the first one's place, and the way to the next. (The
// divisions are made once; inside the copies' loops, which run once per tile between the rows' chains, a step is an addition.)
struct PieceWalk {
  int per_row, r0, c0, dr, dc;
  __device__ __forceinline__ explicit PieceWalk(int n) : per_row(n > 0 ? n : 1) {
    r0 = threadIdx.x / per_row;
    c0 = threadIdx.x - r0 * per_row;
    dr = blockDim.x / per_row;
    dc = blockDim.x - dr * per_row;
  }
};

// n_rows rows into shared memory, asynchronously in 16-byte pieces or element by element
template <typename T>
__device__ __forceinline__ void stage_rows(T* dst, int dst_stride, const T* src, long long src_stride, const PieceWalk& w, int n_rows, bool pieces) {
  constexpr int PER = 16 / int(sizeof(T));
  for (int r = w.r0, c = w.c0; r < n_rows;) {
    if (pieces) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst + r * dst_stride + c * PER)), "l"(src + r * src_stride + c * PER) : "memory");
    else dst[r * dst_stride + c] = src[r * src_stride + c];
    r += w.dr;
    c += w.dc;
    if (c >= w.per_row) {
      c -= w.per_row;
      ++r;
    }
  }
}

// n_rows staged rows, times `scale`, as floats (the walk's pieces; both sides on 16-byte boundaries)
template <typename T>
__device__ __forceinline__ void spread_rows(float* dst, int dst_stride, const T* src, int src_stride, const PieceWalk& w, int n_rows, float scale) {
  constexpr int PER = 16 / int(sizeof(T));
  for (int r = w.r0, c = w.c0; r < n_rows;) {
    const uint4 bits = *reinterpret_cast<const uint4*>(src + r * src_stride + c * PER);
    const T* v = reinterpret_cast<const T*>(&bits);
    float* to = dst + r * dst_stride + c * PER;
#pragma unroll
    for (int u = 0; u < PER; u += 4)
      *reinterpret_cast<float4*>(to + u) = make_float4(to_float(v[u]) * scale, to_float(v[u + 1]) * scale, to_float(v[u + 2]) * scale, to_float(v[u + 3]) * scale);
    r += w.dr;
    c += w.dc;
    if (c >= w.per_row) {
      c -= w.per_row;
      ++r;
    }
  }
}

// Two floats side by side: one instruction for both, each rounded as the single one rounds.
__device__ __forceinline__ uint64_t pair_of(float lo, float hi) {
  uint64_t p;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(lo), "f"(hi));
  return p;
}
__device__ __forceinline__ float2 both(uint64_t p) {
  float2 v;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ uint64_t mul_pair(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t fma_pair(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// Four rows' sums over a column's G >= 4 lanes, G / 2 lanes apart first: at the first two steps a lane gives half of its rows away, so
// that four rows take 3 + log2(G) - 2 shuffles instead of 4 log2(G). Every sum has the terms and the order of the shuffles row by row.
// -> the sum of row 2 [g & G/2] + [g & G/4].
__device__ __forceinline__ float sums_of_four(float y0, float y1, float y2, float y3, int g, int G) {
  const bool late = (g & (G >> 1)) != 0, odd = (g & (G >> 2)) != 0;
  const float other0 = __shfl_xor_sync(0xffffffffu, late ? y0 : y2, G >> 1), other1 = __shfl_xor_sync(0xffffffffu, late ? y1 : y3, G >> 1);
  const float a0 = (late ? y2 : y0) + other0, a1 = (late ? y3 : y1) + other1;
  float y = (odd ? a1 : a0) + __shfl_xor_sync(0xffffffffu, odd ? a0 : a1, G >> 2);
  for (int o = G >> 3; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
  return y;
}

}  // namespace
