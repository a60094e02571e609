// The two ends of a step that runs as a CUDA graph: its batch comes from pinned host memory and its tokens go there, by kernels instead of
// copy nodes. A copy node is a hand-over from the SMs to a copy engine and back: inside a step 6 to 8 us each for a few KB (one in front, two
// at the end), where a kernel that reads or writes the host's memory itself takes one trip over PCIe.
#include "common.cuh"

// dev[i] = host batch[i] of the two host batches that a graph's replays take in turn (`turn` counts the replays on the device), 16 bytes a
// thread. Kernels of the step read the batch's arrays ahead of their waits, so the launch behind this one must not be a programmatic one.
__global__ void __launch_bounds__(128)
fetch_batch_kernel(const uint4* even, const uint4* odd, uint4* __restrict__ dev, int n, const unsigned* turn) {
  const uint4* host = (*turn & 1u) ? odd : even;
  for (int i = blockIdx.x * 128 + threadIdx.x; i < n; i += gridDim.x * 128) {
    uint4 v;
    asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(host + i));
    dev[i] = v;
  }
}

// The sampled tokens and the device's error word into pinned host memory; one replay more has run.
__global__ void __launch_bounds__(128)
finish_step_kernel(const int32_t* __restrict__ tokens, int n, int32_t* host_tokens, const int32_t* error, int n_error, int32_t* host_error, unsigned* turn) {
  pdl_wait();
  for (int i = threadIdx.x; i < n; i += 128) host_tokens[i] = tokens[i];
  if (int(threadIdx.x) < n_error) host_error[threadIdx.x] = error[threadIdx.x];
  if (threadIdx.x == 0) *turn += 1u;
}

// The device's address of pinned host memory, or null where the device cannot reach it.
extern "C" void* r2_host_address(void* host) {
  void* p = nullptr;
  if (cudaHostGetDevicePointer(&p, host, 0) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return p;
}

// n_ints int32 (a multiple of 4; all three addresses multiples of 16 bytes).
extern "C" int r2_fetch_batch(const void* even, const void* odd, void* dev, int n_ints, const unsigned* turn, cudaStream_t stream) {
  if (n_ints <= 0) return R2_OK;
  if (n_ints % 4 != 0 || ((reinterpret_cast<uintptr_t>(even) | reinterpret_cast<uintptr_t>(odd) | reinterpret_cast<uintptr_t>(dev)) & 15)) return R2_BAD_ALIGN;
  const int pieces = n_ints / 4, blocks = (pieces + 127) / 128;
  fetch_batch_kernel<<<blocks < 148 ? blocks : 148, 128, 0, stream>>>(static_cast<const uint4*>(even), static_cast<const uint4*>(odd), static_cast<uint4*>(dev), pieces, turn);
  return launch_status();
}

extern "C" int r2_finish_step(const int32_t* tokens, int n, int32_t* host_tokens, const int32_t* error, int n_error, int32_t* host_error, unsigned* turn,
                              cudaStream_t stream) {
  if (n < 0 || n_error < 0 || n_error > 128) return R2_BAD_SHAPE;
  r2_launch(finish_step_kernel, dim3(1), dim3(128), size_t(0), stream, tokens, n, host_tokens, error, n_error, host_error, turn);
  return launch_status();
}
