// Host buffers of the host-pointer entry points.
//
// On the B200 hosts measured, the copy engines moved page-locked host memory
// at about 24 GB/s, while kernels reading the same memory through its
// device mapping reached about 55 GB/s (PCIe 5.0 x16). So when a caller's
// buffer is page-locked and mapped (cudaPointerGetAttributes: host memory
// with a device address), outputs are written by the compute kernel straight
// into the host buffer, and inputs are either read in place by the compute
// kernel (the radiance estimate, which fetches each query record one query
// ahead) or fetched by a streaming copy kernel (the index search); other
// (pageable) buffers go through cudaMemcpyAsync.
#include "pm_hostio.cuh"

namespace pm {

const void* mapped_host(const void* p) {
  if (!p) return nullptr;
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return a.type == cudaMemoryTypeHost ? a.devicePointer : nullptr;
}

// Grid-stride copy of n16 16-byte words, 4 loads in flight per thread.
__global__ void __launch_bounds__(256)
    stream_copy_kernel(uint4* __restrict__ dst, const uint4* __restrict__ src, size_t n16) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  for (; i + 3 * stride < n16; i += 4 * stride) {
    const uint4 a = src[i], b = src[i + stride], c = src[i + 2 * stride], d = src[i + 3 * stride];
    dst[i] = a;
    dst[i + stride] = b;
    dst[i + 2 * stride] = c;
    dst[i + 3 * stride] = d;
  }
  for (; i < n16; i += stride) dst[i] = src[i];
}

cudaError_t copy_in(void* dst, const void* host, size_t bytes, int num_sms, cudaStream_t st) {
  if (bytes == 0) return cudaSuccess;
  const void* src = mapped_host(host);
  if (src && bytes % 16 == 0 && ((uintptr_t)src & 15) == 0 && ((uintptr_t)dst & 15) == 0) {
    const size_t n16 = bytes / 16;
    size_t blocks = (n16 + 255) / 256;
    const size_t cap = (size_t)num_sms * 8;
    if (blocks > cap) blocks = cap;
    stream_copy_kernel<<<(unsigned)blocks, 256, 0, st>>>((uint4*)dst, (const uint4*)src, n16);
    return cudaGetLastError();
  }
  return cudaMemcpyAsync(dst, host, bytes, cudaMemcpyHostToDevice, st);
}

cudaError_t copy_out(void* host, const void* src, size_t bytes, int num_sms, cudaStream_t st) {
  if (bytes == 0) return cudaSuccess;
  void* dst = const_cast<void*>(mapped_host(host));
  if (dst && bytes % 16 == 0 && ((uintptr_t)src & 15) == 0 && ((uintptr_t)dst & 15) == 0) {
    const size_t n16 = bytes / 16;
    size_t blocks = (n16 + 255) / 256;
    const size_t cap = (size_t)num_sms * 8;
    if (blocks > cap) blocks = cap;
    stream_copy_kernel<<<(unsigned)blocks, 256, 0, st>>>((uint4*)dst, (const uint4*)src, n16);
    return cudaGetLastError();
  }
  return cudaMemcpyAsync(host, src, bytes, cudaMemcpyDeviceToHost, st);
}

}  // namespace pm
