// What the float32 CUDA-core kernels share: copies of four elements of a row into shared memory, and the launch helpers.
#pragma once

#include "common.cuh"

#include <atomic>

// Of 4 elements of a row, the first `count` as float32 into shared memory and zeros behind them. ASYNC: float32 rows whose
// every fourth element is 16-byte aligned, copied without passing through registers (only what is counted is read).
template <bool ASYNC, typename T>
__device__ __forceinline__ void stage4(float* dst, const T* src, int count) {
  if (ASYNC) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(4 * count) : "memory");
  } else {
    float4 v;
    v.x = count > 0 ? to_f32(src[0]) : 0.f;
    v.y = count > 1 ? to_f32(src[1]) : 0.f;
    v.z = count > 2 ? to_f32(src[2]) : 0.f;
    v.w = count > 3 ? to_f32(src[3]) : 0.f;
    *reinterpret_cast<float4*>(dst) = v;
  }
}
__device__ __forceinline__ int count4(int k, int K) { return max(0, min(4, K - k)); }
__device__ __forceinline__ void commit_group() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void wait_groups() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ float part(const float4& v, int e) { return e == 0 ? v.x : e == 1 ? v.y : e == 2 ? v.z : v.w; }

static inline int simt_sm_count() {
  static const int count = [] {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    return n;
  }();
  return count;
}

// More than 48 KB of shared memory has to be asked for, once a kernel and device (`done`: a bit a device).
template <typename K>
static inline void allow_smem(K kernel, int bytes, std::atomic<unsigned long long>& done) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return;
  if (dev < 64 && (done.load(std::memory_order_relaxed) >> dev & 1ull)) return;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess && dev < 64) done.fetch_or(1ull << dev);
}
