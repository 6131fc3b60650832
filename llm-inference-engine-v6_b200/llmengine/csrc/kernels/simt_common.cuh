// What the float32 CUDA-core kernels share: copies of four elements of a row into shared memory, and the launch helpers.
#pragma once

#include "common.cuh"

#include <atomic>

// Of 4 elements of a row, the first `count` as float32 and zeros behind them (only what is counted is read).
template <typename T>
__device__ __forceinline__ float4 fetch4(const T* src, int count) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (count > 0) v.x = to_f32(src[0]);
  if (count > 1) v.y = to_f32(src[1]);
  if (count > 2) v.z = to_f32(src[2]);
  if (count > 3) v.w = to_f32(src[3]);
  return v;
}
// The same of bfloat16 rows whose every fourth element begins on 8 bytes; count is 0 or 4.
__device__ __forceinline__ float4 fetch4_aligned(const bf16* src, int count) {
  uint2 raw = make_uint2(0u, 0u);
  if (count > 0) raw = *reinterpret_cast<const uint2*>(src);
  return make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u), __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u));
}
// The same of float32 rows whose every fourth element begins on 16 bytes, into shared memory without passing through registers.
__device__ __forceinline__ void copy4(float* dst, const float* src, int count) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(4 * count) : "memory");
}
// Parts of N rows into shared memory as float32, zeros where nothing counts: dst(i), src(i) and count(i) say where part i goes, where
// it comes from and how many of its numbers count. ALIGNED: four numbers side by side, as copy4 (float32) or fetch4_aligned
// (bfloat16) need them; else E numbers GAP apart. Where the loads pass through registers, all are on their way before the first is
// stored: one latency, not N.
template <bool ALIGNED, int N, int E, int GAP, typename T, typename Dst, typename Src, typename Count>
__device__ __forceinline__ void stage_rows(Dst dst, Src src, Count count) {
  if constexpr (ALIGNED && sizeof(T) == 4) {
#pragma unroll
    for (int i = 0; i < N; ++i) copy4(dst(i), src(i), count(i));
  } else if constexpr (ALIGNED) {
    float4 v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = fetch4_aligned(src(i), count(i));
#pragma unroll
    for (int i = 0; i < N; ++i) *reinterpret_cast<float4*>(dst(i)) = v[i];
  } else {
    float v[N][E];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const T* from = src(i);
      const int n = count(i);
#pragma unroll
      for (int e = 0; e < E; ++e) v[i][e] = e < n ? to_f32(from[e * GAP]) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
      float* to = dst(i);
#pragma unroll
      for (int e = 0; e < E; ++e) to[e * GAP] = v[i][e];
    }
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
