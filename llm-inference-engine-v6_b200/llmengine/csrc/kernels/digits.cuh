// float32 rows as whole numbers in four digits of base 256, the operands of gemm_digits.cu, which says what they are.
#pragma once

#include "common.cuh"

namespace {

// In the place of a row's exponent: the row does not fit the form, and its results are formed another way; one of them is NaN, and so they are.
constexpr int EXACT_ROW = 0x7ffffffe, NAN_ROW = 0x7fffffff;

// e with every |x| of the row below 2^e and its largest whole number clear of the top digit's last value
__device__ __forceinline__ int row_exponent(uint32_t largest) {  // the bits of the row's largest magnitude
  if (largest == 0u) return 0;
  if (largest > 0x7f800000u) return NAN_ROW;
  if (largest == 0x7f800000u || largest < 0x12800000u) return EXACT_ROW;  // infinities; below 2^-90
  return (int)(largest >> 23) - 126 + ((largest & 0x7fffffu) >= 0x7e0000u ? 1 : 0);
}
__device__ __forceinline__ float power_of_two(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }  // -126 <= e <= 127
__device__ __forceinline__ float row_scale_of(int e) { return e >= EXACT_ROW ? 0.f : power_of_two(31 - e); }

__device__ __forceinline__ uint32_t whole(float x, float scale) { return (uint32_t)__float2int_rn(x * scale); }
// Four words, the digits of a number each, into word p with digit p of each.
__device__ __forceinline__ void sort_digits(uint32_t t0, uint32_t t1, uint32_t t2, uint32_t t3, uint32_t (&p)[4]) {
  const uint32_t lo01 = __byte_perm(t0, t1, 0x5140), hi01 = __byte_perm(t0, t1, 0x7362);
  const uint32_t lo23 = __byte_perm(t2, t3, 0x5140), hi23 = __byte_perm(t2, t3, 0x7362);
  p[0] = __byte_perm(lo01, lo23, 0x5410);
  p[1] = __byte_perm(lo01, lo23, 0x7632);
  p[2] = __byte_perm(hi01, hi23, 0x5410);
  p[3] = __byte_perm(hi01, hi23, 0x7632);
}
__device__ __forceinline__ uint32_t magnitude4(float4 v) {
  return max(max(__float_as_uint(v.x) & 0x7fffffffu, __float_as_uint(v.y) & 0x7fffffffu),
             max(__float_as_uint(v.z) & 0x7fffffffu, __float_as_uint(v.w) & 0x7fffffffu));
}


// Four numbers of an activation row as digits, balanced: word d has digit d of each. Returns their sum as whole numbers.
__device__ __forceinline__ long long balanced_digits(float4 x, float scale, uint32_t (&d)[4]) {
  uint32_t q[4] = {whole(x.x, scale), whole(x.y, scale), whole(x.z, scale), whole(x.w, scale)};
  long long sum = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    sum += (int)q[i];
    q[i] = (q[i] + 0x808080u) ^ 0x808080u;
  }
  sort_digits(q[0], q[1], q[2], q[3], d);
  return sum;
}
// The weights' constant times a row's sum, in the unit of the results, 2^24.
__device__ __forceinline__ long long constant_share(long long sum) { return (long long)(((__int128)sum * 0x808080 + (1 << 23)) >> 24); }

// Four numbers, the part-th of a row, into its digits [k / 64][digit][64].
__device__ __forceinline__ void put_digits(uint8_t* row, int part, const uint32_t (&d)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) *reinterpret_cast<uint32_t*>(row + (part >> 4) * 256 + i * 64 + (part & 15) * 4) = d[i];
}

// Where rows go as digits: digits [row][ceil(dim / 64)][4][64], exps and sums a number a row.
struct DigitRows {
  uint8_t* digits;
  int* exps;
  long long* sums;
};
// A row that a block has in registers, four numbers a thread at (thread + k * threads) * 4, dim % 4 == 0. Every thread calls.
template <int R>
__device__ __forceinline__ void put_digit_row(const float4 (&x)[R], int dim, int row, const DigitRows& to) {
  __shared__ uint32_t s_max[32];
  __shared__ long long s_sum[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (blockDim.x + 31) >> 5, parts = (dim + 63) / 64 * 16;
  uint32_t largest = 0u;
#pragma unroll
  for (int k = 0; k < R; ++k)
    if ((threadIdx.x + k * blockDim.x) * 4 < dim) largest = max(largest, magnitude4(x[k]));  // (what lies beyond the row may be NaN)
  largest = __reduce_max_sync(0xffffffffu, largest);
  if (lane == 0) s_max[warp] = largest;
  __syncthreads();
  largest = __reduce_max_sync(0xffffffffu, lane < warps ? s_max[lane] : 0u);
  const int e = row_exponent(largest);
  const float scale = row_scale_of(e);
  uint8_t* at = to.digits + (size_t)row * parts * 16;
  long long sum = 0;
  uint32_t d[4];
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const int part = threadIdx.x + k * blockDim.x;
    if (part * 4 < dim) {
      sum += balanced_digits(x[k], scale, d);
      put_digits(at, part, d);
    }
  }
  const uint32_t none[4] = {0u, 0u, 0u, 0u};
  for (int part = dim / 4 + threadIdx.x; part < parts; part += blockDim.x) put_digits(at, part, none);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0) s_sum[warp] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < warps; ++i) sum += s_sum[i];
    to.exps[row] = e;
    to.sums[row] = constant_share(sum);
  }
}

}  // namespace
