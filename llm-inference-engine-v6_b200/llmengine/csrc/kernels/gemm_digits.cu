// float32 products on the 5th-generation tensor cores, exact in whole numbers.
//
//   out[m, n] = sum_k a[m, k] * w[n, k]          a: [M, K] activations, w: [N, K] weights, both float32
//
// Every row of a and of w is written as whole numbers of 31 bits and sign on a scale of its own, x = q * 2^(e - 31) with 2^e just
// above the row's largest magnitude, and q in four digits of base 256 between -128 and 127. A digit of a times a digit of w is a
// product of 8-bit whole numbers, which tcgen05.mma kind::i8 sums in 32 bits without rounding; products whose digits' places add up to
// the same power share an accumulator. Kept are the ten products of places 3 to 6 (2^24 to 2^48) in four accumulators, which hold at
// most K * 65,536 < 2^31 (K < 32,768). The four are put together in 64 bits, exactly, and rounded to float32 once.
//   digits of a: balanced, q = sum d_i 256^i, the bytes of q + 0x808080 with the lower three turned by 0x80;
//   digits of w: the bytes of q with the lower three turned by 0x80, one operation: q = 0x808080 + sum d_i 256^i. The constant's share of
//                the result, 0x808080 * sum_k q_a, is one number a row of a and comes with its digits.
//
// Error: of each operand at most half a step, 2^-32 of its row's largest magnitude, and the six products left out, some 2^-31 of the
// largest times sqrt(K); a row's largest magnitude is at most sqrt(K) times its root mean square. Then the one rounding of the result.
// Against float64 2.6e-8 of the result's size with normal numbers, 3.1e-8 where those of a are cubed in size (the activation of
// gate and up is of that kind); chains of multiply-adds with carried errors (gemm_simt.cu) 7.8e-8 in both. Sums of whole numbers do not
// depend on their order: a row's result is the same bits whatever else is in the batch, whatever the tile, and however K is cut.
//
// Rows that do not fit the form, with infinities, NaN or a largest magnitude below 2^-90, are marked. A weight that has one
// stays float32 on CUDA cores; the results of such a row of activations are NaN where it holds one, else summed by the thread that writes
// them with fused multiply-adds in ascending k. (No weight but zero becomes the whole number zero, so that an infinity times it is one.)
//
// The weights are written as digits once, when a model is loaded, in 4 bytes a number as before: tiles of 128 rows x 64 k, 32 KB each, lie
// in memory as they are to lie in shared memory (two planes of 64 bytes a row of the 128-byte swizzle), so a tile is two bulk copies
// of what memory gives fastest, one piece. (Made into digits on their way into shared memory by sixteen warps they came at 5.2 TB/s in the
// longest product and 1.3 to 3.8 in a layer's.) The activations are written as digits by a kernel of their own and come by TMA, plane
// behind plane (64-byte swizzle) with the highest first: the planes i + j >= 3 that a weight digit i meets are the first i + 1, its products
// with them lie in neighbouring accumulators, and one instruction forms them all: 4 for 32 k, not 10. Tiles have at most 64 tokens, so
// that two CTAs share a multiprocessor and one's products run while the other waits for its copies or writes its results: 2,048 rows by
// 16,384 outputs of 2,048 inputs 632 us, 3,800 multiply-adds a clock and multiprocessor (tiles of 128 tokens, one CTA: 781); 300 rows
// 140 us (as three or four tiles of more than 64: 162, 182). The rate of the unit bounds the product from about 64 tokens on.
// The reference computes the same products with a scalar loop (matmul_f32, src/kernels.cpp:33-57).
#include "digits.cuh"
#include "tc_common.cuh"

#include <cooperative_groups.h>

#include <atomic>

namespace {

constexpr int READERS = 8, WARP_COPY = READERS, WARP_MMA = READERS + 1;  // warps that read the accumulators; one thread each for copies, products
constexpr int DIGIT_THREADS = (READERS + 2) * 32;
constexpr int W_BYTES = 4 * BM * BK;  // of a tile of weights (BK = 64 k)
constexpr int LEVELS = 4;
constexpr int MAX_TOKENS = 64;     // of a tile: four accumulators of 64 columns, and two CTAs, are tensor memory's 512

// A block's largest of one number a thread (256 threads).
__device__ __forceinline__ uint32_t block_largest(uint32_t v, uint32_t* red) {
  v = __reduce_max_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i) v = max(v, red[i]);
  return v;
}

template <bool ALIGNED>
__device__ __forceinline__ float4 row_part(const float* row, int k, int K) {
  if (ALIGNED && k + 4 <= K) return *reinterpret_cast<const float4*>(row + k);
  return make_float4(k < K ? row[k] : 0.f, k + 1 < K ? row[k + 1] : 0.f, k + 2 < K ? row[k + 2] : 0.f, k + 3 < K ? row[k + 3] : 0.f);
}

// Weights, once when a model is loaded. Exponents: a block a row.
__global__ void __launch_bounds__(256) weight_exponents_kernel(const float* __restrict__ w, int K, long long ldw, int* __restrict__ exps) {
  __shared__ uint32_t red[8];
  dep_launch();
  dep_wait();
  const float* row = w + (size_t)blockIdx.x * ldw;
  uint32_t v = 0u;
  for (int k = threadIdx.x; k < K; k += 256) v = max(v, __float_as_uint(row[k]) & 0x7fffffffu);
  v = block_largest(v, red);
  if (threadIdx.x == 0) exps[blockIdx.x] = row_exponent(v);
}
// Where digit d of number kk (0..63) of row r lies in a tile.
__host__ __device__ __forceinline__ uint32_t tile_offset(int r, int kk, int d) {
  return (uint32_t)((d >> 1) * (BM * 128) + r * 128 + ((((d & 1) * 4 + (kk >> 4)) ^ (r & 7)) << 4) + (kk & 15));
}
// Digits: a block a tile, tiles[n / 128][k / 64]; rows and k that are not there are the digits of zero.
__global__ void __launch_bounds__(256) weight_digits_kernel(const float* __restrict__ w, int N, int K, long long ldw, const int* __restrict__ exps,
                                                            uint8_t* __restrict__ tiles, int k_blocks) {
  dep_launch();
  dep_wait();
  const int n0 = (int)(blockIdx.x / k_blocks) * BM, k0 = (int)(blockIdx.x % k_blocks) * BK;
  uint8_t* to = tiles + (size_t)blockIdx.x * W_BYTES;
  for (int i = threadIdx.x; i < BM * BK / 4; i += 256) {
    const int r = i / (BK / 4), kk = i % (BK / 4) * 4, n = n0 + r;
    const float scale = n < N ? row_scale_of(exps[n]) : 0.f;
    uint32_t q[4], d[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float x = n < N && k0 + kk + e < K ? w[(size_t)n * ldw + k0 + kk + e] : 0.f;
      q[e] = whole(x, scale);
      if (q[e] == 0u && x != 0.f) q[e] = x > 0.f ? 1u : 0xffffffffu;
      q[e] ^= 0x808080u;
    }
    sort_digits(q[0], q[1], q[2], q[3], d);
#pragma unroll
    for (int e = 0; e < 4; ++e) *reinterpret_cast<uint32_t*>(to + tile_offset(r, kk, e)) = d[e];
  }
}

// Activation rows as digits, a block a row; a row of up to 8,192 numbers is read once: digits[row][k / 64][digit][64], zeros behind K.
// sums[row]: its constant_share.
template <bool ALIGNED>
__global__ void __launch_bounds__(256) row_digits_kernel(const float* __restrict__ a, long long lda, int K, int k_blocks,
                                                         uint8_t* __restrict__ digits, int* __restrict__ exps, long long* __restrict__ sums) {
  __shared__ uint32_t red[8];
  __shared__ long long part_sums[8];
  constexpr int KEEP = 8;
  dep_launch();
  dep_wait();
  const float* row = a + (size_t)blockIdx.x * lda;
  float4 keep[KEEP];
  uint32_t v = 0u;
#pragma unroll
  for (int i = 0; i < KEEP; ++i) {
    keep[i] = row_part<ALIGNED>(row, (i * 256 + (int)threadIdx.x) * 4, K);
    v = max(v, magnitude4(keep[i]));
  }
  for (int k = (KEEP * 256 + (int)threadIdx.x) * 4; k < K; k += 1024) v = max(v, magnitude4(row_part<ALIGNED>(row, k, K)));
  v = block_largest(v, red);
  const int e = row_exponent(v);
  const float scale = row_scale_of(e);
  uint8_t* to = digits + (size_t)blockIdx.x * k_blocks * 256;
  long long sum = 0;
  auto put = [&](int part, float4 x) {
    uint32_t d[4];
    sum += balanced_digits(x, scale, d);
    put_digits(to, part, d);
  };
#pragma unroll
  for (int i = 0; i < KEEP; ++i)
    if (i * 256 + (int)threadIdx.x < k_blocks * 16) put(i * 256 + threadIdx.x, keep[i]);
  for (int part = KEEP * 256 + threadIdx.x; part < k_blocks * 16; part += 256) put(part, row_part<ALIGNED>(row, part * 4, K));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0) part_sums[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; ++i) sum += part_sums[i];
    exps[blockIdx.x] = e;
    sums[blockIdx.x] = constant_share(sum);
  }
}

struct DigitArgs {
  const float* a;
  long long lda;
  const uint8_t* w;  // tiles of digits
  const int *a_exp, *w_exp;
  const long long* a_sum;
  float* out;
  long long ldo;
  int M, N, K;
  int k_blocks, per_cut;  // of 64 k: in all, and of a CTA
  int bn, t_tiles;        // tokens of a tile, tiles of tokens
  int stages, tmem_cols;
  int* error_out;
};

// kind::i8: signed 8-bit x signed 8-bit -> 32-bit whole numbers, both operands K-major, M = 128, N = n
__device__ __forceinline__ uint32_t digit_instr_desc(int n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}
// K-major tile with 64-byte swizzle: rows 64 bytes apart, groups of 8 rows 512 bytes apart
__device__ __forceinline__ uint64_t smem_desc_sw64(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)4 << 61;
}
__device__ __forceinline__ void mma_i8(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_request8(uint32_t taddr, int (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
// sum = result in units of 2^(24 + ea - 31 + ew - 31); rounded once where the result is a normal number
__device__ __forceinline__ float digits_value(long long sum, int ea, int ew) {
  const int e = ea + ew - 38, half = e >> 1;  // (a factor of 2^e may lie outside of float32 where the result does not)
  return __ll2float_rn(sum) * power_of_two(half) * power_of_two(e - half);
}
// A weight from its digits.
__device__ __forceinline__ float weight_at(const uint8_t* w, int k_blocks, int n, int k, int e) {
  const uint8_t* tile = w + ((size_t)(n / BM) * k_blocks + k / BK) * W_BYTES;
  uint32_t q = 0u;
#pragma unroll
  for (int d = 0; d < 4; ++d) q |= (uint32_t)tile[tile_offset(n % BM, k % BK, d)] << (8 * d);
  return (float)(int)(q ^ 0x808080u) * power_of_two(e - 31);
}
// The result of a row that does not fit the form.
__device__ __noinline__ float row_product(const DigitArgs& p, int m, int n, int mark) {
  if (mark == NAN_ROW) return __uint_as_float(0x7fffffffu);
  const float* a = p.a + (size_t)m * p.lda;
  const int e = p.w_exp[n];
  float s = 0.f;
  for (int k = 0; k < p.K; ++k) s = fmaf(a[k], weight_at(p.w, p.k_blocks, n, k, e), s);
  return s;
}
__device__ __forceinline__ void put_result(const DigitArgs& p, int m, int n, long long sum) {
  if (m >= p.M || n >= p.N) return;
  const int ea = p.a_exp[m];
  p.out[(size_t)m * p.ldo + n] = ea >= EXACT_ROW ? row_product(p, m, n, ea) : digits_value(sum + p.a_sum[m], ea, p.w_exp[n]);
}

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes),
               "r"(smem_u32(bar))
               : "memory");
}

// grid: tiles x cuts, the cuts of a tile a cluster. The token tiles of a weight tile are neighbours: they read the same weights, once from
// memory.
__global__ void __launch_bounds__(DIGIT_THREADS, 2) gemm_digits_kernel(const __grid_constant__ CUtensorMap map_a, const DigitArgs p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int a_bytes = 4 * p.bn * BK, stage_bytes = W_BYTES + a_bytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)p.stages * stage_bytes);
  uint64_t* empty = full + p.stages;
  uint64_t* acc_ready = empty + p.stages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_ready + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int cuts = (int)cluster.num_blocks(), cut = (int)cluster.block_rank(), tile = (int)blockIdx.x / cuts;
  const int m0 = tile % p.t_tiles * p.bn, n_tile = tile / p.t_tiles, n0 = n_tile * BM;
  const int kb0 = cut * p.per_cut, n_iter = max(0, min(p.k_blocks, kb0 + p.per_cut) - kb0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_ready, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == WARP_MMA) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(p.tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  dep_launch();

  if (warp == WARP_COPY && lane == 0) {
    // ---------------------------------------------------------------- copies: weights, which the stream does not produce, ahead of the wait
    const uint8_t* from = p.w + ((size_t)n_tile * p.k_blocks + kb0) * W_BYTES;
    auto load_w = [&](int s, int it) {
      mbar_expect_tx(&full[s], (uint32_t)stage_bytes);
      bulk_load(smem + s * stage_bytes, from + (size_t)it * W_BYTES, W_BYTES / 2, &full[s]);
      bulk_load(smem + s * stage_bytes + W_BYTES / 2, from + (size_t)it * W_BYTES + W_BYTES / 2, W_BYTES / 2, &full[s]);
    };
    auto load_a = [&](int s, int it) {
#pragma unroll
      for (int d = 0; d < 4; ++d) tma_load_2d(smem + s * stage_bytes + W_BYTES + (3 - d) * p.bn * BK, &map_a, ((kb0 + it) * 4 + d) * (BK / 2), m0, &full[s]);
    };
    const int early = min(p.stages, n_iter);
    for (int it = 0; it < early; ++it) load_w(it, it);
    dep_wait();
    for (int it = 0; it < early; ++it) load_a(it, it);
    bool ok = true;
    int issued = early;
    RingPos ring(p.stages, 0, 1u);
    for (int it = early; it < n_iter; ++it, ring.next()) {
      ok = mbar_wait(&empty[ring.s], ring.ph ^ 1u, abort_flag, p.error_out, ERR_PRODUCER);
      if (!ok) break;
      load_w(ring.s, it);
      load_a(ring.s, it);
      issued = it + 1;
    }
    if (!ok || *abort_flag)  // copies on their way land before the CTA leaves
      for (int it = max(0, issued - p.stages); it < issued; ++it) mbar_drain(&full[it % p.stages], (uint32_t)(it / p.stages) & 1u, p.error_out);
  } else if (warp == WARP_MMA && lane == 0) {
    // ---------------------------------------------------------------- products
    // (what does not change is worked out before the loop: made anew, descriptors took the thread 200 clocks an instruction)
    const uint64_t desc_w = smem_desc_sw128(smem_u32(smem)), desc_a = smem_desc_sw64(smem_u32(smem) + W_BYTES);
    uint32_t idesc[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) idesc[i] = digit_instr_desc((i + 1) * p.bn);
    RingPos ring(p.stages);
    for (int it = 0; it < n_iter; ++it, ring.next()) {
      if (!mbar_wait(&full[ring.s], ring.ph, abort_flag, p.error_out, ERR_MMA)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t at = (uint32_t)(ring.s * stage_bytes) >> 4;  // in the descriptors' unit
#pragma unroll
      for (int half = 0; half < 2; ++half) {  // 32 k = 32 bytes = +2 in the address field; the second plane of two in a row: +4
#pragma unroll
        for (int i = 3; i >= 0; --i) {  // (digit 3 first: it meets all four planes, and so begins every accumulator)
          const uint64_t dw = desc_w + (at + (uint32_t)((i >> 1) * (BM * 128 / 16) + (i & 1) * 4 + half * 2)), da = desc_a + (at + (uint32_t)(half * 2));
          const uint32_t more = it > 0 || half > 0 || i < 3 ? 1u : 0u;
          mma_i8(tmem_base + (uint32_t)((3 - i) * p.bn), dw, da, idesc[i], more);
        }
      }
      mma_commit(&empty[ring.s]);
    }
    if (n_iter > 0) mma_commit(acc_ready);  // also when a wait gave up: arrives once every product issued above has finished
  }
  __syncwarp();
  dep_wait();

  // ------------------------------------------------------------------ the accumulators put together, and the cuts of K
  bool ready = n_iter > 0;
  if (ready) ready = mbar_wait(acc_ready, 0, abort_flag, p.error_out, ERR_EPILOGUE);
  ready = __all_sync(0xffffffffu, ready);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  long long* sums = reinterpret_cast<long long*>(smem);  // (cuts) [token][128 outputs], in the place of the operands
  if (cuts > 1) __syncthreads();                         // every warp's wait has come back: all products have read their operands
  const int tokens = min(p.bn, p.M - m0);
  if (warp < READERS) {
    const int r = (warp & 3) * 32 + lane;
    const uint32_t tmem = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll 1
    for (int c0 = (warp >> 2) * 8; c0 < tokens; c0 += 16) {
      int lev[LEVELS][8];
      if (ready) {
#pragma unroll
        for (int l = 0; l < LEVELS; ++l) tmem_request8(tmem + (uint32_t)(l * p.bn + c0), lev[l]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      } else {
#pragma unroll
        for (int l = 0; l < LEVELS; ++l)
#pragma unroll
          for (int i = 0; i < 8; ++i) lev[l][i] = 0;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        long long sum = lev[0][i];  // places 6, 5, 4, 3
#pragma unroll
        for (int l = 1; l < LEVELS; ++l) sum = sum * 256 + lev[l][i];
        if (cuts > 1) sums[(c0 + i) * BM + r] = sum;
        else put_result(p, m0 + c0 + i, n0 + r, sum);
      }
    }
  }
  if (cuts > 1) {
    cluster.sync();
    for (int e = cut * DIGIT_THREADS + (int)threadIdx.x; e < tokens * BM; e += cuts * DIGIT_THREADS) {
      long long piece[8], sum = 0;
#pragma unroll
      for (int c = 0; c < 8; ++c) piece[c] = c < cuts ? cluster.map_shared_rank(sums, c)[e] : 0;
#pragma unroll
      for (int c = 0; c < 8; ++c) sum += piece[c];
      put_result(p, m0 + e / BM, n0 + e % BM, sum);
    }
    cluster.sync();  // nobody leaves while its sums are being read
  }
  if (!ready && n_iter > 0 && threadIdx.x == 0) mbar_drain(acc_ready, 0, p.error_out);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == WARP_MMA) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(p.tmem_cols) : "memory");
  }
}

// ------------------------------------------------------------------------------------------------ few rows
// Up to eight rows: the same whole numbers straight from memory into mma.sync (m16n8k32, whose operands are registers), sixteen rows of
// weights by the activations as its eight columns. A CTA a multiprocessor stays and takes sixteen rows of weights at a time, all of K,
// the activations' digits in its shared memory. A warp has every sixteenth k-block; a lane has 16 k of two rows in every
// plane, FEW_DEPTH k-blocks on their way in registers. The order of k inside an instruction is the same for both operands, and else
// free: the four words of a lane's 16 bytes are two instructions' operands. 128,256 outputs of 2,048 inputs, 1 to 8 rows: 150 us, 7 TB/s
// (on tcgen05 175; the activations as the sixteen rows, twice the instructions: 175; four products at a time with dp4a: one row
// 145, two 207, four 378).
constexpr int FEW_WARPS = 16, FEW_M = 8, FEW_ROWS = 16, FEW_DEPTH = 2, FEW_SMEM = 180 * 1024;
struct FewArgs {
  DigitArgs d;
  const uint8_t* digits;
  int units, items;  // groups of sixteen weight rows; k-blocks of a warp
  int copied;        // whether the digits go to shared memory
};
__device__ __forceinline__ void mma_16x8x32(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__global__ void __launch_bounds__(FEW_WARPS * 32, 1) gemm_digits_few_kernel(const FewArgs p) {
  constexpr int OUTS = FEW_ROWS * FEW_M, THREADS = FEW_WARPS * 32;
  extern __shared__ __align__(16) uint8_t digits[];  // [row][k / 64][digit][64], rows 64 bytes further apart than they are long: other banks
  __shared__ long long s_part[2][FEW_WARPS][OUTS];
  __shared__ uint64_t arrived;
  __shared__ int aborted;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int kb_n = p.d.k_blocks, row_bytes = kb_n * 256 + 64;
  if (tid == 0) {
    mbar_init(&arrived, 1);
    aborted = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }

  int load_unit = blockIdx.x, load_item = 0;
  uint4 buf[FEW_DEPTH][2][4];  // by plane, of rows g and g + 8
  auto load = [&](uint4 (&v)[2][4]) {
    if (load_unit >= p.units) return;
    const int kb = warp + load_item * FEW_WARPS, row0 = load_unit * FEW_ROWS;
    const uint8_t* from = p.d.w + ((size_t)(row0 / BM) * kb_n + kb) * W_BYTES + (row0 % BM + g) * 128;
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int d = 0; d < 4; ++d)
        v[r][d] = kb < kb_n ? __ldcs(reinterpret_cast<const uint4*>(from + (d >> 1) * (BM * 128) + r * 1024 + ((((d & 1) * 4 + t) ^ g) << 4))) : make_uint4(0u, 0u, 0u, 0u);
    if (++load_item == p.items) {
      load_item = 0;
      load_unit += gridDim.x;
    }
  };
#pragma unroll
  for (int u = 0; u < FEW_DEPTH; ++u) load(buf[u]);  // weights are not produced by the stream
  dep_launch();
  __syncthreads();
  dep_wait();
  if (tid == 0 && p.copied) {
    mbar_expect_tx(&arrived, (uint32_t)(p.d.M * kb_n * 256));
    for (int m = 0; m < p.d.M; ++m) bulk_load(digits + m * row_bytes, p.digits + (size_t)m * kb_n * 256, (uint32_t)(kb_n * 256), &arrived);
  }
  const int my_m = tid / FEW_ROWS % FEW_M;  // the row whose results this thread may write
  const int my_exp = my_m < p.d.M ? p.d.a_exp[my_m] : 0;
  const long long my_sum = my_m < p.d.M ? p.d.a_sum[my_m] : 0;
  if (p.copied && !mbar_wait(&arrived, 0, &aborted, p.d.error_out, ERR_MMA)) mbar_drain(&arrived, 0, p.d.error_out);

  int acc[LEVELS][4];  // places 6, 5, 4, 3
#pragma unroll
  for (int l = 0; l < LEVELS; ++l)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[l][i] = 0;
  // (results of rows that are not there are not written; digits that do not fit are read where they are: 8 rows, 2,048 outputs of 8,192
  // inputs 16.3 us, on tcgen05 23.5)
  const uint8_t* row = (p.copied ? digits + min(g, p.d.M - 1) * row_bytes : p.digits + (size_t)min(g, p.d.M - 1) * kb_n * 256) + t * 16;
  int unit = blockIdx.x, item = 0, turn = 0;
  while (unit < p.units) {
#pragma unroll
    for (int u = 0; u < FEW_DEPTH; ++u) {
      if (unit >= p.units) break;
      const uint8_t* at = row + min(warp + item * FEW_WARPS, kb_n - 1) * 256;
#pragma unroll
      for (int j = 3; j >= 0; --j) {
        const uint4 x = *reinterpret_cast<const uint4*>(at + j * 64);
#pragma unroll
        for (int d = 3; d >= 3 - j; --d) {
          const uint4 v = buf[u][0][d], w = buf[u][1][d];
          mma_16x8x32(acc[6 - d - j], v.x, w.x, v.y, w.y, x.x, x.y);
          mma_16x8x32(acc[6 - d - j], v.z, w.z, v.w, w.w, x.z, x.w);
        }
      }
      load(buf[u]);
      if (++item == p.items) {
        // a lane's results: activations 2 t and 2 t + 1, weight rows g and g + 8
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          long long mine = acc[0][i];
#pragma unroll
          for (int l = 1; l < LEVELS; ++l) mine = mine * 256 + acc[l][i];
          s_part[turn][warp][(2 * t + (i & 1)) * FEW_ROWS + g + 8 * (i >> 1)] = mine;
        }
#pragma unroll
        for (int l = 0; l < LEVELS; ++l)
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[l][i] = 0;
        __syncthreads();
        const int n = unit * FEW_ROWS + tid % FEW_ROWS;
        if (tid / OUTS == unit % (THREADS / OUTS) && my_m < p.d.M && n < p.d.N) {  // four warps finish the results, others next time
          long long sum = my_sum;
#pragma unroll
          for (int i = 0; i < FEW_WARPS; ++i) sum += s_part[turn][i][tid % OUTS];
          p.d.out[(size_t)my_m * p.d.ldo + n] = my_exp >= EXACT_ROW ? row_product(p.d, my_m, n, my_exp) : digits_value(sum, my_exp, p.d.w_exp[n]);
        }
        turn ^= 1;  // (the other half: those warps may still be reading this one, and come to the next barrier when they have)
        item = 0;
        unit += gridDim.x;
      }
    }
  }
}

constexpr int SMS = 148;  // of a B200

// Tokens of a tile and pieces that K is cut into (a cluster), by the clocks that the last CTA is done after: rounds of two CTAs a
// multiprocessor, or of one where they do not suffice. A k-block takes the longer of its weights' way from memory, 1,400 at the rate that
// all have together, and its products, twenty of a clock a token; the two-stage ring of a CTA alone leaves some 600 in which nothing
// runs. A CTA's beginning and end are some 4,000, the exchange of a cluster's sums 1,500. Of more than 64 tokens tiles of 48 are tried as
// well, which fill the last round better (us with 64, with 48: 160 x 16,384 x 2,048 94, 84; 1,024 x 3,072 x 2,048 94, 79; 300 x 2,048 x 8,192
// 85, 76; but 2,048 x 16,384 x 2,048 632, 731).
void choose_tiles(int M, int n_tiles, int k_blocks, int only_cuts, int* bn, int* t_tiles, int* cuts) {
  long long best = 1LL << 62;
  const int splits[2] = {(M + MAX_TOKENS - 1) / MAX_TOKENS, M > MAX_TOKENS ? (M + 47) / 48 : 1};
  for (int t : splits) {
    const int tokens = ((M + t - 1) / t + 15) / 16 * 16;
    const long long tiles = (long long)n_tiles * t;
    for (int c = 1; c <= 8; c *= 2) {
      if (only_cuts ? c != only_cuts : c > 1 && (tiles * c > 2 * SMS || 2 * c > k_blocks)) continue;
      const long long per = (k_blocks + c - 1) / c, ctas = tiles * c, ends = c > 1 ? 5500 : 4000;
      const long long clocks = ctas <= SMS ? per * (std::max(1400, 20 * tokens) + (tokens > 16 ? 600 : 0)) + ends
                                           : (ctas + 2 * SMS - 1) / (2 * SMS) * 2 * (per * std::max(t == 1 ? 1400 : 0, 20 * tokens) + ends);
      if (clocks < best) best = clocks, *bn = tokens, *t_tiles = t, *cuts = c;
    }
  }
}

// Boxes of a plane of a k-block of box_rows rows, 64 bytes each. Made at each call (host work of well under a microsecond): workspaces
// hand out the same address for matrices of other sizes.
bool digits_map(const void* digits, int M, int k_blocks, int box_rows, CUtensorMap* out) {
  const cuuint64_t dims[2] = {(cuuint64_t)k_blocks * 128, (cuuint64_t)M}, strides[1] = {(cuuint64_t)k_blocks * 256};
  const cuuint32_t box[2] = {BK / 2, (cuuint32_t)box_rows}, step[2] = {1, 1};
  return encode_fn()(out, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(digits), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool rows_on_16_bytes(const void* p, long long ld) { return reinterpret_cast<uintptr_t>(p) % 16 == 0 && ld % 4 == 0; }

}  // namespace

// Whether a weight matrix of these sizes may be taken as digits: sums that fit.
extern "C" int llm_weight_digits_supported(int N, int K) { return N > 0 && K > 0 && K < 32768 && encode_fn() != nullptr; }

// A weight as digits: exps int32 [N], tiles uint8 [ceil(N / 128)][ceil(K / 64)][32768], 16-byte aligned. A row that does not fit the form
// has an exponent of 0x7ffffffe or more: the caller looks for one and keeps the weight as it is.
extern "C" int llm_weight_digits(const float* w, int N, int K, long long ldw, void* tiles, int* exps, cudaStream_t stream) {
  LLM_REQUIRE(llm_weight_digits_supported(N, K) && ldw >= K && reinterpret_cast<uintptr_t>(tiles) % 16 == 0, "weight_digits: sizes not taken: N=%d K=%d", N, K);
  const int k_blocks = (K + BK - 1) / BK;
  launch_kernel(weight_exponents_kernel, N, 256, 0, stream, w, K, ldw, exps);
  launch_kernel(weight_digits_kernel, (unsigned)((N + BM - 1) / BM) * k_blocks, 256, 0, stream, w, N, K, ldw, (const int*)exps, (uint8_t*)tiles, k_blocks);
  LLM_CHECK_LAUNCH("weight_digits");
  return LLM_OK;
}

// digits: uint8 [M][ceil(K / 64)][4][64], 16-byte aligned; exps: int32 [M]; sums: int64 [M]
extern "C" int llm_row_digits(const float* a, int M, int K, long long lda, void* digits, int* exps, long long* sums, cudaStream_t stream) {
  if (M == 0) return LLM_OK;
  LLM_REQUIRE(M > 0 && K > 0 && K < 32768 && lda >= K, "row_digits: bad sizes M=%d K=%d", M, K);
  const int k_blocks = (K + BK - 1) / BK;
  auto kernel = rows_on_16_bytes(a, lda) ? row_digits_kernel<true> : row_digits_kernel<false>;
  launch_kernel(kernel, M, 256, 0, stream, a, lda, K, k_blocks, (uint8_t*)digits, exps, sums);
  LLM_CHECK_LAUNCH("row_digits");
  return LLM_OK;
}

// out [M, N] float32 = a . w^T, a as digits (llm_row_digits) and as it is (for rows that do not fit the form), w as llm_weight_digits wrote
// it. cuts: pieces of K, 1, 2, 4 or 8 (the results are the same bits), or 0: as many as the sizes want.
extern "C" int llm_gemm_digits(const void* digits, const int* a_exp, const long long* a_sum, const float* a, const void* w_tiles, const int* w_exp,
                               float* out, int M, int N, int K, long long lda, long long ldo, int cuts, cudaStream_t stream) {
  if (M == 0 || N == 0) return LLM_OK;
  LLM_REQUIRE(M > 0 && llm_weight_digits_supported(N, K), "gemm_digits: sizes not taken: M=%d N=%d K=%d", M, N, K);
  LLM_REQUIRE(lda >= K && ldo >= N && (reinterpret_cast<uintptr_t>(digits) | reinterpret_cast<uintptr_t>(w_tiles)) % 16 == 0, "gemm_digits: row strides or alignment");
  LLM_REQUIRE(cuts == 0 || cuts == 1 || cuts == 2 || cuts == 4 || cuts == 8, "gemm_digits: %d cuts", cuts);
  LLM_REQUIRE(error_word() != nullptr, "gemm_digits: cannot allocate the error word");
  DigitArgs p{a, lda, (const uint8_t*)w_tiles, a_exp, w_exp, a_sum, out, ldo, M, N, K, (K + BK - 1) / BK};
  const int n_tiles = (N + BM - 1) / BM;
  choose_tiles(M, n_tiles, p.k_blocks, cuts, &p.bn, &p.t_tiles, &cuts);
  LLM_REQUIRE((long long)n_tiles * p.t_tiles * 8 < (1LL << 31), "gemm_digits: M=%d N=%d too large", M, N);
  p.per_cut = (p.k_blocks + cuts - 1) / cuts;
  p.stages = p.bn <= 16 ? 3 : 2;  // two CTAs a multiprocessor
  p.tmem_cols = p.bn <= 16 ? 64 : p.bn <= 32 ? 128 : 256;
  p.error_out = error_word();
  CUtensorMap ma;
  LLM_REQUIRE(digits_map(digits, M, p.k_blocks, p.bn, &ma), "gemm_digits: cuTensorMapEncodeTiled failed");
  static std::atomic<unsigned long long> done{0};  // more than 48 KB of shared memory has to be asked for, once a device
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && !(dev < 64 && (done.load(std::memory_order_relaxed) >> dev & 1ull))) {
    LLM_REQUIRE(cudaFuncSetAttribute(gemm_digits_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) == cudaSuccess,
                "gemm_digits: cannot reserve shared memory");
    if (dev < 64) done.fetch_or(1ull << dev);
  }
  const size_t smem = 1024 + (size_t)p.stages * (W_BYTES + 4 * (size_t)p.bn * BK) + (2 * p.stages + 1) * 8 + 16;
  launch_kernel_cluster(gemm_digits_kernel, dim3((unsigned)(n_tiles * p.t_tiles * cuts)), DIGIT_THREADS, smem, dim3((unsigned)cuts), stream, ma, p);
  LLM_CHECK_LAUNCH("gemm_digits");
  return LLM_OK;
}

// The same for up to eight rows: the same bits as llm_gemm_digits.
extern "C" int llm_gemm_digits_few(const void* digits, const int* a_exp, const long long* a_sum, const float* a, const void* w_tiles, const int* w_exp,
                                   float* out, int M, int N, int K, long long lda, long long ldo, cudaStream_t stream) {
  if (M == 0 || N == 0) return LLM_OK;
  LLM_REQUIRE(llm_weight_digits_supported(N, K) && M > 0 && M <= FEW_M, "gemm_digits_few: sizes not taken: M=%d N=%d K=%d", M, N, K);
  LLM_REQUIRE(lda >= K && ldo >= N && (reinterpret_cast<uintptr_t>(digits) | reinterpret_cast<uintptr_t>(w_tiles)) % 16 == 0, "gemm_digits_few: row strides or alignment");
  LLM_REQUIRE(error_word() != nullptr, "gemm_digits_few: cannot allocate the error word");
  FewArgs p{};
  p.d = DigitArgs{a, lda, (const uint8_t*)w_tiles, a_exp, w_exp, a_sum, out, ldo, M, N, K, (K + BK - 1) / BK};
  p.d.error_out = error_word();
  p.digits = (const uint8_t*)digits;
  p.units = (N + FEW_ROWS - 1) / FEW_ROWS;
  p.items = (p.d.k_blocks + FEW_WARPS - 1) / FEW_WARPS;
  static std::atomic<unsigned long long> done{0};
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && !(dev < 64 && (done.load(std::memory_order_relaxed) >> dev & 1ull))) {
    // Loads on their way to registers are held in L1, so no more of it than this may become shared memory: behind a kernel that wants all
    // of it (float32 decoding attention) the multiprocessors would be left as they are, and 16,384 outputs of 2,048 inputs take 31 us, not 21.
    LLM_REQUIRE(cudaFuncSetAttribute(gemm_digits_few_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FEW_SMEM) == cudaSuccess &&
                    cudaFuncSetAttribute(gemm_digits_few_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 45) == cudaSuccess,
                "gemm_digits_few: cannot reserve shared memory");
    if (dev < 64) done.fetch_or(1ull << dev);
  }
  const long long bytes = (long long)M * (p.d.k_blocks * 256 + 64);
  p.copied = bytes <= FEW_SMEM;
  launch_kernel(gemm_digits_few_kernel, std::min(p.units, SMS), FEW_WARPS * 32, p.copied ? (size_t)bytes : 0, stream, p);
  LLM_CHECK_LAUNCH("gemm_digits_few");
  return LLM_OK;
}
