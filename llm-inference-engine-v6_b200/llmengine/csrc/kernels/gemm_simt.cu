// out[m,n] = sum_k a[m,k] * w[n,k]   (W row-major [N,K], as checkpoints store linear layers)
//
// CUDA-core matrix product with float32 multiply-adds: the true 32-bit path of the engine, and the
// path that takes every shape (any M, N, K and row strides) in bfloat16 when the tensor-core
// kernel refuses one. The dot itself is the reference's matmul_f32 (src/kernels.cpp:33-57); no bias
// (src/engine.cpp:319-341).
//
// Order of the sums, a function of K alone, the same in both kernels below, so that a row's result does not depend on
// what else is in the batch or on which kernel ran:
//   * 16 neighbouring k are a chain of fused multiply-adds from zero, ascending ("block");
//   * K is cut in two halves at half_of(K), a multiple of 64; in each half the blocks whose index is g modulo 4 are
//     added in ascending order ("stream" g = 0..3), the rounding error of every addition carried along (two-sum);
//   * the streams of a half are added in order 0..3, then the second half to the first, sums and carried errors apart, by
//     two-sum again; result = sum + carried errors, rounded once.
// Long inner sizes therefore cost no accuracy: what is left is the rounding inside chains of 16. (Sums in float64 would be
// six additions fewer a block, but the conversion of a float32 runs at a few a clock and multiprocessor.)
//
// w is a weight: its first chunks are fetched before the dependency wait, so no kernel launched ahead on the stream that releases
// its dependents early (all of this library's do) may be writing it. a is read behind the wait. (Fetching w behind it too: a float32
// decode step of 8 requests at the Llama 3.2 1B sizes 2.44 ms instead of 2.36, a tiny model's 130 us instead of 125.)
#include "simt_common.cuh"

#include <cooperative_groups.h>

#include <type_traits>

namespace {

__host__ __device__ __forceinline__ int half_of(int K) { return ((K + 1) / 2 + 63) & ~63; }

// sum += b with what the addition rounds away added to lost; of two numbers at once (the packed additions are a result each
// of the same rounding, and half the instructions)
__device__ __forceinline__ void two_sum(float& sum, float& lost, float b) {
  const float a = sum, s = a + b, bv = s - a;
  lost += (a - (s - bv)) + (b - bv);
  sum = s;
}
// (sum, lost) += (b.x, b.y), a sum and its carried errors
__device__ __forceinline__ void add_pair(float2& a, float2 b) {
  two_sum(a.x, a.y, b.x);
  a.y += b.y;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 r;
  asm("{.reg .b64 a, b, r; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; add.rn.f32x2 r, a, b; mov.b64 {%0, %1}, r;}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {  // as b * -1 + a: there is no packed subtraction
  float2 r;
  asm("{.reg .b64 a, b, m, r; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; mov.b64 m, {%6, %6}; fma.rn.f32x2 r, b, m, a; mov.b64 {%0, %1}, r;}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(-1.0f));
  return r;
}
__device__ __forceinline__ void two_sum2(float2& sum, float2& lost, float2 b) {
  const float2 a = sum, s = add2(a, b), bv = sub2(s, a);
  lost = add2(lost, add2(sub2(a, sub2(s, bv)), sub2(b, bv)));
  sum = s;
}
// ------------------------------------------------------------------------------------------------ many rows
// A tile of 64 x 32 results a CTA, four groups of 64 threads: group g owns stream g (16 of every 64 k), a thread 8 x 4
// results of it, so that two CTAs of eight warps fit a multiprocessor (64 x 64 and one CTA: 25 against 27 TFLOP/s at 2,048
// rows). The two halves of K are the two CTAs of a cluster, which halves the unit of work: at 300 rows a product with 2,048
// outputs has 320 tiles for 296 places. Bound by instruction issue: multiply-adds are half of it, the packed two-sums, the
// moves around them and the reads of shared memory the rest. Rows in shared memory are 64 + 4 numbers long: 8 rows read 16
// bytes each from different banks. 300 rows, 16,384 outputs of 2,048 inputs: 787 us (25.6 TFLOP/s), 1,480 us as one tile of
// 64 x 64 with scalar loads; 2,048 rows: 27.7 TFLOP/s. Rows that do not begin on four numbers, and bfloat16 ones, go through registers:
// of odd length 700 rows, 2,048 outputs of 2,049 inputs in bfloat16 take 344 us (17 TFLOP/s; the 64 x 64 tile, which loads two thirds
// as much for a multiply-add, 315), of a multiple of 4 by 8 bytes 300 rows, 8,192 of 2,052 inputs 466 us (21.6 TFLOP/s).
constexpr int BM = 64, BN = 32, BK = 64, ROW = BK + 4, TILE_STAGES = 4, TJ = BN / 8;
constexpr int Q_ROW = BN + 4;  // a row of the tile's sums
constexpr int TILE_SMEM = TILE_STAGES * (BM + BN) * ROW * 4;
static_assert(TILE_SMEM >= BM * Q_ROW * 8, "the sums take the place of the operands");

template <typename T, typename TO, bool ALIGNED>
__global__ void __launch_bounds__(256, 2)
    gemm_simt_tile_kernel(const T* __restrict__ a, const T* __restrict__ w, TO* __restrict__ out, int M, int N, int K, int m_tiles,
                          long long lda, long long ldw, long long ldo) {
  extern __shared__ __align__(16) float smem[];
  dep_launch();
  const int tid = threadIdx.x, g = tid >> 6, tn = tid & 7, tm = (tid >> 3) & 7;
  const int half = blockIdx.x & 1, tile = blockIdx.x >> 1;
  // row tiles of one column of tiles are neighbours: they read the same weight rows, once from memory
  const int m0 = (tile % m_tiles) * BM, n0 = (tile / m_tiles) * BN;
  const int kh = half_of(K), k_begin = half ? kh : 0, k_end = half ? K : min(kh, K);
  const int n_iter = k_end > k_begin ? (k_end - k_begin + BK - 1) / BK : 0;

  // a thread copies 4 k of rows lr, lr + RS, ...: side by side, or (rows without alignment) 32 apart, so that a warp's loads of single
  // numbers are side by side
  constexpr int RS = ALIGNED ? 16 : 8, ROWS_A = BM / RS, ROWS_W = BN / RS;
  const int lr = ALIGNED ? tid >> 4 : tid >> 5, lk = ALIGNED ? (tid & 15) * 4 : tid & 31;
  const T* wp = w + (size_t)min(n0 + lr, N - 1) * ldw;
  const T* ap = a + (size_t)min(m0 + lr, M - 1) * lda;
  // COUNT rows from FIRST on of the ROWS_A rows of a and then the ROWS_W of w that a thread copies (a row beyond the matrix, or a k
  // beyond the half, reads nothing; its address is that of the thread's first row)
  auto load = [&](int it, auto first_of, auto count_of) {
    constexpr int FIRST = decltype(first_of)::value, COUNT = decltype(count_of)::value;
    float* dst = smem + (it % TILE_STAGES) * (BM + BN) * ROW + lr * ROW + lk;
    const int k = k_begin + it * BK + lk, count = ALIGNED ? count4(k, k_end) : max(0, min(2, (k_end - k + 31) / 32)), at = count ? k : 0;
    auto inside = [&](int i) { return i < ROWS_A ? m0 + lr + RS * i < M : n0 + lr + RS * (i - ROWS_A) < N; };
    stage_rows<ALIGNED, COUNT, 2, 32, T>([&](int i) { return dst + (FIRST + i) * RS * ROW; },
                                         [&](int i) {
                                           i += FIRST;
                                           return i < ROWS_A ? ap + (inside(i) ? at + i * RS * lda : 0) : wp + (inside(i) ? at + (i - ROWS_A) * RS * ldw : 0);
                                         },
                                         [&](int i) { return inside(FIRST + i) ? count : 0; });
  };
  using std::integral_constant;
  auto load_w = [&](int it) { load(it, integral_constant<int, ROWS_A>{}, integral_constant<int, ROWS_W>{}); };
  auto load_a = [&](int it) { load(it, integral_constant<int, 0>{}, integral_constant<int, ROWS_A>{}); };
  const int early = min(TILE_STAGES - 1, n_iter);
  for (int it = 0; it < early; ++it) load_w(it);  // weights are not produced by the stream
  dep_wait();
  for (int it = 0; it < TILE_STAGES - 1; ++it) {
    if (it < early) load_a(it);
    commit_group();  // (the first group holds all early weights too)
  }

  float2 acc[8][TJ / 2], lost[8][TJ / 2];  // the running sums and what their additions rounded away
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < TJ / 2; ++j) acc[i][j] = lost[i][j] = make_float2(0.f, 0.f);

  for (int it = 0; it < n_iter; ++it) {
    wait_groups<TILE_STAGES - 2>();
    __syncthreads();
    if (it + TILE_STAGES - 1 < n_iter) {
      load(it + TILE_STAGES - 1, integral_constant<int, 0>{}, integral_constant<int, ROWS_A + ROWS_W>{});
    }
    commit_group();
    const float* as = smem + (it % TILE_STAGES) * (BM + BN) * ROW + tm * ROW + g * 16;
    const float* ws = smem + (it % TILE_STAGES) * (BM + BN) * ROW + (BM + tn) * ROW + g * 16;
    float blk[8][TJ];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < TJ; ++j) blk[i][j] = 0.f;
#pragma unroll
    for (int kk = 0; kk < 16; kk += 4) {
      float4 wv[TJ];
#pragma unroll
      for (int j = 0; j < TJ; ++j) wv[j] = *reinterpret_cast<const float4*>(ws + j * 8 * ROW + kk);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 av = *reinterpret_cast<const float4*>(as + i * 8 * ROW + kk);
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int j = 0; j < TJ; ++j) blk[i][j] = fmaf(part(av, e), part(wv[j], e), blk[i][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < TJ / 2; ++j) two_sum2(acc[i][j], lost[i][j], make_float2(blk[i][2 * j], blk[i][2 * j + 1]));
  }
  wait_groups<0>();
  float2* q = reinterpret_cast<float2*>(smem);
#pragma unroll
  for (int s = 0; s < 4; ++s) {  // stream 0, then 1, 2 and 3 added to it
    __syncthreads();
    if (g == s) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TJ; ++j) {
          float2* at = q + (tm + 8 * i) * Q_ROW + tn + 8 * j;
          const float2 mine = j & 1 ? make_float2(acc[i][j / 2].y, lost[i][j / 2].y) : make_float2(acc[i][j / 2].x, lost[i][j / 2].x);
          float2 sum = mine;
          if (s > 0) {
            sum = *at;
            add_pair(sum, mine);
          }
          *at = sum;
        }
    }
  }
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  cluster.sync();
  const float2* other = cluster.map_shared_rank(q, half ^ 1);
#pragma unroll
  for (int i = 0; i < BM / 2 * BN / 256; ++i) {  // CTA `half` of the two finishes 32 of the 64 rows
    const int r = half * (BM / 2) + i * (256 / BN) + tid / BN, c = tid % BN;
    const float2 mine = q[r * Q_ROW + c], his = other[r * Q_ROW + c];
    float2 sum = half == 0 ? mine : his;
    add_pair(sum, half == 0 ? his : mine);
    if (m0 + r < M && n0 + c < N) out[(size_t)(m0 + r) * ldo + n0 + c] = from_f32<TO>(sum.x + sum.y);
  }
  cluster.sync();  // nobody leaves while its sums are being read
}

// ------------------------------------------------------------------------------------------------ few rows
// Up to 16 rows: the product streams the weights, so it is bound by memory (one row: 5.8 TB/s of 6.5 with 128,256 outputs), with
// more rows by instruction issue (8 rows: 3.1 TB/s). A CTA a multiprocessor stays and walks over tiles of 16 outputs with all
// of K; operands come in chunks of 512 k by cp.async, chunks of the next tile behind those of this one, so that 32 to 96 KB
// of weights a multiprocessor are on their way at any time. A thread has TN outputs x TM rows of one block; the blocks' sums
// go through shared memory to the threads that own a (stream, result), which add them while the next chunk's blocks are
// formed. 8 rows, 16,384 outputs of 2,048 inputs: 45 us; 730 us in tiles of 64 rows, as larger steps run.
// A row of a chunk takes 512 + 4 numbers in shared memory: the 8 threads of a 16-byte read are 4 neighbouring outputs and 2
// neighbouring blocks, all in different banks.
constexpr int NT = 16, KC = 512, BLOCKS = KC / 16, ROW_C = KC + 4;
template <int MT, int TN, int TM>
constexpr int few_threads() { return BLOCKS * (NT / TN) * (MT / TM); }

template <int MT>
constexpr int few_stages() { return MT <= 4 ? 4 : MT <= 8 ? 3 : 2; }
template <int MT>
constexpr int few_smem() { return (few_stages<MT>() * (NT + MT) * ROW_C + 2 * BLOCKS * (NT * MT + 4)) * 4; }

template <typename T, typename TO, int MT, int TN, int TM, bool ALIGNED>
__global__ void __launch_bounds__(few_threads<MT, TN, TM>(), 1)
    gemm_simt_few_kernel(const T* __restrict__ a, const T* __restrict__ w, TO* __restrict__ out, int M, int N, int K,
                         long long lda, long long ldw, long long ldo) {
  constexpr int FEW_THREADS = few_threads<MT, TN, TM>();
  constexpr int STAGES = few_stages<MT>(), STAGE = (NT + MT) * ROW_C, OUTS = NT * MT, SUMS = OUTS + 4;
  constexpr int OWN = (4 * OUTS + FEW_THREADS - 1) / FEW_THREADS;  // (stream, result) pairs a thread owns
  extern __shared__ __align__(16) float smem[];
  float* const sums = smem + STAGES * STAGE;  // [chunk & 1][block][output][row]
  dep_launch();
  const int tid = threadIdx.x, ng = tid % (NT / TN), blk = tid / (NT / TN) % BLOCKS, mg = tid / (NT / TN) / BLOCKS;
  // (a thread's outputs are ng, ng + NT / TN, ...: neighbouring threads read neighbouring rows)
  const int n_tiles = (N + NT - 1) / NT, chunks = (K + KC - 1) / KC, kh = half_of(K);
  const int mine = (int)blockIdx.x < n_tiles ? (n_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const long long n_iter = (long long)mine * chunks;
  // a thread's four numbers of a row's chunk, side by side or (several rows without alignment) KC / 4 apart, and its first row
  constexpr bool BESIDE = ALIGNED || MT == 1;
  constexpr int GAP = BESIDE ? 1 : KC / 4;
  const int lk = BESIDE ? tid % (KC / 4) * 4 : tid % (KC / 4), lr = tid / (KC / 4);
  constexpr int LOAD_ROWS = FEW_THREADS / (KC / 4);
  const int at = lr * ROW_C + lk;
  constexpr int ROWS_X = MT / LOAD_ROWS, ROWS_W = NT / LOAD_ROWS;
  static_assert(MT % LOAD_ROWS == 0 && NT % LOAD_ROWS == 0, "whole rows a thread");
  const T* ap[ROWS_X];
#pragma unroll
  for (int i = 0; i < ROWS_X; ++i) ap[i] = a + (size_t)min(i * LOAD_ROWS + lr, M - 1) * lda;
  int load_tile = blockIdx.x, load_chunk = 0, load_stage = 0;  // of the next chunk to be requested
  // COUNT of the ROWS_W rows of w and then the ROWS_X of a that a thread copies, from row FIRST of them on
  auto load = [&](int tile, int chunk, int stage, auto first_of, auto count_of) {
    constexpr int FIRST = decltype(first_of)::value, COUNT = decltype(count_of)::value;
    const T* wp = w + (size_t)min(tile * NT + lr, N - 1) * ldw;
    float* dst = smem + stage * STAGE + at;
    const int k = chunk * KC + lk, count = max(0, min(4, (K - k + GAP - 1) / GAP)), from = count ? k : 0;
    auto inside = [&](int i) { return i < ROWS_W ? tile * NT + i * LOAD_ROWS + lr < N : (i - ROWS_W) * LOAD_ROWS + lr < M; };
    stage_rows<ALIGNED, COUNT, 4, GAP, T>([&](int i) { return dst + (FIRST + i) * LOAD_ROWS * ROW_C; },
                                             [&](int i) {
                                               i += FIRST;
                                               return i < ROWS_W ? wp + (inside(i) ? from + i * LOAD_ROWS * ldw : 0) : ap[i < ROWS_W ? 0 : i - ROWS_W] + from;
                                             },
                                             [&](int i) { return inside(FIRST + i) ? count : 0; });
  };
  using std::integral_constant;
  auto load_w = [&](int tile, int chunk, int stage) { load(tile, chunk, stage, integral_constant<int, 0>{}, integral_constant<int, ROWS_W>{}); };
  auto load_x = [&](int chunk, int stage) { load(0, chunk, stage, integral_constant<int, ROWS_W>{}, integral_constant<int, ROWS_X>{}); };
  auto step_load = [&]() {
    if (++load_chunk == chunks) {
      load_chunk = 0;
      load_tile += gridDim.x;
    }
    if (++load_stage == STAGES) load_stage = 0;
  };
  const int early = (int)(n_iter < STAGES - 1 ? n_iter : STAGES - 1);
  for (int it = 0; it < early; ++it) {  // weights are not produced by the stream
    load_w(load_tile, load_chunk, load_stage);
    step_load();
  }
  dep_wait();
  for (int it = 0, chunk = 0; it < STAGES - 1; ++it) {
    if (it < early) load_x(chunk, it);
    commit_group();  // (the first group holds all early weights too)
    if (++chunk == chunks) chunk = 0;
  }

  float2 st[OWN], h0[OWN];  // streams of the half that is being added: sum and carried errors; of the first half
#pragma unroll
  for (int o = 0; o < OWN; ++o) st[o] = h0[o] = make_float2(0.f, 0.f);
  int tile = blockIdx.x, chunk = 0, stage = 0;  // chunk and tile: of the sums that are being added
  for (long long it = 0; it <= n_iter; ++it) {
    wait_groups<STAGES - 2>();
    __syncthreads();
    float acc[TN][TM];
    if (it < n_iter) {
      if (it + STAGES - 1 < n_iter) {  // into the stage that the iteration before this one has read
        load(load_tile, load_chunk, load_stage, integral_constant<int, 0>{}, integral_constant<int, ROWS_W + ROWS_X>{});
        step_load();
      }
      commit_group();
      const float* ws = smem + stage * STAGE + ng * ROW_C + blk * 16;
      const float* xs = smem + stage * STAGE + (NT + mg * TM) * ROW_C + blk * 16;
#pragma unroll
      for (int j = 0; j < TN; ++j)
#pragma unroll
        for (int m = 0; m < TM; ++m) acc[j][m] = 0.f;
#pragma unroll
      for (int kk = 0; kk < 16; kk += 4) {
        float4 wv[TN];
#pragma unroll
        for (int j = 0; j < TN; ++j) wv[j] = *reinterpret_cast<const float4*>(ws + j * (NT / TN) * ROW_C + kk);
#pragma unroll
        for (int m = 0; m < TM; ++m) {
          const float4 xv = *reinterpret_cast<const float4*>(xs + m * ROW_C + kk);
#pragma unroll
          for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[j][m] = fmaf(part(xv, e), part(wv[j], e), acc[j][m]);
        }
      }
      float* to = sums + (it & 1) * BLOCKS * SUMS + blk * SUMS + ng * MT + mg * TM;
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        float* row = to + j * (NT / TN) * MT;
        if constexpr (TM % 4 == 0) {
#pragma unroll
          for (int m = 0; m < TM; m += 4) *reinterpret_cast<float4*>(row + m) = make_float4(acc[j][m], acc[j][m + 1], acc[j][m + 2], acc[j][m + 3]);
        } else {
#pragma unroll
          for (int m = 0; m < TM; ++m) row[m] = acc[j][m];
        }
      }
      if (++stage == STAGES) stage = 0;
    }
    if (it == 0) continue;
    // the sums of the chunk before, of (chunk, tile)
    float* from = sums + ((it - 1) & 1) * BLOCKS * SUMS;
    const int k0 = chunk * KC;
#pragma unroll
    for (int o = 0; o < OWN; ++o) {
      const int id = o * FEW_THREADS + tid, g = id / OUTS;
      if (4 * OUTS % FEW_THREADS != 0 && id >= 4 * OUTS) continue;
      const float* s = from + g * SUMS + id % OUTS;
      if (k0 <= kh && kh < k0 + KC) {  // the second half begins in this chunk
        const int first = (kh - k0) / 16;
#pragma unroll 1
        for (int b = 0; b < BLOCKS; b += 4) {
          if (b == first) {
            h0[o] = st[o];
            st[o] = make_float2(0.f, 0.f);
          }
          two_sum(st[o].x, st[o].y, s[b * SUMS]);
        }
      } else {
#pragma unroll
        for (int b = 0; b < BLOCKS; b += 4) two_sum(st[o].x, st[o].y, s[b * SUMS]);  // (blocks beyond K are zero)
      }
    }
    if (chunk == chunks - 1) {
      __syncthreads();  // the sums have been read: their place takes the streams [half][stream][result]
      float2* fin = reinterpret_cast<float2*>(from);
      const bool two = chunks * KC > kh;  // whether the second half has begun
#pragma unroll
      for (int o = 0; o < OWN; ++o) {
        const int id = o * FEW_THREADS + tid;
        if (4 * OUTS % FEW_THREADS != 0 && id >= 4 * OUTS) continue;
        fin[id] = two ? h0[o] : st[o];
        fin[4 * OUTS + id] = two ? st[o] : make_float2(0.f, 0.f);
        st[o] = make_float2(0.f, 0.f);
      }
      __syncthreads();
#pragma unroll
      for (int id = tid; id < OUTS; id += FEW_THREADS) {
        const int n = tile * NT + id / MT, m = id % MT;
        float2 half[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          half[h] = fin[h * 4 * OUTS + id];
#pragma unroll
          for (int g = 1; g < 4; ++g) add_pair(half[h], fin[(h * 4 + g) * OUTS + id]);
        }
        add_pair(half[0], half[1]);
        if (n < N && m < M) out[(size_t)m * ldo + n] = from_f32<TO>(half[0].x + half[0].y);
      }
    }
    if (++chunk == chunks) {
      chunk = 0;
      tile += gridDim.x;
    }
  }
}

// Up to 16 rows the kernel for few rows is the faster one, and up to 32, in two pieces, where K is long: two pieces of 16 rows take 25 us
// with 2,048 outputs of 2,048 inputs and 81 us with 2,048 of 8,192, a tile of 64 rows, whatever part of it is there, 39 and 150 us; with 64 of
// 64 inputs 8.3 and 5.6 us. Without copies that run by themselves a piece is bound by its loads: only where every tile of outputs has a
// CTA of its own (2,048 of 2,049 in bfloat16 52 and 59 us, 8,192 of 2,049 194 and 130 us).
bool few_rows(int M, int N, int K, bool copies) { return M <= 16 || (M <= 32 && K > 256 && (copies || ceil_div(N, NT) <= simt_sm_count())); }

template <typename T, typename TO, int MT, int TN, int TM, bool ALIGNED>
void launch_few(const T* a, const T* w, TO* out, int M, int N, int K, long long lda, long long ldw, long long ldo, cudaStream_t stream) {
  auto kernel = gemm_simt_few_kernel<T, TO, MT, TN, TM, ALIGNED>;
  constexpr int smem = few_smem<MT>();
  static_assert(smem <= 227 * 1024, "shared memory of a CTA");
  static std::atomic<unsigned long long> done{0};
  allow_smem(kernel, smem, done);
  launch_kernel(kernel, min(ceil_div(N, NT), simt_sm_count()), few_threads<MT, TN, TM>(), smem, stream, a, w, out, M, N, K, lda, ldw, ldo);
}

template <typename T, typename TO, bool ALIGNED>
void launch(const T* a, const T* w, TO* out, int M, int N, int K, long long lda, long long ldw, long long ldo, cudaStream_t stream) {
  if (few_rows(M, N, K, ALIGNED && sizeof(T) == 4)) {
    for (int m = 0; m < M; m += 16) {
      const int rows = min(16, M - m);
      const T* am = a + (size_t)m * lda;
      TO* om = out + (size_t)m * ldo;
      if (rows == 1) launch_few<T, TO, 1, 4, 1, ALIGNED>(am, w, om, rows, N, K, lda, ldw, ldo, stream);
      else if (rows <= 4) launch_few<T, TO, 4, 2, 4, ALIGNED>(am, w, om, rows, N, K, lda, ldw, ldo, stream);
      else if (rows <= 8) launch_few<T, TO, 8, 2, 8, ALIGNED>(am, w, om, rows, N, K, lda, ldw, ldo, stream);
      else launch_few<T, TO, 16, 4, 8, ALIGNED>(am, w, om, rows, N, K, lda, ldw, ldo, stream);
    }
    return;
  }
  auto kernel = gemm_simt_tile_kernel<T, TO, ALIGNED>;
  static std::atomic<unsigned long long> done{0};
  allow_smem(kernel, TILE_SMEM, done);
  const int m_tiles = ceil_div(M, BM);
  launch_kernel_cluster(kernel, dim3(2u * (unsigned)m_tiles * (unsigned)ceil_div(N, BN)), 256, TILE_SMEM, dim3(2), stream, a, w, out, M, N, K,
                        m_tiles, lda, ldw, ldo);
}

template <typename T, typename TO>
void choose(const void* a, const void* w, void* out, int M, int N, int K, long long lda, long long ldw, long long ldo, cudaStream_t stream) {
  // groups of four k at once: rows that begin on four numbers; in bfloat16 of whole groups of four
  const uintptr_t at = reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w);
  if (at % (4 * sizeof(T)) == 0 && lda % 4 == 0 && ldw % 4 == 0 && (sizeof(T) == 4 || K % 4 == 0))
    return launch<T, TO, true>((const T*)a, (const T*)w, (TO*)out, M, N, K, lda, ldw, ldo, stream);
  launch<T, TO, false>((const T*)a, (const T*)w, (TO*)out, M, N, K, lda, ldw, ldo, stream);
}

}  // namespace

// in_dtype: element type of both a and w; out_dtype: element type of out.
extern "C" int llm_gemm_simt(const void* a, const void* w, void* out, int M, int N, int K, long long lda,
                             long long ldw, long long ldo, int in_dtype, int out_dtype, cudaStream_t stream) {
  if (M == 0 || N == 0) return LLM_OK;
  LLM_REQUIRE(M > 0 && N > 0 && K > 0, "gemm_simt: bad sizes M=%d N=%d K=%d", M, N, K);
  LLM_REQUIRE(lda >= K && ldw >= K && ldo >= N, "gemm_simt: row strides smaller than the rows");
  LLM_REQUIRE(ceil_div(M, BM) <= 65535, "gemm_simt: M=%d too large", M);
  if (in_dtype == LLM_F32 && out_dtype == LLM_F32)
    choose<float, float>(a, w, out, M, N, K, lda, ldw, ldo, stream);
  else if (in_dtype == LLM_BF16 && out_dtype == LLM_BF16)
    choose<bf16, bf16>(a, w, out, M, N, K, lda, ldw, ldo, stream);
  else if (in_dtype == LLM_BF16 && out_dtype == LLM_F32)
    choose<bf16, float>(a, w, out, M, N, K, lda, ldw, ldo, stream);
  else
    LLM_REQUIRE(false, "gemm_simt: unsupported dtypes in=%d out=%d", in_dtype, out_dtype);
  LLM_CHECK_LAUNCH("gemm_simt");
  return LLM_OK;
}
