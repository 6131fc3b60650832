// Per-expert products of a routed feed-forward for prompt-sized steps, on tcgen05.
//
// The step's (token, choice) pairs lie sorted by expert in tiles of 128 rows of one expert (group_kernel in routed.cu; the
// used tiles come first). gather_rows copies the rows that the pairs read into that order once, so that a tile of 128 rows is
// a TMA box; the first product writes its results in the same order, so the second one needs no gathering, and the second
// writes each pair's row at the pair's own index. The product itself is the persistent kernel of gemm_tc.cu (one CTA a
// multiprocessor, tiles of 128 x 256, two accumulators in tensor memory, the epilogue of a tile beside the products of the
// next); which expert's weight rows a tile multiplies with, and how many tiles there are, is read from memory.
//
// 2,048 tokens, 4 of 16 experts, 2,048 x 2,048 (68.7 GFLOP a product): 88 us with the gelu, 93 with the weights, as mma.sync tiles of
// 128 x 128 (routed_mma.cu) 306 and 282 us; bound like the dense product by the rate at which a multiprocessor takes a 128 x 256
// tile's operands in (0.5 us a k-block). gather_rows: 7.6 us (8 MB read, 33 MB written).
#include "common.cuh"
#include "tc_common.cuh"

#include <algorithm>
#include <atomic>

namespace {

constexpr int ROWS = BM, BN = 256, THREADS = 192, STAGES = 4;
constexpr int B_BYTES = BN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;

__global__ void __launch_bounds__(256)
    gather_rows_kernel(const bf16* __restrict__ a, long long lda, int a_div, const int* __restrict__ tile_expert, const int* __restrict__ tile_rows,
                       bf16* __restrict__ out, int groups) {
  dep_launch();
  dep_wait();
  const int tile = blockIdx.x / (ROWS / 8), row = blockIdx.x % (ROWS / 8) * 8 + (threadIdx.x >> 5);  // a warp a row
  if (tile_expert[tile] < 0) return;
  const size_t at = (size_t)tile * ROWS + row;
  const int pair = tile_rows[at];
  if (pair < 0) return;  // (a row that nobody reads)
  const uint4* src = reinterpret_cast<const uint4*>(a + (size_t)(pair / a_div) * lda);
  uint4* dst = reinterpret_cast<uint4*>(out) + at * groups;
#pragma unroll 4
  for (int g = threadIdx.x & 31; g < groups; g += 32) dst[g] = src[g];
}

// The (tile of rows, column block, k-block) triples of a persistent CTA in order, without a division but one a tile.
struct Walk {
  const int* tile_expert;
  int tile, kt, a_row0, b_row0, step, total, k_tiles, used, N;
  __device__ __forceinline__ Walk(const int* te, int first, int step_, int total_, int k_tiles_, int used_, int N_)
      : tile_expert(te), kt(0), step(step_), total(total_), k_tiles(k_tiles_), used(used_), N(N_) { set(first); }
  __device__ __forceinline__ void set(int t) {
    tile = t;
    if (t >= total) return;
    const int n = t / used, m = t - n * used;
    a_row0 = m * ROWS;
    b_row0 = tile_expert[m] * N + n * BN;
  }
  __device__ __forceinline__ void next() {
    if (++kt == k_tiles) {
      kt = 0;
      set(tile + step);
    }
  }
};

// How many tiles at the front are in use.
__device__ __forceinline__ int used_tiles(const int* tile_expert, int max_tiles) {
  int lo = 0, hi = max_tiles;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (tile_expert[mid] >= 0) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

template <int N16>
__device__ __forceinline__ void store_bf16(bf16* dst, const float* v, int valid, bool aligned) {
  if (valid >= N16 && aligned) {
    uint32_t p[N16 / 2];
#pragma unroll
    for (int i = 0; i < N16 / 2; ++i) {
      __nv_bfloat162 t = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      p[i] = *reinterpret_cast<uint32_t*>(&t);
    }
#pragma unroll
    for (int i = 0; i < N16 / 8; ++i) reinterpret_cast<uint4*>(dst)[i] = make_uint4(p[4 * i], p[4 * i + 1], p[4 * i + 2], p[4 * i + 3]);
  } else {
    for (int i = 0; i < min(valid, N16); ++i) dst[i] = __float2bfloat16_rn(v[i]);
  }
}

// EPI as in routed_mma.cu. 0: exact gelu; 1: times share[pair] (null: as it is), float32 at the pair's own row; 2: gate and up
// rows in turn, gated_value; 3: max(share[pair] * z, 0)^2. 0, 2, 3: bfloat16 at the row's place in the sorted order.
template <int EPI>
__global__ void __launch_bounds__(THREADS)
    routed_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const int* __restrict__ tile_expert,
                     const int* __restrict__ tile_rows, int max_tiles, void* __restrict__ out, long long ldo, int N, int k_tiles, int n_tiles,
                     const float* __restrict__ share, int act, float p0, float p1, int* __restrict__ error_out) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;  // [2] the tensor cores have finished a tile in accumulator b
  uint64_t* acc_empty = acc_full + 2;   // [2] the epilogue warps have read accumulator b
  uint64_t* mma_done = acc_empty + 2;   // every product this CTA issued has finished (committed last, also after giving up)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mma_done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 4);  // one arrival per epilogue warp
    }
    mbar_init(mma_done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;

  dep_launch();
  dep_wait();  // the list of tiles and the rows are the stream's
  const int used = used_tiles(tile_expert, max_tiles), total = used * n_tiles;
  const int my_tiles = (int)blockIdx.x < total ? (total - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;

  if (warp == 4) {
    if (lane == 0) {
      // ---------------------------------------------------------------- producer: TMA loads
      const long long n_iter = (long long)my_tiles * k_tiles;
      Walk walk(tile_expert, blockIdx.x, gridDim.x, total, k_tiles, used, N);
      long long issued = 0;
      bool ok = true;
      RingPos ring(STAGES);
      for (long long it = 0; it < n_iter; ++it, ring.next(), walk.next()) {
        const int s = ring.s;
        if (it >= STAGES) ok = mbar_wait(&empty[s], ring.ph ^ 1u, abort_flag, error_out, ERR_PRODUCER);
        if (!ok) break;
        uint8_t* sa = smem + (size_t)s * STAGE_BYTES;
        mbar_expect_tx(&full[s], STAGE_BYTES);
        tma_load_2d(sa, &map_a, walk.kt * BK, walk.a_row0, &full[s]);
        tma_load_2d(sa + A_BYTES, &map_b, walk.kt * BK, walk.b_row0, &full[s]);
        issued = it + 1;
      }
      if (!ok || *abort_flag) {
        // wait (bounded) for the copies already issued, so that none lands after the CTA has left
        const long long first = issued > STAGES ? issued - STAGES : 0;
        for (long long it = first; it < issued; ++it) {
          const long long t0 = clock64();
          while (!mbar_try_wait(&full[it % STAGES], (uint32_t)(it / STAGES) & 1u)) {
            if (clock64() - t0 > WAIT_CYCLES) {
              atomicCAS(error_out, 0, ERR_DRAIN);
              break;
            }
          }
        }
      }
    }
  } else if (warp == 5) {
    if (lane == 0) {
      // ---------------------------------------------------------------- tensor-core issue
      constexpr uint32_t idesc = instr_desc(BN);
      bool ok = true;
      RingPos ring(STAGES);
      for (int t = 0; t < my_tiles && ok; ++t) {
        const int b = t & 1;
        if (t >= 2) {  // the epilogue of the tile that used this accumulator two tiles ago
          ok = mbar_wait(&acc_empty[b], (uint32_t)((t >> 1) - 1) & 1u, abort_flag, error_out, ERR_MMA);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        const uint32_t acc = tmem_base + (uint32_t)(b * BN);
        for (int kt = 0; kt < k_tiles && ok; ++kt, ring.next()) {
          const int s = ring.s;
          ok = mbar_wait(&full[s], ring.ph, abort_flag, error_out, ERR_MMA);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t sa = smem_u32(smem + (size_t)s * STAGE_BYTES);
          const uint64_t da = smem_desc_sw128(sa), db = smem_desc_sw128(sa + A_BYTES);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            mma_f16(acc, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (kt > 0 || k > 0) ? 1u : 0u);
          mma_commit(&empty[s]);
        }
        if (ok) mma_commit(&acc_full[b]);
      }
      mma_commit(mma_done);
    }
  } else {
    // ------------------------------------------------------------------ epilogue: warps 0-3
    bool ok = true;
    for (int t = 0; t < my_tiles; ++t) {
      const int b = t & 1;
      ok = mbar_wait(&acc_full[b], (uint32_t)(t >> 1) & 1u, abort_flag, error_out, ERR_EPILOGUE);
      ok = __all_sync(0xffffffffu, ok);  // a warp reads tensor memory together or not at all
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int tile = blockIdx.x + t * gridDim.x, n = tile / used, m = tile - n * used, n0 = n * BN;
      const size_t row = (size_t)m * ROWS + warp * 32 + lane;
      const int pair = tile_rows[row];
      const float sc = ((EPI == 1 || EPI == 3) && share != nullptr && pair >= 0) ? share[pair] : 1.0f;
      const uint32_t acc = tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)(b * BN);
#pragma unroll 1
      for (int c0 = 0; c0 < BN; c0 += 16) {
        float v[16];
        __syncwarp();  // (lanes of padding rows come back early)
        tmem_load16(acc + (uint32_t)c0, v);
        const int col = n0 + c0;
        if (pair < 0 || col >= N) continue;  // (a row of padding, columns of the next expert)
        if (EPI == 1) {
          float* dst = (float*)out + (size_t)pair * ldo + col;
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] *= sc;
          if (col + 16 <= N && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) reinterpret_cast<float4*>(dst)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
          } else {
            for (int i = 0; i < min(16, N - col); ++i) dst[i] = v[i];
          }
        } else if (EPI == 2) {
          bf16* dst = (bf16*)out + row * ldo + col / 2;
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = gated_value(v[2 * i], v[2 * i + 1], act, p0, p1);
          store_bf16<8>(dst, v, (N - col) / 2, (reinterpret_cast<uintptr_t>(dst) & 15u) == 0);
        } else {
          bf16* dst = (bf16*)out + row * ldo + col;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            if (EPI == 0) v[i] = 0.5f * v[i] * (1.0f + erff(v[i] * 0.70710678118654752440f));
            if (EPI == 3) {
              const float z = fmaxf(v[i] * sc, 0.f);
              v[i] = z * z;
            }
          }
          store_bf16<16>(dst, v, N - col, (reinterpret_cast<uintptr_t>(dst) & 15u) == 0);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[b]);
    }
    // Tensor memory and the stages belong to the products in flight until the last of them is done.
    if (threadIdx.x == 0) mbar_drain(mma_done, 0, error_out);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
}

int tc_sm_count() {
  static const int count = [] {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    return n;
  }();
  return count;
}

template <int EPI>
int launch_routed(const CUtensorMap& ma, const CUtensorMap& mb, const int* tile_expert, const int* tile_rows, int max_tiles, void* out, long long ldo,
                  int N, int K, const float* share, int act, float p0, float p1, cudaStream_t stream) {
  constexpr int smem = STAGES * STAGE_BYTES + (2 * STAGES + 5) * 8 + 16 + 1024;
  static std::atomic<unsigned long long> done{0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return LLM_ERR_LAUNCH;
  if (dev >= 64 || !(done.load() >> dev & 1ull)) {
    if (cudaFuncSetAttribute(routed_tc_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
      llm_set_error("routed_tc: cannot raise the shared memory limit");
      return LLM_ERR_LAUNCH;
    }
    if (dev < 64) done.fetch_or(1ull << dev);
  }
  const int n_tiles = (N + BN - 1) / BN, k_tiles = (K + BK - 1) / BK;
  const int grid = (int)std::min<long long>((long long)max_tiles * n_tiles, tc_sm_count());
  launch_kernel(routed_tc_kernel<EPI>, grid, THREADS, smem, stream, ma, mb, tile_expert, tile_rows, max_tiles, out, ldo, N, k_tiles, n_tiles, share,
                act, p0, p1, error_word());
  return LLM_OK;
}

}  // namespace

// out [max_tiles * 128, K] = the rows that the pairs of the tiles read, in the tiles' order (rows of padding are left as they are).
extern "C" int llm_routed_gather(const void* a, long long lda, int a_div, int K, const int* tile_expert, const int* tile_rows, int max_tiles,
                                 void* out, cudaStream_t stream) {
  if (max_tiles == 0) return LLM_OK;
  LLM_REQUIRE(max_tiles > 0 && max_tiles <= (1 << 24) && a_div > 0 && K > 0 && K % 8 == 0 && lda % 8 == 0, "routed_gather: bad sizes");
  LLM_REQUIRE(((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0, "routed_gather: rows must begin on 16 bytes");
  launch_kernel(gather_rows_kernel, max_tiles * (ROWS / 8), 256, 0, stream, (const bf16*)a, lda, a_div, tile_expert, tile_rows, (bf16*)out, K / 8);
  LLM_CHECK_LAUNCH("routed_gather");
  return LLM_OK;
}

// rows [max_tiles * 128, K] in the tiles' order, w [E, N, K]; tiles of 128 rows. epilogue, share, act, p0, p1: as
// llm_routed_product_mma; epilogue 1 writes float32 at the pairs' own rows of out, the others bfloat16 in the tiles' order.
extern "C" int llm_routed_product_tc(const void* rows, const void* w, int E, int N, int K, const int* tile_expert, const int* tile_rows, int max_tiles,
                                     void* out, long long ldo, int epilogue, const float* share, int act, float p0, float p1, cudaStream_t stream) {
  if (max_tiles == 0) return LLM_OK;
  LLM_REQUIRE(N > 0 && K > 0 && E > 0 && max_tiles > 0 && K % 8 == 0, "routed_product_tc: bad sizes");
  LLM_REQUIRE(epilogue >= 0 && epilogue <= 3 && (epilogue != 2 || N % 2 == 0), "routed_product_tc: unknown epilogue %d", epilogue);
  LLM_REQUIRE(act >= 0 && act <= 2, "routed_product_tc: unknown activation %d", act);
  LLM_REQUIRE((long long)max_tiles * ((N + BN - 1) / BN) < (1LL << 30) && (long long)E * N < (1LL << 31), "routed_product_tc: sizes too large");
  LLM_REQUIRE(((reinterpret_cast<uintptr_t>(rows) | reinterpret_cast<uintptr_t>(w)) & 15u) == 0, "routed_product_tc: operands must begin on 16 bytes");
  LLM_REQUIRE(error_word() != nullptr, "routed_product_tc: cannot allocate the error word");
  CUtensorMap ma, mb;
  LLM_REQUIRE(tensor_map_for(rows, (long long)max_tiles * ROWS, K, K, ROWS, &ma) && tensor_map_for(w, (long long)E * N, K, K, BN, &mb),
              "routed_product_tc: cuTensorMapEncodeTiled failed");
  int rc;
  if (epilogue == 0) rc = launch_routed<0>(ma, mb, tile_expert, tile_rows, max_tiles, out, ldo, N, K, share, act, p0, p1, stream);
  else if (epilogue == 1) rc = launch_routed<1>(ma, mb, tile_expert, tile_rows, max_tiles, out, ldo, N, K, share, act, p0, p1, stream);
  else if (epilogue == 2) rc = launch_routed<2>(ma, mb, tile_expert, tile_rows, max_tiles, out, ldo, N, K, share, act, p0, p1, stream);
  else rc = launch_routed<3>(ma, mb, tile_expert, tile_rows, max_tiles, out, ldo, N, K, share, act, p0, p1, stream);
  if (rc != LLM_OK) return rc;
  LLM_CHECK_LAUNCH("routed_product_tc");
  return LLM_OK;
}
