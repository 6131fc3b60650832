// Causal grouped-query attention over the paged cache, CUDA cores, float32 arithmetic: the true 32-bit path, and bfloat16 at
// sizes the tensor-core kernels refuse.
//
// The rows of a request and key/value head are its (token of the step, query head of the group) pairs in order; a CTA takes a
// tile of them, so that every key and value it fetches serves all rows of the tile, and walks over the keys in segments of
// 128 at absolute positions. A row's arithmetic is the same whatever tile it lies in:
//   score = (q . k) * scale, the dot a chain of fused multiply-adds over ascending dimensions; in a segment the largest score
//   m, p = exp(score - m), their sum l (4 neighbouring keys a lane, then the warp's tree) and sum p * v over ascending keys;
//   segments are merged one after the other in ascending order.
// So a token's output does not depend on how its request was cut into steps, on the rest of the batch, on page numbers, or on
// whether one CTA walks over all segments or each segment has a CTA of its own and a second kernel merges them (steps with
// few rows: a CTA a segment is what fills the device).
//
// Bound by latency with few rows, by reads of shared memory and multiply-adds with many. A layer at the Llama 3.2 1B sizes:
// 8 single tokens behind 256 to 768 keys 17 us and 7 for the merge (a warp a token and head, a lane a key: 630 us; in float32 such steps
// run on attention_one.cu, up to some thousand keys); a prompt of 300 tokens 36 us and 7 (417 us).
// Only keys that some row of the tile sees are fetched and scored, so a few tokens' prompt costs what it has: 5 tokens 6.1 us, a warp a
// token and head 6.1, all 128 keys of the segment 13.9.
//
// Formula of the reference's attention_f32 (src/kernels.cpp:413-474): kv head = q head / (nq/nkv), score = (q . k) *
// (1/sqrt(head_dim)) with the scale applied after the dot, softmax in float32, output = sum_t p_t * V[t].
#include "attention_simt.cuh"

#include <type_traits>

using namespace simt_attention;

namespace {

constexpr int KT = 64;  // keys of a tile in shared memory
constexpr int MAX_HD = 256;

// ROWS rows a CTA; a thread has KM keys x RM rows of the scores and KM dimensions x RM rows of the output in each 64
// dimensions; DC: how many times 64 dimensions.
template <typename T, int ROWS, int KM, int RM, int DC, bool ALIGNED>
__global__ void __launch_bounds__((KT / KM) * (ROWS / RM))
    paged_attention_simt_kernel(const AttArgs p) {
  constexpr int TX = KT / KM, THREADS = TX * (ROWS / RM), WARPS = THREADS / 32;
  extern __shared__ __align__(16) float smem[];
  __shared__ long long s_key[SEG];
  __shared__ float s_m[ROWS], s_l[ROWS];
  dep_launch();
  dep_wait();
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX, lane = tid & 31, warp = tid >> 5;
  const int seq = blockIdx.x / p.row_tiles, kvh = blockIdx.y % p.nkv, only = p.scratch != nullptr ? (int)blockIdx.y / p.nkv : -1;
  const int group = p.nq / p.nkv, row0 = (blockIdx.x % p.row_tiles) * ROWS, n_rows = min(ROWS, p.seq_ntok[seq] * group - row0);
  if (n_rows <= 0) return;
  const int start = p.seq_start[seq], tok0 = p.seq_qoff[seq];
  const int first_pos = start + row0 / group, last_pos = start + (row0 + n_rows - 1) / group;
  const int lo = p.window > 0 ? max(0, first_pos - p.window + 1) : 0;  // the tile's first key
  int seg = lo / SEG, seg_end = last_pos / SEG + 1;
  if (only >= 0) {
    if (only < seg || only >= seg_end) return;
    seg = only;
    seg_end = only + 1;
  }
  const int hp = (p.hd + 3) & ~3, row_len = hp + 4, chunks = hp / 4;
  float* tiles = smem;                         // [2][KT][row_len]: keys, then values
  float* qs = smem + 2 * KT * row_len;         // [ROWS][row_len]
  float* ss = qs + ROWS * row_len;             // [ROWS][S_ROW]
  const int* table = p.table + (size_t)seq * p.max_blocks;

  for (int i0 = tid; i0 < n_rows * chunks; i0 += 4 * THREADS) {  // (rows beyond the tile's are read by nobody whose result is kept)
    float4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * THREADS, r = i / chunks, c = i - r * chunks;
      const T* src = (const T*)p.q + (size_t)(tok0 + (row0 + r) / group) * p.ld_q + (size_t)(kvh * group + (row0 + r) % group) * p.hd;
      v[u] = fetch4(src + 4 * c, i < n_rows * chunks ? count4(4 * c, p.hd) : 0);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * THREADS, r = i / chunks, c = i - r * chunks;
      if (i < n_rows * chunks) *reinterpret_cast<float4*>(qs + r * row_len + 4 * c) = v[u];
    }
  }

  float acc[DC][KM][RM], m_run[RM], l_run[RM];
#pragma unroll
  for (int j = 0; j < RM; ++j) {
    m_run[j] = -INFINITY;
    l_run[j] = 0.f;
#pragma unroll
    for (int c = 0; c < DC; ++c)
#pragma unroll
      for (int i = 0; i < KM; ++i) acc[c][i][j] = 0.f;
  }

  // step s of a segment: 0, 1 its key tiles, 2, 3 its value tiles; keys up to the tile's last one (what lies behind it is masked)
  auto load = [&](int s, int n_keys) {
    const T* base = (const T*)(s < 2 ? p.k : p.v);
    float* dst = tiles + (s & 1) * KT * row_len;
    const int total = n_keys * chunks;
    constexpr int U = ALIGNED && sizeof(T) == 4 ? 1 : ALIGNED && DC == 4 ? 8 : 4;  // loads through registers: several on their way
    for (int i0 = tid; i0 < total; i0 += U * THREADS) {
      int key[U], c[U];
      long long off[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = min(i0 + u * THREADS, total - 1);  // (beyond the end: the last group again, the same bytes to the same place)
        key[u] = i / chunks;
        c[u] = i - key[u] * chunks;
        off[u] = s_key[(s & 1) * KT + key[u]];
      }
      stage_rows<ALIGNED, U, 4, 1, T>([&](int u) { return dst + key[u] * row_len + 4 * c[u]; }, [&](int u) { return off[u] >= 0 ? base + off[u] + 4 * c[u] : base; },
                                [&](int u) { return off[u] >= 0 ? count4(4 * c[u], p.hd) : 0; });
    }
    commit_group();
  };

  for (; seg < seg_end; ++seg) {
    const int k0 = seg * SEG;
    auto keys_of = [&](int half) { return max(0, min(KT, last_pos - (k0 + half * KT) + 1)); };
    __syncthreads();  // the segment before this one has been read
    for (int i = tid; i < SEG; i += THREADS) {
      const int key = k0 + i;
      long long off = -1;
      if (key >= lo && key <= last_pos) {
        const int page = table[key / p.page];
        off = (((long long)page * p.nkv + kvh) * p.page + key % p.page) * p.hd;
      }
      s_key[i] = off;
    }
    __syncthreads();
    load(0, keys_of(0));
    load(1, keys_of(1));
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      wait_groups<1>();  // (the other key tile, then the first value tile, is on its way)
      __syncthreads();
      const int n_keys = keys_of(half);
      float s[KM][RM];
#pragma unroll
      for (int i = 0; i < KM; ++i)
#pragma unroll
        for (int j = 0; j < RM; ++j) s[i][j] = 0.f;
      const float* kt = tiles + half * KT * row_len + tx * row_len;
      const float* qt = qs + ty * RM * row_len;
      auto scores = [&](auto used) {  // of the first `used` of the thread's keys
        constexpr int USED = decltype(used)::value;
        for (int d = 0; d < hp; d += 4) {
          float4 kv[USED];
#pragma unroll
          for (int i = 0; i < USED; ++i) kv[i] = *reinterpret_cast<const float4*>(kt + i * TX * row_len + d);
#pragma unroll
          for (int j = 0; j < RM; ++j) {
            const float4 qv = *reinterpret_cast<const float4*>(qt + j * row_len + d);
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
              for (int i = 0; i < USED; ++i) s[i][j] = fmaf(part(qv, e), part(kv[i], e), s[i][j]);
          }
        }
      };
      if (ty * RM < n_rows && n_keys > 0) {
        if (KM > 1 && n_keys <= TX) scores(std::integral_constant<int, 1>{});
        else if (KM > 2 && n_keys <= 2 * TX) scores(std::integral_constant<int, (KM > 2 ? 2 : KM)>{});
        else scores(std::integral_constant<int, KM>{});
      }
#pragma unroll
      for (int i = 0; i < KM; ++i)
#pragma unroll
        for (int j = 0; j < RM; ++j) ss[(ty * RM + j) * S_ROW + half * KT + tx + i * TX] = s[i][j] * p.scale;
      __syncthreads();
      load(2 + half, n_keys);  // over the key tile that has just been read
    }
    // softmax of the segment, a warp a row
    for (int r = warp; r < n_rows; r += WARPS) {
      const int pos = start + (row0 + r) / group, from = p.window > 0 ? max(0, pos - p.window + 1) : 0;
      float4 v = *reinterpret_cast<const float4*>(ss + r * S_ROW + 4 * lane);
      const int key = k0 + 4 * lane;
      v.x = key >= from && key <= pos ? v.x : -INFINITY;
      v.y = key + 1 >= from && key + 1 <= pos ? v.y : -INFINITY;
      v.z = key + 2 >= from && key + 2 <= pos ? v.z : -INFINITY;
      v.w = key + 3 >= from && key + 3 <= pos ? v.w : -INFINITY;
      const float m = warp_max(fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)));
      v.x = v.x == -INFINITY ? 0.f : expf(v.x - m);
      v.y = v.y == -INFINITY ? 0.f : expf(v.y - m);
      v.z = v.z == -INFINITY ? 0.f : expf(v.z - m);
      v.w = v.w == -INFINITY ? 0.f : expf(v.w - m);
      const float l = warp_sum((v.x + v.y) + (v.z + v.w));
      *reinterpret_cast<float4*>(ss + r * S_ROW + 4 * lane) = v;
      if (lane == 0) {
        s_m[r] = m;
        s_l[r] = l;
      }
    }
    // sums of probabilities times values; a key that a row does not see is passed over, whatever its value
    const bool whole = k0 + SEG - 1 <= first_pos && (p.window == 0 || k0 >= last_pos - p.window + 1);
    float av[DC][KM][RM];
#pragma unroll
    for (int c = 0; c < DC; ++c)
#pragma unroll
      for (int i = 0; i < KM; ++i)
#pragma unroll
        for (int j = 0; j < RM; ++j) av[c][i][j] = 0.f;
    int pos_of[RM];
#pragma unroll
    for (int j = 0; j < RM; ++j) pos_of[j] = start + (row0 + ty * RM + j) / group;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      if (half == 0) wait_groups<1>();
      else wait_groups<0>();
      __syncthreads();
      if (ty * RM >= n_rows) continue;
      const float* vt = tiles + half * KT * row_len + tx * KM;
      const float* pt = ss + ty * RM * S_ROW + half * KT;
      const int n_keys = keys_of(half);
      for (int key = 0; key < n_keys; key += 4) {
        float4 pv[RM];
#pragma unroll
        for (int j = 0; j < RM; ++j) pv[j] = *reinterpret_cast<const float4*>(pt + j * S_ROW + key);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int at = k0 + half * KT + key + e;
#pragma unroll
          for (int c = 0; c < DC; ++c) {
            if (64 * c + tx * KM >= hp) continue;
            float vv[KM];
            if constexpr (KM == 4) {
              const float4 v4 = *reinterpret_cast<const float4*>(vt + (key + e) * row_len + 64 * c);
              vv[0] = v4.x; vv[1] = v4.y; vv[2] = v4.z; vv[3] = v4.w;
            } else {
#pragma unroll
              for (int i = 0; i < KM; ++i) vv[i] = vt[(key + e) * row_len + 64 * c + i];
            }
#pragma unroll
            for (int j = 0; j < RM; ++j) {
              const bool sees = whole || (at <= pos_of[j] && (p.window == 0 || at > pos_of[j] - p.window));
#pragma unroll
              for (int i = 0; i < KM; ++i) av[c][i][j] = sees ? fmaf(part(pv[j], e), vv[i], av[c][i][j]) : av[c][i][j];
            }
          }
        }
      }
    }
    if (only >= 0) {  // a segment's own results, for the merging kernel
#pragma unroll
      for (int j = 0; j < RM; ++j) {
        const int r = ty * RM + j;
        if (r >= n_rows) continue;
        const size_t item = (size_t)(tok0 + (row0 + r) / group) * p.nq + kvh * group + (row0 + r) % group;
        float* o = p.scratch + (item * p.n_seg + only) * (p.hd + 2);
#pragma unroll
        for (int c = 0; c < DC; ++c)
#pragma unroll
          for (int i = 0; i < KM; ++i) {
            const int d = 64 * c + tx * KM + i;
            if (d < p.hd) o[d] = av[c][i][j];
          }
        if (tx == 0) {
          o[p.hd] = s_m[r];
          o[p.hd + 1] = s_l[r];
        }
      }
      return;
    }
#pragma unroll
    for (int j = 0; j < RM; ++j) {
      if (k0 > pos_of[j] || (p.window > 0 && k0 + SEG - 1 <= pos_of[j] - p.window)) continue;  // the row sees no key of this segment
      float m_new, a, b;
      join_weights(m_run[j], s_m[ty * RM + j], m_new, a, b);
      m_run[j] = m_new;
      l_run[j] = join(l_run[j], a, s_l[ty * RM + j], b);
#pragma unroll
      for (int c = 0; c < DC; ++c)
#pragma unroll
        for (int i = 0; i < KM; ++i) acc[c][i][j] = join(acc[c][i][j], a, av[c][i][j], b);
    }
  }
#pragma unroll
  for (int j = 0; j < RM; ++j) {
    const int r = ty * RM + j;
    if (r >= n_rows) continue;
    const float inv = 1.0f / l_run[j];
    T* o = (T*)p.out + (size_t)(tok0 + (row0 + r) / group) * p.ld_out + (size_t)(kvh * group + (row0 + r) % group) * p.hd;
#pragma unroll
    for (int c = 0; c < DC; ++c)
#pragma unroll
      for (int i = 0; i < KM; ++i) {
        const int d = 64 * c + tx * KM + i;
        if (d < p.hd) o[d] = from_f32<T>(acc[c][i][j] * inv);
      }
  }
}

// Segments of a (token, query head), merged in ascending order: a warp an item, 4 items a CTA.
template <typename T>
__global__ void __launch_bounds__(128) paged_attention_simt_merge_kernel(const AttArgs p, const int* __restrict__ positions, int n_tokens) {
  dep_launch();
  dep_wait();
  const int lane = threadIdx.x & 31;
  const long long item = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (item >= (long long)n_tokens * p.nq) return;
  const int tok = (int)(item / p.nq), head = (int)(item - (long long)tok * p.nq), pos = positions[tok];
  const int first = p.window > 0 ? max(0, pos - p.window + 1) / SEG : 0;
  const float* from = p.scratch + item * p.n_seg * (p.hd + 2);
  float acc[MAX_HD / 32], m = -INFINITY, l = 0.f;
#pragma unroll
  for (int i = 0; i < MAX_HD / 32; ++i) acc[i] = 0.f;
  for (int s = first; s <= pos / SEG; ++s) {
    const float* o = from + (size_t)s * (p.hd + 2);
    const float m_s = o[p.hd], l_s = o[p.hd + 1];
    float m_new, a, b;
    join_weights(m, m_s, m_new, a, b);
    m = m_new;
    l = join(l, a, l_s, b);
#pragma unroll
    for (int i = 0; i < MAX_HD / 32; ++i)
      if (32 * i + lane < p.hd) acc[i] = join(acc[i], a, o[32 * i + lane], b);
  }
  const float inv = 1.0f / l;
  T* out = (T*)p.out + (size_t)tok * p.ld_out + (size_t)head * p.hd;
#pragma unroll
  for (int i = 0; i < MAX_HD / 32; ++i)
    if (32 * i + lane < p.hd) out[32 * i + lane] = from_f32<T>(acc[i] * inv);
}

template <typename T, int ROWS, int KM, int RM, int DC, bool ALIGNED>
void launch_rows(AttArgs p, int n_seqs, int max_rows, cudaStream_t stream) {
  p.row_tiles = ceil_div(max_rows, ROWS);
  const int row_len = ((p.hd + 3) & ~3) + 4, smem = (2 * KT * row_len + ROWS * (row_len + S_ROW)) * 4;
  auto kernel = paged_attention_simt_kernel<T, ROWS, KM, RM, DC, ALIGNED>;
  static std::atomic<unsigned long long> done{0};
  constexpr int most = (2 * KT * (64 * DC + 4) + ROWS * (64 * DC + 4 + S_ROW)) * 4;
  static_assert(most <= 224 * 1024, "shared memory of a CTA");
  allow_smem(kernel, most, done);
  launch_kernel(kernel, dim3((unsigned)p.row_tiles * (unsigned)n_seqs, p.nkv * (p.scratch != nullptr ? p.n_seg : 1)), (KT / KM) * (ROWS / RM), smem, stream, p);
}

template <typename T, bool ALIGNED>
void launch(const AttArgs& p, int n_seqs, int max_rows, bool wide, cudaStream_t stream) {
  if (wide) {
    if (p.hd <= 64) launch_rows<T, 64, 4, 4, 1, ALIGNED>(p, n_seqs, max_rows, stream);
    else launch_rows<T, 64, 4, 4, 2, ALIGNED>(p, n_seqs, max_rows, stream);
  } else if (p.hd <= 64) launch_rows<T, 8, 1, 2, 1, ALIGNED>(p, n_seqs, max_rows, stream);
  else if (p.hd <= 128) launch_rows<T, 8, 1, 2, 2, ALIGNED>(p, n_seqs, max_rows, stream);
  else launch_rows<T, 8, 1, 2, 4, ALIGNED>(p, n_seqs, max_rows, stream);
}

// Tiles of 64 rows where a request brings more than 8 (and two key tiles, 64 queries and their scores fit beside one another):
// a prompt of 300 tokens with 4 heads a group takes 19 tiles a key/value head instead of 150, each of which would fetch all keys. Not
// where tiles of 8 rows, and segments with CTAs of their own, would leave multiprocessors without one (a
// prompt of 5 tokens, 24 heads on 8 of 128: 9.7 us as one tile of 64 rows a key/value head, 7.1 as two of 8; of 40 tokens, 12 heads on 1 of
// 80 in bfloat16: 22 and 10.6 us).
bool wide_rows(int max_rows, int hd, long long pairs, int n_seg) {
  return max_rows > 8 && hd <= 128 && (long long)ceil_div(max_rows, 8) * pairs * n_seg > simt_sm_count();
}

// Whether every segment gets a CTA of its own: where CTAs that walk over all of them would not fill the device twice, as long
// as the segments' results stay small.
int segments(int n_seqs, int n_tokens, int max_new, int max_len, int nq, int nkv, int hd) {
  const int n_seg = ceil_div(max_len, SEG), max_rows = max_new * (nq / nkv);
  const long long ctas = (long long)ceil_div(max_rows, wide_rows(max_rows, hd, (long long)nkv * n_seqs, n_seg) ? 64 : 8) * nkv * n_seqs;
  const long long floats = (long long)n_tokens * nq * n_seg * (hd + 2);
  return n_seg > 1 && ctas < 2LL * simt_sm_count() && floats <= (16LL << 20) && (long long)nkv * n_seg <= 65535 ? n_seg : 1;
}

}  // namespace

// CTAs of the aligned tiles of 8 rows, heads of up to 64 numbers, that a multiprocessor holds at a time.
extern "C" int llm_paged_attention_simt_resident(int dtype) {
  const int row_len = 64 + 4, smem = (2 * KT * row_len + 8 * (row_len + S_ROW)) * 4;
  int n = 0;
  const cudaError_t rc = dtype == LLM_F32
                             ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, paged_attention_simt_kernel<float, 8, 1, 2, 1, true>, KT * 4, smem)
                             : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, paged_attention_simt_kernel<bf16, 8, 1, 2, 1, true>, KT * 4, smem);
  return rc == cudaSuccess ? n : 0;
}

// float32 numbers of scratch that a step needs (0: none). rows16: float32 queries, keys and values whose rows begin on 16 bytes.
extern "C" long long llm_paged_attention_simt_scratch(int n_seqs, int n_tokens, int max_new, int max_len, int nq, int nkv, int hd, int rows16) {
  if (n_seqs <= 0 || n_tokens <= 0 || nkv <= 0 || nq < nkv || hd <= 0) return 0;
  if (rows16 && one_token(n_seqs, max_new, max_len, nq, nkv, hd)) return 0;
  const int n_seg = segments(n_seqs, n_tokens, max_new, max_len, nq, nkv, hd);
  return n_seg > 1 ? (long long)n_tokens * nq * n_seg * (hd + 2) : 0;
}

extern "C" int llm_paged_attention_simt(const void* q, long long ld_q, const void* kcache, const void* vcache, int dtype, const int* positions,
                                        const int* seq_start, const int* seq_ntok, const int* seq_qoff, const int* block_table, int max_blocks,
                                        void* out, long long ld_out, int n_seqs, int n_tokens, int max_new, int max_len, int nq, int nkv, int hd,
                                        int page_size, float scale, int window, float* scratch, cudaStream_t stream) {
  if (n_tokens == 0 || n_seqs == 0) return LLM_OK;
  LLM_REQUIRE(n_tokens > 0 && nq > 0 && nkv > 0 && nq % nkv == 0, "attention: bad head counts nq=%d nkv=%d", nq, nkv);
  LLM_REQUIRE(hd > 0 && hd <= MAX_HD, "attention: head_dim %d not in 1..%d", hd, MAX_HD);
  LLM_REQUIRE(page_size > 0 && max_blocks > 0 && window >= 0, "attention: bad page_size/max_blocks/window");
  LLM_REQUIRE(n_seqs > 0 && max_new > 0 && max_len > 0, "attention: bad n_seqs/max_new/max_len");
  const uintptr_t at = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(kcache) | reinterpret_cast<uintptr_t>(vcache);
  if (dtype == LLM_F32 && at % 16 == 0 && ld_q % 4 == 0 && one_token(n_seqs, max_new, max_len, nq, nkv, hd)) {
    const AttArgs p{q, kcache, vcache, out, seq_start, seq_ntok, seq_qoff, block_table, nullptr, ld_q, ld_out,
                    max_blocks, nq, nkv, hd, page_size, window, 1, 0, scale};
    launch_one_token(p, n_seqs, max_len, stream);
    LLM_CHECK_LAUNCH("paged_attention_simt");
    return LLM_OK;
  }
  const int n_seg = segments(n_seqs, n_tokens, max_new, max_len, nq, nkv, hd), max_rows = max_new * (nq / nkv);
  LLM_REQUIRE(n_seg == 1 || scratch != nullptr, "attention: this step needs scratch");
  const AttArgs p{q, kcache, vcache, out, seq_start, seq_ntok, seq_qoff, block_table, n_seg > 1 ? scratch : nullptr, ld_q, ld_out,
                  max_blocks, nq, nkv, hd, page_size, window, n_seg, 0, scale};
  const bool wide = wide_rows(max_rows, hd, (long long)nkv * n_seqs, ceil_div(max_len, SEG));
  if (dtype == LLM_F32) {
    // 16-byte copies of cache rows: a row is hd float32
    if (hd % 4 == 0 && ((reinterpret_cast<uintptr_t>(kcache) | reinterpret_cast<uintptr_t>(vcache)) & 15u) == 0) launch<float, true>(p, n_seqs, max_rows, wide, stream);
    else launch<float, false>(p, n_seqs, max_rows, wide, stream);
    if (n_seg > 1) launch_kernel(paged_attention_simt_merge_kernel<float>, ceil_div((long long)n_tokens * nq, 4), 128, 0, stream, p, positions, n_tokens);
  } else if (dtype == LLM_BF16) {
    if (hd % 4 == 0 && ((reinterpret_cast<uintptr_t>(kcache) | reinterpret_cast<uintptr_t>(vcache)) & 7u) == 0) launch<bf16, true>(p, n_seqs, max_rows, wide, stream);
    else launch<bf16, false>(p, n_seqs, max_rows, wide, stream);
    if (n_seg > 1) launch_kernel(paged_attention_simt_merge_kernel<bf16>, ceil_div((long long)n_tokens * nq, 4), 128, 0, stream, p, positions, n_tokens);
  } else
    LLM_REQUIRE(false, "attention: unknown dtype %d", dtype);
  LLM_CHECK_LAUNCH("paged_attention_simt");
  return LLM_OK;
}
