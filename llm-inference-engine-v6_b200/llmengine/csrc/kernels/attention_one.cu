// Float32 attention of steps in which every request brings one token, on CUDA cores: up to 8 query heads a key/value head, rows of four
// float32 on 16 bytes. The arithmetic of attention_simt.cu, so its bits, with one latency after the other taken out. The CTAs of a request
// and key/value head are a cluster that shares its segments (segment s is CTA s modulo its size's) and merges them out of one another's
// shared memory, without scratch and a second kernel; tables are read ahead of the wait (they are the step's own input), all keys and values
// of a segment are requested at once, a thread has a key's scores, then a dimension's sums of a row. Calls one
// behind the other, us, against segments and a merge or CTAs that walk: 8 key/value heads of 64, 4 query heads each, 8 tokens behind 512 keys 11.5,
// 21.6; 4 behind 4,000 38.7, 68.0; 64 behind 1,000 93.4, 135.9; 1 behind 8,000 47.3, 75.4; 1 head of 32, 6 query heads, 4 tokens behind 64 4.6, 8.0.
// Of 316 sizes of 1 to 64 tokens behind 64 to 8,000 keys all were faster.
//
// A file of its own: in one with the kernels of attention_simt.cu the compiler gave those 77 registers a thread instead of 64, three CTAs a
// multiprocessor instead of four, and 64 tokens behind 2,000 keys took 391 us a layer instead of 268.
#include "attention_simt.cuh"

#include <cooperative_groups.h>

using namespace simt_attention;

namespace {

constexpr int ONE_THREADS = 256, ONE_ROWS = 8, ONE_CTAS = 8, ONE_SLOTS = 8;  // segments of a CTA at most

// RM: rows of a thread's scores; NO: rows of a thread's sums.
template <int RM, int NO>
__global__ void __launch_bounds__(ONE_THREADS, NO <= 2 ? 4 : 2) paged_attention_simt_one_kernel(const AttArgs p) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) float smem[];
  __shared__ long long s_key[SEG];
  cg::cluster_group cluster = cg::this_cluster();
  const int ctas = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int kvh = blockIdx.y, seq = blockIdx.z, group = p.nq / p.nkv, hd = p.hd, chunks = hd / 4, row_len = hd + 4;
  float* keys = smem;                          // [SEG][row_len]
  float* values = keys + SEG * row_len;        // [SEG / 2][hd]: of the first half of the segment; the second takes the keys' place
  float* qs = values + SEG / 2 * hd;           // [group][row_len]
  float* ss = qs + group * row_len;            // [group][S_ROW]
  float* found = ss + group * S_ROW;           // [slot][group][row_len]: a segment's sums, its largest score, its sum of weights
  dep_launch();
  const bool there = p.seq_ntok[seq] > 0;
  const int pos = p.seq_start[seq], tok = p.seq_qoff[seq];
  const int from = p.window > 0 ? max(0, pos - p.window + 1) : 0, first = from / SEG, last = there ? pos / SEG : first - 1;
  const int* table = p.table + (size_t)seq * p.max_blocks;
  const int at_key = tid / chunks, at_dim = (tid - at_key * chunks) * 4, at_once = ONE_THREADS / chunks;  // a thread copies four dimensions of every so many keys
  auto find_keys = [&](int seg) {
    for (int i = tid; i < SEG; i += ONE_THREADS) {
      const int key = seg * SEG + i;
      s_key[i] = key >= from && key <= pos ? (((long long)table[key / p.page] * p.nkv + kvh) * p.page + key % p.page) * hd : -1;
    }
    __syncthreads();
  };
  int seg = first + (rank - first % ctas + ctas) % ctas;  // the first of this CTA's: seg % ctas == rank
  if (seg <= last) find_keys(seg);
  dep_wait();
  for (int i = tid; i < group * chunks; i += ONE_THREADS) {
    const int r = i / chunks, c = i - r * chunks;
    if (there) copy4(qs + r * row_len + 4 * c, (const float*)p.q + (size_t)tok * p.ld_q + (size_t)(kvh * group + r) * hd + 4 * c, 4);
  }
  for (int turn = 0; seg <= last; seg += ctas, ++turn) {
    const int k0 = seg * SEG, lo = max(from - k0, 0), n_keys = min(SEG, pos - k0 + 1);  // the segment's keys lo .. n_keys - 1 are seen
    if (turn > 0) {
      __syncthreads();  // the segment before this one has been read
      find_keys(seg);
    }
    auto load = [&](const void* cache, float* dst, int stride, int begin, int end) {  // key `begin` of the segment goes to dst
      if (at_key < at_once)
        for (int key = begin + at_key; key < end; key += at_once) copy4(dst + (key - begin) * stride + at_dim, (const float*)cache + s_key[key] + at_dim, 4);
      commit_group();
    };
    const int middle = max(lo, min(SEG / 2, n_keys));
    load(p.k, keys + lo * row_len, row_len, lo, n_keys);
    load(p.v, values, hd, lo, middle);
    wait_groups<1>();
    __syncthreads();
    {
      const int key = tid % SEG, r0 = tid / SEG;  // rows r0, r0 + 2, ...
      float s[RM];
#pragma unroll
      for (int j = 0; j < RM; ++j) s[j] = 0.f;
      if (key >= lo && key < n_keys) {
        const float* kt = keys + key * row_len;
        const float* qt = qs + r0 * row_len;
#pragma unroll 4
        for (int d = 0; d < hd; d += 4) {
          const float4 kv = *reinterpret_cast<const float4*>(kt + d);
#pragma unroll
          for (int j = 0; j < RM; ++j) {
            const float4 qv = *reinterpret_cast<const float4*>(qt + min(2 * j, group - 1 - r0) * row_len + d);
#pragma unroll
            for (int e = 0; e < 4; ++e) s[j] = fmaf(part(qv, e), part(kv, e), s[j]);
          }
        }
      }
#pragma unroll
      for (int j = 0; j < RM; ++j)
        if (r0 + 2 * j < group) ss[(r0 + 2 * j) * S_ROW + key] = key >= lo && key < n_keys ? s[j] * p.scale : -INFINITY;
    }
    __syncthreads();
    load(p.v, keys, hd, middle, n_keys);
    float* mine = found + turn * group * row_len;
    if (warp < group) {
      float4 v = *reinterpret_cast<const float4*>(ss + warp * S_ROW + 4 * lane);
      const float m = warp_max(fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)));
      v.x = v.x == -INFINITY ? 0.f : expf(v.x - m);
      v.y = v.y == -INFINITY ? 0.f : expf(v.y - m);
      v.z = v.z == -INFINITY ? 0.f : expf(v.z - m);
      v.w = v.w == -INFINITY ? 0.f : expf(v.w - m);
      const float l = warp_sum((v.x + v.y) + (v.z + v.w));
      *reinterpret_cast<float4*>(ss + warp * S_ROW + 4 * lane) = v;
      if (lane == 0) {
        mine[warp * row_len + hd] = m;
        mine[warp * row_len + hd + 1] = l;
      }
    }
    // a thread has a dimension of NO rows
    float av[NO];
    const int sums = tid / hd, dim = tid - sums * hd;
    const float* pt[NO];
#pragma unroll
    for (int o = 0; o < NO; ++o) {
      av[o] = 0.f;
      pt[o] = ss + min(sums * NO + o, group - 1) * S_ROW;
    }
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      if (half == 0) wait_groups<1>();
      else wait_groups<0>();
      __syncthreads();
      if (sums * NO >= group) continue;
      const int begin = half ? middle : lo, end = half ? n_keys : middle;
      const float* vt = (half ? keys : values) - begin * hd + dim;
      int key = begin;
      for (; key < end && key % 8 != 0; ++key)
#pragma unroll
        for (int o = 0; o < NO; ++o) av[o] = fmaf(pt[o][key], vt[key * hd], av[o]);
      for (; key + 8 <= end; key += 8) {
        float x[8];
        float4 w[NO][2];
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = vt[(key + e) * hd];
#pragma unroll
        for (int o = 0; o < NO; ++o) {
          w[o][0] = *reinterpret_cast<const float4*>(pt[o] + key);
          w[o][1] = *reinterpret_cast<const float4*>(pt[o] + key + 4);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e)
#pragma unroll
          for (int o = 0; o < NO; ++o) av[o] = fmaf(part(w[o][e / 4], e % 4), x[e], av[o]);
      }
      for (; key < end; ++key)
#pragma unroll
        for (int o = 0; o < NO; ++o) av[o] = fmaf(pt[o][key], vt[key * hd], av[o]);
    }
#pragma unroll
    for (int o = 0; o < NO; ++o)
      if (sums * NO + o < group) mine[(sums * NO + o) * row_len + dim] = av[o];
  }
  cluster.sync();
  for (int at = rank * ONE_THREADS + tid; there && at < group * hd; at += ctas * ONE_THREADS) {
    const int r = at / hd, d = at - r * hd;
    float acc = 0.f, m = -INFINITY, l = 0.f;
    for (int s0 = first; s0 <= last; s0 += 8) {
      float o[8], m_s[8], l_s[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (s0 + i > last) break;
        const int owner = (s0 + i) % ctas, slot = (s0 + i - (first + (owner - first % ctas + ctas) % ctas)) / ctas;
        const float* row = cluster.map_shared_rank(found, owner) + (slot * group + r) * row_len;
        o[i] = row[d];
        m_s[i] = row[hd];
        l_s[i] = row[hd + 1];
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (s0 + i > last) break;
        float m_new, a, b;
        join_weights(m, m_s[i], m_new, a, b);
        m = m_new;
        l = join(l, a, l_s[i], b);
        acc = join(acc, a, o[i], b);
      }
    }
    const float inv = 1.0f / l;
    ((float*)p.out)[(size_t)tok * p.ld_out + (size_t)kvh * group * hd + at] = acc * inv;
  }
  cluster.sync();  // nobody leaves while its sums are being read
}

// CTAs of a cluster: a segment each, as long as all clusters run at a time (four CTAs a multiprocessor with heads of 64): what a
// context does not need of them they hold for nothing.
int one_ctas(int n_seqs, int max_len, int nkv) {
  return max(1, min(min(ceil_div(max_len, SEG), ONE_CTAS), (int)(4LL * simt_sm_count() / ((long long)n_seqs * nkv))));
}
template <int RM, int NO>
void launch_one(const AttArgs& p, int n_seqs, int max_len, cudaStream_t stream) {
  const int n_seg = ceil_div(max_len, SEG), ctas = one_ctas(n_seqs, max_len, p.nkv), slots = ceil_div(n_seg, ctas), group = p.nq / p.nkv, row_len = p.hd + 4;
  const int smem = (SEG * row_len + SEG / 2 * p.hd + group * (row_len + S_ROW) + slots * group * row_len) * 4;
  auto kernel = paged_attention_simt_one_kernel<RM, NO>;
  static std::atomic<unsigned long long> done{0};
  constexpr int most = (SEG * 132 + SEG / 2 * 128 + ONE_ROWS * (132 + S_ROW) + ONE_SLOTS * ONE_ROWS * 132) * 4;
  static_assert(most <= 224 * 1024, "shared memory of a CTA");
  static_assert(4 * (ONE_THREADS / 128) >= ONE_ROWS, "sets of four rows take every group");
  allow_smem(kernel, most, done);
  launch_kernel_cluster(kernel, dim3((unsigned)ctas, (unsigned)p.nkv, (unsigned)n_seqs), ONE_THREADS, smem, dim3((unsigned)ctas), stream, p);
}

}  // namespace

// Whether a step runs on the kernel above: one token a request and at most ONE_SLOTS segments a CTA of the largest cluster.
bool simt_attention::one_token(int n_seqs, int max_new, int max_len, int nq, int nkv, int hd) {
  return max_new == 1 && n_seqs <= 65535 && nkv <= 65535 && nq / nkv <= ONE_ROWS && hd % 4 == 0 && hd <= 128 &&
         ceil_div(max_len, SEG) <= one_ctas(n_seqs, max_len, nkv) * ONE_SLOTS;
}

// A row's sums take hd whole threads: ONE_THREADS / hd sets of them, one, two or four rows each (four always suffice: hd <= 128).
void simt_attention::launch_one_token(const AttArgs& p, int n_seqs, int max_len, cudaStream_t stream) {
  const int group = p.nq / p.nkv, sets = ONE_THREADS / p.hd, rm = group <= 2 ? 0 : group <= 4 ? 1 : 2, no = group == 1 ? 0 : 2 * sets >= group ? 1 : 2;
  constexpr void (*const forms[3][3])(const AttArgs&, int, int, cudaStream_t) = {{launch_one<1, 1>, launch_one<1, 2>, launch_one<1, 4>},
                                                                                 {launch_one<2, 1>, launch_one<2, 2>, launch_one<2, 4>},
                                                                                 {launch_one<4, 1>, launch_one<4, 2>, launch_one<4, 4>}};
  forms[rm][no](p, n_seqs, max_len, stream);
}
