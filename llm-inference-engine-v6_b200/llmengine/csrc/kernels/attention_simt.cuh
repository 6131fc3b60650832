// What the two files of float32 attention on CUDA cores share: attention_simt.cu and attention_one.cu.
#pragma once

#include "simt_common.cuh"

#include <cfloat>
#include <cmath>

namespace simt_attention {

constexpr int SEG = 128;  // keys of a segment
constexpr int S_ROW = SEG + 4;

struct AttArgs {
  const void *q, *k, *v;
  void* out;
  const int *seq_start, *seq_ntok, *seq_qoff, *table;
  float* scratch;  // [token, query head][segment][hd + 2]: sums, m, l; null: one CTA walks over all segments
  long long ld_q, ld_out;
  int max_blocks, nq, nkv, hd, page, window, n_seg, row_tiles;
  float scale;
};

// acc and l of the segments so far, with the largest score m, joined with those of one more segment. A largest score of -inf does not
// say that a segment holds nothing: NaNs are passed over by a maximum and stay in l and the sums, which keep them whatever their weight.
__device__ __forceinline__ void join_weights(float m, float m_s, float& m_new, float& a, float& b) {
  m_new = fmaxf(m, m_s);
  a = m == -INFINITY ? 0.f : expf(m - m_new);
  b = m_s == -INFINITY ? 0.f : expf(m_s - m_new);
}
__device__ __forceinline__ float join(float x, float a, float x_s, float b) { return fmaf(x, a, __fmul_rn(x_s, b)); }

// attention_one.cu: whether a step of float32 rows on 16 bytes runs on its kernel, and the launch (of AttArgs without scratch).
bool one_token(int n_seqs, int max_new, int max_len, int nq, int nkv, int hd);
void launch_one_token(const AttArgs& p, int n_seqs, int max_len, cudaStream_t stream);

}  // namespace simt_attention
