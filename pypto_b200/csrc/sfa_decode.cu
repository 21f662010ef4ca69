// Sparse MLA attention over the rows selected by the indexer (decode and prefill entries): which kernel takes a call,
// and the merge of split partials.
//
// Per query token (b, i):  n = clamp(S_b - s1 + 1 + i, 0, topk); for the first n indices
//   r_j = block_table[b, idx_j / bs] * bs + idx_j % bs
//   kn  = int8 latent[r_j] * scale[r_j, c / 128],   K = [kn | rope[r_j]]  (576 wide)
//   s   = fp32(q . K^T) * softmax_scale;  P = softmax(s);  O = bf16( P . kn )           (512 wide)
// (reference: examples/models/deepseek_v32_exp/sparse_flash_attention_quant_impl.py:45-207; golden
// deepseekv32_sparse_flash_attention_quant.py:169-254; packed rows
// sparse_attention_antiquant_impl.py:45-243.)
#include "common.cuh"
#include "sfa_common.cuh"

namespace pto {

namespace {

constexpr int kDV = 512;  // v width

// Merge of the split partials: O = sum_i O_i 2^(m_i - m) / sum_i l_i 2^(m_i - m), rounded once to bf16.
// One row is a token's head: 512 values of each split. What bounds it is the chain wait -> read -> write behind the
// attention kernel, so a warp asks for the splits' maxima and sums and for the rows of up to kGroup splits at once, weighs
// them by shuffles (no barrier), and a split without rows, whose partial was never written, is dropped behind the load.
// kWarps warps per row: four where there are more than four splits (few tokens: rows are few, splits many), else one, so that
// the rows of many tokens are one wave of blocks: the attention kernel's registers leave these blocks no room before it
// ends. (One block per row, maxima first: 8.9 us behind the attention kernel at 33 tokens x 2 splits, 3.7 at 2 x 16.)
constexpr int kMaxSplit = 32;
template <int kWarps>
__global__ void __launch_bounds__(128)
sfa_combine_kernel(SfaParams p, int rows) {
  constexpr int kVec = 4 / kWarps;                 // float4 per lane and split
  constexpr int kGroup = kWarps == 1 ? 4 : 16;     // splits asked for together
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int th = blockIdx.x * (4 / kWarps) + warp / kWarps;  // (token - split_begin) * nq + head
  pdl_wait();  // launched with programmatic serialization behind the kernel that writes the partials
  if (th >= rows) return;
  const int pt = th / p.nq, ti = p.split_begin + pt, head = th % p.nq;
  const int64_t prow0 = static_cast<int64_t>(pt) * p.n_split * p.nq + head;  // row of split 0; splits are nq rows apart
  const int col = (warp % kWarps) * 128 + lane * 4;                          // first value of this lane; the next float4 128 on
  float mi = -INFINITY, li = 0.f;
  if (lane < p.n_split) {
    const float2 ml = *reinterpret_cast<const float2*>(p.part_ml + (prow0 + static_cast<int64_t>(lane) * p.nq) * 2);
    mi = ml.x;
    li = ml.y;
  }
  float4 acc[kVec];
#pragma unroll
  for (int c = 0; c < kVec; ++c) acc[c] = make_float4(0.f, 0.f, 0.f, 0.f);
  float w_lane = 0.f, inv = 0.f;
  for (int s0 = 0; s0 < p.n_split; s0 += kGroup) {
    float4 v[kGroup][kVec];
#pragma unroll
    for (int u = 0; u < kGroup; ++u) {
      const float* src = p.part_o + (prow0 + static_cast<int64_t>(s0 + u) * p.nq) * kDV + col;
#pragma unroll
      for (int c = 0; c < kVec; ++c) {
        v[u][c] = s0 + u < p.n_split ? *reinterpret_cast<const float4*>(src + 128 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    if (s0 == 0) {
      float m = mi;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      w_lane = (li > 0.f && m != -INFINITY) ? ex2f(mi - m) : 0.f;
      float l = li * w_lane;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
      inv = l > 0.f ? 1.f / l : 0.f;
    }
#pragma unroll
    for (int u = 0; u < kGroup; ++u) {
      const float w = __shfl_sync(0xffffffffu, w_lane, (s0 + u) & 31);
      if (s0 + u >= p.n_split || w == 0.f) continue;
#pragma unroll
      for (int c = 0; c < kVec; ++c) {
        acc[c].x += v[u][c].x * w;
        acc[c].y += v[u][c].y * w;
        acc[c].z += v[u][c].z * w;
        acc[c].w += v[u][c].w * w;
      }
    }
  }
  __nv_bfloat16* dst = p.out + (static_cast<int64_t>(ti) * p.nq_total + p.head_begin + head) * kDV + col;
#pragma unroll
  for (int c = 0; c < kVec; ++c) {
    uint2 pk;
    pk.x = pack_bf16x2(acc[c].x * inv, acc[c].y * inv);
    pk.y = pack_bf16x2(acc[c].z * inv, acc[c].w * inv);
    *reinterpret_cast<uint2*>(dst + 128 * c) = pk;
  }
}

}  // namespace

cudaError_t launch_sfa(const SfaParams& p, int num_sms, cudaStream_t stream) {
  const int t = p.b * p.s1;
  // all 128 heads of a token: a pair of SMs that shares every MMA (sfa_pair.cu; int8, packed and bf16 caches); other
  // head counts: one SM per token and block of 16 or 32 heads, the rows as the M dimension (sfa_slice.cu)
  cudaError_t e = p.nq == 128 ? launch_sfa_pair(p, stream) : launch_sfa_slice(p, num_sms, stream);
  if (e != cudaSuccess) return e;
  if (p.n_split > 1) {
    if (p.n_split > kMaxSplit) return cudaErrorInvalidValue;
    count_launch();
    // may be scheduled while the attention kernel drains; its first instruction waits for that grid
    const int rows = (t - p.split_begin) * p.nq;
    e = p.n_split > 4 ? launch_maybe_pdl(sfa_combine_kernel<4>, dim3(rows), dim3(128), 0, stream, true, p, rows)
                      : launch_maybe_pdl(sfa_combine_kernel<1>, dim3((rows + 3) / 4), dim3(128), 0, stream, true, p, rows);
  }
  return e;
}

}  // namespace pto
