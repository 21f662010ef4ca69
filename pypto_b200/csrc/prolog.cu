// MLA + lightning-indexer prolog: everything between the projections (the weight-streaming products of
// prolog_gemm.cu and prolog_sgemm.cu, issued by the C entry point) — RMSNorm / LayerNorm, rope, Hadamard rotation, dynamic int8 quantisation, dequantisation of
// the int32 products, and the scatter of the new token's rows into the paged caches.
//
// Arithmetic follows the reference's torch goldens step by step, including every intermediate rounding to
// bf16 (examples/models/deepseek_v32_exp/deepseekv32_mla_indexer_prolog_quant.py: `quant` :35-53,
// `rms_norm` :56-73, `apply_rotary_pos_emb_v2` :106-131, `single_rope` :140-152, `layer_norm` :155-162,
// `mla_prolog_quant_v32_compute` :409-541, `indexer_prolog` :544-614). Products and sums that the goldens
// round separately are kept separate here (`__fmul_rn` / `__fadd_rn`, no contraction into FMAs).
#include "common.cuh"

namespace pto {

namespace {

constexpr int kHeads = 128;     // attention heads
constexpr int kNope = 128;      // per-head query width before absorption
constexpr int kRope = 64;       // rope width (attention and indexer)
constexpr int kLora = 512;      // latent KV width
constexpr int kIdxHeads = 64;   // indexer heads
constexpr int kIdxDim = 128;    // indexer head width
constexpr int kQHead = kNope + kRope;
constexpr int kPackedRow = kLora + 2 * kRope + 16;  // 656 bytes: int8 latent | bf16 rope | 4 fp32 scales

__device__ __forceinline__ float bf16_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ float ld_bf16(const __nv_bfloat16* p) { return __bfloat162float(*p); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Block-wide reductions over up to 32 warps; `red` holds 32 floats. The result is returned to every thread.
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();  // `red` may still be read from a previous reduction
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float r = lane < nw ? red[lane] : 0.f;
  return warp_sum(r);
}
__device__ __forceinline__ float block_max(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float r = lane < nw ? red[lane] : 0.f;  // maxima of absolute values: 0 is neutral
  return warp_max(r);
}

// round(x * 127/max) -> int32 -> fp16 -> trunc -> int8: integers up to 127 are exact in fp16, so the chain
// after the round-half-even is the identity
__device__ __forceinline__ int8_t quant_one(float v, float scale_q) {
  return static_cast<int8_t>(__float2int_rn(__fmul_rn(v, scale_q)));
}

// ---- query down-projection: bf16 rounding, RMSNorm, then per-token int8 (kQuant) or the bf16 row itself ----
// grid = tokens, 512 threads, dynamic shared memory = q_lora floats (16-byte aligned rows: ld and q_lora multiples of 4)
template <bool kQuant>
__global__ void __launch_bounds__(512)
prolog_qnorm_kernel(const float* qa, int ld, int n_split, long long split_stride,
                    const __nv_bfloat16* __restrict__ gamma, int q_lora, float eps, int8_t* __restrict__ q_norm,
                    float* __restrict__ q_norm_scale, __nv_bfloat16* __restrict__ q_norm_bf16) {
  extern __shared__ __align__(16) float row[];
  __shared__ float red[32];
  // First the trigger: the product behind this kernel fills its rings with weights meanwhile. What is no kernel's result is
  // requested before the wait too: while weights stream, a read that misses L2 takes some microseconds. (Here and below.)
  if (threadIdx.x == 0) pdl_trigger();
  uint2 gm0 = make_uint2(0u, 0u);  // four bf16
  if (threadIdx.x < (q_lora >> 2)) gm0 = __ldg(reinterpret_cast<const uint2*>(gamma) + threadIdx.x);
  pdl_wait();  // the projection before it may still be running when this grid is scheduled
  const int ti = blockIdx.x;
  const float4* src = reinterpret_cast<const float4*>(qa + static_cast<int64_t>(ti) * ld);
  float4* row4 = reinterpret_cast<float4*>(row);
  const int groups = q_lora >> 2;  // four values per step: at q_lora = 1536 every thread makes one trip to memory
  const float inv_n = 1.0f / static_cast<float>(q_lora);
  float ss = 0.f;
  for (int g = threadIdx.x; g < groups; g += blockDim.x) {
    float4 part[8];  // K-split partials of the projection (n_split <= 8): requested together, added in split order
#pragma unroll
    for (int sp = 0; sp < 8; ++sp) {
      part[sp] = sp < n_split ? src[g + sp * (split_stride >> 2)] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float4 v = part[0];
#pragma unroll
    for (int sp = 1; sp < 8; ++sp) {
      if (sp < n_split) {
        v.x = __fadd_rn(v.x, part[sp].x);
        v.y = __fadd_rn(v.y, part[sp].y);
        v.z = __fadd_rn(v.z, part[sp].z);
        v.w = __fadd_rn(v.w, part[sp].w);
      }
    }
    v.x = bf16_round(v.x);
    v.y = bf16_round(v.y);
    v.z = bf16_round(v.z);
    v.w = bf16_round(v.w);
    row4[g] = v;
    ss = __fadd_rn(ss, __fmul_rn(__fmul_rn(v.x, v.x), inv_n));
    ss = __fadd_rn(ss, __fmul_rn(__fmul_rn(v.y, v.y), inv_n));
    ss = __fadd_rn(ss, __fmul_rn(__fmul_rn(v.z, v.z), inv_n));
    ss = __fadd_rn(ss, __fmul_rn(__fmul_rn(v.w, v.w), inv_n));
  }
  const float rms = sqrtf(block_sum(ss, red) + eps);
  float amax = 0.f;
  for (int g = threadIdx.x; g < groups; g += blockDim.x) {
    float4 v = row4[g];
    const uint2 gm = g == threadIdx.x ? gm0 : __ldg(reinterpret_cast<const uint2*>(gamma) + g);
    v.x = bf16_round(__fmul_rn(__fdiv_rn(v.x, rms), __uint_as_float(gm.x << 16)));
    v.y = bf16_round(__fmul_rn(__fdiv_rn(v.y, rms), __uint_as_float(gm.x & 0xffff0000u)));
    v.z = bf16_round(__fmul_rn(__fdiv_rn(v.z, rms), __uint_as_float(gm.y << 16)));
    v.w = bf16_round(__fmul_rn(__fdiv_rn(v.w, rms), __uint_as_float(gm.y & 0xffff0000u)));
    if constexpr (kQuant) {
      row4[g] = v;
      amax = fmaxf(fmaxf(amax, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
    } else {
      uint2 o;  // the values are bf16 already: their upper halves are the row
      o.x = (__float_as_uint(v.x) >> 16) | (__float_as_uint(v.y) & 0xffff0000u);
      o.y = (__float_as_uint(v.z) >> 16) | (__float_as_uint(v.w) & 0xffff0000u);
      reinterpret_cast<uint2*>(q_norm_bf16 + static_cast<int64_t>(ti) * q_lora)[g] = o;
    }
  }
  if constexpr (!kQuant) return;
  amax = block_max(amax, red);
  const float scale_q = __fdiv_rn(127.0f, amax);
  char4* dst = reinterpret_cast<char4*>(q_norm + static_cast<int64_t>(ti) * q_lora);
  for (int g = threadIdx.x; g < groups; g += blockDim.x) {
    const float4 v = row4[g];
    char4 q;
    q.x = quant_one(v.x, scale_q);
    q.y = quant_one(v.y, scale_q);
    q.z = quant_one(v.z, scale_q);
    q.w = quant_one(v.w, scale_q);
    dst[g] = q;
  }
  if (threadIdx.x == 0) q_norm_scale[ti] = __fdiv_rn(1.0f, scale_q);
}

// The same for many tokens and rows of at most kNormRow values: 128 threads a row, which stays in registers. The kernel above holds two
// rows an SM at a time (registers), so 1000 tokens were three and a half rounds of loads and block reductions; here all rows of 1000
// tokens are on the chip at once (22 -> 7 us from the projections' end; whole prolog, us: 512 tokens 93.7 -> 93.6, 600 112.8 -> 109.5,
// 1000 148.2 -> 141.6, 4096 522 -> 498). With few rows it loses (200 63.6 -> 65.9, 384 83.7 -> 85.4): K is split more often there, and
// this kernel asks for two of the partials at a time. Sums in the same order, the same bits: the 128 values of group w of 32 threads there are those of
// step w / 4 of warp w % 4 here.
constexpr int kNormRow = 2048, kNormManyRows = 512;
template <bool kQuant>
__global__ void __launch_bounds__(128)
prolog_qnorm_many_kernel(const float* qa, int ld, int n_split, long long split_stride, const __nv_bfloat16* __restrict__ gamma, int q_lora,
                         float eps, int8_t* __restrict__ q_norm, float* __restrict__ q_norm_scale, __nv_bfloat16* __restrict__ q_norm_bf16) {
  constexpr int kSteps = kNormRow / 512;
  __shared__ float red[32];
  if (threadIdx.x == 0) pdl_trigger();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int groups = q_lora >> 2;
  uint2 gm[kSteps];  // four bf16 each
#pragma unroll
  for (int j = 0; j < kSteps; ++j) {
    const int g = threadIdx.x + 128 * j;
    gm[j] = g < groups ? __ldg(reinterpret_cast<const uint2*>(gamma) + g) : make_uint2(0u, 0u);
  }
  if (threadIdx.x < 32) red[threadIdx.x] = 0.f;
  pdl_wait();
  const int ti = blockIdx.x;
  const float4* src = reinterpret_cast<const float4*>(qa + static_cast<int64_t>(ti) * ld);
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 v[kSteps], next[kSteps];  // K-split partials, added in split order; the next ones are on their way meanwhile
#pragma unroll
  for (int j = 0; j < kSteps; ++j) {
    const int g = threadIdx.x + 128 * j;
    v[j] = g < groups ? src[g] : zero;
    next[j] = g < groups && n_split > 1 ? src[g + (split_stride >> 2)] : zero;
  }
  for (int sp = 1; sp < n_split; ++sp) {
#pragma unroll
    for (int j = 0; j < kSteps; ++j) {
      const int g = threadIdx.x + 128 * j;
      v[j].x = __fadd_rn(v[j].x, next[j].x);
      v[j].y = __fadd_rn(v[j].y, next[j].y);
      v[j].z = __fadd_rn(v[j].z, next[j].z);
      v[j].w = __fadd_rn(v[j].w, next[j].w);
      if (g < groups && sp + 1 < n_split) next[j] = src[g + (sp + 1) * (split_stride >> 2)];
    }
  }
  const float inv_n = 1.0f / static_cast<float>(q_lora);
  float ss[kSteps];
#pragma unroll
  for (int j = 0; j < kSteps; ++j) {
    v[j] = make_float4(bf16_round(v[j].x), bf16_round(v[j].y), bf16_round(v[j].z), bf16_round(v[j].w));
    ss[j] = __fmul_rn(__fmul_rn(v[j].x, v[j].x), inv_n);
    ss[j] = __fadd_rn(ss[j], __fmul_rn(__fmul_rn(v[j].y, v[j].y), inv_n));
    ss[j] = __fadd_rn(ss[j], __fmul_rn(__fmul_rn(v[j].z, v[j].z), inv_n));
    ss[j] = __fadd_rn(ss[j], __fmul_rn(__fmul_rn(v[j].w, v[j].w), inv_n));
    ss[j] = warp_sum(ss[j]);
  }
  __syncthreads();  // `red` is zero
  if (lane == 0) {
#pragma unroll
    for (int j = 0; j < kSteps; ++j) red[4 * j + warp] = ss[j];
  }
  __syncthreads();
  const float rms = sqrtf(warp_sum(red[lane]) + eps);
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < kSteps; ++j) {
    const int g = threadIdx.x + 128 * j;
    if (g >= groups) break;
    v[j].x = bf16_round(__fmul_rn(__fdiv_rn(v[j].x, rms), __uint_as_float(gm[j].x << 16)));
    v[j].y = bf16_round(__fmul_rn(__fdiv_rn(v[j].y, rms), __uint_as_float(gm[j].x & 0xffff0000u)));
    v[j].z = bf16_round(__fmul_rn(__fdiv_rn(v[j].z, rms), __uint_as_float(gm[j].y << 16)));
    v[j].w = bf16_round(__fmul_rn(__fdiv_rn(v[j].w, rms), __uint_as_float(gm[j].y & 0xffff0000u)));
    if constexpr (kQuant) {
      amax = fmaxf(fmaxf(amax, fmaxf(fabsf(v[j].x), fabsf(v[j].y))), fmaxf(fabsf(v[j].z), fabsf(v[j].w)));
    } else {
      uint2 o;  // the values are bf16 already: their upper halves are the row
      o.x = (__float_as_uint(v[j].x) >> 16) | (__float_as_uint(v[j].y) & 0xffff0000u);
      o.y = (__float_as_uint(v[j].z) >> 16) | (__float_as_uint(v[j].w) & 0xffff0000u);
      reinterpret_cast<uint2*>(q_norm_bf16 + static_cast<int64_t>(ti) * q_lora)[g] = o;
    }
  }
  if constexpr (!kQuant) return;
  amax = block_max(amax, red);
  const float scale_q = __fdiv_rn(127.0f, amax);
  char4* dst = reinterpret_cast<char4*>(q_norm + static_cast<int64_t>(ti) * q_lora);
#pragma unroll
  for (int j = 0; j < kSteps; ++j) {
    const int g = threadIdx.x + 128 * j;
    if (g >= groups) break;
    char4 q;
    q.x = quant_one(v[j].x, scale_q);
    q.y = quant_one(v[j].y, scale_q);
    q.z = quant_one(v[j].z, scale_q);
    q.w = quant_one(v[j].w, scale_q);
    dst[g] = q;
  }
  if (threadIdx.x == 0) q_norm_scale[ti] = __fdiv_rn(1.0f, scale_q);
}

// Hadamard rotation of 16 rows (bf16, row pitch kIdxPitch, shared memory) by the warps' own matrix instruction (m16n8k16):
// 64 columns from col0, 16 * kSteps values of the contraction from k0; with kOneRow only row 0 is there. For few tokens only: the 128-row tile of the
// tensor-memory path would be mostly empty and its set-up costs as much as the kernels here take. The instruction wants two
// neighbours along k in one register where the matrix has two columns: a lane reads eight columns of four rows, 16 bytes each
// and exchanges halves in registers; column g of tile n is column 8 g + n of the 64. `h`: the matrix, rows
// kPitch apart: in global memory, or where the call waits for it in shared memory (pitch kIdxPitch, conflict-free for these
// reads), requested at once by hadamard_fetch: from L2 step by step each trip takes over a microsecond while weights stream.
// acc[n]: of row lane / 4 (first two) and lane / 4 + 8: columns 16 (lane % 4) + n and 16 (lane % 4) + 8 + n.
constexpr int kIdxPitch = kIdxDim + 8;  // the eight rows of a fragment fall into different banks
template <int kSteps, int kPitch, bool kOneRow>
__device__ __forceinline__ void hadamard_rows(const __nv_bfloat16* h, int k0, int col0, const __nv_bfloat16* rows,
                                              int lane, float (&acc)[8][4]) {
  const int g = lane >> 2, l4 = lane & 3;
#pragma unroll
  for (int n = 0; n < 8; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
#pragma unroll
  for (int ks = 0; ks < kSteps; ++ks) {
    const int k = k0 + ks * 16;
    uint32_t b[2][8];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const __nv_bfloat16* src = h + (k + half * 8 + 2 * l4) * kPitch + col0 + 8 * g;
      const uint4 even = *reinterpret_cast<const uint4*>(src);
      const uint4 odd = *reinterpret_cast<const uint4*>(src + kPitch);
      const uint32_t e[4] = {even.x, even.y, even.z, even.w}, o[4] = {odd.x, odd.y, odd.z, odd.w};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        b[half][2 * c] = __byte_perm(e[c], o[c], 0x5410);
        b[half][2 * c + 1] = __byte_perm(e[c], o[c], 0x7632);
      }
    }
    uint32_t a[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t* row = reinterpret_cast<const uint32_t*>(rows + (kOneRow ? 0 : (g + 8 * (i & 1)) * kIdxPitch) + k + 8 * (i >> 1) + 2 * l4);
      a[i] = !kOneRow || (g == 0 && (i & 1) == 0) ? *row : 0u;
    }
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
          : "+f"(acc[n][0]), "+f"(acc[n][1]), "+f"(acc[n][2]), "+f"(acc[n][3])
          : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0][n]), "r"(b[1][n]));
    }
  }
}
constexpr int kHadBytes = kIdxDim * kIdxPitch * 2;  // 34 KB
__device__ __forceinline__ void hadamard_fetch(const __nv_bfloat16* __restrict__ src, __nv_bfloat16* dst, int i, int n) {
  for (int u = i; u < kIdxDim * kIdxDim / 8; u += n) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst + (u >> 4) * kIdxPitch + (u & 15) * 8)), "l"(src + u * 8) : "memory");
  }
}
// `bytes` (a multiple of 128) at `p` into L2, by `n` threads of which this one is number `i`
__device__ __forceinline__ void prefetch_l2(const void* p, int bytes, int i, int n) {
  for (int at = i * 128; at < bytes; at += n * 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const uint8_t*>(p) + at));
}

// ---- query up-projection: int32 -> bf16, rope of the 64-wide tail ----------------------------------------
// grid = (16 head groups, tokens), block = 256: eight heads (1536 values) per block
constexpr int kQbHeadsPerBlock = 8;
__global__ void __launch_bounds__(256)
prolog_qb_dequant_rope_kernel(const int32_t* qb_i32, const float* q_norm_scale, const float* __restrict__ w_scale,
                              const __nv_bfloat16* __restrict__ cos, const __nv_bfloat16* __restrict__ sin,
                              __nv_bfloat16* __restrict__ q_b, __nv_bfloat16* __restrict__ q_rope) {
  // (the results of the kernels before this one are not __restrict__: loads of what nothing may write could be moved in
  // front of pdl_wait())
  __shared__ float pe[kQbHeadsPerBlock][kRope];
  const int ti = blockIdx.y, tid = threadIdx.x;
  // (CTAs of the product behind this kernel fill their rings while the up-projections end; the other stream's kernels are
  // first in line for what room there is)
  if (tid == 0) pdl_trigger();
  const int hg = blockIdx.x;
  const int64_t col0 = static_cast<int64_t>(hg) * kQbHeadsPerBlock * kQHead;
  const int64_t row0 = static_cast<int64_t>(ti) * kHeads * kQHead;
  float ws[kQbHeadsPerBlock * kQHead / 256];
#pragma unroll
  for (int u = 0; u < kQbHeadsPerBlock * kQHead / 256; ++u) ws[u] = __ldg(w_scale + col0 + u * 256 + tid);
  static_assert(256 % kRope == 0, "a thread rotates one dim of several heads");
  const int c = tid % kRope;
  const float cs = ld_bf16(cos + ti * kRope + c), sn = ld_bf16(sin + ti * kRope + c);
  pdl_wait();
  const float rs = q_norm_scale[ti];
  int32_t product[kQbHeadsPerBlock * kQHead / 256];
#pragma unroll
  for (int u = 0; u < kQbHeadsPerBlock * kQHead / 256; ++u) product[u] = qb_i32[row0 + col0 + u * 256 + tid];
#pragma unroll
  for (int u = 0; u < kQbHeadsPerBlock * kQHead / 256; ++u) {
    const int e = u * 256 + tid;  // element of the block's 8 x 192 slice
    const int64_t col = col0 + e;
    const float v = bf16_round(__fmul_rn(__fmul_rn(static_cast<float>(product[u]), rs), ws[u]));
    q_b[row0 + col] = __float2bfloat16_rn(v);
    const int hh = e / kQHead, d = e % kQHead;
    if (d >= kNope) pe[hh][d - kNope] = v;
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kQbHeadsPerBlock * kRope / 256; ++u) {
    const int hh = (u * 256 + tid) / kRope;
    // de-interleaved layout: first half = even dims, second half = odd dims; rotate_half = (-second, first)
    const int j = c & 31;
    const float even = pe[hh][2 * j], odd = pe[hh][2 * j + 1];
    const float x = c < 32 ? even : odd;
    const float rot = c < 32 ? -odd : even;
    q_rope[(static_cast<int64_t>(ti) * kHeads + hg * kQbHeadsPerBlock + hh) * kRope + c] =
        __float2bfloat16_rn(__fadd_rn(__fmul_rn(x, cs), __fmul_rn(rot, sn)));
  }
}

// ---- indexer query of few tokens: int32 -> bf16, rope, Hadamard rotation, per-head int8 -------------------------
// grid = tokens, block = 256: all 64 heads; a warp rotates 16 heads x 64 columns. On a second stream beside the absorbed
// query; its blocks (53 KB) find room on the SMs that hold three of that product's 512 CTAs instead of four. On CUDA cores with the matrix in
// shared memory (41 KB, eight heads a block) it waited for those CTAs and took 12.6 us at 64 tokens (7.9 at 3): it ended the call.
__global__ void __launch_bounds__(256)
prolog_idxq_kernel(const int32_t* __restrict__ qi_i32, const float* __restrict__ q_norm_scale,
                   const float* __restrict__ w_scale, const __nv_bfloat16* __restrict__ cos,
                   const __nv_bfloat16* __restrict__ sin, const __nv_bfloat16* __restrict__ hadamard_q,
                   int8_t* __restrict__ q_int8, __half* __restrict__ q_scale) {
  extern __shared__ __align__(16) __nv_bfloat16 had[];
  __shared__ __align__(16) __nv_bfloat16 q[kIdxHeads][kIdxPitch];
  __shared__ float half_amax[2][kIdxHeads];
  const int ti = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, l4 = lane & 3;
  hadamard_fetch(hadamard_q, had, tid, 256);
  {
    const int l = tid & 15;  // dims l, l + 16, ... of a head: a dim and its partner of the rotation are in one thread
    const float rs = q_norm_scale[ti];
    float cs[4], sn[4], scale[kIdxHeads / 16][8];
    int32_t product[kIdxHeads / 16][8];  // all requested before the first is used
#pragma unroll
    for (int u = 0; u < kIdxHeads / 16; ++u) {
      const int hh = u * 16 + (tid >> 4);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const void* a = qi_i32 + (static_cast<int64_t>(ti) * kIdxHeads + hh) * kIdxDim + l + 16 * j;
        const void* b = w_scale + hh * kIdxDim + l + 16 * j;
        asm volatile("ld.global.b32 %0, [%1];" : "=r"(product[u][j]) : "l"(a));
        asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(scale[u][j]) : "l"(b));
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      cs[j] = ld_bf16(cos + ti * kRope + l + 16 * j);
      sn[j] = ld_bf16(sin + ti * kRope + l + 16 * j);
    }
#pragma unroll
    for (int u = 0; u < kIdxHeads / 16; ++u) {
      const int hh = u * 16 + (tid >> 4);
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = bf16_round(__fmul_rn(__fmul_rn(static_cast<float>(product[u][j]), rs), scale[u][j]));
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float o = v[j];
        if (j < 4) {
          const float rot = j < 2 ? -v[j + 2] : v[j - 2];
          o = __fadd_rn(__fmul_rn(v[j], cs[j]), __fmul_rn(rot, sn[j]));
        }
        q[hh][l + 16 * j] = __float2bfloat16_rn(o);
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const int head0 = (warp >> 1) * 16, half = warp & 1;
  float acc[8][4];
  hadamard_rows<8, kIdxPitch, false>(had, 0, half * 64, &q[head0][0], lane, acc);
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    float m = 0.f;
#pragma unroll
    for (int n = 0; n < 8; ++n) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        acc[n][2 * r + e] = bf16_round(acc[n][2 * r + e]);
        m = fmaxf(m, fabsf(acc[n][2 * r + e]));
      }
    }
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
    if (l4 == 0) half_amax[half][head0 + g + 8 * r] = m;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int hh = head0 + g + 8 * r;
    const float sq = __fdiv_rn(127.0f, fmaxf(half_amax[0][hh], half_amax[1][hh]));
    const int64_t head = static_cast<int64_t>(ti) * kIdxHeads + hh;
    __align__(16) int8_t out[16];
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      out[n] = quant_one(acc[n][2 * r], sq);
      out[8 + n] = quant_one(acc[n][2 * r + 1], sq);
    }
    int8_t* dst = q_int8 + head * kIdxDim + half * 64 + 16 * l4;
    if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
      *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(out);
    } else {
#pragma unroll
      for (int e = 0; e < 16; ++e) dst[e] = out[e];
    }
    if (half == 0 && l4 == 0) q_scale[head] = __float2half_rn(__fdiv_rn(1.0f, sq));
  }
}

// ---- per token: latent KV row, rope key, indexer key, indexer weights; scatter into the caches ---------
// grid = tokens, block = 128 (thread i owns latent dims 4i..4i+3: warp w = 128-wide quantisation tile w). kMany: 64 registers, so
// that eight blocks share an SM and 1184 tokens are one round (the up-projections' CTAs need whole SMs and wait for the last block:
// whole prolog 770 tokens 131.7 -> 129.2 us, 1000 142.0 -> 140.1, 1100 168.7 -> 165.5; 600 109.9 -> 109.5; 32 bytes of a thread spill for it)
template <bool kMany>
__global__ void __launch_bounds__(128, kMany ? 8 : 0)
prolog_kv_kernel(const float* __restrict__ kv, const float* __restrict__ ki, const float* __restrict__ wp, int ld,
                 int n_split, long long split_stride, const __nv_bfloat16* __restrict__ gamma_ckv, const __nv_bfloat16* __restrict__ cos,
                 const __nv_bfloat16* __restrict__ sin, const __nv_bfloat16* __restrict__ ln_gamma,
                 const __nv_bfloat16* __restrict__ ln_beta, const __nv_bfloat16* __restrict__ hadamard_k,
                 const int64_t* __restrict__ cache_index, int64_t cache_rows, float eps_ckv, float ln_eps,
                 int8_t* __restrict__ kv_cache, __nv_bfloat16* __restrict__ kr_cache, float* __restrict__ kv_scale_cache,
                 int8_t* __restrict__ idx_k_cache, __half* __restrict__ idx_k_scale_cache, __half* __restrict__ weights,
                 int8_t* __restrict__ packed_cache, const void* next_hadamard, const void* next_scale, int32_t* status) {
  __shared__ float red[32];
  __shared__ float pe[kRope];
  __shared__ float kvec[kIdxDim];
  __shared__ __align__(16) __nv_bfloat16 krow[kIdxDim];  // the rotation's operand
  __shared__ float kpart[2][kIdxDim];
  const int ti = blockIdx.x, i = threadIdx.x, lane = i & 31, warp = i >> 5;
  if (!kMany || ti < 128) prefetch_l2(hadamard_k, 2 * kIdxDim * kIdxDim, i, 128);
  // for the indexer query's kernel, which would miss L2 while weights stream (some microseconds); each block a share
  prefetch_l2(next_hadamard, 2 * kIdxDim * kIdxDim, ti * 128 + i, gridDim.x * 128);
  prefetch_l2(next_scale, 4 * kIdxHeads * kIdxDim, ti * 128 + i, gridDim.x * 128);
  const int64_t row = cache_index[ti];
  float gm[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) gm[e] = ld_bf16(gamma_ckv + 4 * i + e);
  const float cs = ld_bf16(cos + ti * kRope + i % kRope), sn = ld_bf16(sin + ti * kRope + i % kRope);
  const float lg = ld_bf16(ln_gamma + i), lb = ld_bf16(ln_beta + i);
  const bool row_ok = row >= 0 && row < cache_rows;
  if (!row_ok && i == 0) set_status(status, PTO_ST_BAD_PAGE, static_cast<int>(row), 60);

  // a projection value: its K-split partials added in split order
  auto proj = [&](const float* p) {
    float part[8];  // all partials requested before the first is used (n_split <= 8)
#pragma unroll
    for (int sp = 0; sp < 8; ++sp) part[sp] = sp < n_split ? __ldg(p + sp * split_stride) : 0.f;
    float a = part[0];
#pragma unroll
    for (int sp = 1; sp < 8; ++sp) {
      if (sp < n_split) a = __fadd_rn(a, part[sp]);
    }
    return a;
  };
  // latent part: bf16 rounding, RMSNorm, int8 per 128-wide tile. Everything that the thread reads of the projections is
  // requested here, before the first sum over the block.
  const float* src = kv + static_cast<int64_t>(ti) * ld;
  const float x = proj(ki + static_cast<int64_t>(ti) * ld + i);
  const float tail = i < kRope ? proj(src + kLora + i) : proj(wp + static_cast<int64_t>(ti) * ld + (i - kRope));
  float v[4];
  float ss = 0.f;
#pragma unroll
  for (int e = 0; e < 4; ++e) v[e] = bf16_round(proj(src + 4 * i + e));
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    ss = __fadd_rn(ss, __fmul_rn(__fmul_rn(v[e], v[e]), 1.0f / kLora));
  }
  const float rms = sqrtf(block_sum(ss, red) + eps_ckv);
  float amax = 0.f;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    v[e] = bf16_round(__fmul_rn(__fdiv_rn(v[e], rms), gm[e]));
    amax = fmaxf(amax, fabsf(v[e]));
  }
  amax = warp_max(amax);
  const float scale_q = __fdiv_rn(127.0f, amax);
  if (row_ok) {
    char4 q;
    q.x = quant_one(v[0], scale_q);
    q.y = quant_one(v[1], scale_q);
    q.z = quant_one(v[2], scale_q);
    q.w = quant_one(v[3], scale_q);
    *reinterpret_cast<char4*>(kv_cache + row * kLora + 4 * i) = q;
    const float dq = __fdiv_rn(1.0f, scale_q);
    if (lane == 0) kv_scale_cache[row * 4 + warp] = dq;
    if (packed_cache != nullptr) {  // the same row in the packed layout: 512 int8 | 64 bf16 | 4 f32
      *reinterpret_cast<char4*>(packed_cache + row * kPackedRow + 4 * i) = q;
      if (lane == 0) *reinterpret_cast<float*>(packed_cache + row * kPackedRow + kLora + 2 * kRope + 4 * warp) = dq;
    }
  }

  // rope key: the 64 values after the latent part, de-interleaved rope
  if (i < kRope) pe[i] = bf16_round(tail);
  __syncthreads();
  if (i < kRope && row_ok) {
    const int j = i & 31;
    const float even = pe[2 * j], odd = pe[2 * j + 1];
    const float x = i < 32 ? even : odd;
    const float rot = i < 32 ? -odd : even;
    const __nv_bfloat16 kr = __float2bfloat16_rn(__fadd_rn(__fmul_rn(x, cs), __fmul_rn(rot, sn)));
    kr_cache[row * kRope + i] = kr;
    if (packed_cache != nullptr) *reinterpret_cast<__nv_bfloat16*>(packed_cache + row * kPackedRow + kLora + 2 * i) = kr;
  }

  // indexer key: LayerNorm in fp32 -> bf16, rope on the first 64 dims (halves, no de-interleave), Hadamard, int8
  const float mean = block_sum(x, red) * (1.0f / kIdxDim);
  const float dx = x - mean;
  const float var = block_sum(__fmul_rn(dx, dx), red) * (1.0f / kIdxDim);
  const float y = __fdiv_rn(dx, sqrtf(var + ln_eps));
  kvec[i] = bf16_round(__fadd_rn(__fmul_rn(y, lg), lb));
  __syncthreads();
  float k = kvec[i];
  if (i < kRope) {
    const float rot = i < 32 ? -kvec[i + 32] : kvec[i - 32];
    k = bf16_round(__fadd_rn(__fmul_rn(k, cs), __fmul_rn(rot, sn)));
  }
  krow[i] = __float2bfloat16_rn(k);
  __syncthreads();  // (and kvec has been read)
  {
    float acc[8][4];
    const int half = warp & 1, part = warp >> 1;  // warp: 64 columns, half of the contraction
    hadamard_rows<4, kIdxDim, true>(hadamard_k, part * 64, half * 64, krow, lane, acc);
    if (lane < 4) {
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        kpart[part][half * 64 + 16 * lane + n] = acc[n][0];
        kpart[part][half * 64 + 16 * lane + 8 + n] = acc[n][1];
      }
    }
  }
  __syncthreads();
  const float hk = bf16_round(__fadd_rn(kpart[0][i], kpart[1][i]));
  const float kmax = block_max(fabsf(hk), red);
  const float ksq = __fdiv_rn(127.0f, kmax);
  if (row_ok) {
    idx_k_cache[row * kIdxDim + i] = quant_one(hk, ksq);
    if (i == 0) idx_k_scale_cache[row] = __float2half_rn(__fdiv_rn(1.0f, ksq));
  }

  // indexer weights: bf16 rounding, then heads^-1/2 and dim^-1/2 in fp32, fp16 out
  if (i >= kRope) {
    const float w = bf16_round(tail);
    weights[static_cast<int64_t>(ti) * kIdxHeads + i - kRope] =
        __float2half_rn(__fmul_rn(__fmul_rn(w, 0.125f), 0.08838834764831845f));
  }
}

// ==== the two prologs of the non-quantised chain ===========================================================
// Arithmetic of the system tests' goldens: `mla_prolog_compute` without quantisation
// (framework/tests/st/operator/src/test_deepseek_v3.2_exp/gen_mla_prolog_golden_v32.py:176-303) and the
// non-quantised `indexer_prolog` (.../gen_lightning_indexer_prolog.py:253-293); operators
// `MlaPrologComputeV32` (framework/src/operator/models/deepseek_v3.2_exp/dynamic_mla_v32.cpp:187-345) and
// `LightningIndexerPrologCompute` (.../lightning_indexer_prolog.cpp:129-227). Every rope here de-interleaves
// (even dims first), the indexer's too; there is no Hadamard rotation and the weights are not scaled.

// de-interleaving rope of 64 values held in shared memory: output element c
__device__ __forceinline__ float rope_deinterleaved(const float* pe, int c, float cs, float sn) {
  const int j = c & 31;
  const float even = pe[2 * j], odd = pe[2 * j + 1];
  const float x = c < 32 ? even : odd;
  const float rot = c < 32 ? -odd : even;
  return __fadd_rn(__fmul_rn(x, cs), __fmul_rn(rot, sn));
}

// ---- per token: bf16 latent row, rope key, indexer key, indexer weights; scatter into the bf16 caches -----
// grid = tokens, block = 128 (thread i owns latent dims 4i..4i+3 and indexer-key dim i)
__global__ void __launch_bounds__(128)
prolog_kv_bf16_kernel(const float* __restrict__ kv, const float* __restrict__ ki, const float* __restrict__ wp, int ld,
                      int n_split, long long split_stride, const __nv_bfloat16* __restrict__ gamma_ckv,
                      const __nv_bfloat16* __restrict__ cos, const __nv_bfloat16* __restrict__ sin,
                      const __nv_bfloat16* __restrict__ ln_gamma, const __nv_bfloat16* __restrict__ ln_beta,
                      const int64_t* __restrict__ cache_index, int64_t cache_rows, float eps_ckv, float ln_eps,
                      __nv_bfloat16* __restrict__ kv_cache, __nv_bfloat16* __restrict__ kr_cache,
                      __nv_bfloat16* __restrict__ idx_k_cache, __nv_bfloat16* __restrict__ weights, int32_t* status) {
  __shared__ float red[32];
  __shared__ float pe[kRope];
  __shared__ float kpe[kRope];
  const int ti = blockIdx.x, i = threadIdx.x;
  const int64_t row = cache_index[ti];
  const bool row_ok = row >= 0 && row < cache_rows;
  if (!row_ok && i == 0) set_status(status, PTO_ST_BAD_PAGE, static_cast<int>(row), 61);
  auto proj = [&](const float* p) {
    float part[8];
#pragma unroll
    for (int sp = 0; sp < 8; ++sp) part[sp] = sp < n_split ? __ldg(p + sp * split_stride) : 0.f;
    float a = part[0];
#pragma unroll
    for (int sp = 1; sp < 8; ++sp) {
      if (sp < n_split) a = __fadd_rn(a, part[sp]);
    }
    return a;
  };
  // latent part: bf16 rounding, RMSNorm, bf16
  const float* src = kv + static_cast<int64_t>(ti) * ld;
  float v[4];
  float ss = 0.f;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    v[e] = bf16_round(proj(src + 4 * i + e));
    ss = __fadd_rn(ss, __fmul_rn(__fmul_rn(v[e], v[e]), 1.0f / kLora));
  }
  const float rms = sqrtf(block_sum(ss, red) + eps_ckv);
  if (row_ok) {
    __nv_bfloat16 o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      o[e] = __float2bfloat16_rn(__fmul_rn(__fdiv_rn(v[e], rms), ld_bf16(gamma_ckv + 4 * i + e)));
    }
    *reinterpret_cast<uint2*>(kv_cache + row * kLora + 4 * i) = *reinterpret_cast<const uint2*>(o);
  }
  // rope key and indexer key: the values to rotate go through shared memory
  if (i < kRope) pe[i] = bf16_round(proj(src + kLora + i));
  const float x = proj(ki + static_cast<int64_t>(ti) * ld + i);
  const float mean = block_sum(x, red) * (1.0f / kIdxDim);
  const float dx = x - mean;
  const float var = block_sum(__fmul_rn(dx, dx), red) * (1.0f / kIdxDim);
  const float y = __fdiv_rn(dx, sqrtf(var + ln_eps));
  const float k = bf16_round(__fadd_rn(__fmul_rn(y, ld_bf16(ln_gamma + i)), ld_bf16(ln_beta + i)));
  if (i < kRope) kpe[i] = k;
  __syncthreads();
  if (row_ok) {
    float ko = k;
    if (i < kRope) {
      const float cs = ld_bf16(cos + ti * kRope + i), sn = ld_bf16(sin + ti * kRope + i);
      kr_cache[row * kRope + i] = __float2bfloat16_rn(rope_deinterleaved(pe, i, cs, sn));
      ko = rope_deinterleaved(kpe, i, cs, sn);
    }
    idx_k_cache[row * kIdxDim + i] = __float2bfloat16_rn(ko);
  }
  if (i < kIdxHeads) {
    weights[static_cast<int64_t>(ti) * kIdxHeads + i] = __float2bfloat16_rn(proj(wp + static_cast<int64_t>(ti) * ld + i));
  }
}

// ---- ropes of the two up-projections -----------------------------------------------------------------
// grid = (24 head groups, tokens), block = 256, two values per thread: groups 0..15 take eight attention heads
// each (q_b[t, head, 128:192] -> q_rope[t, head, :]), groups 16..23 eight indexer heads each
// (idx_query[t, head, 0:64] rotated in place; the other 64 dims of a head stay as the product wrote them)
__global__ void __launch_bounds__(256)
prolog_rope_bf16_kernel(const __nv_bfloat16* q_b, const __nv_bfloat16* __restrict__ cos,
                        const __nv_bfloat16* __restrict__ sin, __nv_bfloat16* __restrict__ q_rope, __nv_bfloat16* idx_query) {
  // (q_b not __restrict__, as above)
  __shared__ float pe[8][kRope];
  if (threadIdx.x == 0) pdl_trigger();
  const int rc = threadIdx.x % kRope;  // a thread rotates one dim of several heads
  const float cs = ld_bf16(cos + blockIdx.y * kRope + rc), sn = ld_bf16(sin + blockIdx.y * kRope + rc);
  pdl_wait();
  const int g = blockIdx.x, ti = blockIdx.y;
  const bool att = g < kHeads / 8;
  const int head0 = att ? g * 8 : (g - kHeads / 8) * 8;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int e = u * 256 + threadIdx.x;
    const int hh = e >> 6, c = e & 63;
    const __nv_bfloat16* src = att ? q_b + (static_cast<int64_t>(ti) * kHeads + head0 + hh) * kQHead + kNope + c
                                   : idx_query + (static_cast<int64_t>(ti) * kIdxHeads + head0 + hh) * kIdxDim + c;
    pe[hh][c] = __bfloat162float(*src);
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int e = u * 256 + threadIdx.x;
    const int hh = e >> 6, c = e & 63;
    const __nv_bfloat16 o = __float2bfloat16_rn(rope_deinterleaved(pe[hh], c, cs, sn));
    if (att) {
      q_rope[(static_cast<int64_t>(ti) * kHeads + head0 + hh) * kRope + c] = o;
    } else {
      idx_query[(static_cast<int64_t>(ti) * kIdxHeads + head0 + hh) * kIdxDim + c] = o;
    }
  }
}

// ---- split caches -> packed 656-byte rows: one warp per row, 41 16-byte pieces ----------------------------
__global__ void __launch_bounds__(256)
kv_pack_rows_kernel(const int8_t* __restrict__ kv, const __nv_bfloat16* __restrict__ kr, const float* __restrict__ sc,
                    int64_t rows, int8_t* __restrict__ packed) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); r < rows; r += warps) {
    uint4* dst = reinterpret_cast<uint4*>(packed + r * kPackedRow);
    dst[lane] = __ldg(reinterpret_cast<const uint4*>(kv + r * kLora) + lane);
    if (lane < 8) dst[32 + lane] = __ldg(reinterpret_cast<const uint4*>(kr + r * kRope) + lane);
    if (lane == 8) dst[40] = __ldg(reinterpret_cast<const uint4*>(sc + r * 4));
  }
}

}  // namespace

cudaError_t launch_kv_pack_rows(const int8_t* kv, const void* kr, const float* sc, int64_t rows, int8_t* packed,
                                int num_sms, cudaStream_t stream) {
  const int64_t want = (rows + 7) / 8;
  const int grid = static_cast<int>(want < static_cast<int64_t>(num_sms) * 8 ? (want < 1 ? 1 : want) : num_sms * 8);
  count_launch();
  kv_pack_rows_kernel<<<grid, 256, 0, stream>>>(kv, reinterpret_cast<const __nv_bfloat16*>(kr), sc, rows, packed);
  return cudaGetLastError();
}

cudaError_t launch_prolog_qnorm_quant(const float* qa, int ld, int n_split, long long split_stride, const void* gamma_cq,
                                      int t, int q_lora, float eps, int8_t* q_norm, float* q_norm_scale,
                                      cudaStream_t stream, bool pdl) {
  if (t > kNormManyRows && q_lora <= kNormRow) {
    count_launch();
    return launch_maybe_pdl(prolog_qnorm_many_kernel<true>, dim3(t), dim3(128), 0, stream, pdl, qa, ld, n_split, split_stride,
                            reinterpret_cast<const __nv_bfloat16*>(gamma_cq), q_lora, eps, q_norm, q_norm_scale,
                            static_cast<__nv_bfloat16*>(nullptr));
  }
  const size_t dyn = static_cast<size_t>(q_lora) * sizeof(float);
  if (dyn > 40 * 1024) {  // beyond what fits the default 48 KB next to the kernel's static shared memory
    cudaError_t e = cudaFuncSetAttribute(prolog_qnorm_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(dyn));
    if (e != cudaSuccess) return e;
  }
  count_launch();
  return launch_maybe_pdl(prolog_qnorm_kernel<true>, dim3(t), dim3(512), dyn, stream, pdl, qa, ld, n_split, split_stride,
                          reinterpret_cast<const __nv_bfloat16*>(gamma_cq), q_lora, eps, q_norm, q_norm_scale,
                          static_cast<__nv_bfloat16*>(nullptr));
}

cudaError_t launch_prolog_qnorm_bf16(const float* qa, int ld, int n_split, long long split_stride, const void* gamma_cq,
                                     int t, int q_lora, float eps, void* q_norm, cudaStream_t stream, bool pdl) {
  if (t > kNormManyRows && q_lora <= kNormRow) {
    count_launch();
    return launch_maybe_pdl(prolog_qnorm_many_kernel<false>, dim3(t), dim3(128), 0, stream, pdl, qa, ld, n_split, split_stride,
                            reinterpret_cast<const __nv_bfloat16*>(gamma_cq), q_lora, eps, static_cast<int8_t*>(nullptr), static_cast<float*>(nullptr),
                            reinterpret_cast<__nv_bfloat16*>(q_norm));
  }
  const size_t dyn = static_cast<size_t>(q_lora) * sizeof(float);
  if (dyn > 40 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(prolog_qnorm_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(dyn));
    if (e != cudaSuccess) return e;
  }
  count_launch();
  return launch_maybe_pdl(prolog_qnorm_kernel<false>, dim3(t), dim3(512), dyn, stream, pdl, qa, ld, n_split,
                          split_stride, reinterpret_cast<const __nv_bfloat16*>(gamma_cq), q_lora, eps,
                          static_cast<int8_t*>(nullptr), static_cast<float*>(nullptr),
                          reinterpret_cast<__nv_bfloat16*>(q_norm));
}

cudaError_t launch_prolog_qb_dequant_rope(const int32_t* qb_i32, const float* q_norm_scale, const float* w_scale,
                                          const void* cos, const void* sin, int t, void* q_b, void* q_rope,
                                          cudaStream_t stream, bool pdl) {
  count_launch();
  return launch_maybe_pdl(prolog_qb_dequant_rope_kernel, dim3(kHeads / kQbHeadsPerBlock, t), dim3(256), 0, stream, pdl,
                          qb_i32, q_norm_scale, w_scale, reinterpret_cast<const __nv_bfloat16*>(cos),
                          reinterpret_cast<const __nv_bfloat16*>(sin), reinterpret_cast<__nv_bfloat16*>(q_b),
                          reinterpret_cast<__nv_bfloat16*>(q_rope));
}

cudaError_t launch_prolog_kv(const float* kv, const float* ki, const float* wp, int ld, int n_split,
                             long long split_stride, const void* gamma_ckv, const void* cos,
                             const void* sin, const void* ln_gamma, const void* ln_beta, const void* hadamard_k,
                             const int64_t* cache_index, int64_t cache_rows, int t, float eps_ckv, float ln_eps,
                             int8_t* kv_cache, void* kr_cache, float* kv_scale_cache, int8_t* idx_k_cache,
                             void* idx_k_scale_cache, void* weights, int8_t* packed_cache, const void* next_hadamard,
                             const void* next_scale, int32_t* status, cudaStream_t stream) {
  count_launch();
  (t > kNormManyRows ? prolog_kv_kernel<true> : prolog_kv_kernel<false>)<<<t, 128, 0, stream>>>(
      kv, ki, wp, ld, n_split, split_stride, reinterpret_cast<const __nv_bfloat16*>(gamma_ckv),
      reinterpret_cast<const __nv_bfloat16*>(cos),
      reinterpret_cast<const __nv_bfloat16*>(sin), reinterpret_cast<const __nv_bfloat16*>(ln_gamma),
      reinterpret_cast<const __nv_bfloat16*>(ln_beta), reinterpret_cast<const __nv_bfloat16*>(hadamard_k), cache_index,
      cache_rows, eps_ckv, ln_eps, kv_cache, reinterpret_cast<__nv_bfloat16*>(kr_cache), kv_scale_cache, idx_k_cache,
      reinterpret_cast<__half*>(idx_k_scale_cache), reinterpret_cast<__half*>(weights), packed_cache,
      next_hadamard, next_scale, status);
  return cudaGetLastError();
}

cudaError_t launch_prolog_kv_bf16(const float* kv, const float* ki, const float* wp, int ld, int n_split,
                                  long long split_stride, const void* gamma_ckv, const void* cos, const void* sin,
                                  const void* ln_gamma, const void* ln_beta, const int64_t* cache_index,
                                  int64_t cache_rows, int t, float eps_ckv, float ln_eps, void* kv_cache, void* kr_cache,
                                  void* idx_k_cache, void* weights, int32_t* status, cudaStream_t stream) {
  count_launch();
  prolog_kv_bf16_kernel<<<t, 128, 0, stream>>>(
      kv, ki, wp, ld, n_split, split_stride, reinterpret_cast<const __nv_bfloat16*>(gamma_ckv),
      reinterpret_cast<const __nv_bfloat16*>(cos), reinterpret_cast<const __nv_bfloat16*>(sin),
      reinterpret_cast<const __nv_bfloat16*>(ln_gamma), reinterpret_cast<const __nv_bfloat16*>(ln_beta), cache_index,
      cache_rows, eps_ckv, ln_eps, reinterpret_cast<__nv_bfloat16*>(kv_cache), reinterpret_cast<__nv_bfloat16*>(kr_cache),
      reinterpret_cast<__nv_bfloat16*>(idx_k_cache), reinterpret_cast<__nv_bfloat16*>(weights), status);
  return cudaGetLastError();
}

cudaError_t launch_prolog_rope_bf16(const void* q_b, const void* cos, const void* sin, int t, void* q_rope,
                                    void* idx_query, cudaStream_t stream, bool pdl) {
  count_launch();
  return launch_maybe_pdl(prolog_rope_bf16_kernel, dim3((kHeads + kIdxHeads) / 8, t), dim3(256), 0, stream, pdl,
                          reinterpret_cast<const __nv_bfloat16*>(q_b), reinterpret_cast<const __nv_bfloat16*>(cos),
                          reinterpret_cast<const __nv_bfloat16*>(sin), reinterpret_cast<__nv_bfloat16*>(q_rope),
                          reinterpret_cast<__nv_bfloat16*>(idx_query));
}

cudaError_t launch_prolog_idxq(const int32_t* qi_i32, const float* q_norm_scale, const float* w_scale, const void* cos,
                               const void* sin, const void* hadamard_q, int t, int8_t* q_int8, void* q_scale,
                               cudaStream_t stream) {
  count_launch();
  cudaError_t e = cudaFuncSetAttribute(prolog_idxq_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kHadBytes);
  if (e != cudaSuccess) return e;
  prolog_idxq_kernel<<<t, 256, kHadBytes, stream>>>(
      qi_i32, q_norm_scale, w_scale, reinterpret_cast<const __nv_bfloat16*>(cos),
      reinterpret_cast<const __nv_bfloat16*>(sin), reinterpret_cast<const __nv_bfloat16*>(hadamard_q), q_int8,
      reinterpret_cast<__half*>(q_scale));
  return cudaGetLastError();
}

}  // namespace pto
