// Lightning-indexer score stage.
//
//   d[h, pos]  = int32( q[h, :] . k[pos, :] )                    64 heads x 128 dims, int8
//   h16        = fp16( relu(d) * 2^-11 )
//   score[pos] = k_scale[pos] * sum_h fp32(ws_h) * fp32(h16),    ws_h = q_scale_h * weight_h
//
// (reference: examples/models/deepseek_v32_exp/lightning_indexer_quant_impl.py:138-194; golden
// deepseekv32_lightning_indexer_quant.py:205-241).
//
// Tensor-core kernel: persistent CTAs, each owning a contiguous range of the flattened
// (token group, sequence, page) list. Per page: one TMA load of the 16 KB key page (128 keys x 128 B,
// 128-byte swizzle) and its key scales; per page and pair of query tokens (an item): four tcgen05.mma kind::i8
// (M = 128 keys, N = 64 or 128 heads, K = 32) into a TMEM accumulator -> epilogue warps read their key's
// row (one TMEM lane = one key), apply ReLU/2^-11/fp16 rounding and the weighted head sum, and write the fp32 score.
// With two and more query tokens per pass the head sum is a second product (kLiQuantTc): the epilogue writes the fp16
// values back over the accumulator, tcgen05.mma kind::f16 takes them as its A operand from TMEM (K = 64 heads), B is the
// weights, and what comes back is the key's score. The weights of a token are fp32, scaled to 2^13 by a power of two: B holds
// them as three fp16 limbs. The tensor core truncates where it adds, so a column of the product takes sixteen heads of one limb
// (one step of K; zeros elsewhere), its twelve columns are added here, and the first limb has six bits, multiples of 2^8 for
// all heads: its products, which are the large ones, share a grid that the sum has room for. (With 11 bits, each limb as many of
// a weight as it could hold, the scores were a third further from 64 bits than the fp32 sum on CUDA cores, and too small: relative error 6.7e-8 rms with a mean of -2.0e-8,
// now 3.8e-8 without one, the fp32 sum 5.1e-8. Of a weight below 2^-7 of the token's largest the limbs hold 22 bits.) On
// CUDA cores the head sum was the kernel's bound: unpacking the fp16 values and the multiply-adds were 1.5 of its 3.5
// instructions per (key, head) and kept the half-rate FP16 / packed-FP32 pipe 70 % busy (16 x 65536 keys, two query
// tokens 39.6 -> 37.4 us, four 66.0 -> 59.0; 256 tokens over 65536 keys 230 -> 192 us). With one query token the key
// pages bound the kernel and the second product only adds to an item's latency (64 x 32768 keys 50.4 -> 51.9 us).
// Warp roles: warp 0 TMA producer, warps 1..2 MMA issuers (alternate items; warp 1 owns TMEM),
// warps 3..18 epilogue (four groups of four warps that take items round-robin; a single warp is
// latency-bound on the conversion chain, so thread-level parallelism has to come from many warps).
// Two rings: key pages in shared memory (8), freed by the MMAs that read them, and accumulators in TMEM (8 of 64
// columns, 4 of 128), freed by the epilogue. With one ring for both, a page's load was requested only when the epilogue
// had let go of an accumulator, and every slot paid load latency + product + epilogue in turn: 1117 cycles per page with
// two query tokens, where the page's bytes take 750 at the memory's rate. Items of at most two tokens keep all four
// epilogue groups at work when a pass takes three or four tokens of a sequence (with 256 columns per item two of
// them had no accumulator to serve). All waits are bounded.
//
// Non-quantised formulation (bf16 queries, keys and weights; reference LightningIndexerTopkImpl with isQuant =
// false, framework/src/operator/models/deepseek_v3.2_exp/lightning_indexer.cpp:113-147, golden
// indexer_topk_compute(is_quant=False), framework/tests/st/operator/src/test_deepseek_v3.2_exp/
// gen_lightning_indexer.py:189-279):   score[pos] = sum_h fp32(w_h) * relu( fp32( q[h, :] . k[pos, :] ) ).
// Same kernel and rings, mode kLiBf16: a key page is 32 KB (two 128-byte-swizzled halves of the 128 dims), the
// product is tcgen05.mma kind::f16 (bf16 x bf16 -> fp32, eight MMAs of K = 16 per page), four pages, at
// most two query tokens of a sequence per pass, and the epilogue is max/fma on the fp32 accumulators.
#include <cuda.h>

#include "sfa_common.cuh"

namespace pto {

namespace {

constexpr int kLiStages = 8;           // ring of key pages in shared memory
constexpr int kLiAccs = 8;             // accumulators of 64 columns (4 of 128)
constexpr int kLiScaleRing = 16;       // key scales of the pages in flight, see the producer
constexpr int kPageKeys = 128;
constexpr int kPageBytes = kPageKeys * 128;
constexpr int kScaleBytes = 512;                // the page's 128 key scales
constexpr int kHeads = 64;
constexpr int kQBytesPerToken = kHeads * 128;
constexpr int kLiMmaWarps = 2;         // warps 1..2: issuer for pages n with n % 2 == warp - 1
constexpr int kLiEpilogueGroups = 4;   // groups of four warps; an accumulator is always served by the same group (below)
constexpr int kLiEpilogueWarp0 = 1 + kLiMmaWarps;
constexpr int kLiThreads = 32 * (kLiEpilogueWarp0 + 4 * kLiEpilogueGroups);
constexpr int kMaxS1 = 4;
constexpr int kMaxSeqPerLaunch = 2048;
constexpr int kTmemCols = 512;
// score formulations the tensor-core kernel is instantiated for
enum { kLiQuant = 0, kLiChain = 1, kLiBf16 = 2, kLiQuantTc = 3 };  // kLiQuantTc: the head sum on the tensor cores
constexpr int kBf16PageBytes = kPageKeys * 256;  // one stage of the bf16 ring: the page's two 16 KB halves
constexpr int kBf16Stages = 4;                   // 4 x 32 KB where the int8 ring keeps 8 x 16 KB
constexpr int kBf16MaxS1 = 2;                    // 2 tokens x 64 heads x 256 B of queries fit the int8 Q area
static_assert(kBf16Stages * kBf16PageBytes <= kLiStages * kPageBytes, "bf16 ring exceeds the stage area");
static_assert(kLiScaleRing >= kLiStages + kLiAccs, "a page's scales are read until its items' accumulators are free again");
static_assert(kBf16MaxS1 * kHeads * 256 <= kMaxS1 * kQBytesPerToken, "bf16 queries exceed the Q area");

struct LiCtl {
  uint64_t full[kLiStages];    // TMA bytes of the page (and its scales) landed
  uint64_t kempty[kLiStages];  // all MMAs that read the page completed (tcgen05.commit, one per item of the page)
  uint64_t accfull[kLiAccs];   // the item's MMAs completed (tcgen05.commit)
  uint64_t accempty[kLiAccs];  // the item's epilogue warps have read the accumulator
  uint64_t sumfull[kLiAccs];   // the item's head sums completed (tcgen05.commit; int8 formulation)
  uint64_t qfull;
  uint32_t tmem_base;
  int abort;
  int prefix[kMaxSeqPerLaunch + 1];
  __align__(16) float ws[kMaxS1 * kHeads];
  unsigned int wmax[kMaxS1][2];  // bit patterns of the largest |ws| of each half of a token's heads
  float winv[kMaxS1];            // power of two that undoes the scaling of the limbs
};

constexpr size_t kLiHistSmemBytes = static_cast<size_t>(kLiHistMaxS1) * kLiHistBins * sizeof(unsigned int) + 16;  // 32 KB (+ alignment of its start)
constexpr int kLimbBytes = 16 * 128;  // B operand of the head sum per token: 16 rows (limb x sixteen heads, four of zeros) of 64 heads
constexpr int kLiSmemScales = kLiStages * kPageBytes, kLiSmemLimbs = kLiSmemScales + kLiScaleRing * kScaleBytes;
constexpr int kLiSmemQ = kLiSmemLimbs + kMaxS1 * kLimbBytes;
constexpr int kLiSmemCtl = kLiSmemQ + kMaxS1 * kQBytesPerToken;
static_assert(kLiSmemQ % 1024 == 0, "swizzled query tile");
constexpr size_t kLiSmemBytes = 1024 /*alignment slack*/ + kLiSmemCtl + sizeof(LiCtl);
static_assert(kLiSmemBytes + kLiHistSmemBytes <= 227 * 1024, "score kernel shared memory");

__device__ __forceinline__ float load_scale(const void* base, int dtype, int64_t i) {
  if (dtype == PTO_DT_F16) return __half2float(reinterpret_cast<const __half*>(base)[i]);
  return reinterpret_cast<const float*>(base)[i];
}

// ws = q_scale * weight, the product taken in the tensors' own dtype (fp16 product is rounded to
// fp16 before widening, as the golden does).
__device__ __forceinline__ float load_ws(const void* qs, const void* w, int dtype, int64_t i) {
  if (dtype == PTO_DT_F16) {
    return __half2float(__hmul(reinterpret_cast<const __half*>(qs)[i], reinterpret_cast<const __half*>(w)[i]));
  }
  return __fmul_rn(reinterpret_cast<const float*>(qs)[i], reinterpret_cast<const float*>(w)[i]);
}

// relu(d) * 2^-11 rounded to fp16, for two dots at once; exact for |d| < 2^21:
// adding d to the bit pattern of 6144.0f (ulp 2^-11) and subtracting 6144 gives d * 2^-11.
__device__ __forceinline__ uint32_t relu_scale_half2(int d0, int d1) {
  // the two subtractions as one packed fp32 instruction (each half is an ordinary IEEE subtraction)
  const float2 f = __fadd2_rn(make_float2(__int_as_float(0x45C00000 + d0), __int_as_float(0x45C00000 + d1)),
                              make_float2(-6144.0f, -6144.0f));
  uint32_t packed;  // round to fp16 and clamp negatives to zero in one conversion (f.x in the low half)
  asm("cvt.rn.relu.f16x2.f32 %0, %1, %2;" : "=r"(packed) : "f"(f.y), "f"(f.x));
  return packed;
}

// The same values weighted and summed on CUDA cores, 32 heads of one key.
__device__ __forceinline__ float weighted_sum_32(const uint32_t (&v)[32], const float* ws) {
  // four running sums as two packed pairs: one packed FMA per two heads (the same four chains of ordinary FMAs)
  float2 a01 = make_float2(0.f, 0.f), a23 = make_float2(0.f, 0.f);
#pragma unroll
  for (int c = 0; c < 32; c += 4) {
    const float4 w = *reinterpret_cast<const float4*>(ws + c);
    const uint32_t hx = relu_scale_half2(static_cast<int>(v[c]), static_cast<int>(v[c + 1]));
    const uint32_t hy = relu_scale_half2(static_cast<int>(v[c + 2]), static_cast<int>(v[c + 3]));
    a01 = __ffma2_rn(make_float2(w.x, w.y), __half22float2(*reinterpret_cast<const __half2*>(&hx)), a01);
    a23 = __ffma2_rn(make_float2(w.z, w.w), __half22float2(*reinterpret_cast<const __half2*>(&hy)), a23);
  }
  return (a01.x + a01.y) + (a23.x + a23.y);
}

// named barrier of kThreads threads that returns the OR of their predicates: the same answer in every thread, so whoever
// meets at later barriers stays together
template <int kThreads>
__device__ __forceinline__ bool li_vote(int id, bool pred) {
  uint32_t any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %2, 0;\n\tbarrier.cta.red.or.pred q, %1, %3, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(any)
      : "r"(id), "r"(pred ? 1u : 0u), "n"(kThreads)
      : "memory");
  return any != 0;
}

// the twelve columns of a head sum (limb l of heads 16 s .. 16 s + 15 at 4 l + s) -> the sum in units of the largest limb
__device__ __forceinline__ float limb_sum(const uint32_t (&r)[16]) {
  float v[3];
#pragma unroll
  for (int l = 0; l < 3; ++l) {
    v[l] = (__uint_as_float(r[4 * l]) + __uint_as_float(r[4 * l + 1])) + (__uint_as_float(r[4 * l + 2]) + __uint_as_float(r[4 * l + 3]));
  }
  return fmaf(fmaf(v[2], 1.0f / 2048.0f, v[1]), 1.0f / 128.0f, v[0]);
}

// The older formulation for 32 heads of one key: table entries come in pairs, (q_scale_2p, q_scale_2p+1) and
// (weight_2p, weight_2p+1) as half2 bit patterns; d * 2^-11 is exact by the same magic number as above.
__device__ __forceinline__ float chain_sum_32(const uint32_t (&v)[32], const float* table, __half2 ks2) {
  const uint32_t* tb = reinterpret_cast<const uint32_t*>(table);
  float acc = 0.f;
#pragma unroll
  for (int c = 0; c < 32; c += 2) {
    const float f0 = __int_as_float(0x45C00000 + static_cast<int>(v[c])) - 6144.0f;
    const float f1 = __int_as_float(0x45C00000 + static_cast<int>(v[c + 1])) - 6144.0f;
    const uint32_t qs_bits = tb[c], w_bits = tb[c + 1];
    const __half2 qs2 = *reinterpret_cast<const __half2*>(&qs_bits);
    const __half2 w2 = *reinterpret_cast<const __half2*>(&w_bits);
    __half2 a = __hmul2(__hmul2(__floats2half2_rn(f0, f1), qs2), ks2);
    a = __hmax2(a, __float2half2_rn(0.0f));
    const float2 m = __half22float2(__hmul2(a, w2));
    acc = __fadd_rn(__fadd_rn(acc, m.x), m.y);
  }
  return acc;
}

// Non-quantised formulation, 32 heads of one key: the accumulators are fp32 dots.
__device__ __forceinline__ float weighted_relu_sum_32(const uint32_t (&v)[32], const float* ws) {
  float2 a01 = make_float2(0.f, 0.f), a23 = make_float2(0.f, 0.f);
#pragma unroll
  for (int c = 0; c < 32; c += 4) {
    const float4 w = *reinterpret_cast<const float4*>(ws + c);
    a01 = __ffma2_rn(make_float2(w.x, w.y),
                     make_float2(fmaxf(__uint_as_float(v[c]), 0.f), fmaxf(__uint_as_float(v[c + 1]), 0.f)), a01);
    a23 = __ffma2_rn(make_float2(w.z, w.w),
                     make_float2(fmaxf(__uint_as_float(v[c + 2]), 0.f), fmaxf(__uint_as_float(v[c + 3]), 0.f)), a23);
  }
  return (a01.x + a01.y) + (a23.x + a23.y);
}

template <int kMode, bool kGroups>  // kGroups: takes launches of more than one token group
__global__ void __launch_bounds__(kLiThreads, 1)
li_score_tc_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_q, LiParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw);
  const uint32_t stage_base = base;
  const uint32_t q_base = base + kLiSmemQ;
  LiCtl* ctl = reinterpret_cast<LiCtl*>(smem + kLiSmemCtl);
  // per-CTA histogram of the current sequence's scores (present only when the launch asked for it)
  unsigned int* hist_sm = reinterpret_cast<unsigned int*>(smem + kLiSmemCtl + ((sizeof(LiCtl) + 15) & ~size_t(15)));
  const bool with_hist = p.hist != nullptr;

  constexpr bool kChain = kMode == kLiChain;
  constexpr bool kBf16 = kMode == kLiBf16;
  constexpr uint32_t kStage = kBf16 ? kBf16PageBytes : kPageBytes;
  constexpr uint32_t kStages = kBf16 ? kBf16Stages : kLiStages;
  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  // this kernel is launched the ordinary way (everything before it has completed); the top-k kernel behind it
  // may be scheduled as soon as SMs drain and waits there for this grid to complete
  if (tid == 0) pdl_trigger();
  const int s1 = kMode == kLiQuant ? 1 : p.s1;  // (that formulation is launched for one token)
  const int items_per_page = s1 > 2 ? 2 : 1;                     // an item: one or two query tokens of a page
  const uint32_t unit_cols = s1 > 1 ? 2 * kHeads : kHeads;       // columns of an accumulator
  const uint32_t n_accs = kTmemCols / unit_cols;                 // 8 or 4
  const uint32_t acc_shift = s1 > 1 ? 2 : 3;                     // log2 of it
  if (tid == 0) {
    for (int i = 0; i < kLiStages; ++i) {
      mbar_init(smem_u32(&ctl->full[i]), 1);
      mbar_init(smem_u32(&ctl->kempty[i]), static_cast<uint32_t>(items_per_page));
    }
    for (int i = 0; i < kLiAccs; ++i) {
      mbar_init(smem_u32(&ctl->accfull[i]), 1);
      mbar_init(smem_u32(&ctl->accempty[i]), 4);
      mbar_init(smem_u32(&ctl->sumfull[i]), 1);
    }
    mbar_init(smem_u32(&ctl->qfull), 1);
    ctl->abort = 0;
    fence_mbar_init();
    fence_proxy_async();
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_q);
  }
  if (with_hist) {
    for (int j = tid; j < s1 * kLiHistBins; j += kLiThreads) hist_sm[j] = 0u;
  }
  if (kMode == kLiQuantTc) {  // (what is not written below stays zero)
    for (int j = tid; j < kMaxS1 * kLimbBytes / 16; j += kLiThreads) {
      *reinterpret_cast<uint4*>(smem + kLiSmemLimbs + j * 16) = make_uint4(0, 0, 0, 0);
    }
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&ctl->tmem_base), kTmemCols);
    tmem_relinquish();
  }
  // A chunk of one prompt whose scores only the selection reads: a token group needs the pages up to its last token's causal end, and
  // the list below is one of groups instead of sequences. (All pages for every group: twice the work where the chunk is the prompt.)
  // The CTAs share it by cost: a group's queries and weights take as long as `kGroupCost` of its pages, and the first groups have
  // few of these (by pages alone the first CTA got seventy groups of a chunk of 4096). 4096 tokens that are the prompt 208 -> 119 us,
  // behind 12288 keys 756 -> 642, 512 tokens 12.4 -> 11.0; with few tokens behind many keys there is nothing to leave out.
  // The cost in pages, 0 / 1 / 2 / 3 / 4 / 6 / 8, selection included, us: int8, 4096 tokens that are the prompt 305 / 228 / 186 / 171 / 172 / 177 /
  // 181, 3000 176 / 129 / 103 / 101 / 102 / 105 / 109; bf16, whose groups are two tokens, 4000 414 / 305 / 245 / 210 / 192 / 180 / 183, 2000 121 / 76 /
  // 62 / 56 / 53 / 54 / 56; behind other keys and up to 1000 tokens the same within a percent from 1 to 4.
  // (kGroups: kernels of their own, since calls that have nothing to leave out lose by the code for it; whole steps with inputs that are not
  // in L2: 10 sequences of three tokens 79.3 / 77.9 us, 40 of one 109.5 / 108.2; a bf16 layer of 16 95.0 / 93.7.)
  const bool by_group = kGroups && p.causal != 0 && p.b == 1 && p.groups > 1 && p.groups <= kMaxSeqPerLaunch;
  const int n_lists = by_group ? p.groups : p.b;
  constexpr int kGroupCost = kBf16 ? 6 : 3;
  const int head = by_group ? kGroupCost : 0;  // units of cost before a list's first page
  if (warp == kLiEpilogueWarp0) {
    // exclusive prefix of pages per sequence (or token group)
    int carry = 0;
    const int first_end = by_group ? p.act_seq[0] - p.s1_total + p.tok_offset + s1 : 0;  // causal end of the first group
    for (int b0 = 0; b0 < n_lists; b0 += 32) {
      int v = 0;
      if (b0 + lane < n_lists) {
        int s = by_group ? first_end + (b0 + lane) * s1 : p.act_seq[b0 + lane];
        s = max(s, 0);
        v = min((s + kPageKeys - 1) / kPageKeys, p.max_blocks);
        if (kGroups && v > 0) v += head;
      }
      int incl = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int n = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += n;
      }
      if (b0 + lane < n_lists) ctl->prefix[b0 + lane] = carry + incl - v;
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) ctl->prefix[n_lists] = carry;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;

  // pages of all sequences, once per token group
  const int total = ctl->prefix[n_lists];
  const long long all = static_cast<long long>(total) * (by_group ? 1 : p.groups);
  const long long it0 = all * blockIdx.x / gridDim.x, it1 = all * (blockIdx.x + 1) / gridDim.x;

  const uint32_t idesc1 = kBf16 ? umma_idesc(kCFmtF32, kABFmtBF16, kABFmtBF16, 0, 0, 128, kHeads)
                                : umma_idesc(kCFmtS32, kABFmtS8, kABFmtS8, 0, 0, 128, kHeads);
  const uint32_t idesc2 = kBf16 ? umma_idesc(kCFmtF32, kABFmtBF16, kABFmtBF16, 0, 0, 128, 2 * kHeads)
                                : umma_idesc(kCFmtS32, kABFmtS8, kABFmtS8, 0, 0, 128, 2 * kHeads);
  const uint32_t scale_bytes = kBf16 ? 0u : kPageKeys * (p.scale_dtype == PTO_DT_F16 ? 2u : 4u);
  const uint32_t q_half_bytes = static_cast<uint32_t>(s1 * kHeads) * 128u;  // bf16: one 64-dim half of the query tile

  long long cur = it0;
  int li = 0, group = 0;  // list (sequence or token group)
  if (cur < it1) {
    group = static_cast<int>(cur / total);
    const int lc = static_cast<int>(cur - static_cast<long long>(group) * total);
    int lo = 0, hi = n_lists;  // largest list with prefix[lo] <= lc
    while (hi - lo > 1) {
      int mid = (lo + hi) >> 1;
      if (ctl->prefix[mid] <= lc) lo = mid; else hi = mid;
    }
    li = lo;
  }
  uint32_t n_page = 0;  // pages and items of the segments before
  uint32_t n_item = 0;
  uint32_t seg = 0;
  int64_t prev_tok0 = 0;
  // adds this CTA's counts of the tokens tok_first .. tok_first + s1 - 1 into the global histogram and clears them
  auto flush_hist = [&](int64_t tok_first) {
    // (not the producer warp: it does not take part in the barrier that orders the flush before new counts)
    for (int j = tid - 32; j >= 0 && j < s1 * kLiHistBins; j += kLiThreads - 32) {
      const unsigned int c = hist_sm[j];
      if (c != 0u) {
        atomicAdd(p.hist + tok_first * kLiHistBins + j, c);
        hist_sm[j] = 0u;
      }
    }
  };

  while (cur < it1) {
    int lc = static_cast<int>(cur - static_cast<long long>(group) * total);
    if (lc >= total) {  // next token group, from the first sequence
      ++group;
      li = 0;
      lc = 0;
    }
    while (ctl->prefix[li + 1] <= lc) ++li;
    const int cost = static_cast<int>(min(it1 - cur, static_cast<long long>(ctl->prefix[li + 1] - lc)));
    const int page0 = kGroups ? max(0, lc - ctl->prefix[li] - head) : lc - ctl->prefix[li];
    const int npages = kGroups ? max(0, lc - ctl->prefix[li] - head + cost) - page0 : cost;
    if (kGroups && npages == 0) {  // (the same in every thread)
      cur += cost;
      continue;
    }
    const int bi = by_group ? 0 : li;
    const int seq_len = p.act_seq[bi];
    const int tok_first = p.tok_offset + (by_group ? li : group) * s1;  // first query token of the segment within its sequence
    const int64_t tok0 = static_cast<int64_t>(bi) * p.s1_total + tok_first;

    // The producer warp takes no part in the two barriers of a segment: the ring's own barriers order its loads, so
    // the next segment's first pages are on their way while this one drains and the scale products are fetched.
    // previous segment fully drained: Q tile and ws may be overwritten
    bool aborted = ctl->abort != 0;
    if (warp != 0) aborted = li_vote<kLiThreads - 32>(1, aborted);
    if (with_hist && seg > 0) flush_hist(prev_tok0);  // (the barrier below orders it before the next segment's counts)
    prev_tok0 = tok0;
    if (!aborted) {
      if (warp == 1 && lane == 0) {
        if (kBf16) {
          mbar_arrive_expect_tx(smem_u32(&ctl->qfull), 2 * q_half_bytes);
          tma_load_2d(q_base, &tmap_q, 0, static_cast<int>(tok0) * kHeads, smem_u32(&ctl->qfull));
          tma_load_2d(q_base + q_half_bytes, &tmap_q, 128, static_cast<int>(tok0) * kHeads, smem_u32(&ctl->qfull));
        } else {
          mbar_arrive_expect_tx(smem_u32(&ctl->qfull), s1 * kQBytesPerToken);
          tma_load_2d(q_base, &tmap_q, 0, static_cast<int>(tok0) * kHeads, smem_u32(&ctl->qfull));
        }
      }
      const int e = tid - 32 * kLiEpilogueWarp0;
      if (e >= 0 && e < s1 * kHeads) {
        if (kBf16) {
          ctl->ws[e] = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.weight)[tok0 * kHeads + e]);
        } else if (kChain) {
          // pairs of heads: even slot = the two query scales, odd slot = the two weights (fp16 bit patterns)
          const __half* src = reinterpret_cast<const __half*>((e & 1) ? p.weight : p.q_scale) + tok0 * kHeads + (e & ~1);
          const __half2 two = __halves2half2(src[0], src[1]);
          reinterpret_cast<uint32_t*>(ctl->ws)[e] = *reinterpret_cast<const uint32_t*>(&two);
        } else {
          const float w = load_ws(p.q_scale, p.weight, p.scale_dtype, tok0 * kHeads + e);
          ctl->ws[e] = w;
          const unsigned int m = __reduce_max_sync(0xffffffffu, __float_as_uint(w) & 0x7fffffffu);  // (whole warps: 64 heads)
          if (lane == 0) ctl->wmax[e >> 6][(e >> 5) & 1] = m;
        }
      }
    }
    if (kMode == kLiQuantTc) {
      if (warp != 0) asm volatile("bar.sync 1, %0;" ::"n"(kLiThreads - 32) : "memory");
      const int e = tid - 32 * kLiEpilogueWarp0;
      if (!aborted && e >= 0 && e < s1 * kHeads) {
        const int i = e >> 6, h = e & 63;
        const unsigned int m = max(ctl->wmax[i][0], ctl->wmax[i][1]);
        const int ex = max(-100, min(127, static_cast<int>(m >> 23) - 127));  // 2^ex <= largest weight < 2^(ex + 1)
        float r = ctl->ws[e] * __int_as_float((127 + 13 - ex) << 23);
#pragma unroll
        for (int l = 0; l < 3; ++l) {  // exact splitting: what a limb leaves over, scaled up by 2^7 or 2^11, goes to the next
          // (the first: multiples of 2^8)
          const __half w = __float2half_rn(l == 0 ? __fsub_rn(__fadd_rn(r, 3221225472.0f), 3221225472.0f) : r);
          // row (limb, sixteen heads) of 128 bytes (64 heads), 128-byte swizzle
          const int rw = l * 4 + (h >> 4);
          *reinterpret_cast<__half*>(smem + kLiSmemLimbs + i * kLimbBytes + rw * 128 + (((h >> 3) ^ (rw & 7)) << 4) + (h & 7) * 2) = w;
          // (nothing is left over of an infinite weight: its product decides alone, as in a sum of fp32 products)
          r = __hisinf(w) != 0 ? 0.f : (r - __half2float(w)) * (l == 0 ? 128.0f : 2048.0f);
        }
        if (h == 0) ctl->winv[i] = __int_as_float((127 + ex - 13) << 23);
        fence_proxy_async();
      }
    }
    // the scale products are visible to the MMA and epilogue warps
    if (warp != 0) asm volatile("bar.sync 1, %0;" ::"n"(kLiThreads - 32) : "memory");

    if (!aborted) {
      if (warp == 0) {
        // ---------------- TMA producer ----------------
        const int32_t* bt = p.block_table + static_cast<int64_t>(bi) * p.max_blocks + page0;
        // key pages that are read once are the first to leave L2, so that the score rows written for the selection stay
        // there (a prompt chunk reads them once per token group)
        const uint64_t stream_policy = l2_policy_evict_first();
        const bool once = p.groups == 1;
        bool ok = true;
        for (int j0 = 0; j0 < npages && ok; j0 += 32) {
          const int mine = (j0 + lane < npages) ? bt[j0 + lane] : 0;
          const int cnt = min(32, npages - j0);
          for (int jj = 0; jj < cnt; ++jj) {
            int phys = __shfl_sync(0xffffffffu, mine, jj);
            if (lane == 0) {
              const uint32_t n = n_page + j0 + jj;
              const uint32_t slot = n % kStages;
              const uint32_t ph = (n / kStages) & 1u;
              if (!mbar_wait(smem_u32(&ctl->kempty[slot]), ph ^ 1u)) {
                ok = false;
                ctl->abort = 1;
                set_status(p.status, PTO_ST_WAIT_EXPIRED, static_cast<int>(n), 1);
              } else {
                int scale_page = phys;
                if (phys < 0 || phys >= p.block_num) {
                  set_status(p.status, PTO_ST_BAD_PAGE, phys, 1);
                  phys = p.block_num;  // out of range of the tensor map: the page reads as zeros
                  scale_page = 0;      // any valid scales: the dots are zero
                }
                const uint32_t bar = smem_u32(&ctl->full[slot]);
                const uint32_t dst = stage_base + slot * kStage;
                if (kBf16) {
                  mbar_arrive_expect_tx(bar, kBf16PageBytes);
                  if (once) {
                    tma_load_2d_hint(dst, &tmap_k, 0, phys * kPageKeys, bar, stream_policy);
                    tma_load_2d_hint(dst + kPageBytes, &tmap_k, 128, phys * kPageKeys, bar, stream_policy);
                  } else {
                    tma_load_2d(dst, &tmap_k, 0, phys * kPageKeys, bar);
                    tma_load_2d(dst + kPageBytes, &tmap_k, 128, phys * kPageKeys, bar);
                  }
                } else {
                  mbar_arrive_expect_tx(bar, kPageBytes + scale_bytes);
                  if (once) tma_load_2d_hint(dst, &tmap_k, 0, phys * kPageKeys, bar, stream_policy);
                  else tma_load_2d(dst, &tmap_k, 0, phys * kPageKeys, bar);
                  // The place of these scales was last used by page n - 16. Its epilogue has read them: the MMAs of every
                  // page up to n - 8 are complete (the waits above), so the accumulators that they overwrote, those of the
                  // items up to 8 before each, have been read.
                  bulk_load_1d(base + kLiSmemScales + (n % kLiScaleRing) * kScaleBytes,
                               reinterpret_cast<const uint8_t*>(p.k_scale) + static_cast<int64_t>(scale_page) * scale_bytes,
                               scale_bytes, bar);
                }
              }
            }
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            if (!ok) break;
          }
        }
      } else if (warp < kLiEpilogueWarp0) {
        // ---------------- MMA issuers: warp w takes items n with n % 2 == w - 1 ----------------
        // (the warp stays converged and an elected lane issues: the descriptors stay in uniform registers)
        bool ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&ctl->qfull), seg & 1u));
        if (!ok && lane == 0) set_status(p.status, PTO_ST_WAIT_EXPIRED, static_cast<int>(seg), 2);
        const uint64_t b_desc0 = umma_desc_kmajor_sw128(q_base);
        const uint64_t a_desc0 = umma_desc_kmajor_sw128(stage_base);
        const int n_items = npages * items_per_page;
        for (int j = static_cast<int>((n_item + static_cast<uint32_t>(warp - 1)) & 1u); j < n_items && ok; j += kLiMmaWarps) {
          const uint32_t n = n_item + j;
          const int half = items_per_page == 2 ? j & 1 : 0;
          const uint32_t np = n_page + static_cast<uint32_t>(items_per_page == 2 ? j >> 1 : j);
          const uint32_t stage = np % kStages, acc = n & (n_accs - 1u);
          ok = mbar_wait(smem_u32(&ctl->accempty[acc]), ((n >> acc_shift) & 1u) ^ 1u) &&
               mbar_wait(smem_u32(&ctl->full[stage]), (np / kStages) & 1u);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) {
            if (lane == 0) set_status(p.status, PTO_ST_WAIT_EXPIRED, static_cast<int>(n), 3);
            break;
          }
          tc_fence_after();
          const uint64_t a_desc = a_desc0 + ((stage * kStage) >> 4);
          const uint64_t b_desc = b_desc0 + (static_cast<uint32_t>(half * 2 * kQBytesPerToken) >> 4);  // (int8; bf16 has one item)
          const uint32_t idesc = s1 - 2 * half >= 2 ? idesc2 : idesc1;
          const uint32_t d = tmem_base + acc * unit_cols;
          if (elect_one()) {
            if (kBf16) {
              // K = 16 bf16 (32 bytes) per instruction: four steps inside each 64-dim half
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                const uint64_t a = a_desc + ((k >> 2) * (kPageBytes >> 4)) + 2 * (k & 3);
                const uint64_t bq = b_desc + ((k >> 2) * (q_half_bytes >> 4)) + 2 * (k & 3);
                mma_f16_ss(d, a, bq, idesc, k > 0 ? 1u : 0u);
              }
            } else {
#pragma unroll
              for (int k = 0; k < 4; ++k) mma_i8_ss(d, a_desc + 2 * k, b_desc + 2 * k, idesc, k > 0 ? 1u : 0u);
            }
            tc_commit(smem_u32(&ctl->accfull[acc]));
            tc_commit(smem_u32(&ctl->kempty[stage]));
          }
          __syncwarp();
        }
        if (!ok && lane == 0) ctl->abort = 1;
        __syncwarp();
      } else {
        // ---------------- epilogue ----------------
        const int grp = (warp - kLiEpilogueWarp0) >> 2;
        const int quarter = warp & 3;  // TMEM lane quarter this warp may read
        const int row = quarter * 32 + lane;
        // Group g takes the items n with n % 4 == g: there are 4 or 8 accumulators, so an accumulator belongs to one group,
        // which sees every use of it, and consecutive waits on its barriers alternate in parity. (A group that met only
        // every second use of an accumulator would wait twice in a row on the same parity, and the second wait would
        // return at once, before the products are there.)
        const int n_items = npages * items_per_page;
        bool ok = true;
        for (int j = (grp - static_cast<int>(n_item % kLiEpilogueGroups) + kLiEpilogueGroups) % kLiEpilogueGroups; j < n_items;
             j += kLiEpilogueGroups) {
          const uint32_t n = n_item + j;
          const uint32_t acc = n & (n_accs - 1u);
          const int half = items_per_page == 2 ? j & 1 : 0;
          const int page = items_per_page == 2 ? j >> 1 : j;
          const uint32_t np = n_page + static_cast<uint32_t>(page);
          const int cnt = min(2, s1 - 2 * half);  // query tokens of the item
          ok = ok && mbar_wait(smem_u32(&ctl->accfull[acc]), (n >> acc_shift) & 1u);
          if (!ok) {
            ctl->abort = 1;
            set_status(p.status, PTO_ST_WAIT_EXPIRED, static_cast<int>(n), 4);
            if (kMode != kLiQuantTc) break;
          }
          tc_fence_after();
          // the page's scales came in with the page; its `full` phase has completed (the MMA issuer waited on it). Observing
          // it here orders this thread after the bulk copy, unless the stage has been loaded again since: then the
          // wait is for another page, which a bounded probe must not sit out, and the chain issuer -> accumulator orders
          // the copy
          if (!kBf16) mbar_test_wait(smem_u32(&ctl->full[np % kStages]), (np / kStages) & 1u);
          const uint8_t* sc_smem = smem + kLiSmemScales + (np % kLiScaleRing) * kScaleBytes;
          float ks = 1.f;
          if (!kBf16) {
            ks = (p.scale_dtype == PTO_DT_F16) ? __half2float(reinterpret_cast<const __half*>(sc_smem)[row])
                                               : reinterpret_cast<const float*>(sc_smem)[row];
          }
          __half2 ks2 = __float2half2_rn(0.f);
          if (kChain) ks2 = __half2half2(reinterpret_cast<const __half*>(sc_smem)[row]);
          const int pos = (page0 + page) * kPageKeys + row;
          const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * unit_cols;
          const float* ws = ctl->ws + half * 2 * kHeads;
          float res[2];
          if constexpr (kMode == kLiQuantTc) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              if (i < cnt) {
                // The key's 64 values: K elements 2c, 2c + 1 of column c. Sixteen dots at a time, which overwrite columns already
                // read: with all 64 in registers the loop spilled, and a spilled register costs a trip to L2 here (a chunk of 4096
                // tokens over 131072 keys 6.16 -> 5.85 ms).
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  uint32_t v[16], h[8];
                  tmem_ld_32x32b_x16(taddr + i * kHeads + 16 * u, v);
                  tc_wait_ld();
#pragma unroll
                  for (int c = 0; c < 8; ++c) h[c] = relu_scale_half2(static_cast<int>(v[2 * c]), static_cast<int>(v[2 * c + 1]));
                  tmem_st_32x32b_x8(taddr + i * kHeads + 8 * u, h);
                }
              }
            }
            tc_wait_st();
            tc_fence_before();
            // the group's four warps have written theirs; a wait that expired in one of them ends the loop for all four
            if (li_vote<128>(2 + grp, !ok)) break;
            if (((warp - kLiEpilogueWarp0) & 3) == 0) {
              tc_fence_after();
              constexpr uint32_t idesc_sum = umma_idesc(kCFmtF32, 0, 0, 0, 0, 128, 16);  // fp16 x fp16
              const uint64_t w_desc = umma_desc_kmajor_sw128(base + kLiSmemLimbs) + ((half * 2 * kLimbBytes) >> 4);
              const uint32_t unit = tmem_base + acc * unit_cols;
              if (elect_one()) {
                for (int i = 0; i < cnt; ++i) {
#pragma unroll
                  for (int k = 0; k < 4; ++k) {  // K = 16 heads: eight columns of A, 32 bytes of B's rows
                    mma_f16_ts(unit + i * kHeads + 32, unit + i * kHeads + 8 * k, w_desc + i * (kLimbBytes >> 4) + 2 * k, idesc_sum,
                               k > 0 ? 1u : 0u);
                  }
                }
                tc_commit(smem_u32(&ctl->sumfull[acc]));
              }
              __syncwarp();
            }
            ok = mbar_wait(smem_u32(&ctl->sumfull[acc]), (n >> acc_shift) & 1u);
            if (!ok) {  // the group leaves together, at its next barrier
              ctl->abort = 1;
              set_status(p.status, PTO_ST_WAIT_EXPIRED, static_cast<int>(n), 6);
            }
            tc_fence_after();
            uint32_t r[2][16];
            tmem_ld_32x32b_x16(taddr + 32, r[0]);
            if (cnt > 1) tmem_ld_32x32b_x16(taddr + kHeads + 32, r[1]);
            tc_wait_ld();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&ctl->accempty[acc]));
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              if (i < cnt) res[i] = limb_sum(r[i]) * ctl->winv[half * 2 + i] * ks;
            }
          } else {
#pragma unroll
          for (int i = 0; i < (kMode == kLiQuant ? 1 : 2); ++i) {
            if (i < cnt) {
              // One half of the heads after the other: with both in registers, and the code of several tokens in the formulation that
              // is launched for one, these modes spilled (64 sequences of up to 65536 keys 54.6 -> 53.4 us, 8 x 32768 10.9 -> 10.3,
              // bf16 16 x 8192 11.0 -> 10.6).
              float part[2];
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                uint32_t v[32];
                tmem_ld_32x32b_x32(taddr + i * kHeads + 32 * h, v);
                tc_wait_ld();
                if (h == 1 && i == cnt - 1) {
                  // TMEM and the scale row are read: hand the accumulator back before the arithmetic
                  tc_fence_before();
                  __syncwarp();
                  if (lane == 0) mbar_arrive(smem_u32(&ctl->accempty[acc]));
                }
                const float* w = ws + i * kHeads + 32 * h;
                part[h] = kBf16 ? weighted_relu_sum_32(v, w) : (kMode == kLiQuant ? weighted_sum_32(v, w) : chain_sum_32(v, w, ks2));
              }
              res[i] = kChain ? __fadd_rn(part[0], part[1]) : (part[0] + part[1]) * (kBf16 ? 1.f : ks);
            }
          }
          }
          if (pos < seq_len) {
#pragma unroll
            for (int i = 0; i < (kMode == kLiQuant ? 1 : 2); ++i) {
              if (i < cnt) p.scores[(tok0 + 2 * half + i) * p.row_stride + pos] = res[i];
            }
          }
          if (with_hist) {
            // counts for the top-k kernel: positions below the token's causal end
#pragma unroll
            for (int i = 0; i < (kMode == kLiQuant ? 1 : kLiHistMaxS1); ++i) {
              if (i < s1) {
                const int eff = seq_len - (p.s1_total - 1 - (tok_first + i));
                if (pos < eff) atomicAdd(&hist_sm[i * kLiHistBins + (li_float_order(res[i]) >> kLiHistShift)], 1u);
              }
            }
          }
        }
      }
    }
    n_page += npages;
    n_item += npages * items_per_page;
    cur += cost;
    ++seg;
  }

  // teardown
  tc_fence_before();
  __syncthreads();
  if (with_hist && seg > 0) flush_hist(prev_tok0);
  if (ctl->abort) {
    // give copies still in flight time to land before the CTA's shared memory is released
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// ------------------------------------------------------------------------------------------------
// CUDA-core variant (dp4a), one thread per key position. Used to cross-check the tensor-core
// kernel bit for bit and to produce the `first_mm` debug tile.
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128)
li_score_simt_kernel(LiParams p) {
  __shared__ __align__(16) int8_t qs[kMaxS1 * kQBytesPerToken];
  __shared__ float ws[kMaxS1 * kHeads];
  __shared__ __half qsc[kMaxS1 * kHeads], wgt[kMaxS1 * kHeads];  // older formulation: scales and weights apart
  const int bi = blockIdx.y;
  const int page = blockIdx.x;
  const int seq_len = p.act_seq[bi];
  if (page * kPageKeys >= seq_len) return;
  const int s1 = p.s1;
  const int tid = threadIdx.x;
  {
    const int64_t tok0 = static_cast<int64_t>(bi) * p.s1_total + p.tok_offset;
    const int4* src = reinterpret_cast<const int4*>(p.q + tok0 * kQBytesPerToken);
    int4* dst = reinterpret_cast<int4*>(qs);
    for (int i = tid; i < s1 * kQBytesPerToken / 16; i += blockDim.x) dst[i] = src[i];
    for (int e = tid; e < s1 * kHeads; e += blockDim.x) {
      if (p.fp16_chain) {
        qsc[e] = reinterpret_cast<const __half*>(p.q_scale)[tok0 * kHeads + e];
        wgt[e] = reinterpret_cast<const __half*>(p.weight)[tok0 * kHeads + e];
      } else {
        ws[e] = load_ws(p.q_scale, p.weight, p.scale_dtype, tok0 * kHeads + e);
      }
    }
  }
  __syncthreads();
  const int phys = p.block_table[static_cast<int64_t>(bi) * p.max_blocks + page];
  const int pos = page * kPageKeys + tid;
  if (phys < 0 || phys >= p.block_num) {
    // a rejected page scores 0 for every token, as in the tensor-core kernel (where the page reads as zeros):
    // the top-k stage never ranks what an earlier call left in the buffer
    if (tid == 0) set_status(p.status, PTO_ST_BAD_PAGE, phys, 5);
    if (pos < seq_len) {
      for (int i = 0; i < s1; ++i) {
        p.scores[(static_cast<int64_t>(bi) * p.s1_total + p.tok_offset + i) * p.row_stride + pos] = 0.f;
      }
    }
    return;
  }
  if (pos >= seq_len) return;
  int4 kreg[8];
  const int4* krow = reinterpret_cast<const int4*>(p.k_cache + (static_cast<int64_t>(phys) * kPageKeys + tid) * 128);
#pragma unroll
  for (int c = 0; c < 8; ++c) kreg[c] = krow[c];
  const float ks = load_scale(p.k_scale, p.scale_dtype, static_cast<int64_t>(phys) * kPageKeys + tid);
  for (int i = 0; i < s1; ++i) {
    float acc = 0.f;
    for (int h = 0; h < kHeads; ++h) {
      const int4* qrow = reinterpret_cast<const int4*>(qs + (i * kHeads + h) * 128);
      int d = 0;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const int4 qv = qrow[c];
        d = __dp4a(kreg[c].x, qv.x, d);
        d = __dp4a(kreg[c].y, qv.y, d);
        d = __dp4a(kreg[c].z, qv.z, d);
        d = __dp4a(kreg[c].w, qv.w, d);
      }
      if (p.fp16_chain) {
        const __half ksh = reinterpret_cast<const __half*>(p.k_scale)[static_cast<int64_t>(phys) * kPageKeys + tid];
        __half a = __hmul(__hmul(__float2half_rn(static_cast<float>(d) * (1.0f / 2048.0f)), qsc[i * kHeads + h]), ksh);
        a = __hmax(a, __float2half_rn(0.0f));
        acc = __fadd_rn(acc, __half2float(__hmul(a, wgt[i * kHeads + h])));
        continue;
      }
      const float f = fmaxf(static_cast<float>(d), 0.f) * (1.0f / 2048.0f);
      const __half hh = __float2half_rn(f);
      if (p.first_mm != nullptr) {
        reinterpret_cast<__half*>(p.first_mm)[((static_cast<int64_t>(bi) * p.s1_total + p.tok_offset + i) * kHeads + h) * p.row_stride + pos] = hh;
      }
      acc = fmaf(ws[i * kHeads + h], __half2float(hh), acc);
    }
    p.scores[(static_cast<int64_t>(bi) * p.s1_total + p.tok_offset + i) * p.row_stride + pos] = p.fp16_chain ? acc : acc * ks;
  }
}

}  // namespace

cudaError_t launch_li_score_tc(const LiParams& p, const void* tmap_k, const void* tmap_q, int num_sms,
                               cudaStream_t stream) {
  auto kernel = p.bf16 ? li_score_tc_kernel<kLiBf16, false>
                       : (p.fp16_chain ? li_score_tc_kernel<kLiChain, false>
                                       : (p.s1 > 1 ? li_score_tc_kernel<kLiQuantTc, false> : li_score_tc_kernel<kLiQuant, false>));
  // Of one token group, the int8 kernel of several tokens runs faster with the code for groups in it, which it does not use, where pages are
  // many (registers lie otherwise; whole steps, without -> with, us: 128 x 131072 keys, two tokens 815 -> 804, 32 x 131072 218.5 -> 215.2, 64 x 65536,
  // three 398.7 -> 395.8, 16 x 65536, four 133.0 -> 132.3; from 13 to 33 pages a CTA the same; 2 x 8000, two 36.3 -> 37.0). The others gain without.
  constexpr long long kManyPages = 32;  // per CTA
  const bool many_pages = !p.bf16 && !p.fp16_chain && p.s1 > 1 && static_cast<long long>(p.b) * p.max_blocks > kManyPages * num_sms;
  if (p.groups > 1 || many_pages) {  // (a launch of one token has one group)
    kernel = p.bf16 ? li_score_tc_kernel<kLiBf16, true> : (p.fp16_chain ? li_score_tc_kernel<kLiChain, true> : li_score_tc_kernel<kLiQuantTc, true>);
  }
  if (p.hist != nullptr && p.s1 > kLiHistMaxS1) return cudaErrorInvalidValue;
  const size_t smem_bytes = kLiSmemBytes + (p.hist != nullptr ? kLiHistSmemBytes : 0);
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(kLiSmemBytes + kLiHistSmemBytes));
  if (e != cudaSuccess) return e;
  const long long max_items = static_cast<long long>(p.b) * p.max_blocks * p.groups;
  int gx = static_cast<int>(max_items < num_sms ? max_items : num_sms);
  if (gx < 1) gx = 1;
  const dim3 grid(static_cast<unsigned>(gx), 1, 1);
  count_launch();
  kernel<<<grid, kLiThreads, smem_bytes, stream>>>(*reinterpret_cast<const CUtensorMap*>(tmap_k),
                                                                 *reinterpret_cast<const CUtensorMap*>(tmap_q), p);
  return cudaGetLastError();
}

cudaError_t launch_li_score_simt(const LiParams& p, cudaStream_t stream) {
  dim3 grid(p.max_blocks, p.b);
  count_launch();
  li_score_simt_kernel<<<grid, 128, 0, stream>>>(p);
  return cudaGetLastError();
}

int li_max_s1() { return kMaxS1; }
int li_max_s1_bf16() { return kBf16MaxS1; }
int li_max_sequences() { return kMaxSeqPerLaunch; }

}  // namespace pto
