// Sparse MLA attention for a slice of a token's heads (16 .. 112, a device's share of a head-sharded call), on
// tcgen05 with the operands swapped: the selected rows are the M dimension of both products, the heads their N.
//
// Arithmetic as in sfa_pair.cu (reference: examples/models/deepseek_v32_exp/sparse_flash_attention_quant_impl.py:45-207;
// golden deepseekv32_sparse_flash_attention_quant.py:169-254; packed rows sparse_attention_antiquant_impl.py:45-243):
//   S^T[key, head] = K . q^T      M = 128 lanes (kTK keys used), N = kHB heads, K = 576
//   O^T[dim, head] = V^T . P^T    four blocks of M = 128 dims,   N = kHB heads, K = kTK keys
// With few heads a product with the heads as M would pad 16 rows to 128 (the mma.sync kernel this one replaced padded
// them to 64 and took 6.53 ms for 4096 tokens x 2048 rows x 16 heads). Swapped, nothing is padded but the lanes above
// kTK of the score product, and a row is converted ONCE: the bf16 tile [key][64-dim chunk of 128 bytes], 128-byte
// swizzled, is a K-major A operand for S^T and, the same bytes, an MN-major A operand for O^T.
//
// The latent bytes are converted without their scale: an int8 is exact in bf16. The scale of a (row, 128-dim tile) is
// applied where there are few values: to the four partial scores of the row's tiles (one accumulator per tile, the rope
// part a fifth), and, for O^T, whose four M blocks are those same tiles, to the probabilities: block c multiplies
// bf16(p * scale_c). One rounding per (row, tile, head) instead of one per value and one per probability.
//
// Persistent CTAs, one per SM, walk (token, head block, split) items; tiles of kTK rows alternate between two buffers
// and run on across items, so that only the query tile and the output are handed over at an item's end.
//   warp 0          issues the score MMAs of a tile        warp 1   issues the value MMAs of a tile
//   warps 2..3      query tile of the next item (cp.async) warps 4..11 softmax and output (TMEM lane = key / dim), in two
//                   groups of four warps, half of the heads each
//   warps 12..      producers, four rows of a tile each: gather, int8 -> bf16, swizzled stores
// What bounds it: the chain gather -> conversion -> scores -> softmax -> products over two tile buffers. 4096 tokens x 2048 rows
// x 16 heads take 1.82 ms, i.e. 4.8 k cycles per tile of 80 rows, of which the MMAs' issue is 2184 (one with N = 16 takes 39
// cycles, measured in isolation, 32 of them for the 128 lanes of its A operand at the shared memory's 128 bytes a clock; there are
// 36 + 4 kTK/16 of them). No unit is more than half busy: with all MMAs left out it takes 1.35, with all work of the producers left out
// 1.5. All heads in four softmax warps 2.11 ms, two groups of them 2.00; look-ahead before the row loads 1.90; tiles handed over and
// given back in halves, and 48 registers for the issuing warps, which spilled with 40, 1.84; 32-byte loads 1.82.
// Why bf16: a form that multiplied the rows as int8, queries and probabilities as fixed-point limbs, took 1.24 ms, but a
// fixed-point probability has an absolute error: beside a row with 0.96 of the weight the others rounded to zero (rel-L2
// against 64 bits 0.22, 16 heads; this form 0.0020, the mma.sync kernel before it 0.0024).
// kTK: as many rows as leave room for two tile buffers (80 with 16 heads, 64 with 32).
// All waits are bounded.
#include "common.cuh"
#include "sfa_common.cuh"

namespace pto {

namespace {

constexpr int kSliceChunks = 9;  // 8 latent chunks of 64 dims + the rope chunk

template <int kHB, int kTK>
struct SliceCfg {
  static constexpr int kChunk = kTK * 128;                  // kTK rows x 64 bf16
  static constexpr int kTile = kSliceChunks * kChunk;
  static constexpr int kQChunk = kHB * 128;
  static constexpr int kPBytes = kTK * kHB * 2;             // one scaled copy of P^T
  static constexpr int kSmemTile = 0;
  static constexpr int kSmemQ = 2 * kTile;
  static constexpr int kSmemP = kSmemQ + kSliceChunks * kQChunk;  // [buffer][tile c]
  static constexpr int kSmemCtl = kSmemP + 2 * 4 * kPBytes;
  static constexpr int kProdWarps = kTK / 4;
  static constexpr int kH = kHB / 2;                        // heads of a softmax group
  static constexpr int kThreads = 32 * (12 + kProdWarps);
  static constexpr uint32_t kColS = 0;                      // S buffer b, accumulator c at (b * 5 + c) * kHB
  static constexpr uint32_t kColO = 2 * 5 * kHB;            // O block c at kColO + c * kHB
  static constexpr uint32_t kTmemCols = kHB == 16 ? 256 : 512;
  static_assert(kColO + 4 * kHB <= kTmemCols, "tensor memory");
  // registers per thread: at launch, issuers / loaders, softmax, producers (nothing spills: a spilled register costs a trip to L2)
  static constexpr int kRegLaunch = kHB == 16 ? 64 : 72;
  static constexpr int kRegIssue = kHB == 16 ? 48 : 56, kRegSoftmax = kHB == 16 ? 72 : 96, kRegProd = 64;
  static_assert(128 * kRegIssue + 256 * kRegSoftmax + 32 * kProdWarps * kRegProd <= kThreads * kRegLaunch, "register split");
};

template <int kHB, int kTK>
struct SliceCtl {
  __align__(16) float scales[2][kTK][4];  // the tile's row scales
  float live[2][kTK];                     // 1: a row to attend to, 0: padding or rejected
  __align__(16) float mref[kHB];          // reference maximum of a head (log2 units)
  __align__(16) float alpha[kHB];
  float red[4][kHB];
  // Halves of a tile: chunks 0-3, then chunks 4-7, rope part and scales. Each is handed over as it is filled and given back as it is
  // read, so that the scores of the first run beside the conversion of the second.
  uint64_t full[2][2];  // [buffer][half] filled                      (producer warps)
  uint64_t done[2][2];  // P.V of the half complete (commit); of the second: P buffer free, O at rest
  uint64_t sfull[2];  // scores of the tile complete                 (commit)
  uint64_t sfree[2];  // scores read                                 (8 softmax warps)
  uint64_t pfull[2];  // P^T of the tile written                     (8 softmax warps)
  uint64_t qfull;     // query tile of the item loaded               (2 loader warps)
  uint64_t qfree;     // last score product of the item complete     (commit)
  uint64_t ofree;     // output of the item read from tensor memory  (8 softmax warps)
  uint32_t tmem_base;
  int abort;
};

// what a role needs to know of a work item
struct SliceItem {
  int ti, bi, sp, head0, begin, end, ntiles;
};

template <int kTK>
__device__ __forceinline__ SliceItem slice_item(const SfaParams& p, int hb_heads, int item) {
  SliceItem it;
  const int n_hb = (p.nq + hb_heads - 1) / hb_heads;
  it.sp = item % p.n_split;
  item /= p.n_split;
  it.head0 = (item % n_hb) * hb_heads;
  it.ti = item / n_hb;
  it.bi = it.ti / p.s1;
  int n = __ldg(p.act_seq + it.bi) - p.s1 + 1 + it.ti % p.s1;
  n = max(0, min(n, p.topk_k));
  const int tiles_total = (n + kTK - 1) / kTK;
  const int tiles_per_split = (tiles_total + p.n_split - 1) / p.n_split;
  it.begin = min(n, it.sp * tiles_per_split * kTK);
  it.end = min(n, (it.sp + 1) * tiles_per_split * kTK);
  it.ntiles = (it.end - it.begin + kTK - 1) / kTK;
  return it;
}

__device__ __forceinline__ bool slice_wait(uint32_t bar, uint32_t parity) {  // whole warp, bounded, uniform outcome
  if (__all_sync(0xffffffffu, mbar_test_wait(bar, parity))) return true;
  const long long t0 = clock64();
  while (true) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    if (__any_sync(0xffffffffu, clock64() - t0 > kWaitBudgetCycles)) return false;
  }
}

// MN-major B operand of kHB = 16 / 32 heads: rows (keys) of 32 / 64 bytes, 32- / 64-byte swizzle, eight rows per atom
template <int kHB>
__device__ __forceinline__ uint64_t slice_desc_p(uint32_t smem_addr) {
  constexpr uint32_t row = kHB * 2;
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>(1) << 16;                 // one group along the heads
  d |= static_cast<uint64_t>((8 * row) >> 4) << 32;    // eight keys
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(kHB == 16 ? 6 : 4) << 61;  // SWIZZLE_32B / SWIZZLE_64B
  return d;
}

// four int8 -> two bf16 pairs, exact. With the byte b in the low half of a bf16 0x43bb, bits 0-6 are the integers 128 + (b &
// 127) (exponent 2^7, one unit per mantissa step) and bit 7 alone is 128 or 256; their difference is the signed byte.
__device__ __forceinline__ uint2 slice_cvt4(uint32_t w) {
  uint2 o;
  const uint32_t a = __byte_perm(w, 0x43434343u, 0x4140), b = __byte_perm(w, 0x43434343u, 0x4342);
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(o.x) : "r"(a & 0xff7fff7fu), "r"(a & 0xff80ff80u));
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(o.y) : "r"(b & 0xff7fff7fu), "r"(b & 0xff80ff80u));
  return o;
}

// ================================ producers =====================================================
// Warp w owns rows 4w .. 4w+3 of every tile. A gather instruction reads half the latent bytes of two rows (four whole
// 128-byte lines); the eight lanes of a quarter-warp hold four 16-byte units of two neighbouring rows, whose swizzle
// terms differ in the lowest bit, so their stores hit eight different bank groups. (kWide, latent rows on
// 32-byte boundaries: half the latent bytes of all four rows, 32 bytes a lane; eight lanes hold both halves of a 64-dim chunk of
// four rows.) Lane r % 4 walks the look-ahead chain
// of row 4w + r: selected index three tiles ahead, block-table entry two, L2 prefetch of the row two, the row itself
// one tile ahead (into registers, as soon as the tile before it is converted). The chain runs on across items.
template <int kHB, int kTK, bool kPacked, bool kWide>
__device__ __forceinline__ void slice_role_producer(const SfaParams& p, SliceCtl<kHB, kTK>* ctl, uint32_t base, int n_items) {
  using Cfg = SliceCfg<kHB, kTK>;
  const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) - 12;
  const int r = lane & 3, rsel = (lane >> 2) & 1;
  const int src_off = (((lane & 3) | ((lane >> 3) << 2)) << 4);  // this lane's 16 bytes of a half row
  // (the base pointers are read from the parameter block where they are used: they would otherwise occupy six registers)
#define SLICE_KN reinterpret_cast<const uint8_t*>(p.kn)
#define SLICE_KR (kPacked ? SLICE_KN + 512 : reinterpret_cast<const uint8_t*>(p.kr))
#define SLICE_KS (kPacked ? SLICE_KN + 640 : reinterpret_cast<const uint8_t*>(p.kn_scales))
  constexpr int stride_n = kPacked ? 656 : 512, stride_r = kPacked ? 656 : 128, stride_s = kPacked ? 656 : 16;

  int cur_item = blockIdx.x, cur_j = 0;
  SliceItem it = slice_item<kTK>(p, kHB, cur_item);
  // index of this lane's row in the next tile of this CTA (false: no further tile; the same answer in every lane)
  auto fetch = [&](int& idx, int& bi) -> bool {
    while (cur_j >= it.ntiles) {
      cur_item += gridDim.x;
      if (cur_item >= n_items) return false;
      it = slice_item<kTK>(p, kHB, cur_item);
      cur_j = 0;
    }
    const int pos = it.begin + cur_j * kTK + 4 * w + r;
    idx = pos < it.end ? ldg_pinned_i32(p.topk + static_cast<int64_t>(it.ti) * p.topk_k + pos) : -1;
    bi = it.bi;
    ++cur_j;
    return true;
  };
  uint4 d[2][2];  // [row pair][half]: this lane's 16 bytes of row 2 pair + rsel (kWide: [0, 1][half]: its 32 bytes of row r4)
  const int part = lane & 1, r4 = (lane >> 1) & 3;  // kWide
  uint4 rope;     // unit lane % 8 of row lane / 8
  float4 sc;      // the four scales of row r
  int row_loaded = -1;
  // a padding or rejected row reads row 0; it is masked out of the softmax (`live`), its rope part is zeroed
  auto issue_loads = [&](int phys) {
    row_loaded = phys;
    if constexpr (kWide) {
      const int pm = max(__shfl_sync(0xffffffffu, phys, r4), 0);
      const uint8_t* src = SLICE_KN + static_cast<int64_t>(pm) * stride_n + (2 * (lane >> 3) + part) * 32;
      ldg_pinned_v8(src, d[0][0], d[1][0]);
      ldg_pinned_v8(src + 256, d[0][1], d[1][1]);
    } else {
#pragma unroll
      for (int pr = 0; pr < 2; ++pr) {
        const int pm = max(__shfl_sync(0xffffffffu, phys, 2 * pr + rsel), 0);
        const uint8_t* src = SLICE_KN + static_cast<int64_t>(pm) * stride_n + src_off;
        d[pr][0] = ldg_pinned_v4(src);
        d[pr][1] = ldg_pinned_v4(src + 256);
      }
    }
    const int px = __shfl_sync(0xffffffffu, phys, lane >> 3);
    rope = make_uint4(0, 0, 0, 0);
    if (px >= 0) rope = ldg_pinned_v4(SLICE_KR + static_cast<int64_t>(px) * stride_r + (lane & 7) * 16);
    uint4 s4 = make_uint4(0, 0, 0, 0);
    if (phys >= 0) s4 = ldg_pinned_v4(SLICE_KS + static_cast<int64_t>(phys) * stride_s);
    sc = make_float4(__uint_as_float(s4.x), __uint_as_float(s4.y), __uint_as_float(s4.z), __uint_as_float(s4.w));
  };
  auto prefetch_row = [&](int phys) {  // lanes r, r+4, ...: one line of the row each
    if (phys < 0) return;
    const int l = lane >> 2;
    if (kPacked) {
      if (l < 6) asm volatile("prefetch.global.L2 [%0];" ::"l"(SLICE_KN + static_cast<int64_t>(phys) * 656 + min(l * 128, 640)));
    } else {
      if (l < 4) asm volatile("prefetch.global.L2 [%0];" ::"l"(SLICE_KN + static_cast<int64_t>(phys) * 512 + l * 128));
      else if (l == 4) asm volatile("prefetch.global.L2 [%0];" ::"l"(SLICE_KR + static_cast<int64_t>(phys) * 128));
      else if (l == 5) asm volatile("prefetch.global.L2 [%0];" ::"l"(SLICE_KS + static_cast<int64_t>(phys) * 16));
    }
  };

  int idx_n = -1, bi_n = 0, idx_a = -1, bi_a = 0, entry_a = kTableSkip, row_n = -1;
  bool has = false, has_n = false, has_a = false;
  {
    int idx0 = -1, bi0 = 0;
    has = fetch(idx0, bi0);
    has_n = has && fetch(idx_n, bi_n);
    has_a = has_n && fetch(idx_a, bi_a);
    const int e0 = has ? tc_table_entry(p, bi0, idx0) : kTableSkip;
    const int e1 = has_n ? tc_table_entry(p, bi_n, idx_n) : kTableSkip;
    if (has_a) entry_a = tc_table_entry(p, bi_a, idx_a);
    if (has) issue_loads(tc_row_from_entry(p, idx0, e0));
    if (has_n) {
      row_n = tc_row_from_entry(p, idx_n, e1);
      prefetch_row(row_n);
    }
  }
  bool ok = true;
  for (uint32_t t = 0; has; ++t) {
    const uint32_t b = t & 1;
    // the tile after the next: index (requested now, used at the end of this step) and block-table entry
    int idx_b = -1, bi_b = 0;
    const bool has_b = has_a && fetch(idx_b, bi_b);
    const uint32_t tile = base + Cfg::kSmemTile + b * Cfg::kTile;
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      if (t >= 2) {
        ok = slice_wait(smem_u32(&ctl->done[b][hf]), ((t >> 1) - 1) & 1);
        if (!ok) break;
      }
#pragma unroll
      for (int pr = 0; pr < 2; ++pr) {
        const int row = 4 * w + (kWide ? r4 : 2 * pr + rsel), x = row & 7;
        const uint32_t dst = tile + (4 * hf + (lane >> 3)) * Cfg::kChunk + row * 128;
        const int unit = kWide ? 4 * part + 2 * pr : 2 * (lane & 3);  // first of the two 16-byte units of the chunk's 128 bytes
        const uint32_t a = (unit ^ x) << 4, c = ((unit + 1) ^ x) << 4;
        const uint4 v = d[pr][hf];
        const uint2 v0 = slice_cvt4(v.x), v1 = slice_cvt4(v.y), v2 = slice_cvt4(v.z), v3 = slice_cvt4(v.w);
        sts_v4u(dst + a, make_uint4(v0.x, v0.y, v1.x, v1.y));
        sts_v4u(dst + c, make_uint4(v2.x, v2.y, v3.x, v3.y));
      }
      if (hf == 1) {
        const int row = 4 * w + (lane >> 3);
        sts_v4u(tile + 8 * Cfg::kChunk + row * 128 + (((lane & 7) ^ (row & 7)) << 4), rope);
        if (lane < 4) {
          *reinterpret_cast<float4*>(&ctl->scales[b][4 * w + lane][0]) = sc;
          ctl->live[b][4 * w + lane] = row_loaded >= 0 ? 1.f : 0.f;
        }
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl->full[b][hf]));
    }
    if (!ok) break;
    // The look-ahead comes before the row loads: what it waits for was requested a tile ago, but a wait behind the row loads
    // is a wait for these too (loads share the few scoreboards of a warp).
    has = has_n;
    const int row_next = row_n;
    has_n = has_a;
    if (has_a) {
      row_n = tc_row_from_entry(p, idx_a, entry_a);
      prefetch_row(row_n);
    }
    has_a = has_b;
    idx_a = idx_b;
    if (has_b) entry_a = tc_table_entry(p, bi_b, idx_b);
    if (has) issue_loads(row_next);
  }
  if (!ok && lane == 0) {
    ctl->abort = 1;
    set_status(p.status, PTO_ST_WAIT_EXPIRED, blockIdx.x, 90);
  }
}

// ================================ MMA issuers ====================================================
// What an MMA of this size costs is its issue: measured in isolation, 51-61 cycles whatever the shape when one lane
// issues under `if (lane == 0)`, where the descriptors are moved to uniform registers for every MMA, against 39 (N = 16)
// when the warp stays converged and an elected lane issues. Here, beside 26 busy warps, the descriptors have to be
// constants of the code for that (kBase, the address where a kernel without static shared memory finds its dynamic
// part; kBase = 0 is the same code with the address in a register): 2.25 -> 2.05 ms for 4096 tokens of 16 heads.
constexpr uint32_t kSliceUsualBase = 1024;
template <int kHB, int kTK, int kHalf>
__device__ __forceinline__ void slice_issue_scores(uint32_t d, uint64_t a_desc, uint64_t b_desc) {
  using Cfg = SliceCfg<kHB, kTK>;
  constexpr uint32_t idesc = umma_idesc(kCFmtF32, kABFmtBF16, kABFmtBF16, 0, 0, 128, kHB);
#pragma unroll
  for (int ch = 4 * kHalf; ch < (kHalf == 0 ? 4 : kSliceChunks); ++ch) {  // accumulator ch / 2: one per scale tile, the rope part the fifth
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      mma_f16_ss(d + (ch >> 1) * kHB, a_desc + ch * (Cfg::kChunk >> 4) + 2 * k, b_desc + ch * (Cfg::kQChunk >> 4) + 2 * k,
                 idesc, ((ch & 1) | k) != 0 ? 1u : 0u);
    }
  }
}
template <int kHB, int kTK, int kHalf>
__device__ __forceinline__ void slice_issue_values(uint32_t d, uint64_t a_desc, uint64_t b_desc, uint32_t accumulate) {
  using Cfg = SliceCfg<kHB, kTK>;
  constexpr uint32_t idesc = umma_idesc(kCFmtF32, kABFmtBF16, kABFmtBF16, 1, 1, 128, kHB);
#pragma unroll
  for (int c = 2 * kHalf; c < 2 * kHalf + 2; ++c) {
#pragma unroll
    for (int k = 0; k < kTK / 16; ++k) {  // 16 rows per step: 2 KB of a chunk, 16 rows of the tile's copy of P^T
      mma_f16_ss(d + c * kHB, a_desc + c * (2 * Cfg::kChunk >> 4) + k * (2048 >> 4),
                 b_desc + c * (Cfg::kPBytes >> 4) + k * ((16 * kHB * 2) >> 4), idesc, k > 0 ? 1u : accumulate);
    }
  }
}

template <int kHB, int kTK, uint32_t kBase>
__device__ __forceinline__ void slice_role_scores(const SfaParams& p, SliceCtl<kHB, kTK>* ctl, uint32_t base, uint32_t tmem,
                                                  int n_items) {
  using Cfg = SliceCfg<kHB, kTK>;
  if (kBase != 0) base = kBase;
  const uint64_t a_desc = umma_desc_kmajor_sw128(base + Cfg::kSmemTile), b_desc = umma_desc_kmajor_sw128(base + Cfg::kSmemQ);
  bool ok = true;
  uint32_t t = 0, n = 0;
  for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
    const int ntiles = slice_item<kTK>(p, kHB, item).ntiles;
    if (ntiles == 0) continue;
    ok = slice_wait(smem_u32(&ctl->qfull), n & 1);
    for (int j = 0; j < ntiles && ok; ++j, ++t) {
      const uint32_t b = t & 1;
      if (t >= 2) ok = slice_wait(smem_u32(&ctl->sfree[b]), ((t >> 1) - 1) & 1);
      ok = ok && slice_wait(smem_u32(&ctl->full[b][0]), (t >> 1) & 1);
      if (!ok) break;
      tc_fence_after();
      const uint32_t d = tmem + Cfg::kColS + b * 5 * kHB;
      if (elect_one()) slice_issue_scores<kHB, kTK, 0>(d, a_desc + b * (Cfg::kTile >> 4), b_desc);
      __syncwarp();
      ok = slice_wait(smem_u32(&ctl->full[b][1]), (t >> 1) & 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        slice_issue_scores<kHB, kTK, 1>(d, a_desc + b * (Cfg::kTile >> 4), b_desc);
        tc_commit(smem_u32(&ctl->sfull[b]));
        if (j + 1 == ntiles) tc_commit(smem_u32(&ctl->qfree));
      }
      __syncwarp();
    }
    ++n;
  }
  if (!ok && (threadIdx.x & 31) == 0) {
    ctl->abort = 1;
    set_status(p.status, PTO_ST_WAIT_EXPIRED, blockIdx.x, 91);
  }
  __syncwarp();
}

template <int kHB, int kTK, uint32_t kBase>
__device__ __forceinline__ void slice_role_values(const SfaParams& p, SliceCtl<kHB, kTK>* ctl, uint32_t base, uint32_t tmem,
                                                  int n_items) {
  using Cfg = SliceCfg<kHB, kTK>;
  if (kBase != 0) base = kBase;
  const uint64_t a_desc = desc_mnmajor_sw128(base + Cfg::kSmemTile, Cfg::kChunk, 1024);
  const uint64_t b_desc = slice_desc_p<kHB>(base + Cfg::kSmemP);
  bool ok = true;
  uint32_t t = 0, n = 0;
  for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
    const int ntiles = slice_item<kTK>(p, kHB, item).ntiles;
    if (ntiles == 0) continue;
    if (n > 0) ok = slice_wait(smem_u32(&ctl->ofree), (n - 1) & 1);
    for (int j = 0; j < ntiles && ok; ++j, ++t) {
      const uint32_t b = t & 1;
      ok = slice_wait(smem_u32(&ctl->pfull[b]), (t >> 1) & 1) && slice_wait(smem_u32(&ctl->full[b][1]), (t >> 1) & 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        const uint64_t a = a_desc + b * (Cfg::kTile >> 4), pb = b_desc + b * (4 * Cfg::kPBytes >> 4);
        slice_issue_values<kHB, kTK, 0>(tmem + Cfg::kColO, a, pb, j > 0 ? 1u : 0u);
        tc_commit(smem_u32(&ctl->done[b][0]));
        slice_issue_values<kHB, kTK, 1>(tmem + Cfg::kColO, a, pb, j > 0 ? 1u : 0u);
        tc_commit(smem_u32(&ctl->done[b][1]));
      }
      __syncwarp();
    }
    ++n;
  }
  if (!ok && (threadIdx.x & 31) == 0) {
    ctl->abort = 1;
    set_status(p.status, PTO_ST_WAIT_EXPIRED, blockIdx.x, 92);
  }
  __syncwarp();
}

// ================================ query tile =====================================================
template <int kHB, int kTK>
__device__ __forceinline__ void slice_role_query(const SfaParams& p, SliceCtl<kHB, kTK>* ctl, uint32_t base, int n_items) {
  using Cfg = SliceCfg<kHB, kTK>;
  const int tid = threadIdx.x - 64;  // 0..63
  bool ok = true;
  uint32_t n = 0;
  for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
    const SliceItem it = slice_item<kTK>(p, kHB, item);
    if (it.ntiles == 0) continue;
    const int64_t row0 = static_cast<int64_t>(it.ti) * p.nq_total + p.head_begin + it.head0;
    if (n > 0) {
      // the rows are wanted in L2 by the time the previous item's last score product lets go of the buffer
      for (int e = tid; e < kHB * 8; e += 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.q_nope + row0 * 512 + e * 64));
      for (int e = tid; e < kHB; e += 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.q_rope + row0 * 64 + e * 64));
      ok = slice_wait(smem_u32(&ctl->qfree), (n - 1) & 1);
      if (!ok) break;
    }
    for (int e = tid; e < kHB * 72; e += 64) {
      const int r = e / 72, u = e % 72;
      cp_async_16(base + Cfg::kSmemQ + (u >> 3) * Cfg::kQChunk + r * 128 + (((u & 7) ^ (r & 7)) << 4),
                  u < 64 ? p.q_nope + (row0 + r) * 512 + u * 8 : p.q_rope + (row0 + r) * 64 + (u - 64) * 8, 16u);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    fence_proxy_async();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(smem_u32(&ctl->qfull));
    ++n;
  }
  if (!ok && (threadIdx.x & 31) == 0) {
    ctl->abort = 1;
    set_status(p.status, PTO_ST_WAIT_EXPIRED, blockIdx.x, 93);
  }
}

// ================================ softmax and output =============================================
// Two groups of four warps, each with half of the heads; TMEM lane = key of the tile (warp q of a group holds keys 32q .. +31;
// lanes above kTK take part in the barriers only). A thread has one key's scores for its group's kH heads: the scores ->
// probabilities chain of a tile sits between its two products, and half as many heads are half as long a chain.
// The reference maximum of a head moves only when a score exceeds it by more than 2^8 (first tile: always), which one vote over the
// group finds out; so the reduction over keys, here across lanes, is rare, and the row sums stay per-thread partials until the
// item ends.
constexpr float kSliceRescale = 8.0f;

template <int kH>
__device__ __forceinline__ void slice_ld(uint32_t taddr, float (&v)[kH]) {
  uint32_t r[kH];
  if constexpr (kH == 8) tmem_ld_32x32b_x8(taddr, r);
  else tmem_ld_32x32b_x16(taddr, r);
  tc_wait_ld();
#pragma unroll
  for (int h = 0; h < kH; ++h) v[h] = __uint_as_float(r[h]);
}

__device__ __forceinline__ bool slice_vote(int group, bool pred) {  // OR over the group's four warps; also their barrier
  uint32_t any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %2, 0;\n\tbarrier.cta.red.or.pred q, %1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(any)
      : "r"(1 + group), "r"(pred ? 1u : 0u)
      : "memory");
  return any != 0;
}
__device__ __forceinline__ void slice_meet(int group) { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); }

template <int kHB, int kTK>
__device__ __forceinline__ void slice_role_softmax(const SfaParams& p, SliceCtl<kHB, kTK>* ctl, uint32_t base, uint32_t tmem,
                                                   int n_items) {
  using Cfg = SliceCfg<kHB, kTK>;
  constexpr int kH = Cfg::kH;
  const int lane = threadIdx.x & 31, quarter = (threadIdx.x >> 5) & 3;
  const int group = (threadIdx.x >> 7) - 1, tid = threadIdx.x & 127;  // heads kH group .. + kH - 1 of the block; thread of the group
  const int h0 = kH * group;
  float* const mref = ctl->mref + h0;
  float* const alpha = ctl->alpha + h0;
  const int key = 32 * quarter + lane;
  const uint32_t lane_addr = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
  bool ok = true;
  uint32_t t = 0;
  for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
    const SliceItem it = slice_item<kTK>(p, kHB, item);
    const int64_t orow0 = static_cast<int64_t>(it.ti) * p.nq_total + p.head_begin + it.head0 + h0;
    const int64_t prow0 = (static_cast<int64_t>(it.ti) * p.n_split + it.sp) * p.nq + it.head0 + h0;
    if (it.ntiles == 0) {
      if (p.n_split == 1) {
        for (int e = tid; e < kH * 64; e += 128) *reinterpret_cast<uint4*>(p.out + orow0 * 512 + e * 8) = make_uint4(0, 0, 0, 0);
      } else if (tid < kH) {
        p.part_ml[(prow0 + tid) * 2] = -INFINITY;
        p.part_ml[(prow0 + tid) * 2 + 1] = 0.f;
      }
      continue;
    }
    float l[kH];
#pragma unroll
    for (int h = 0; h < kH; ++h) l[h] = 0.f;
    for (int j = 0; j < it.ntiles; ++j, ++t) {
      const uint32_t b = t & 1;
      // (a wait that expired is voted on below, so that the group's four warps leave together: one that left alone would leave the
      // others at a barrier)
      ok = ok && slice_wait(smem_u32(&ctl->sfull[b]), (t >> 1) & 1) && slice_wait(smem_u32(&ctl->full[b][1]), (t >> 1) & 1);
      tc_fence_after();
      float s[kH];
      float4 sc = make_float4(0.f, 0.f, 0.f, 0.f);
      bool valid = false;
      if (32 * quarter < kTK) {
        const uint32_t col = lane_addr + Cfg::kColS + b * 5 * kHB + h0;
        if (key < kTK) {
          sc = *reinterpret_cast<const float4*>(&ctl->scales[b][key][0]);
          valid = ctl->live[b][key] != 0.f && it.begin + j * kTK + key < it.end;
        }
        slice_ld<kH>(col + 4 * kHB, s);  // rope part
        const float scv[4] = {sc.x, sc.y, sc.z, sc.w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float x[kH];
          slice_ld<kH>(col + c * kHB, x);
#pragma unroll
          for (int h = 0; h < kH; ++h) s[h] = fmaf(x[h], scv[c], s[h]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl->sfree[b]));
      float over = -INFINITY;
#pragma unroll
      for (int h = 0; h < kH; ++h) {
        s[h] = valid ? s[h] * p.scale_log2 : -INFINITY;
        over = fmaxf(over, s[h] - (j > 0 ? mref[h] : 0.f));
      }
      if (slice_vote(group, j == 0 || over > kSliceRescale || !ok)) {
        // ---- new reference maxima --------------------------------------------------------------------
#pragma unroll
        for (int h = 0; h < kH; ++h) {
          float m = s[h];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
          if (lane == 0) ctl->red[quarter][h0 + h] = m;
        }
        if (slice_vote(group, !ok)) {
          ok = false;
          break;
        }
        if (tid < kH) {
          const float old = j > 0 ? mref[tid] : -INFINITY;
          const float m = fmaxf(fmaxf(ctl->red[0][h0 + tid], ctl->red[1][h0 + tid]), fmaxf(ctl->red[2][h0 + tid], ctl->red[3][h0 + tid]));
          const float mn = fmaxf(old, m);
          alpha[tid] = old == -INFINITY ? 0.f : ex2f(old - mn);
          mref[tid] = mn;
        }
        slice_meet(group);
        if (j > 0) {
          ok = slice_wait(smem_u32(&ctl->done[b ^ 1][1]), ((t - 1) >> 1) & 1);  // the output so far is at rest
          if (ok) tc_fence_after();
#pragma unroll
          for (int h = 0; h < kH; ++h) l[h] *= alpha[h];
          if (ok) {
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
              uint32_t o[kH];
              const uint32_t taddr = lane_addr + Cfg::kColO + c * kHB + h0;
              if constexpr (kH == 8) tmem_ld_32x32b_x8(taddr, o);
              else tmem_ld_32x32b_x16(taddr, o);
              tc_wait_ld();
#pragma unroll
              for (int e = 0; e < kH; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha[e]);
              if constexpr (kH == 8) tmem_st_32x32b_x8(taddr, o);
              else tmem_st_32x32b_x16(taddr, o);
            }
            tc_wait_st();
          }
          if (slice_vote(group, !ok)) {  // (alpha is read; a later tile may write it)
            ok = false;
            break;
          }
        }
      }
#pragma unroll
      for (int h = 0; h < kH; ++h) {
        const float m = mref[h];
        s[h] = ex2f(s[h] - (m == -INFINITY ? 0.f : m));
        l[h] += s[h];
      }
      if (t >= 2) {  // the products that read this P buffer are complete
        ok = slice_wait(smem_u32(&ctl->done[b][1]), ((t >> 1) - 1) & 1) && ok;
      }
      if (ok && key < kTK) {
        const float scv[4] = {sc.x, sc.y, sc.z, sc.w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint32_t row = base + Cfg::kSmemP + (b * 4 + c) * Cfg::kPBytes + key * kHB * 2;
#pragma unroll
          for (int u = 0; u < kH / 8; ++u) {
            uint4 w;
            w.x = pack_bf16x2(s[8 * u] * scv[c], s[8 * u + 1] * scv[c]);
            w.y = pack_bf16x2(s[8 * u + 2] * scv[c], s[8 * u + 3] * scv[c]);
            w.z = pack_bf16x2(s[8 * u + 4] * scv[c], s[8 * u + 5] * scv[c]);
            w.w = pack_bf16x2(s[8 * u + 6] * scv[c], s[8 * u + 7] * scv[c]);
            // swizzle: 32-byte rows, unit ^= (row / 4) % 2; 64-byte rows, unit ^= (row / 2) % 4
            const int x = kHB == 16 ? (key >> 2) & 1 : (key >> 1) & 3;
            sts_v4u(row + (((h0 / 8 + u) ^ x) << 4), w);
          }
        }
      }
      fence_proxy_async();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl->pfull[b]));
    }
    // (a `done` that expired at the last tile; the break above comes with the same answer in the whole group)
    if (slice_vote(group, !ok)) {
      ok = false;
      break;
    }
    // ---- output --------------------------------------------------------------------------------------
#pragma unroll
    for (int h = 0; h < kH; ++h) {
      float v = l[h];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) ctl->red[quarter][h0 + h] = v;
    }
    slice_meet(group);
    if (tid < kH) {
      const float tot = (ctl->red[0][h0 + tid] + ctl->red[1][h0 + tid]) + (ctl->red[2][h0 + tid] + ctl->red[3][h0 + tid]);
      if (p.n_split == 1) {
        alpha[tid] = tot > 0.f ? 1.f / tot : 0.f;
      } else {
        alpha[tid] = 1.f;
        p.part_ml[(prow0 + tid) * 2] = mref[tid];
        p.part_ml[(prow0 + tid) * 2 + 1] = tot;
      }
    }
    slice_meet(group);
    ok = slice_wait(smem_u32(&ctl->done[(t - 1) & 1][1]), ((t - 1) >> 1) & 1);
    tc_fence_after();
#pragma unroll
    for (int c = 0; c < 4 && ok; ++c) {  // dim 128 c + key of every head: 32 lanes write consecutive dims of a head's row
      float o[kH];
      slice_ld<kH>(lane_addr + Cfg::kColO + c * kHB + h0, o);
      if (c == 3) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctl->ofree));
      }
#pragma unroll
      for (int h = 0; h < kH; ++h) {
        const float v = o[h] * alpha[h];
        if (p.n_split == 1) p.out[(orow0 + h) * 512 + 128 * c + key] = __float2bfloat16_rn(v);
        else p.part_o[(prow0 + h) * 512 + 128 * c + key] = v;
      }
    }
    if (slice_vote(group, !ok)) ok = false;  // (alpha and mref are read; the next item may write them)
  }
  if (!ok && lane == 0) {
    ctl->abort = 1;
    set_status(p.status, PTO_ST_WAIT_EXPIRED, blockIdx.x, 94);
  }
}

template <int kHB, int kTK>
__global__ void __launch_bounds__(SliceCfg<kHB, kTK>::kThreads, 1)
sfa_slice_kernel(const __grid_constant__ SfaParams p, int n_items) {
  using Cfg = SliceCfg<kHB, kTK>;
  extern __shared__ __align__(1024) uint8_t sfa_slice_smem[];
  const uint32_t base = smem_u32(sfa_slice_smem);
  if ((base & 1023u) != 0) {  // the swizzled operand tiles need a 1024-byte aligned base
    if (threadIdx.x == 0) set_status(p.status, PTO_ST_WAIT_EXPIRED, static_cast<int>(base), 95);
    return;
  }
  auto* ctl = reinterpret_cast<SliceCtl<kHB, kTK>*>(sfa_slice_smem + Cfg::kSmemCtl);
  const int tid = threadIdx.x, warp = tid >> 5;
  if (tid == 0) {
    for (int b = 0; b < 2; ++b) {
      for (int hf = 0; hf < 2; ++hf) {
        mbar_init(smem_u32(&ctl->full[b][hf]), Cfg::kProdWarps);
        mbar_init(smem_u32(&ctl->done[b][hf]), 1);
      }
      mbar_init(smem_u32(&ctl->sfull[b]), 1);
      mbar_init(smem_u32(&ctl->sfree[b]), 8);
      mbar_init(smem_u32(&ctl->pfull[b]), 8);
    }
    mbar_init(smem_u32(&ctl->qfull), 2);
    mbar_init(smem_u32(&ctl->qfree), 1);
    mbar_init(smem_u32(&ctl->ofree), 8);
    ctl->abort = 0;
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(&ctl->tmem_base), Cfg::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ctl->tmem_base;
  pdl_wait();  // the set-up above overlaps the tail of the kernel before this one
  if (tid == 0) pdl_trigger();
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::kRegIssue));
    if (warp < 2 && base == kSliceUsualBase) {
      if (warp == 0) slice_role_scores<kHB, kTK, kSliceUsualBase>(p, ctl, base, tmem, n_items);
      else slice_role_values<kHB, kTK, kSliceUsualBase>(p, ctl, base, tmem, n_items);
    } else if (warp == 0) slice_role_scores<kHB, kTK, 0>(p, ctl, base, tmem, n_items);
    else if (warp == 1) slice_role_values<kHB, kTK, 0>(p, ctl, base, tmem, n_items);
    else slice_role_query<kHB, kTK>(p, ctl, base, n_items);
  } else if (warp < 12) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Cfg::kRegSoftmax));
    slice_role_softmax<kHB, kTK>(p, ctl, base, tmem, n_items);
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::kRegProd));
    if (p.packed) slice_role_producer<kHB, kTK, true, false>(p, ctl, base, n_items);
    else if (p.kn_wide) slice_role_producer<kHB, kTK, false, true>(p, ctl, base, n_items);
    else slice_role_producer<kHB, kTK, false, false>(p, ctl, base, n_items);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, Cfg::kTmemCols);
  }
}

template <int kHB, int kTK>
cudaError_t launch_one(const SfaParams& p, int num_sms, cudaStream_t stream) {
  using Cfg = SliceCfg<kHB, kTK>;
  constexpr size_t smem = Cfg::kSmemCtl + sizeof(SliceCtl<kHB, kTK>);
  static_assert(smem <= 232448, "exceeds the 227 KB of shared memory a CTA may use");
  auto kernel = sfa_slice_kernel<kHB, kTK>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  const long long items = static_cast<long long>(p.b) * p.s1 * (p.nq / kHB) * p.n_split;
  if (items > 0x7fffffffLL) return cudaErrorInvalidValue;
  const int grid = static_cast<int>(items < num_sms ? items : num_sms);
  count_launch();
  return launch_maybe_pdl(kernel, dim3(grid), dim3(Cfg::kThreads), smem, stream, p.pdl != 0, p, static_cast<int>(items));
}

}  // namespace

int sfa_slice_heads(int nq) { return nq % 32 == 0 ? 32 : 16; }

cudaError_t launch_sfa_slice(const SfaParams& p, int num_sms, cudaStream_t stream) {
  return sfa_slice_heads(p.nq) == 32 ? launch_one<32, 64>(p, num_sms, stream) : launch_one<16, 80>(p, num_sms, stream);
}

}  // namespace pto
