// Sparse MLA attention for a slice of a token's heads (16 .. 112, a device's share of a head-sharded call), on
// tcgen05 with the operands swapped and the latent rows left as they are: int8.
//
// Arithmetic as in sfa_pair.cu (reference: examples/models/deepseek_v32_exp/sparse_flash_attention_quant_impl.py:45-207;
// golden deepseekv32_sparse_flash_attention_quant.py:169-254; packed rows sparse_attention_antiquant_impl.py:45-243):
//   S^T[key, head] = K . q^T      M = 128 keys,                N = 16 heads, K = 576
//   O^T[dim, head] = V^T . P^T    four blocks of M = 128 dims, N = 16 heads, K = 128 keys
// With few heads a product with the heads as M would pad 16 rows to 128. Swapped, nothing is padded, and the same tile
// [key][128-byte chunk], 128-byte swizzled, is a K-major A operand for S^T and an MN-major A operand for O^T.
//
// The latent part is multiplied as int8 (kind::i8, exact): the gathered bytes go straight from L2 to the operand tile, no
// conversion stands between. A chunk is one 128-dim tile with its scale, so the scale of a (row, tile) is applied where
// there are few values: to the four partial scores of the row, and, for O^T, to the probabilities of block c.
//   q          per head a fixed-point number of 14 bits and sign below the head's largest |q| (a power of two), as two int8
//              limbs: columns 0-15 and 16-31 of the product, combined in int32. bf16 values down to 2^-6 of the largest are
//              exact, smaller ones are off by at most 2^-14 of it; the bf16 rounding of the dequantised keys (2^-9 of every
//              term) that other forms of this product carry is not there.
//   p scale_c  per tile and chunk a fixed-point number below twice the tile's largest |scale_c|, again as two limbs (the
//              reference maximum of a head follows its scores within a factor of two): 2^-14 of the largest, against 2^-9
//              of each value when the scaled probabilities are bf16.
//   rope part  bf16 x bf16 -> fp32 as before.
// The int32 results of a tile's O^T are added to fp32 accumulators in registers with the tile's factor.
//
// Persistent CTAs, one per SM, walk (token, block of 16 heads, split) items; tiles of 128 rows alternate between two
// buffers and run on across items; the query tile is double-buffered too.
//   warp 0          issues the score MMAs of a tile        warp 1   issues the value MMAs of a tile
//   warps 2..3      query tile of the next item            warps 4..11  softmax (TMEM lane = key, eight heads per warp)
//   warps 12..15    output (TMEM lane = dim)               warps 16..23 producers, 16 rows of a tile each (cp.async)
// What bounds it: the issue of 36 MMAs of 39 cycles per 128 rows (N = 32: any smaller shape costs as much) and the softmax
// warps' instruction stream beside it. History at 4096 tokens x 2048 rows x 16 heads: mma.sync with 64-row tiles 6.53
// ms; swapped, rows converted to bf16 by the producers (5.6 k cycles per 80 rows) 2.10 ms.
// All waits are bounded.
#include "common.cuh"
#include "sfa_common.cuh"

namespace pto {

namespace {

constexpr int kSHeads = 16;                  // heads per work item
constexpr int kSRows = 128;                  // selected rows per tile
constexpr int kSChunk = kSRows * 128;        // 128 rows x 128 bytes: one dim tile of int8, or the bf16 rope part
constexpr int kSTile = 5 * kSChunk;          // chunks 0-3 latent, chunk 4 rope
constexpr int kSQChunk = 2 * kSHeads * 128;  // two limbs of 16 heads x 128 dims
constexpr int kSQRope = kSHeads * 128;
constexpr int kSQ = 4 * kSQChunk + kSQRope;
constexpr int kSPBlock = kSRows * 2 * kSHeads;  // P^T of one dim tile: per key 16 high and 16 low limbs
constexpr int kSSmemTile = 0;
constexpr int kSSmemQ = 2 * kSTile;
constexpr int kSSmemP = kSSmemQ + 2 * kSQ;
constexpr int kSSmemCtl = kSSmemP + 4 * kSPBlock;
constexpr int kSSoftWarp0 = 4, kSSoftWarps = 8, kSOutWarp0 = 12, kSProdWarp0 = 16, kSProdWarps = 8;
constexpr int kSThreads = 32 * (kSProdWarp0 + kSProdWarps);
constexpr uint32_t kSTmemCols = 512;
constexpr uint32_t kSColS = 0, kSSBuf = 4 * 2 * kSHeads + kSHeads;  // S buffer b: four blocks of two limbs, then the rope part
constexpr uint32_t kSColO = 2 * kSSBuf;                             // O block c at kSColO + 32 c
static_assert(kSColO + 4 * 2 * kSHeads <= kSTmemCols, "tensor memory");
// registers per thread: at launch, and after the split (six groups of four warps)
constexpr int kSRegIssue = 56, kSRegSoft = 96, kSRegOut = 120, kSRegProd = 56, kSRegLaunch = 80;
static_assert(kSRegIssue + 2 * kSRegSoft + kSRegOut + 2 * kSRegProd <= 6 * kSRegLaunch, "register split");
constexpr float kSRescale = 1.0f;   // log2 units a score may exceed its head's reference: p <= 2
constexpr float kSPUnit = 8191.0f;  // fixed-point units of p = 1: 2 * 8191 fits 7 + 7 bits

struct SliceCtl {
  __align__(16) float scales[2][kSRows][4];  // the tile's row scales
  float live[2][kSRows];                     // 1: a row to attend to, 0: padding or rejected
  __align__(16) float smax[2][4][4];         // [tile parity][lane quarter][c]: largest |scale_c|
  __align__(16) float fac[2][4];             // [tile parity][c]: value of a unit of the tile's O^T
  __align__(16) float alpha[2][kSHeads];     // [tile parity]: factor for what was summed before
  int rescale[2];
  __align__(16) float mref[kSHeads];         // reference maximum of a head (log2 units)
  __align__(16) float red[4][kSHeads];
  __align__(16) float linv[2][kSHeads];      // [item parity]
  __align__(16) float qunit[4][kSHeads];     // [item % 4]: value of a unit of the head's query limbs
  uint64_t full[2];   // rows of the tile landed                     (8 producer warps)
  uint64_t done[2];   // O^T of the tile complete: tile buffer and P free (commit)
  uint64_t sfull[2];  // scores of the tile complete                 (commit)
  uint64_t sfree[2];  // scores read                                 (8 softmax warps)
  uint64_t pfull;     // P^T of the tile written                     (8 softmax warps)
  uint64_t ofree;     // O^T of the tile read                        (4 output warps)
  uint64_t qfull[2];  // query tile of the item written              (2 query warps)
  uint64_t qfree[2];  // last score product of the item complete     (commit)
  uint64_t lfull[2];  // row sums of the item known                  (8 softmax warps)
  uint32_t tmem_base;
  int abort;
};
static_assert(kSSmemCtl + sizeof(SliceCtl) <= 232448, "exceeds the 227 KB of shared memory a CTA may use");
constexpr size_t kSSmemBytes = kSSmemCtl + sizeof(SliceCtl);

// what a role needs to know of a work item
struct SliceItem {
  int ti, bi, sp, head0, begin, end, ntiles;
};

__device__ __forceinline__ SliceItem slice_item(const SfaParams& p, int item) {
  SliceItem it;
  const int n_hb = p.nq / kSHeads;
  it.sp = item % p.n_split;
  item /= p.n_split;
  it.head0 = (item % n_hb) * kSHeads;
  it.ti = item / n_hb;
  it.bi = it.ti / p.s1;
  int n = __ldg(p.act_seq + it.bi) - p.s1 + 1 + it.ti % p.s1;
  n = max(0, min(n, p.topk_k));
  const int tiles_total = (n + kSRows - 1) / kSRows;
  const int tiles_per_split = (tiles_total + p.n_split - 1) / p.n_split;
  it.begin = min(n, it.sp * tiles_per_split * kSRows);
  it.end = min(n, (it.sp + 1) * tiles_per_split * kSRows);
  it.ntiles = (it.end - it.begin + kSRows - 1) / kSRows;
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

// MN-major B operand of 32 int8 columns: keys of 32 bytes, 32-byte swizzle, eight keys per atom
__device__ __forceinline__ uint64_t slice_desc_p(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>(1) << 16;           // one group along the columns
  d |= static_cast<uint64_t>(256 >> 4) << 32;    // eight keys
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(6) << 61;           // SWIZZLE_32B
  return d;
}

__device__ __forceinline__ void tmem_ld_32x32b_x8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}

// ================================ producers =====================================================
// Warp w owns rows 16w .. 16w+15 of every tile. Nothing passes through registers: an instruction copies one row's 512 latent
// bytes (or four rows' rope parts) from L2 to their swizzled places. The copies of a tile are issued when its buffer
// is free and waited for at the next tile, before that tile's buffer is. Lane r % 16 walks the look-ahead chain of row
// 16w + r: selected index three tiles ahead of the copies, block-table entry two, L2 prefetch one.
template <bool kPacked>
__device__ __forceinline__ void slice_role_producer(const SfaParams& p, SliceCtl* ctl, uint32_t base, int n_items) {
  const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) - kSProdWarp0;
  const int r = lane & 15;
  const uint8_t* const kn = reinterpret_cast<const uint8_t*>(p.kn);
  const uint8_t* const kr = kPacked ? kn + 512 : reinterpret_cast<const uint8_t*>(p.kr);
  const uint8_t* const ks = kPacked ? kn + 640 : reinterpret_cast<const uint8_t*>(p.kn_scales);
  constexpr int stride_n = kPacked ? 656 : 512, stride_r = kPacked ? 656 : 128, stride_s = kPacked ? 656 : 16;

  int cur_item = blockIdx.x, cur_j = 0;
  SliceItem it = slice_item(p, cur_item);
  // index of this lane's row in the next tile of this CTA (false: no further tile; the same answer in every lane)
  auto fetch = [&](int& idx, int& bi) -> bool {
    while (cur_j >= it.ntiles) {
      cur_item += gridDim.x;
      if (cur_item >= n_items) return false;
      it = slice_item(p, cur_item);
      cur_j = 0;
    }
    const int pos = it.begin + cur_j * kSRows + 16 * w + r;
    idx = pos < it.end ? ldg_pinned_i32(p.topk + static_cast<int64_t>(it.ti) * p.topk_k + pos) : -1;
    bi = it.bi;
    ++cur_j;
    return true;
  };
  auto row_of = [&](int idx, int entry) -> int {  // 32 bits: the host side refuses caches of 2^31 rows or more
    return static_cast<int>(tc_row_from_entry(p, idx, entry));
  };
  auto prefetch_row = [&](int phys) {  // two lanes per row
    if (phys < 0) return;
    if (kPacked) {
      if (lane < 16) bulk_prefetch_l2(kn + static_cast<int64_t>(phys) * 656, 656);
    } else {
      const uint8_t* a = kn + static_cast<int64_t>(phys) * 512 + (lane >> 4) * 256;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(a + 128));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(lane < 16 ? kr + static_cast<int64_t>(phys) * 128 : ks + static_cast<int64_t>(phys) * 16));
    }
  };

  int idx_n = -1, bi_n = 0, idx_a = -1, bi_a = 0, entry_n = kTableSkip, row = -1;
  bool has, has_n = false, has_a = false;
  {
    int idx0 = -1, bi0 = 0;
    has = fetch(idx0, bi0);
    has_n = has && fetch(idx_n, bi_n);
    has_a = has_n && fetch(idx_a, bi_a);
    const int e0 = has ? tc_table_entry(p, bi0, idx0) : kTableSkip;
    if (has_n) entry_n = tc_table_entry(p, bi_n, idx_n);
    if (has) row = row_of(idx0, e0);
  }
  bool ok = true;
  uint32_t t = 0;
  for (; has; ++t) {
    const uint32_t b = t & 1;
    int idx_b = -1, bi_b = 0;
    const bool has_b = has_a && fetch(idx_b, bi_b);
    // the tile after this one: into L2
    int row_n = -1;
    if (has_n) {
      row_n = row_of(idx_n, entry_n);
      prefetch_row(row_n);
    }
    if (t >= 1) {  // the tile before this one has had a whole step to arrive
      asm volatile("cp.async.wait_all;" ::: "memory");
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl->full[b ^ 1]));
    }
    if (t >= 2) {
      ok = slice_wait(smem_u32(&ctl->done[b]), ((t >> 1) - 1) & 1);
      if (!ok) break;
    }
    const uint32_t tile = base + kSSmemTile + b * kSTile;
#pragma unroll
    for (int m = 0; m < 16; ++m) {  // row 16w + m: 32 units, eight per chunk (a padding or rejected row reads as zeros)
      const int pm = __shfl_sync(0xffffffffu, row, m);
      cp_async_16(tile + (lane >> 3) * kSChunk + (16 * w + m) * 128 + (((lane & 7) ^ (m & 7)) << 4),
                  kn + (pm >= 0 ? static_cast<int64_t>(pm) * stride_n + lane * 16 : 0), pm >= 0 ? 16u : 0u);
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int x = 4 * m + (lane >> 3);
      const int pm = __shfl_sync(0xffffffffu, row, x);
      cp_async_16(tile + 4 * kSChunk + (16 * w + x) * 128 + (((lane & 7) ^ (x & 7)) << 4),
                  kr + (pm >= 0 ? static_cast<int64_t>(pm) * stride_r + (lane & 7) * 16 : 0), pm >= 0 ? 16u : 0u);
    }
    if (lane < 16) {
      cp_async_16(smem_u32(&ctl->scales[b][16 * w + lane][0]), ks + (row >= 0 ? static_cast<int64_t>(row) * stride_s : 0),
                  row >= 0 ? 16u : 0u);
      ctl->live[b][16 * w + lane] = row >= 0 ? 1.f : 0.f;
    }
    row = row_n;
    has = has_n;
    has_n = has_a;
    idx_n = idx_a;
    if (has_a) entry_n = tc_table_entry(p, bi_a, idx_a);
    has_a = has_b;
    idx_a = idx_b;
    bi_a = bi_b;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (ok && t > 0) {
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&ctl->full[(t - 1) & 1]));
  }
  if (!ok && lane == 0) {
    ctl->abort = 1;
    set_status(p.status, PTO_ST_WAIT_EXPIRED, blockIdx.x, 90);
  }
}

// ================================ MMA issuers ====================================================
// What an MMA of this size costs is its issue: measured in isolation, 51-61 cycles whatever the shape when one lane
// issues under `if (lane == 0)`, where the descriptors are moved to uniform registers for every MMA, against 39 (N = 16)
// when the warp stays converged and an elected lane issues. Beside two dozen busy warps, the descriptors have to be
// constants of the code for that (kBase, the address where a kernel without static shared memory finds its dynamic
// part; kBase = 0 is the same code with the address in a register).
constexpr uint32_t kSliceUsualBase = 1024;
__device__ __forceinline__ void slice_issue_scores(uint32_t d, uint64_t a_desc, uint64_t b_desc) {
  constexpr uint32_t idesc_i8 = umma_idesc(kCFmtS32, kABFmtS8, kABFmtS8, 0, 0, 128, 2 * kSHeads);
  constexpr uint32_t idesc_bf = umma_idesc(kCFmtF32, kABFmtBF16, kABFmtBF16, 0, 0, 128, kSHeads);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      mma_i8_ss(d + c * 2 * kSHeads, a_desc + c * (kSChunk >> 4) + 2 * k, b_desc + c * (kSQChunk >> 4) + 2 * k, idesc_i8, k != 0 ? 1u : 0u);
    }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    mma_f16_ss(d + 4 * 2 * kSHeads, a_desc + 4 * (kSChunk >> 4) + 2 * k, b_desc + 4 * (kSQChunk >> 4) + 2 * k, idesc_bf, k != 0 ? 1u : 0u);
  }
}
__device__ __forceinline__ void slice_issue_values(uint32_t d, uint64_t a_desc, uint64_t b_desc) {
  constexpr uint32_t idesc = umma_idesc(kCFmtS32, kABFmtS8, kABFmtS8, 1, 1, 128, 2 * kSHeads);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {  // 32 keys per step: 4 KB of a chunk, 1 KB of the block's P^T
      mma_i8_ss(d + c * 2 * kSHeads, a_desc + c * (kSChunk >> 4) + k * (4096 >> 4), b_desc + c * (kSPBlock >> 4) + k * (1024 >> 4),
                idesc, k != 0 ? 1u : 0u);
    }
  }
}

template <uint32_t kBase>
__device__ __forceinline__ void slice_role_scores(const SfaParams& p, SliceCtl* ctl, uint32_t base, uint32_t tmem, int n_items) {
  if (kBase != 0) base = kBase;
  const uint64_t a_desc = umma_desc_kmajor_sw128(base + kSSmemTile), b_desc = umma_desc_kmajor_sw128(base + kSSmemQ);
  bool ok = true;
  uint32_t t = 0, n = 0;
  for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
    const int ntiles = slice_item(p, item).ntiles;
    if (ntiles == 0) continue;
    const uint32_t qb = n & 1;
    ok = slice_wait(smem_u32(&ctl->qfull[qb]), (n >> 1) & 1);
    for (int j = 0; j < ntiles && ok; ++j, ++t) {
      const uint32_t b = t & 1;
      if (t >= 2) ok = slice_wait(smem_u32(&ctl->sfree[b]), ((t >> 1) - 1) & 1);
      ok = ok && slice_wait(smem_u32(&ctl->full[b]), (t >> 1) & 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        slice_issue_scores(tmem + kSColS + b * kSSBuf, a_desc + b * (kSTile >> 4), b_desc + qb * (kSQ >> 4));
        tc_commit(smem_u32(&ctl->sfull[b]));
        if (j + 1 == ntiles) tc_commit(smem_u32(&ctl->qfree[qb]));
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

template <uint32_t kBase>
__device__ __forceinline__ void slice_role_values(const SfaParams& p, SliceCtl* ctl, uint32_t base, uint32_t tmem, int n_items) {
  if (kBase != 0) base = kBase;
  const uint64_t a_desc = desc_mnmajor_sw128(base + kSSmemTile, 16, 1024);
  const uint64_t b_desc = slice_desc_p(base + kSSmemP);
  bool ok = true;
  uint32_t t = 0;
  for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
    const int ntiles = slice_item(p, item).ntiles;
    for (int j = 0; j < ntiles && ok; ++j, ++t) {
      const uint32_t b = t & 1;
      ok = slice_wait(smem_u32(&ctl->pfull), t & 1);
      if (ok && t >= 1) ok = slice_wait(smem_u32(&ctl->ofree), (t - 1) & 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        slice_issue_values(tmem + kSColO, a_desc + b * (kSTile >> 4), b_desc);
        tc_commit(smem_u32(&ctl->done[b]));
      }
      __syncwarp();
    }
  }
  if (!ok && (threadIdx.x & 31) == 0) {
    ctl->abort = 1;
    set_status(p.status, PTO_ST_WAIT_EXPIRED, blockIdx.x, 92);
  }
  __syncwarp();
}

// ================================ query tile =====================================================
// Two warps, eight heads each: a head's 512 latent values as fixed-point limbs (lane l holds dims 16l .. 16l+15), its rope part
// as it is.
__device__ __forceinline__ void slice_role_query(const SfaParams& p, SliceCtl* ctl, uint32_t base, int n_items) {
  const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) - 2;
  bool ok = true;
  uint32_t n = 0;
  for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
    const SliceItem it = slice_item(p, item);
    if (it.ntiles == 0) continue;
    const uint32_t qb = n & 1;
    const int64_t row0 = static_cast<int64_t>(it.ti) * p.nq_total + p.head_begin + it.head0 + 8 * w;
    if (n >= 2) {
      ok = slice_wait(smem_u32(&ctl->qfree[qb]), ((n >> 1) - 1) & 1);
      if (!ok) break;
    }
    const uint32_t q = base + kSSmemQ + qb * kSQ;
#pragma unroll 2
    for (int m = 0; m < 8; ++m) {
      const int head = 8 * w + m;
      const uint4* src = reinterpret_cast<const uint4*>(p.q_nope + (row0 + m) * 512) + 2 * lane;
      const uint4 v0 = __ldg(src), v1 = __ldg(src + 1);
      const uint32_t v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
      uint32_t mx = 0;
#pragma unroll
      for (int e = 0; e < 8; ++e) mx = max(mx, max((v[e] << 16) & 0x7fffffffu, v[e] & 0x7fff0000u));
      mx = __reduce_max_sync(0xffffffffu, mx);  // bit pattern of the head's largest |q|
      const int ex = max(-100, static_cast<int>(mx >> 23) - 127);  // 2^ex <= largest < 2^(ex + 1)
      const float up = __int_as_float((127 + 13 - ex) << 23);
      uint32_t hi[4], lo[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        uint32_t y[4];  // low 22 bits: the integer (two's complement)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint32_t word = v[2 * u + (e >> 1)];
          const float x = __uint_as_float((e & 1) ? (word & 0xffff0000u) : (word << 16));
          y[e] = __float_as_uint(fmaf(x, up, 12582912.0f));
        }
        lo[u] = __byte_perm(__byte_perm(y[0], y[1], 0x0040), __byte_perm(y[2], y[3], 0x0040), 0x5410) & 0x7f7f7f7fu;
        hi[u] = __byte_perm(__byte_perm(y[0] << 1, y[1] << 1, 0x0051), __byte_perm(y[2] << 1, y[3] << 1, 0x0051), 0x5410);
      }
      // dims 16 lane ..: chunk lane / 8, unit lane % 8 of rows `head` (high limbs) and 16 + `head`
      const uint32_t at = q + (lane >> 3) * kSQChunk + head * 128 + (((lane & 7) ^ (head & 7)) << 4);
      sts_v4u(at, make_uint4(hi[0], hi[1], hi[2], hi[3]));
      sts_v4u(at + kSHeads * 128, make_uint4(lo[0], lo[1], lo[2], lo[3]));
      if (lane < 8) {
        sts_v4u(q + 4 * kSQChunk + head * 128 + ((lane ^ (head & 7)) << 4),
                __ldg(reinterpret_cast<const uint4*>(p.q_rope + (row0 + m) * 64) + lane));
      }
      // (a query that is not finite makes the head's scores, and with them its output, NaN)
      if (lane == 0) ctl->qunit[n & 3][head] = mx >= 0x7f800000u ? __int_as_float(0x7fffffff) : __int_as_float((127 + ex - 13) << 23);
    }
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&ctl->qfull[qb]));
    ++n;
  }
  if (!ok && lane == 0) {
    ctl->abort = 1;
    set_status(p.status, PTO_ST_WAIT_EXPIRED, blockIdx.x, 93);
  }
}

// ================================ softmax ========================================================
// Eight warps, TMEM lane = key of the tile (warp quarter q holds keys 32q .. +31); warps 4-7 take heads 0-7, warps 8-11 heads
// 8-15. The reference maximum of a head moves only when a score exceeds it by more than a factor of two (first tile:
// always), which one vote over the eight warps finds out; so the reduction over keys, here across lanes, is rare, and
// the row sums stay per-thread partials until the item ends.
__device__ __forceinline__ bool slice_vote(bool pred) {  // OR over the softmax warps; also their barrier
  uint32_t any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, 1, 256, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(any)
      : "r"(pred ? 1u : 0u)
      : "memory");
  return any != 0;
}
__device__ __forceinline__ void slice_meet() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

__device__ __forceinline__ void slice_role_softmax(const SfaParams& p, SliceCtl* ctl, uint32_t base, uint32_t tmem, int n_items) {
  const int lane = threadIdx.x & 31, quarter = (threadIdx.x >> 5) & 3, g = ((threadIdx.x >> 5) - kSSoftWarp0) >> 2;
  const int tid = threadIdx.x - 32 * kSSoftWarp0;
  const int key = 32 * quarter + lane, h0 = 8 * g;
  const uint32_t lane_addr = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
  // this key's 32 bytes of a block of P^T; 32-byte swizzle: unit ^= (key / 4) % 2. High limbs at unit 0, low at unit 1
  const uint32_t p_row = base + kSSmemP + key * 32 + 8 * g;
  const uint32_t u_hi = ((key >> 2) & 1) << 4, u_lo = u_hi ^ 16u;
  bool ok = true;
  uint32_t t = 0, n = 0;
  for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
    const SliceItem it = slice_item(p, item);
    if (it.ntiles == 0) continue;
    float l[8], qunit[8];
#pragma unroll
    for (int h = 0; h < 8; ++h) l[h] = qunit[h] = 0.f;
    for (int j = 0; j < it.ntiles; ++j, ++t) {
      const uint32_t b = t & 1;
      ok = ok && slice_wait(smem_u32(&ctl->sfull[b]), (t >> 1) & 1) && slice_wait(smem_u32(&ctl->full[b]), (t >> 1) & 1);
      // (a wait that expired is voted on below, so that the eight warps leave together)
      tc_fence_after();
      const float4 sc = *reinterpret_cast<const float4*>(&ctl->scales[b][key][0]);
      const float scv[4] = {sc.x, sc.y, sc.z, sc.w};
      const bool valid = ctl->live[b][key] != 0.f && it.begin + j * kSRows + key < it.end;
      if (j == 0) {  // (before the scores are handed back: the slot is written again four items on, behind two more products)
#pragma unroll
        for (int h = 0; h < 8; ++h) qunit[h] = ctl->qunit[n & 3][h0 + h];
      }
      const uint32_t col = lane_addr + kSColS + b * kSSBuf + h0;
      float s[8], rope[8];
#pragma unroll
      for (int h = 0; h < 8; ++h) s[h] = 0.f;
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) {
        uint32_t hi[2][8], lo[2][8], rp[8];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          tmem_ld_32x32b_x8(col + (2 * cc + e) * 2 * kSHeads, hi[e]);
          tmem_ld_32x32b_x8(col + (2 * cc + e) * 2 * kSHeads + kSHeads, lo[e]);
        }
        if (cc == 1) tmem_ld_32x32b_x8(col + 4 * 2 * kSHeads, rp);
        tc_wait_ld();
        if (cc == 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&ctl->sfree[b]));
#pragma unroll
          for (int h = 0; h < 8; ++h) rope[h] = __uint_as_float(rp[h]);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
#pragma unroll
          for (int h = 0; h < 8; ++h) {
            const int d = static_cast<int>(hi[e][h]) * 128 + static_cast<int>(lo[e][h]);
            s[h] = fmaf(static_cast<float>(d), scv[2 * cc + e], s[h]);
          }
        }
      }
      float over = -INFINITY;
#pragma unroll
      for (int h = 0; h < 8; ++h) {
        s[h] = valid ? fmaf(s[h], qunit[h], rope[h]) * p.scale_log2 : -INFINITY;
        over = fmaxf(over, s[h] - (j > 0 ? ctl->mref[h0 + h] : 0.f));
      }
      if (g == 0) {  // largest |scale| of the quarter's rows (zero in rows that are not there)
        float m4[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) m4[c] = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(scv[c]) & 0x7fffffffu));
        if (lane == 0) *reinterpret_cast<float4*>(&ctl->smax[b][quarter][0]) = make_float4(m4[0], m4[1], m4[2], m4[3]);
      }
      const bool fresh = slice_vote(j == 0 || over > kSRescale || !ok);
      if (fresh) {
        // ---- new reference maxima (uniform branch) ----------------------------------------------------
#pragma unroll
        for (int h = 0; h < 8; ++h) {
          const float m = s[h];
          const uint32_t o = li_float_order(m);
          const uint32_t mx = __reduce_max_sync(0xffffffffu, o);
          if (lane == 0) ctl->red[quarter][h0 + h] = __uint_as_float((mx & 0x80000000u) ? (mx & 0x7fffffffu) : ~mx);
        }
        if (slice_vote(!ok)) {
          ok = false;
          break;
        }
        if (tid < kSHeads) {
          const float old = j > 0 ? ctl->mref[tid] : -INFINITY;
          const float m = fmaxf(fmaxf(ctl->red[0][tid], ctl->red[1][tid]), fmaxf(ctl->red[2][tid], ctl->red[3][tid]));
          ctl->mref[tid] = fmaxf(old, m);
          ctl->red[0][tid] = old == -INFINITY ? 0.f : ex2f(old - fmaxf(old, m));
        }
        slice_meet();
        if (j > 0) {
#pragma unroll
          for (int h = 0; h < 8; ++h) l[h] *= ctl->red[0][h0 + h];
        }
      }
#pragma unroll
      for (int h = 0; h < 8; ++h) {
        const float m = ctl->mref[h0 + h];
        s[h] = ex2f(s[h] - (m == -INFINITY ? 0.f : m));
        l[h] += s[h];
      }
      if (t >= 1) {  // the products that read the P^T of the tile before are complete, its O^T has a reader
        ok = slice_wait(smem_u32(&ctl->done[b ^ 1]), ((t - 1) >> 1) & 1) && ok;
      }
      float unit[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        unit[c] = fmaxf(fmaxf(ctl->smax[b][0][c], ctl->smax[b][1][c]), fmaxf(ctl->smax[b][2][c], ctl->smax[b][3][c]));
      }
      if (tid < kSHeads) {
        if (tid == 0) {
          ctl->rescale[b] = fresh && j > 0 ? 1 : 0;
          *reinterpret_cast<float4*>(&ctl->fac[b][0]) =
              make_float4(unit[0] * (1.0f / kSPUnit), unit[1] * (1.0f / kSPUnit), unit[2] * (1.0f / kSPUnit), unit[3] * (1.0f / kSPUnit));
        }
        ctl->alpha[b][tid] = fresh && j > 0 ? ctl->red[0][tid] : 1.f;
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float f = unit[c] > 0.f ? __fdividef(scv[c], unit[c]) * kSPUnit : 0.f;
        uint32_t hi[2], lo[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          uint32_t y[4];  // low 22 bits: round(p * scale in units), two's complement; 7 low bits and the rest are the limbs
#pragma unroll
          for (int e = 0; e < 4; ++e) y[e] = __float_as_uint(fmaf(s[4 * u + e], f, 12582912.0f));
          lo[u] = __byte_perm(__byte_perm(y[0], y[1], 0x0040), __byte_perm(y[2], y[3], 0x0040), 0x5410) & 0x7f7f7f7fu;
          hi[u] = __byte_perm(__byte_perm(y[0] << 1, y[1] << 1, 0x0051), __byte_perm(y[2] << 1, y[3] << 1, 0x0051), 0x5410);
        }
        const uint32_t at = p_row + c * kSPBlock;
        asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(at + u_hi), "r"(hi[0]), "r"(hi[1]) : "memory");
        asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(at + u_lo), "r"(lo[0]), "r"(lo[1]) : "memory");
      }
      fence_proxy_async();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl->pfull));
      // (a `done` that expired is voted on at the next tile, or here at the last one)
      if (j + 1 == it.ntiles) {
        if (slice_vote(!ok)) {
          ok = false;
          break;
        }
      }
    }
    if (!ok) break;
    // ---- row sums ------------------------------------------------------------------------------------
#pragma unroll
    for (int h = 0; h < 8; ++h) {
      float v = l[h];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) ctl->red[quarter][h0 + h] = v;
    }
    slice_meet();
    if (tid < kSHeads) {
      const float tot = (ctl->red[0][tid] + ctl->red[1][tid]) + (ctl->red[2][tid] + ctl->red[3][tid]);
      if (p.n_split == 1) {
        ctl->linv[n & 1][tid] = tot != 0.f ? 1.f / tot : 0.f;
      } else {
        ctl->linv[n & 1][tid] = 1.f;
        const int64_t prow = (static_cast<int64_t>(it.ti) * p.n_split + it.sp) * p.nq + it.head0 + tid;
        p.part_ml[prow * 2] = ctl->mref[tid];
        p.part_ml[prow * 2 + 1] = tot;
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&ctl->lfull[n & 1]));
    slice_meet();  // (red and mref are read; the next item may write them)
    ++n;
  }
  if (!ok && lane == 0) {
    ctl->abort = 1;
    set_status(p.status, PTO_ST_WAIT_EXPIRED, blockIdx.x, 94);
  }
}

// ================================ output =========================================================
// Four warps, TMEM lane = dim of the block: fp32 sums of four blocks x 16 heads in registers.
__device__ __forceinline__ void slice_role_output(const SfaParams& p, SliceCtl* ctl, uint32_t tmem, int n_items) {
  const int lane = threadIdx.x & 31, quarter = (threadIdx.x >> 5) & 3;
  const int dim = 32 * quarter + lane;
  const uint32_t lane_addr = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + kSColO;
  bool ok = true;
  uint32_t t = 0, n = 0;
  for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
    const SliceItem it = slice_item(p, item);
    const int64_t orow0 = static_cast<int64_t>(it.ti) * p.nq_total + p.head_begin + it.head0;
    const int64_t prow0 = (static_cast<int64_t>(it.ti) * p.n_split + it.sp) * p.nq + it.head0;
    if (it.ntiles == 0) {
      const int tid = threadIdx.x - 32 * kSOutWarp0;
      if (p.n_split == 1) {
        for (int e = tid; e < kSHeads * 64; e += 128) *reinterpret_cast<uint4*>(p.out + orow0 * 512 + e * 8) = make_uint4(0, 0, 0, 0);
      } else if (tid < kSHeads) {
        p.part_ml[(prow0 + tid) * 2] = -INFINITY;
        p.part_ml[(prow0 + tid) * 2 + 1] = 0.f;
      }
      continue;
    }
    float o[4][kSHeads];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
#pragma unroll
      for (int h = 0; h < kSHeads; ++h) o[c][h] = 0.f;
    }
    for (int j = 0; j < it.ntiles; ++j, ++t) {
      const uint32_t b = t & 1;
      ok = slice_wait(smem_u32(&ctl->done[b]), (t >> 1) & 1);
      if (!ok) break;
      tc_fence_after();
      if (ctl->rescale[b] != 0) {
#pragma unroll
        for (int h = 0; h < kSHeads; ++h) {
          const float a = ctl->alpha[b][h];
#pragma unroll
          for (int c = 0; c < 4; ++c) o[c][h] *= a;
        }
      }
      const float4 f4 = *reinterpret_cast<const float4*>(&ctl->fac[b][0]);
      const float f[4] = {f4.x, f4.y, f4.z, f4.w};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t v[32];
        tmem_ld_32x32b_x32(lane_addr + c * 2 * kSHeads, v);
        tc_wait_ld();
#pragma unroll
        for (int h = 0; h < kSHeads; ++h) {
          o[c][h] = fmaf(static_cast<float>(static_cast<int>(v[h]) * 128 + static_cast<int>(v[kSHeads + h])), f[c], o[c][h]);
        }
      }
      // the item's row sums are read before its last tile lets go, so that they can be written again two items on
      if (j + 1 == it.ntiles) {
        ok = slice_wait(smem_u32(&ctl->lfull[n & 1]), (n >> 1) & 1);
        if (!ok) break;
#pragma unroll
        for (int h = 0; h < kSHeads; ++h) {
          const float a = ctl->linv[n & 1][h];
#pragma unroll
          for (int c = 0; c < 4; ++c) o[c][h] *= a;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl->ofree));
    }
    if (!ok) break;
#pragma unroll
    for (int c = 0; c < 4; ++c) {  // 32 lanes write consecutive dims of a head's row
#pragma unroll
      for (int h = 0; h < kSHeads; ++h) {
        if (p.n_split == 1) p.out[(orow0 + h) * 512 + 128 * c + dim] = __float2bfloat16_rn(o[c][h]);
        else p.part_o[(prow0 + h) * 512 + 128 * c + dim] = o[c][h];
      }
    }
    ++n;
  }
  if (!ok && lane == 0) {
    ctl->abort = 1;
    set_status(p.status, PTO_ST_WAIT_EXPIRED, blockIdx.x, 96);
  }
}

__global__ void __launch_bounds__(kSThreads, 1)
sfa_slice_kernel(const __grid_constant__ SfaParams p, int n_items) {
  extern __shared__ __align__(1024) uint8_t sfa_slice_smem[];
  const uint32_t base = smem_u32(sfa_slice_smem);
  if ((base & 1023u) != 0) {  // the swizzled operand tiles need a 1024-byte aligned base
    if (threadIdx.x == 0) set_status(p.status, PTO_ST_WAIT_EXPIRED, static_cast<int>(base), 95);
    return;
  }
  SliceCtl* ctl = reinterpret_cast<SliceCtl*>(sfa_slice_smem + kSSmemCtl);
  const int tid = threadIdx.x, warp = tid >> 5;
  if (tid == 0) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&ctl->full[b]), kSProdWarps);
      mbar_init(smem_u32(&ctl->done[b]), 1);
      mbar_init(smem_u32(&ctl->sfull[b]), 1);
      mbar_init(smem_u32(&ctl->sfree[b]), kSSoftWarps);
      mbar_init(smem_u32(&ctl->qfull[b]), 2);
      mbar_init(smem_u32(&ctl->qfree[b]), 1);
      mbar_init(smem_u32(&ctl->lfull[b]), kSSoftWarps);
    }
    mbar_init(smem_u32(&ctl->pfull), kSSoftWarps);
    mbar_init(smem_u32(&ctl->ofree), 4);
    ctl->abort = 0;
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(&ctl->tmem_base), kSTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ctl->tmem_base;
  pdl_wait();  // the set-up above overlaps the tail of the kernel before this one
  if (tid == 0) pdl_trigger();
  if (warp < kSSoftWarp0) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kSRegIssue));
    if (warp < 2 && base == kSliceUsualBase) {
      if (warp == 0) slice_role_scores<kSliceUsualBase>(p, ctl, base, tmem, n_items);
      else slice_role_values<kSliceUsualBase>(p, ctl, base, tmem, n_items);
    } else if (warp == 0) slice_role_scores<0>(p, ctl, base, tmem, n_items);
    else if (warp == 1) slice_role_values<0>(p, ctl, base, tmem, n_items);
    else slice_role_query(p, ctl, base, n_items);
  } else if (warp < kSOutWarp0) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSRegSoft));
    slice_role_softmax(p, ctl, base, tmem, n_items);
  } else if (warp < kSProdWarp0) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSRegOut));
    slice_role_output(p, ctl, tmem, n_items);
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kSRegProd));
    if (p.packed) slice_role_producer<true>(p, ctl, base, n_items);
    else slice_role_producer<false>(p, ctl, base, n_items);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, kSTmemCols);
  }
}

}  // namespace

int sfa_slice_heads() { return kSHeads; }

cudaError_t launch_sfa_slice(const SfaParams& p, int num_sms, cudaStream_t stream) {
  const cudaError_t e = cudaFuncSetAttribute(sfa_slice_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSSmemBytes));
  if (e != cudaSuccess) return e;
  const long long items = static_cast<long long>(p.b) * p.s1 * (p.nq / kSHeads) * p.n_split;
  if (items > 0x7fffffffLL) return cudaErrorInvalidValue;
  const int grid = static_cast<int>(items < num_sms ? items : num_sms);
  count_launch();
  return launch_maybe_pdl(sfa_slice_kernel, dim3(grid), dim3(kSThreads), kSSmemBytes, stream, p.pdl != 0, p, static_cast<int>(items));
}

}  // namespace pto
