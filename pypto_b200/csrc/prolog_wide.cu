// Products of the prologs for many token rows (prompt chunks): out[tok, n] = x[tok, k] . W[k, n] on tcgen05 with the token
// rows as the M dimension, and what follows a product fused into its epilogue:
//
//   kWideF32    fp32 K-split partials (projections of the hidden state)
//   kWideBf16   bf16 rows (absorbed query per head; up-projections of the non-quantised prolog)
//   kWideUp     both int8 up-projections of the normalised query in one launch, int32 -> bf16 dequantisation. Attention: the
//               128-wide nope part of a head goes to the scratch the absorbed product reads, the 64-wide tail is rotated
//               and goes to the output. Indexer: a head's first 64 dims are rotated, the rows go to the Hadamard product
//   kWideHad    indexer rows . Hadamard matrix, bf16 rounding, per-row int8 quantisation (rows = tokens x 64 heads)
//
// (reference: examples/models/deepseek_v32_exp/mla_prolog_quant_impl.py:502-707,
// lightning_indexer_prolog_quant_impl.py:325-504; arithmetic and roundings as in prolog.cu.)
//
// Why tokens as M: a TMEM lane is a token row, so a thread of the epilogue holds neighbouring columns of one row. Row
// scales are per-lane constants and a rope pair or a head's maximum lies inside a thread. A warp passes 128 bytes of each
// of its 32 rows through shared memory and writes whole lines (32-byte stores straight from the lanes, each to a row of
// its own, reached L2 as three times their sectors: 64 -> 41 us for the absorbed query of 1000 tokens). With the weight columns as lanes (prolog_sgemm.cu, made for few rows) every store instruction writes 64
// bytes of one row and everything between the products needs a kernel of its own. 1000 tokens, one kernel each, before
// -> after: dequantisation 33 us -> fused; indexer query 118 us (Hadamard on CUDA cores) -> product of 16 us.
//
// One CTA per SM, persistent. A ring stage is one 128-byte-wide K chunk: x tile [128 rows] (16 KB, K-major) and W tile
// [chunk rows x kN columns] (32 KB at kN = 256, MN-major as it lies in memory), both 128-byte swizzled by TMA; rows and
// columns outside the tensors read as zeros. Two accumulators of kN columns, one per epilogue group of four warps, so
// that one tile is stored while the next is multiplied. Items run over token blocks first: the CTAs that are at work at
// the same time read the same weight columns from L2.
// Of many rows two CTAs on neighbouring SMs take 256 rows x 256 columns together (tcgen05.mma.cta_group::2): each loads its own rows and
// half of the columns, so a stage is 32 KB instead of 48, six fit, and a third less of the operands passes from L2. CTA 0 issues the
// MMAs; each CTA stores its rows (1000 tokens: projections 32.4 -> 28.9 us, 1.14 PFLOP/s; the line is drawn at the launch).
// Roles: warp 0 TMA, warp 1 MMA, warps 2-5 / 6-9 epilogue. All waits are bounded.
#include <cuda.h>

#include <initializer_list>

#include "sfa_common.cuh"

namespace pto {

namespace {

constexpr int kWRows = 128;                  // token rows per tile (MMA M)
constexpr int kWXBytes = kWRows * 128;
constexpr int kWThreads = 320;
constexpr int kWStaging = 8 * 4096;           // per epilogue warp: 128 bytes of 32 rows
constexpr int kHeadQ = 192, kHeadNope = 128;  // widths of an attention head of the up-projection

enum { kWideF32 = 0, kWideBf16 = 1, kWideUp = 2, kWideHad = 3 };

constexpr int kWMaxStages = 6;
struct WideCtl {
  uint64_t full[kWMaxStages];   // (of a pair: in CTA 0, for both CTAs' bytes)
  uint64_t empty[kWMaxStages];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  int abort;
};

struct WideParams {
  int t;                  // rows of x
  int n;                  // valid output columns per problem
  int n_tiles;            // kN-column tiles per problem
  int chunks, per_split, splits;
  int batch;              // problems (heads)
  int row_blocks;         // (of a pair: two blocks of 128 rows)
  int w_batch_rows;       // rows of W between problems
  int x_batch_bytes;      // bytes along a row of x between problems
  long long out_batch;    // output elements between problems
  long long ld_out;       // output elements between rows
  long long split_stride;
  int idx_tiles;          // kWideUp: the first tiles are the indexer's (second tensor map of W), the others the attention's
  void* out;              // kWideUp: nope scratch bf16 [t, 128, 128]; kWideHad: int8 rows
  void* out2;             // kWideUp: query_rope [t, 128, 64]; kWideHad: fp16 scale per row
  void* out_idx;          // kWideUp: indexer rows bf16 [t, 64, 128]
  const float* row_scale; // kWideUp: per token
  const float* col_scale; // per column of the attention's product
  const float* col_scale_idx;
  const __nv_bfloat16* cos;  // [t, 64]
  const __nv_bfloat16* sin;
  PrologWBoxes boxes;     // bf16 products: 64-column boxes of the matrices of W
  int aligned;            // everything the epilogue touches lies on 16-byte boundaries: wide accesses, else single elements
  int32_t* status;
};

template <bool kI8, int kN, bool kPair>
struct WideCfg {
  static constexpr int kStages = kPair ? 6 : 4;
  static constexpr int kChunkK = kI8 ? 128 : 64;     // k per stage: 128 bytes of a row of x
  static constexpr int kGroup = kI8 ? 128 : 64;      // columns per 128-byte box of W
  static constexpr int kBoxBytes = kChunkK * 128;
  static constexpr int kBoxes = kN / kGroup / (kPair ? 2 : 1);  // of a pair, each CTA holds half of the columns
  static constexpr int kWBytes = kBoxes * kBoxBytes;
  static constexpr int kStage = kWXBytes + kWBytes;
  static constexpr int kSmem = kStages * kStage + kWStaging + sizeof(WideCtl) + 1024;
  static_assert(kSmem <= 232448, "exceeds the 227 KB of shared memory a CTA may use");
  static constexpr uint32_t kTmemCols = 2 * kN;
};

struct WideItem {
  int rb, b, tile, split;
};
__device__ __forceinline__ WideItem wide_item(const WideParams& p, int item) {
  WideItem it;
  it.rb = item % p.row_blocks;
  int r = item / p.row_blocks;
  it.split = r % p.splits;
  r /= p.splits;
  it.tile = r % p.n_tiles;
  it.b = r / p.n_tiles;
  return it;
}

// --- a pair of SMs on one tile (tcgen05.mma.cta_group::2) ---
__device__ __forceinline__ uint32_t wide_cta_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t wide_in_cta0(uint32_t local) {  // the same place in the pair's first CTA
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(local));
  return r;
}
__device__ __forceinline__ void wide_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// into this CTA's shared memory, completion on a barrier of either CTA of the pair
__device__ __forceinline__ void wide_load_pair(uint32_t dst_smem, const void* tmap, int x, int y, uint32_t cluster_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst_smem), "l"(tmap), "r"(x), "r"(y), "r"(cluster_bar)
      : "memory");
}
template <bool kI8>
__device__ __forceinline__ void wide_mma_pair(uint32_t d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  if constexpr (kI8) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
  }
}
// arrives on the barrier at this place in both CTAs once all MMAs issued so far have completed
__device__ __forceinline__ void wide_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(static_cast<uint16_t>(3))
               : "memory");
}
__device__ __forceinline__ void wide_arrive_cluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ bool wide_wait_cluster(uint32_t bar, uint32_t parity) {  // bounded; arrivals from both CTAs
  const long long t0 = clock64();
  while (true) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok != 0) return true;
    if (clock64() - t0 > kWaitBudgetCycles) return false;
  }
}

__device__ __forceinline__ float wide_bf16_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// This warp's rows: lane l holds 128 bytes of row l, which go to its staging area. 16-byte unit u of row r comes back from there.
__device__ __forceinline__ void stage_rows(uint32_t stage, const uint32_t (&w)[32]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    sts_v4u(stage + lane * 128 + ((i ^ (lane & 7)) << 4), make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]));
  }
  __syncwarp();
}
__device__ __forceinline__ uint4 staged_unit(uint32_t stage, int r, int u) { return lds_v4u(stage + r * 128 + ((u ^ (r & 7)) << 4)); }
template <bool kAligned>
__device__ __forceinline__ void store_unit(uint8_t* at, const uint4& v) {
  if constexpr (kAligned) {
    *reinterpret_cast<uint4*>(at) = v;
  } else {
    const uint32_t x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int e = 0; e < 16; ++e) at[e] = static_cast<uint8_t>(x[e >> 2] >> (8 * (e & 3)));
  }
}
// The rows go to `dst` + l * `pitch` through the staging area, four whole lines per store instruction. `n_rows`: rows that
// exist; `n_bytes`: bytes that exist of each (a multiple of 16).
template <bool kAligned>
__device__ __forceinline__ void store_rows(uint32_t stage, const uint32_t (&w)[32], uint8_t* dst, int64_t pitch, int n_rows,
                                           int n_bytes) {
  const int lane = threadIdx.x & 31;
  stage_rows(stage, w);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = 4 * i + (lane >> 3), u = lane & 7;
    const uint4 v = staged_unit(stage, r, u);
    if (r < n_rows && u * 16 < n_bytes) store_unit<kAligned>(dst + r * pitch + u * 16, v);
  }
  __syncwarp();
}
// eight of a token's 64 cosines or sines, two to a word
template <bool kAligned>
__device__ __forceinline__ uint4 load_bf16_8(const __nv_bfloat16* p) {
  if constexpr (kAligned) return ldg_pinned_v4(p);
  const unsigned short* q = reinterpret_cast<const unsigned short*>(p);
  uint32_t w[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) w[e] = q[2 * e] | static_cast<uint32_t>(q[2 * e + 1]) << 16;
  return make_uint4(w[0], w[1], w[2], w[3]);
}
// The same for rows of 64 bf16 that are rotated on the way: out[j] = a[j] cos[j] - b[j] sin[j], out[32 + j] = b[j] cos[32 + j] +
// a[j] sin[32 + j]. kPairs: a and b are the even and the odd dims (the outputs are de-interleaved), else the halves. The lane that
// stores eight outputs computes them, so a load of cosines touches the four lines that its store does; with a row to a lane every
// load touched 32 (1000 tokens: both up-projections 57.8 -> 53.7 us).
template <bool kAligned, bool kPairs>
__device__ __forceinline__ void store_rows_rotated(const WideParams& p, uint32_t stage, const uint32_t (&w)[32], int row0, uint8_t* dst,
                                                   int64_t pitch, int n_rows) {
  const int lane = threadIdx.x & 31, u = lane & 7;
  const bool first = u < 4;
  stage_rows(stage, w);
#pragma unroll
  for (int h = 0; h < 8; h += 4) {  // (all sixteen loads at once are 64 registers: spills)
    uint4 cs[4], sn[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int64_t at = static_cast<int64_t>(min(row0 + 4 * (h + i) + (lane >> 3), p.t - 1)) * 64 + 8 * u;
      cs[i] = load_bf16_8<kAligned>(p.cos + at);
      sn[i] = load_bf16_8<kAligned>(p.sin + at);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = 4 * (h + i) + (lane >> 3);
      const uint4 v0 = staged_unit(stage, r, kPairs ? 2 * (u & 3) : u), v1 = staged_unit(stage, r, kPairs ? 2 * (u & 3) + 1 : u ^ 4);
      float x[8], y[8];  // the dim that meets the cosine, and the one that meets the sine
      const uint32_t a[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        if constexpr (kPairs) {
          x[e] = first ? bf16_lo(a[e]) : bf16_hi(a[e]);
          y[e] = first ? -bf16_hi(a[e]) : bf16_lo(a[e]);
        } else {
          x[e] = (e & 1) != 0 ? bf16_hi(a[e >> 1]) : bf16_lo(a[e >> 1]);
          const float o = (e & 1) != 0 ? bf16_hi(a[4 + (e >> 1)]) : bf16_lo(a[4 + (e >> 1)]);
          y[e] = first ? -o : o;
        }
      }
      const uint32_t c[4] = {cs[i].x, cs[i].y, cs[i].z, cs[i].w}, s[4] = {sn[i].x, sn[i].y, sn[i].z, sn[i].w};
      uint32_t o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        o[e] = pack_bf16x2(__fadd_rn(__fmul_rn(x[2 * e], bf16_lo(c[e])), __fmul_rn(y[2 * e], bf16_lo(s[e]))),
                           __fadd_rn(__fmul_rn(x[2 * e + 1], bf16_hi(c[e])), __fmul_rn(y[2 * e + 1], bf16_hi(s[e]))));
      }
      if (r < n_rows) store_unit<kAligned>(dst + r * pitch + u * 16, make_uint4(o[0], o[1], o[2], o[3]));
    }
  }
  __syncwarp();
}

// The column scales of a tile of 256: lane l holds those of columns 8l .. 8l + 7. They are asked for before the tile's products are there;
// loaded where they were used, the same addresses in all lanes, they came from L2 eight times a tile, as there is next to no L1
// (whole prolog, us: 300 tokens 79.7 -> 78.5, 512 94.2 -> 92.8, 1000 140.0 -> 137.7, 4096 499 -> 493).
template <bool kAligned>
__device__ __forceinline__ void load_col_scales(const float* col_scale, float (&sc)[8]) {
  const float* sp = col_scale + 8 * (threadIdx.x & 31);
  if constexpr (kAligned) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(sp)), b = __ldg(reinterpret_cast<const float4*>(sp) + 1);
    sc[0] = a.x;
    sc[1] = a.y;
    sc[2] = a.z;
    sc[3] = a.w;
    sc[4] = b.x;
    sc[5] = b.y;
    sc[6] = b.z;
    sc[7] = b.w;
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) sc[e] = __ldg(sp + e);
  }
}
// int32 accumulators of 64 columns, from column c of the tile on -> bf16 products with the row and column scales, two to a word
__device__ __forceinline__ void wide_dequant_64(uint32_t taddr, float rs, const float (&sc)[8], int c, uint32_t (&v)[32]) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t r[32];
    tmem_ld_32x32b_x32(taddr + c + 32 * h, r);
    tc_wait_ld();
#pragma unroll
    for (int e = 0; e < 32; e += 2) {
      const int from = (c >> 3) + 4 * h + (e >> 3);
      const float w0 = __shfl_sync(0xffffffffu, sc[e & 7], from), w1 = __shfl_sync(0xffffffffu, sc[(e & 7) + 1], from);
      v[16 * h + e / 2] = pack_bf16x2(__fmul_rn(__fmul_rn(static_cast<float>(static_cast<int>(r[e])), rs), w0),
                                      __fmul_rn(__fmul_rn(static_cast<float>(static_cast<int>(r[e + 1])), rs), w1));
    }
  }
}

// One tile's rows out of tensor memory: this warp's 32 rows start at `row0`, `taddr` is its lanes of the tile's accumulator. The
// alignment is a template parameter: with a branch at each of the scales' and cosines' loads they came one after the other, a trip to
// L2 each (1000 tokens: both up-projections 70 -> 57 us, absorbed query 47.5 -> 43.3, the whole prolog 174 -> 158). Of the int8
// up-projections' 168 registers two words of a thread spill.
template <int kEpi, int kN, bool kAligned>
__device__ __forceinline__ void wide_epilogue(const WideParams& p, const WideItem& w, const float (&sc)[8], uint32_t taddr, int row0,
                                              uint32_t stage) {
  const int n_rows = p.t - row0;                 // (may be more than 32, or none)
  const int row = min(row0 + static_cast<int>(threadIdx.x & 31), p.t - 1);
  const int n0 = w.tile * kN;
  if (n_rows <= 0) return;
  if constexpr (kEpi == kWideF32 || kEpi == kWideBf16) {
    constexpr int kEl = kEpi == kWideF32 ? 4 : 2;
    constexpr int kCols = 128 / kEl;
    uint8_t* dst = reinterpret_cast<uint8_t*>(p.out) + (static_cast<long long>(row0) * p.ld_out + static_cast<long long>(w.b) * p.out_batch +
                   n0 + static_cast<long long>(w.split) * p.split_stride) * kEl;
#pragma unroll 1
    for (int c = 0; c < kN; c += kCols) {
      if (n0 + c >= p.n) break;  // (uniform)
      uint32_t o[32];
      if constexpr (kEpi == kWideF32) {
        tmem_ld_32x32b_x32(taddr + c, o);
        tc_wait_ld();
      } else {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(taddr + c + 32 * h, r);
          tc_wait_ld();
#pragma unroll
          for (int e = 0; e < 16; ++e) o[16 * h + e] = pack_bf16x2(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1]));
        }
      }
      // (n is a multiple of 16, so a cut-off piece ends on a 16-byte boundary)
      store_rows<kAligned>(stage, o, dst + c * kEl, p.ld_out * kEl, n_rows, min(128, (p.n - n0 - c) * kEl));
    }
  } else if (kEpi == kWideUp && w.tile >= p.idx_tiles) {
    const float rs = __ldg(p.row_scale + row);
#pragma unroll 1
    for (int c = 0; c < kN; c += 64) {
      const int col = n0 - p.idx_tiles * kN + c;  // 64 columns are the low or high half of a head's nope part or its rope tail
      const int head = col / kHeadQ, part = (col % kHeadQ) >> 6;
      uint32_t v[32];
      wide_dequant_64(taddr, rs, sc, c, v);
      if (part < 2) {
        store_rows<kAligned>(stage, v, reinterpret_cast<uint8_t*>(p.out) + ((static_cast<int64_t>(row0) * 128 + head) * kHeadNope + 64 * part) * 2,
                   128 * kHeadNope * 2, n_rows, 128);
      } else {
        // de-interleaved layout: outputs 0-31 from the even dims, 32-63 from the odd ones; rotate_half = (-second, first)
        store_rows_rotated<kAligned, true>(p, stage, v, row0, reinterpret_cast<uint8_t*>(p.out2) + (static_cast<int64_t>(row0) * 128 + head) * 128,
                                           128 * 128, n_rows);
      }
    }
  } else if (kEpi == kWideUp) {
    const float rs = __ldg(p.row_scale + row);
#pragma unroll 1
    for (int c = 0; c < kN; c += 64) {
      uint32_t v[32];
      wide_dequant_64(taddr, rs, sc, c, v);
      uint8_t* dst = reinterpret_cast<uint8_t*>(p.out_idx) + (static_cast<int64_t>(row0) * 64 * 128 + n0 + c) * 2;
      // rope on the head's first 64 dims: halves, no de-interleave
      if ((c & 64) == 0) store_rows_rotated<kAligned, false>(p, stage, v, row0, dst, 64 * 128 * 2, n_rows);
      else store_rows<kAligned>(stage, v, dst, 64 * 128 * 2, n_rows, 128);
    }
  } else {  // kWideHad: two readings of the row's 128 accumulators, one for the maximum, one to quantise
    static_assert(kEpi != kWideHad || kN == 128, "a Hadamard row is 128 wide");
    float amax = 0.f;
#pragma unroll 1
    for (int c = 0; c < kN; c += 32) {
      uint32_t r[32];
      tmem_ld_32x32b_x32(taddr + c, r);
      tc_wait_ld();
#pragma unroll
      for (int e = 0; e < 32; ++e) amax = fmaxf(amax, fabsf(wide_bf16_round(__uint_as_float(r[e]))));
    }
    const float sq = __fdiv_rn(127.0f, amax);
    uint32_t o[32];
#pragma unroll
    for (int c = 0; c < kN; c += 32) {
      uint32_t r[32];
      tmem_ld_32x32b_x32(taddr + c, r);
      tc_wait_ld();
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        uint32_t word = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int q = static_cast<int8_t>(__float2int_rn(__fmul_rn(wide_bf16_round(__uint_as_float(r[4 * u + e])), sq)));
          word |= (static_cast<uint32_t>(q) & 0xffu) << (8 * e);
        }
        o[c / 4 + u] = word;
      }
    }
    store_rows<kAligned>(stage, o, reinterpret_cast<uint8_t*>(p.out) + static_cast<int64_t>(row0) * 128, 128, n_rows, 128);
    if (static_cast<int>(threadIdx.x & 31) < n_rows) reinterpret_cast<__half*>(p.out2)[row] = __float2half_rn(__fdiv_rn(1.0f, sq));
  }
}

template <bool kI8, int kEpi, int kN, bool kPair>
__global__ void __launch_bounds__(kWThreads, 1)
prolog_wide_kernel(const __grid_constant__ PrologWMaps maps_w,  // int8: map 0 attention, map 1 indexer
                   const __grid_constant__ CUtensorMap tmap_x, const WideParams p) {
  using Cfg = WideCfg<kI8, kN, kPair>;
  constexpr int kWStages = Cfg::kStages;
  extern __shared__ uint8_t wide_smem_raw[];
  const uint32_t raw = smem_u32(wide_smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  WideCtl* ctl = reinterpret_cast<WideCtl*>(wide_smem_raw + (base - raw) + kWStages * Cfg::kStage + kWStaging);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_items = p.row_blocks * p.batch * p.n_tiles * p.splits;
  const uint32_t rank = kPair ? wide_cta_rank() : 0u;
  constexpr int kShift = kPair ? 1 : 0;  // CTAs per worker

  if (tid == 0) {
    for (int i = 0; i < kWStages; ++i) {
      mbar_init(smem_u32(&ctl->full[i]), 1);
      mbar_init(smem_u32(&ctl->empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&ctl->acc_full[i]), 1);
      mbar_init(smem_u32(&ctl->acc_empty[i]), kPair ? 8 : 4);
    }
    ctl->abort = 0;
    fence_mbar_init();
    fence_proxy_async();
    for (int i = 0; i < (kEpi == kWideF32 ? 4 : (kEpi == kWideUp ? 2 : 1)); ++i) tma_prefetch_desc(&maps_w.map[i]);
    tma_prefetch_desc(&tmap_x);
  }
  if (warp == 1) {
    if constexpr (kPair) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)), "r"(Cfg::kTmemCols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      tmem_alloc(smem_u32(&ctl->tmem_base), Cfg::kTmemCols);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (kPair) wide_cluster_sync();  // both CTAs' barriers are there
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;
  pdl_wait();  // the set-up above overlaps the tail of the kernel before this one
  if (tid == 0) pdl_trigger();

  if (warp == 0) {
    // ---------------- producer ----------------
    bool ok = true;
    uint32_t it = 0;
    for (int item = blockIdx.x >> kShift; item < n_items && ok; item += gridDim.x >> kShift) {
      const WideItem w = wide_item(p, item);
      const int k0 = w.split * p.per_split;
      const int kn = min(p.per_split, p.chunks - k0);
      const bool idx = kEpi == kWideUp && w.tile < p.idx_tiles;
      constexpr int kBoxes = Cfg::kBoxes;
      const int box0 = static_cast<int>(rank) * kBoxes;  // first of this CTA's boxes of the tile
      const CUtensorMap* tm[kBoxes];
      int col[kBoxes];  // bytes
#pragma unroll
      for (int g = 0; g < kBoxes; ++g) {
        if (kI8) {
          tm[g] = &maps_w.map[idx ? 1 : 0];
          col[g] = (idx ? w.tile : w.tile - p.idx_tiles) * kN + (box0 + g) * 128;
        } else {
          tm[g] = prolog_w_box(maps_w, p.boxes, w.tile * (kN / Cfg::kGroup) + box0 + g, &col[g]);
        }
      }
      for (int c = 0; c < kn; ++c, ++it) {
        const uint32_t s = it % kWStages;
        if (it >= kWStages) ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&ctl->empty[s]), ((it / kWStages) - 1) & 1));
        if (!ok) break;
        if (elect_one()) {
          const uint32_t bar = smem_u32(&ctl->full[s]);
          const uint32_t dst = base + s * Cfg::kStage;
          const int krow = w.b * p.w_batch_rows + (k0 + c) * Cfg::kChunkK;
          if constexpr (kPair) {
            if (rank == 0) mbar_arrive_expect_tx(bar, 2 * Cfg::kStage);
            const uint32_t bar0 = wide_in_cta0(bar);
            wide_load_pair(dst, &tmap_x, w.b * p.x_batch_bytes + (k0 + c) * 128, (2 * w.rb + static_cast<int>(rank)) * kWRows, bar0);
#pragma unroll
            for (int g = 0; g < kBoxes; ++g) wide_load_pair(dst + kWXBytes + g * Cfg::kBoxBytes, tm[g], col[g], krow, bar0);
          } else {
            mbar_arrive_expect_tx(bar, Cfg::kStage);
            tma_load_2d(dst, &tmap_x, w.b * p.x_batch_bytes + (k0 + c) * 128, w.rb * kWRows, bar);
#pragma unroll
            for (int g = 0; g < kBoxes; ++g) tma_load_2d(dst + kWXBytes + g * Cfg::kBoxBytes, tm[g], col[g], krow, bar);
          }
        }
        __syncwarp();
      }
    }
    if (!ok && lane == 0) {
      ctl->abort = 1;
      set_status(p.status, PTO_ST_WAIT_EXPIRED, blockIdx.x, 80);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    constexpr int kM = kPair ? 2 * kWRows : kWRows;
    constexpr uint32_t idesc = kI8 ? umma_idesc(kCFmtS32, kABFmtS8, kABFmtS8, 0, 1, kM, kN)
                                   : umma_idesc(kCFmtF32, kABFmtBF16, kABFmtBF16, 0, 1, kM, kN);
    bool ok = true;
    uint32_t it = 0, ti = 0;
    for (int item = rank == 0 ? blockIdx.x >> kShift : n_items; item < n_items && ok; item += gridDim.x >> kShift, ++ti) {  // (of a pair: CTA 0 for both)
      const WideItem w = wide_item(p, item);
      const int kn = min(p.per_split, p.chunks - w.split * p.per_split);
      const uint32_t acc = ti & 1;
      if (ti >= 2) {
        const uint32_t bar = smem_u32(&ctl->acc_empty[acc]), ph = ((ti >> 1) - 1) & 1;
        ok = __all_sync(0xffffffffu, kPair ? wide_wait_cluster(bar, ph) : mbar_wait(bar, ph));
      }
      if (!ok) break;
      tc_fence_after();
      const uint32_t d = tmem_base + acc * kN;
      for (int c = 0; c < kn; ++c, ++it) {
        const uint32_t s = it % kWStages;
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&ctl->full[s]), (it / kWStages) & 1));
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
          const uint32_t a = base + s * Cfg::kStage;
          const uint64_t a_desc = umma_desc_kmajor_sw128(a);
          const uint64_t b_desc = desc_mnmajor_sw128(a + kWXBytes, Cfg::kBoxBytes, 1024);
#pragma unroll
          for (int j = 0; j < 4; ++j) {  // 32 bytes along x's rows; 32 (int8) or 16 (bf16) rows of W
            if (kPair) wide_mma_pair<kI8>(d, a_desc + 2 * j, b_desc + j * ((kI8 ? 4096 : 2048) >> 4), idesc, (c | j) != 0 ? 1u : 0u);
            else if (kI8) mma_i8_ss(d, a_desc + 2 * j, b_desc + j * (4096 >> 4), idesc, (c | j) != 0 ? 1u : 0u);
            else mma_f16_ss(d, a_desc + 2 * j, b_desc + j * (2048 >> 4), idesc, (c | j) != 0 ? 1u : 0u);
          }
          if constexpr (kPair) {
            wide_commit_pair(smem_u32(&ctl->empty[s]));
            if (c + 1 == kn) wide_commit_pair(smem_u32(&ctl->acc_full[acc]));
          } else {
            tc_commit(smem_u32(&ctl->empty[s]));
            if (c + 1 == kn) tc_commit(smem_u32(&ctl->acc_full[acc]));
          }
        }
        __syncwarp();
      }
    }
    if (!ok && lane == 0) {
      ctl->abort = 1;
      set_status(p.status, PTO_ST_WAIT_EXPIRED, blockIdx.x, 81);
    }
  } else {
    // ---------------- epilogue: group g stores the tiles of accumulator g ----------------
    const int q = warp & 3;  // TMEM lanes 32q .. 32q+31
    const uint32_t g = static_cast<uint32_t>(warp - 2) >> 2;
    bool ok = true;
    uint32_t ti = 0;
    for (int item = blockIdx.x >> kShift; item < n_items; item += gridDim.x >> kShift, ++ti) {
      if ((ti & 1) != g) continue;
      const WideItem w = wide_item(p, item);
      float sc[8];
      if constexpr (kEpi == kWideUp) {
        const float* scales = w.tile < p.idx_tiles ? p.col_scale_idx + w.tile * kN : p.col_scale + (w.tile - p.idx_tiles) * kN;
        if (p.aligned) load_col_scales<true>(scales, sc);
        else load_col_scales<false>(scales, sc);
      }
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&ctl->acc_full[g]), (ti >> 1) & 1));
      if (!ok) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + g * kN;
      const uint32_t stage = base + kWStages * Cfg::kStage + static_cast<uint32_t>(warp - 2) * 4096u;
      const int row0 = (kPair ? 2 * w.rb + static_cast<int>(rank) : w.rb) * kWRows + q * 32;
      if (p.aligned) wide_epilogue<kEpi, kN, true>(p, w, sc, taddr, row0, stage);
      else wide_epilogue<kEpi, kN, false>(p, w, sc, taddr, row0, stage);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (!kPair || rank == 0) mbar_arrive(smem_u32(&ctl->acc_empty[g]));
        else wide_arrive_cluster(wide_in_cta0(smem_u32(&ctl->acc_empty[g])));
      }
    }
    if (!ok && lane == 0) {
      ctl->abort = 1;
      set_status(p.status, PTO_ST_WAIT_EXPIRED, blockIdx.x, 82);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (ctl->abort) {
    // give copies still in flight time to land before the CTA's shared memory is released
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if constexpr (kPair) wide_cluster_sync();  // neither CTA leaves while the other's loads, MMAs or arrivals may still reach it
  if (warp == 1) {
    tc_fence_after();
    if constexpr (kPair) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(Cfg::kTmemCols) : "memory");
    else tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
}

int wide_aligned(std::initializer_list<const void*> ptrs) {
  for (const void* q : ptrs) {
    if ((reinterpret_cast<uintptr_t>(q) & 15u) != 0) return 0;
  }
  return 1;
}

template <bool kI8, int kEpi, int kN, bool kPair>
cudaError_t wide_launch_as(const PrologWMaps& maps_w, const void* tmap_x, WideParams& p, int k, int num_sms, cudaStream_t stream, bool pdl) {
  using Cfg = WideCfg<kI8, kN, kPair>;
  p.n_tiles = (p.n + kN - 1) / kN;
  p.chunks = (k + Cfg::kChunkK - 1) / Cfg::kChunkK;
  p.per_split = (p.chunks + p.splits - 1) / p.splits;
  if ((p.chunks + p.per_split - 1) / p.per_split != p.splits) return cudaErrorInvalidValue;  // a split without work
  constexpr int kRows = kPair ? 2 * kWRows : kWRows, kCtas = kPair ? 2 : 1;
  p.row_blocks = (p.t + kRows - 1) / kRows;
  auto kernel = prolog_wide_kernel<kI8, kEpi, kN, kPair>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem);
  if (e != cudaSuccess) return e;
  const long long items = static_cast<long long>(p.row_blocks) * p.batch * p.n_tiles * p.splits;
  if (items > 0x7fffffffLL) return cudaErrorInvalidValue;
  const int units = num_sms / kCtas;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(kCtas * (items < units ? static_cast<int>(items) : units)), 1, 1);
  cfg.blockDim = dim3(kWThreads, 1, 1);
  cfg.dynamicSmemBytes = Cfg::kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kCtas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 2 : 1;
  count_launch();
  return cudaLaunchKernelEx(&cfg, kernel, maps_w, *reinterpret_cast<const CUtensorMap*>(tmap_x), static_cast<const WideParams&>(p));
}

// Pairs of SMs from four blocks of 128 rows on; with fewer, whole prologs lost (two blocks up to 1.4 us, three up to 4.9). What a pair saves
// of a tile has to outweigh the work of the last pair's missing block, if the number of blocks is odd. The projections and the bf16
// up-projections save enough at any count: whole prolog by blocks, a CTA per tile -> pairs, us: projections 5 112.2 -> 109.4, 8 145.7 -> 139.8,
// 16 261.5 -> 252.3; bf16 up-projections 4 115.5 -> 110.7, 5 138.0 -> 137.2, 7 168.2 -> 165.2, 8 185.2 -> 174.5, 16 343 -> 322. Those of
// int8 save about a sixteenth, so pairs where the empty share is no more: 4 94.4 -> 92.8, 8 145.7 -> 144.4, 16 261.5 -> 256.8, but 5 112.2 ->
// 114.7, 7 136.5 -> 138.7, 9 173.7 -> 175.4, 13 228.0 -> 230.3; 15 249.8 -> 248.9, 21 363.5 -> 359.7. The absorbed query has two chunks of K per tile
// and is bound by its stores (pairs 47 -> 51), the Hadamard matrix fits one CTA's tile.
template <bool kI8, int kEpi, int kN>
cudaError_t wide_launch(const PrologWMaps& maps_w, const void* tmap_x, WideParams& p, int k, int num_sms, cudaStream_t stream, bool pdl) {
  if constexpr (kEpi != kWideHad) {
    const int blocks = (p.t + kWRows - 1) / kWRows;
    const int empty = blocks & 1;
    const bool pairs = blocks >= 4 && (kEpi != kWideBf16 || k > 128) && (kEpi != kWideUp || 16 * empty <= blocks + empty);
    if (pairs) return wide_launch_as<kI8, kEpi, kN, true>(maps_w, tmap_x, p, k, num_sms, stream, pdl);
  }
  return wide_launch_as<kI8, kEpi, kN, false>(maps_w, tmap_x, p, k, num_sms, stream, pdl);
}

}  // namespace

// The tensor maps are byte matrices: W with a [chunk rows x 128 B] box (64 rows for bf16, 128 for int8), x with a [128 x
// 128 B] box. kind 0: bf16 -> fp32 partials, 1: bf16 -> bf16.
cudaError_t launch_prolog_wide(int kind, const PrologWMaps& maps_w, const PrologWBoxes& boxes, const void* tmap_x, void* out, int t, int n, int k, int batch,
                               int w_batch_rows, int x_batch_bytes, long long out_batch, long long ld_out, int splits,
                               long long split_stride, int num_sms, int32_t* status, cudaStream_t stream, bool pdl) {
  WideParams p{};
  p.boxes = boxes;
  p.t = t;
  p.n = n;
  p.splits = splits < 1 ? 1 : splits;
  p.batch = batch < 1 ? 1 : batch;
  p.w_batch_rows = w_batch_rows;
  p.x_batch_bytes = x_batch_bytes;
  p.out_batch = out_batch;
  p.ld_out = ld_out;
  p.split_stride = split_stride;
  p.out = out;
  p.aligned = wide_aligned({out});
  p.status = status;
  return kind == kWideF32 ? wide_launch<false, kWideF32, 256>(maps_w, tmap_x, p, k, num_sms, stream, pdl)
                          : wide_launch<false, kWideBf16, 256>(maps_w, tmap_x, p, k, num_sms, stream, pdl);
}

// both up-projections: int8 [t, k] . int8 [k, 128 * 192] -> nope parts bf16 [t, 128, 128] and rotated tails [t, 128, 64];
// int8 [t, k] . int8 [k, 64 * 128] -> rotated rows bf16 [t, 64, 128]
cudaError_t launch_prolog_wide_up(const void* tmap_w, const void* tmap_w_idx, const void* tmap_x, int t, int k,
                                  const float* row_scale, const float* col_scale, const float* col_scale_idx, const void* cos,
                                  const void* sin, void* q_nope, void* q_rope, void* idx_rows, int num_sms, int32_t* status,
                                  cudaStream_t stream, bool pdl) {
  WideParams p{};
  p.t = t;
  p.n = 64 * 128 + 128 * kHeadQ;
  p.idx_tiles = 64 * 128 / 256;
  p.splits = p.batch = 1;
  p.out = q_nope;
  p.out2 = q_rope;
  p.out_idx = idx_rows;
  p.row_scale = row_scale;
  p.col_scale = col_scale;
  p.col_scale_idx = col_scale_idx;
  p.cos = reinterpret_cast<const __nv_bfloat16*>(cos);
  p.sin = reinterpret_cast<const __nv_bfloat16*>(sin);
  p.aligned = wide_aligned({q_nope, q_rope, idx_rows, col_scale, col_scale_idx, cos, sin});
  p.status = status;
  PrologWMaps maps;
  maps.map[0] = maps.map[2] = maps.map[3] = *reinterpret_cast<const CUtensorMap*>(tmap_w);
  maps.map[1] = *reinterpret_cast<const CUtensorMap*>(tmap_w_idx);
  return wide_launch<true, kWideUp, 256>(maps, tmap_x, p, k, num_sms, stream, pdl);
}

// rows bf16 [n_rows, 128] . Hadamard bf16 [128, 128] -> int8 rows and an fp16 scale per row
cudaError_t launch_prolog_wide_hadamard(const void* tmap_had, const void* tmap_rows, int n_rows, int8_t* q_int8,
                                        void* q_scale, int num_sms, int32_t* status, cudaStream_t stream) {
  WideParams p{};
  p.t = n_rows;
  p.n = 128;
  p.splits = p.batch = 1;
  p.out = q_int8;
  p.out2 = q_scale;
  p.aligned = wide_aligned({q_int8});
  p.status = status;
  PrologWMaps maps;
  for (int i = 0; i < 4; ++i) maps.map[i] = *reinterpret_cast<const CUtensorMap*>(tmap_had);
  p.boxes = PrologWBoxes{{2, 2, 2, 2}};
  return wide_launch<false, kWideHad, 128>(maps, tmap_rows, p, 128, num_sms, stream, false);
}

}  // namespace pto
