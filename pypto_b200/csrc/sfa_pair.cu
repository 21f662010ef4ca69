// Sparse MLA attention for all 128 heads of a token on a PAIR of SMs that share every matrix product
// (tcgen05.mma.cta_group::2): the two CTAs of a cluster split the token's HEADS, 64 each.
//
// Arithmetic as in sfa_decode.cu (reference:
// examples/models/deepseek_v32_exp/sparse_flash_attention_quant_impl.py:45-207; golden
// deepseekv32_sparse_flash_attention_quant.py:169-254).
//
// Why a pair: the fp32 output of 128 heads x 512 values is 256 KB, all of one SM's tensor memory. With the
// heads split, CTA c keeps O for its 64 heads (256 columns) and two score buffers (2 x 64 columns), and the
// whole 576-wide contraction is local to the pair's MMA: no score ever crosses between the CTAs, and nothing
// else does either except the "ready" notices of a tile (two for K; V with the next tile's rope part; P; scores read). A 2-SM MMA reads half
// of its B operand from each CTA's shared memory:
//   q.K^T  (M = 128 heads, N = 128 keys of a tile, K = 576): A = this CTA's 64 query rows, B = the tile's keys,
//          of which CTA c gathers and dequantises keys [64c, 64c+64) in full width (9 chunks of 64 dims).
//   P.V    (M = 128 heads, N = 256 of the 512 values per MMA, K = 128 keys): A = this CTA's P, B = V, of which
//          CTA c supplies the value columns [256c, 256c+256) of ALL 128 keys. Those of its own 64 keys are the chunks 4c ..
//          4c+3 of its K tile, the same bytes (K-major there, MN-major here). Those of the peer's keys it gathers (an L2
//          hit: the other CTA has just fetched the row) and dequantises itself, since shared memory between the SMs moves
//          about 7 bytes per clock (measured: a 32 KB bulk copy to the peer takes 4-5 k cycles); they go into the other
//          four chunks of the K tile once q.K^T has read those, while the softmax works.
//          So a tile needs 64 + 8 KB of shared memory, two tiles are in flight, and a row is dequantised one and a half
//          times. (With regions of their own for K and V, one tile each, every row was dequantised twice: 4096 tokens x
//          2048 rows 3.75 -> 3.35 ms; of rows in L2, 64 tokens 79 -> 74 us behind a selection, 2 tokens 18.5 -> 16.6 us with the merge.)
// Tensor memory of a 2-SM MMA with 64 rows per CTA: lanes 0-63 hold the first half of the N columns, lanes
// 64-127 the second half (row = lane % 64). So of a score tile lane l holds (head l % 64, keys 64 (l / 64) ..+63),
// and of O lane l holds (head l % 64, values 256 (l / 64) ..+255).
//   warp 0          CTA 0: issues the q.K^T MMAs of a tile as soon as its keys are ready and a score buffer is free
//   warp 2          CTA 0: issues the P.V MMAs of a tile as soon as P is written and the values are ready
//                   (two issuing threads on two schedulers: neither queue waits behind the other's barrier)
//   warps 0, 1, 2   CTA 1: forward the "ready" events of their CTA to CTA 0 (tcgen05.commit arrivals on CTA 0's barriers)
//   warps 4..11     softmax: four threads per head (two TMEM lanes x two column halves), P goes to shared memory
//   warps 12..19    K producers: 16-byte gathers of the CTA's 64 rows, int8 -> bf16 in registers, swizzled stores
//   warps 20..27    V producers: this CTA's half of the value columns of the peer's 64 rows; rope parts of the CTA's own
// Cache formats: int8 latent + bf16 rope + fp32 scales in three arrays, the same as packed 656-byte rows, or bf16
// latent + rope arrays (the non-quantised cache): there the producers dequantise nothing, they copy the rows' bytes
// from L2 to the same swizzled places with cp.async once their part of the buffer is free. The MMAs, the softmax and the
// output are the same code, so the bf16 cache of dequantised values gives the int8 cache's output bit for bit.
// Roles are uniform within each group of four warps so that registers can be moved between them (setmaxnreg):
// 72 per thread at launch (seven warps share one scheduler's file of 512 x 32), then 24 / 104 / 72 / 64:
// nothing spills (a spilled register costs a trip to L2: beside 227 KB of shared memory there is no L1 to speak of).
// All waits are bounded.
#include "common.cuh"
#include "sfa_common.cuh"

namespace pto {

namespace {

constexpr int kPT = 128;                 // selected rows per tile (64 per CTA)
constexpr int kPRows = 64;               // rows a CTA gathers in full width per tile; also heads per CTA
constexpr int kChunk = kPRows * 128;     // 64 rows x 64 bf16 (128-byte rows, 128-byte swizzle): 8 KB
constexpr int kQChunks = 9;              // 8 latent chunks + 1 rope chunk
constexpr int kSmemQ = 0;
constexpr int kSmemT = kSmemQ + kQChunks * kChunk;        // 73,728: two tile buffers of eight latent chunks
constexpr int kTileBytes = 8 * kChunk;
constexpr int kVHalfBytes = 4 * kChunk;                   // 64 keys x 256 values: half of a tile buffer
constexpr int kSmemRope = kSmemT + 2 * kTileBytes;        // 204,800: rope chunk of a tile
constexpr int kSmemP = kSmemRope + kChunk;                // 212,992: two chunks (keys 0-63, keys 64-127)
constexpr int kSmemCtl = kSmemP + 2 * kChunk;             // 229,376
constexpr int kPairSoftmaxWarp0 = 4, kPairSoftmaxWarps = 8;
constexpr int kPairKWarp0 = 12, kPairKWarps = 8;
constexpr int kPairVWarp0 = 20, kPairVWarps = 8;
constexpr int kPairThreads = 32 * 28;
constexpr uint32_t kPairTmemCols = 512;
constexpr uint32_t kPairColO = 0, kPairColS = 256;        // S buffer b at kPairColS + 64 b
constexpr float kPairRescale = 8.0f;

// Tile buffer b = j % 2 of tile j; half h of it = chunks 4h .. 4h+3. In CTA c a half goes through
//   half c:      K of the CTA's own 64 keys (chunks 4c .. 4c+3) for q.K^T, then, the same bytes, V of those keys
//   half 1 - c:  K of its own keys (the other four chunks), then V (columns 256c ..) of the peer's keys
// so that half h holds, in both CTAs, V of the keys 64h .. 64h+63 when P.V reads it. The rope chunk of tile j+1 is copied when
// q.K^T of tile j has read its predecessor, by the V producers along with V of tile j: event j+1 of `vfull` (event 0: rope of
// tile 0). Barriers that may complete for tile j+1 before everybody has waited for tile j exist once per buffer.
struct PairCtl {
  uint64_t kfull[2][2];  // [b][h] K producers filled half h of buffer b               (4 warps)
  uint64_t kread[2];     // the q.K^T MMAs that read half 0 of buffer b are complete   (tcgen05.commit, both CTAs)
  uint64_t vfull[2];     // [event % 2] V of tile event - 1, rope of tile event        (8 warps)
  uint64_t bfree[2][2];  // [b][h] the P.V MMAs that read half h are complete          (tcgen05.commit, both CTAs)
  uint64_t sfull[2];     // q.K^T of a tile complete (score buffer b)                  (tcgen05.commit, both CTAs)
  uint64_t pvdone;       // P.V of a tile complete                                    (tcgen05.commit, both CTAs)
  uint64_t pfull;        // this CTA's P of tile j written                            (8 warps)
  uint64_t sread[2];     // this CTA's softmax warps have the scores in registers     (8 warps)
  // in CTA 0 only: the same events of CTA 1, forwarded (one arrival each)
  uint64_t kpeer[2][2], vpeer[2], ppeer, speer[2];
  uint32_t tmem_base;
  int abort;
  int go[2];           // outcome of the softmax role's latest waits
  float mt[2][4][64];  // [tile parity][key half * 2 + column half][head]: partial maxima; partial sums at the end
};
static_assert(kSmemCtl + sizeof(PairCtl) <= 232448, "exceeds the 227 KB of shared memory a CTA may use");
constexpr size_t kPairSmemBytes = 232448;

__device__ __forceinline__ uint32_t pair_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void pair_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Notice from CTA 1 to CTA 0: a tcgen05.commit of no outstanding operation arrives at once on the mbarrier at this
// offset in CTA 0 (mask 1). It travels on the tensor pipe's own path: measured one way 390 cycles, as fast as an
// asynchronous remote store, but unlike that store it does not queue behind the SM's gathers in the load/store
// unit (under load the store took 2000-3300 cycles to arrive; a remote mbarrier arrive holds the lane ~1400).
__device__ __forceinline__ void pair_signal(uint32_t bar_local) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar_local), "h"(static_cast<uint16_t>(1))
               : "memory");
}

__device__ __forceinline__ void mma2_f16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives (count 1) on the mbarrier at this offset in BOTH CTAs once all MMAs issued so far have completed
__device__ __forceinline__ void tc2_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(static_cast<uint16_t>(3))
               : "memory");
}

// Warp-wide bounded wait. try_wait parks the warp in hardware; probing with sleeps in between takes issue slots and
// shared-memory cycles from the warps that have work.
__device__ __forceinline__ bool pair_wait(uint32_t bar, uint32_t parity) {
  bool ok = true;
  if (!mbar_test_wait(bar, parity)) {
    const long long t0 = clock64();
    while (true) {
      if (mbar_try_wait(bar, parity)) break;
      if (clock64() - t0 > kWaitBudgetCycles) {
        ok = false;
        break;
      }
    }
  }
  return __all_sync(0xffffffffu, ok);
}

// Wait of a whole role (kThreads threads = full warps, named barrier kBarId): only the role's first warp probes the
// mbarrier, the others block at the named barrier without issuing anything. The first warp publishes the outcome
// in one of two slots (alternating: a thread is never more than one wait behind), every thread of the role reads
// the same slot after the barrier, so the whole role takes the same branch; the barrier itself depends on no data
// and every thread of the role reaches it on every path.
template <int kBarId, int kThreads>
__device__ __forceinline__ bool pair_group_wait(PairCtl* ctl, uint32_t& nwait, uint32_t bar, uint32_t parity, bool first_warp) {
  volatile int* go = &ctl->go[nwait & 1u];
  ++nwait;
  if (first_warp) {
    const bool ok = pair_wait(bar, parity);
    if ((threadIdx.x & 31) == 0) *go = ok ? 1 : 0;
  }
  asm volatile("bar.sync %0, %1;" ::"n"(kBarId), "n"(kThreads) : "memory");
  return *go != 0;
}

// 8 int8 (two words) -> 8 bf16 of (value * scale), with the subtraction and the multiplication on pairs (fp32x2 instructions):
// byte^0x80 placed in the mantissa of 2^23 gives 2^23 + 128 + x exactly, subtracting 8388736
// leaves x, one fp32 multiply and one rounding to bf16: bf16(fp32(x) * scale) as the golden computes it.
__device__ __forceinline__ uint4 pair_dequant8(const uint32_t w0, const uint32_t w1, const float scale) {
  const float2 off = make_float2(-8388736.0f, -8388736.0f), sc = make_float2(scale, scale);
  uint4 o;
  {
    const uint32_t w = w0 ^ 0x80808080u;
    float2 a = make_float2(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540)), __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7541)));
    float2 b = make_float2(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7542)), __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7543)));
    a = __fmul2_rn(__fadd2_rn(a, off), sc);
    b = __fmul2_rn(__fadd2_rn(b, off), sc);
    o.x = pack_bf16x2(a.x, a.y);
    o.y = pack_bf16x2(b.x, b.y);
  }
  {
    const uint32_t w = w1 ^ 0x80808080u;
    float2 a = make_float2(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540)), __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7541)));
    float2 b = make_float2(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7542)), __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7543)));
    a = __fmul2_rn(__fadd2_rn(a, off), sc);
    b = __fmul2_rn(__fadd2_rn(b, off), sc);
    o.z = pack_bf16x2(a.x, a.y);
    o.w = pack_bf16x2(b.x, b.y);
  }
  return o;
}

// this lane's 32 bytes of a row: 32 values, half `part` of the chunk's 64
__device__ __forceinline__ void pair_store_wide(uint32_t row_addr, int part, int x, const uint4 lo, const uint4 hi, float scale) {
  sts_v4u(row_addr + (((4 * part) ^ x) << 4), pair_dequant8(lo.x, lo.y, scale));
  sts_v4u(row_addr + (((4 * part + 1) ^ x) << 4), pair_dequant8(lo.z, lo.w, scale));
  sts_v4u(row_addr + (((4 * part + 2) ^ x) << 4), pair_dequant8(hi.x, hi.y, scale));
  sts_v4u(row_addr + (((4 * part + 3) ^ x) << 4), pair_dequant8(hi.z, hi.w, scale));
}

struct PairCtx {
  PairCtl* ctl;
  const int32_t* idx_row;  // this token's selected positions
  int64_t q_row0;          // first query/output row of the token
  uint32_t base, tmem_base, crank;
  int ntiles, begin, end, sp, bi;
  int pt;  // token among those that are split, or -1: the rows are one piece, the output is written as it is
};

// The one meeting of all threads of the pair before the tile loop (barriers initialised, tensor memory allocated, both Q
// halves in shared memory), in two parts. The producers have nothing to show the others and arrive first thing; they wait
// when tile 0 is converted, whose place nobody has used before, so that the index -> block table -> row chain and the
// conversion of the first tile run beside the set-up and the meeting's own latency (1.5-2 k cycles) instead of after them.
// The other twelve warps meet among themselves, then arrive for what they wrote, and wait.
__device__ __forceinline__ void pair_setup_arrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void pair_setup_wait() {
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  tc_fence_after();
}
__device__ __forceinline__ uint32_t pair_setup_sync(PairCtl* ctl) {
  tc_fence_before();
  asm volatile("bar.sync 2, %0;" ::"n"(32 * kPairKWarp0) : "memory");
  pair_setup_arrive();
  pair_setup_wait();
  // the kernel behind this one (the merge of the split partials) may be scheduled from here on; it waits for
  // this grid to complete before it reads anything
  if (threadIdx.x == 0) pdl_trigger();
  return ctl->tmem_base;
}

// ================================ MMA issuers (CTA 0) ===========================================
// Two threads on two different schedulers: warp 0 issues the score products, warp 2 the value products.
//   q.K^T half 0  (chunks 0-3: 16 MMAs)  needs K half 0 of the tile and the score buffer it overwrites read
//   q.K^T half 1  (chunks 4-7: 16 MMAs)  needs K half 1
//   q.K^T rope    (chunk 8: 4 MMAs)      needs the rope chunk; completes the tile's scores
//   P.V half h    (keys 64h .. +63: 8 MMAs)  needs P of the tile and V of the keys; the second completes the tile's P.V
// After each action a commit hands the part it read back to its producers, so that the refill for the next tile
// runs behind the MMAs that read the others. One thread issuing everything was what a tile waited for: 36 + 16 MMAs kept it
// busy for 8.7 k cycles per tile (two threads: 80.1 -> 77.7 us on 64 tokens x 2048 rows). The products of the two threads
// are independent (different accumulators), every dependency between them goes through the mbarriers, and a
// commit covers the MMAs of the thread that executes it.
// (No cluster-scope fence before the MMAs: measured, `fence.acq_rel.cluster` holds a thread for 2000-3700 cycles
// per use. The order is kept by the chain itself: CTA 1's writers fence for the async proxy and arrive on their
// own barrier, its forwarding thread observes that barrier before it sends the notice, and the MMA issued here
// after the notice reads CTA 1's shared memory from CTA 1's side.)
// The issuing warps stay converged and one elected lane issues, with descriptors that are constants of the code (kBase:
// the address where a kernel without static shared memory finds its dynamic part; kBase = 0 is the same code with the
// address in a register). Under `if (lane == 0)` the descriptors are moved to uniform registers for every MMA: measured in
// isolation, K = 16, 51-61 cycles per MMA whatever its shape, against the 39 / 48 / 64 / 128 the tensor core needs for N
// = 16 / 64 / 128 / 256 (cta_group::1); beside two dozen busy warps an address in a register costs about as much.
constexpr uint32_t kPairUsualBase = 1024;
__device__ __forceinline__ bool pair_poll(uint32_t bar, uint32_t parity) {  // whole warp, bounded, uniform outcome
  if (__all_sync(0xffffffffu, mbar_test_wait(bar, parity))) return true;
  const long long t0 = clock64();
  while (true) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    if (__any_sync(0xffffffffu, clock64() - t0 > kWaitBudgetCycles)) return false;
  }
}

// part kPart of the score product of buffer kB into score buffer kB: four latent chunks, or (2) the rope chunk
template <int kB, int kPart>
__device__ __forceinline__ void pair_issue_qk(uint32_t tmem_base, uint64_t a_desc, uint64_t b_desc) {
  constexpr uint32_t idesc_qk = umma_idesc(kCFmtF32, kABFmtBF16, kABFmtBF16, 0, 0, 128, kPT);
#pragma unroll
  for (int ch = 4 * kPart; ch < (kPart == 2 ? kQChunks : 4 * kPart + 4); ++ch) {
    const int kch = kPart == 2 ? (kSmemRope - kSmemT) / kChunk : kB * 8 + ch;  // chunks from the first tile buffer on
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      mma2_f16_ss(tmem_base + kPairColS + 64 * kB, a_desc + ch * (kChunk >> 4) + 2 * k, b_desc + kch * (kChunk >> 4) + 2 * k, idesc_qk,
                  (ch | k) != 0 ? 1u : 0u);
    }
  }
}

template <uint32_t kBase>
__device__ __forceinline__ void pair_role_issue_qk(const SfaParams& p, PairCtx c) {
  if (kBase != 0) c.base = kBase;
  PairCtl* ctl = c.ctl;
  const int ntiles = c.ntiles;
  const uint32_t tmem_base = pair_setup_sync(ctl);
  const uint64_t a_desc = umma_desc_kmajor_sw128(c.base + kSmemQ), b_desc = umma_desc_kmajor_sw128(c.base + kSmemT);
  bool ok = true;
  for (int j = 0; j < ntiles && ok; ++j) {
    const uint32_t b = j & 1, ph = (j >> 1) & 1;
    if (j >= 2) {  // the score buffer it overwrites has been read in both CTAs
      ok = pair_poll(smem_u32(&ctl->sread[b]), ph ^ 1) && pair_poll(smem_u32(&ctl->speer[b]), ph ^ 1);
    }
#define PAIR_QK_PART(part, mine, peer, done)                                                                    \
  ok = ok && pair_poll(smem_u32(&(mine)), ph) && pair_poll(smem_u32(&(peer)), ph);                              \
  if (!ok) break;                                                                                               \
  tc_fence_after();                                                                                             \
  if (elect_one()) {                                                                                            \
    if (b == 0) pair_issue_qk<0, part>(tmem_base, a_desc, b_desc);                                              \
    else pair_issue_qk<1, part>(tmem_base, a_desc, b_desc);                                                     \
    if ((part) != 1) tc2_commit(smem_u32(&(done)));                                                             \
  }                                                                                                             \
  __syncwarp();
    PAIR_QK_PART(0, ctl->kfull[b][0], ctl->kpeer[b][0], ctl->kread[b])
    PAIR_QK_PART(1, ctl->kfull[b][1], ctl->kpeer[b][1], ctl->kread[b])
    PAIR_QK_PART(2, ctl->vfull[b], ctl->vpeer[b], ctl->sfull[b])
#undef PAIR_QK_PART
  }
  if (!ok && (threadIdx.x & 31) == 0) {
    ctl->abort = 1;
    set_status(p.status, PTO_ST_WAIT_EXPIRED, blockIdx.x, 50);
  }
  __syncwarp();
}

// keys 64 kH .. +63 of the tile in buffer kB into both pairs of value columns
template <int kB, int kH>
__device__ __forceinline__ void pair_issue_pv(uint32_t d, uint64_t a_desc, uint64_t b_desc, uint32_t accumulate) {
  constexpr uint32_t idesc_pv = umma_idesc(kCFmtF32, kABFmtBF16, kABFmtBF16, 0, 1, 128, 256);
#pragma unroll
  for (int dp = 0; dp < 2; ++dp) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      mma2_f16_ss(d + 128 * dp, a_desc + kH * (kChunk >> 4) + 2 * k,
                  b_desc + ((kB * kTileBytes + kH * kVHalfBytes + dp * 2 * kChunk + k * 16 * 128) >> 4), idesc_pv,
                  (kH > 0 || k > 0) ? 1u : accumulate);
    }
  }
}

template <uint32_t kBase>
__device__ __forceinline__ void pair_role_issue_pv(const SfaParams& p, PairCtx c) {
  if (kBase != 0) c.base = kBase;
  PairCtl* ctl = c.ctl;
  const int ntiles = c.ntiles;
  const uint32_t tmem_base = pair_setup_sync(ctl);
  const uint64_t a_desc = umma_desc_kmajor_sw128(c.base + kSmemP), b_desc = desc_mnmajor_sw128(c.base + kSmemT, kChunk, 1024);
  bool ok = true;
  for (int j = 0; j < ntiles && ok; ++j) {
    const uint32_t b = j & 1, pp = j & 1, ev = (j + 1) & 1, eph = ((j + 1) >> 1) & 1;
    ok = pair_poll(smem_u32(&ctl->pfull), pp) && pair_poll(smem_u32(&ctl->ppeer), pp);
    // V of the keys that are not a CTA's own: keys 0-63 in CTA 1, 64-127 in CTA 0
#define PAIR_PV_HALF(h, bar)                                                                                    \
  ok = ok && pair_poll(smem_u32(&(bar)), eph);                                                                  \
  if (!ok) break;                                                                                               \
  tc_fence_after();                                                                                             \
  if (elect_one()) {                                                                                            \
    if (b == 0) pair_issue_pv<0, h>(tmem_base + kPairColO, a_desc, b_desc, j > 0 ? 1u : 0u);                    \
    else pair_issue_pv<1, h>(tmem_base + kPairColO, a_desc, b_desc, j > 0 ? 1u : 0u);                           \
    tc2_commit(smem_u32(&ctl->bfree[b][h]));                                                                    \
    if ((h) == 1) tc2_commit(smem_u32(&ctl->pvdone));                                                           \
  }                                                                                                             \
  __syncwarp();
    PAIR_PV_HALF(0, ctl->vpeer[ev])
    PAIR_PV_HALF(1, ctl->vfull[ev])
#undef PAIR_PV_HALF
  }
  if (!ok && (threadIdx.x & 31) == 0) {
    ctl->abort = 1;
    set_status(p.status, PTO_ST_WAIT_EXPIRED, blockIdx.x, 55);
  }
  __syncwarp();
}

// ================================ forwarding (CTA 1) ============================================
// Three warps, one per producer of events: when a per-tile event of this CTA completes, tell CTA 0. The events of a
// role complete in order, so each warp waits for one at a time (a single warp that polled all of them in turn added
// up to 1 k cycles to a notice).
enum { kRelayK = 0, kRelayV = 1, kRelayP = 2 };
template <int kWhat>
__device__ __forceinline__ void pair_role_relay(const SfaParams& p, PairCtx c) {
  PairCtl* ctl = c.ctl;
  const int ntiles = c.ntiles;
  pair_setup_sync(ctl);
  bool ok = true;
  for (int j = 0; j < (kWhat == kRelayV ? ntiles + 1 : ntiles) && ok; ++j) {  // (V: events)
    const uint32_t b = j & 1, ph = (j >> 1) & 1;
    if (kWhat == kRelayP) {
      if (j < ntiles - 2) {  // scores of tile j read: only tiles that have a successor two on
        ok = pair_poll(smem_u32(&ctl->sread[b]), ph);
        if (ok && elect_one()) pair_signal(smem_u32(&ctl->speer[b]));
        __syncwarp();
      }
      ok = ok && pair_poll(smem_u32(&ctl->pfull), j & 1);
      if (ok && elect_one()) pair_signal(smem_u32(&ctl->ppeer));
      __syncwarp();
    } else if (kWhat == kRelayV) {
      ok = pair_poll(smem_u32(&ctl->vfull[b]), ph);
      if (ok && elect_one()) pair_signal(smem_u32(&ctl->vpeer[b]));
      __syncwarp();
    } else {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        ok = ok && pair_poll(smem_u32(&ctl->kfull[b][h]), ph);
        if (ok && elect_one()) pair_signal(smem_u32(&ctl->kpeer[b][h]));
        __syncwarp();
      }
    }
  }
  if (!ok && (threadIdx.x & 31) == 0) {
    ctl->abort = 1;
    set_status(p.status, PTO_ST_WAIT_EXPIRED, blockIdx.x, 54);
  }
  __syncwarp();
}

// ================================ softmax =======================================================
// Thread (TMEM lane L, column half ch): head L % 64, keys 64 (L / 64) + 32 ch .. +31 of the 128-key tile.
__device__ __forceinline__ void pair_role_softmax(const SfaParams& p, PairCtx c) {
  PairCtl* ctl = c.ctl;
  const uint32_t tmem_base = pair_setup_sync(ctl);
  const int ntiles = c.ntiles;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = warp & 3;                            // TMEM lane quarter this warp may access
  const int ch = (warp - kPairSoftmaxWarp0) >> 2;      // column half
  const int kh = sub >> 1;                             // key half of the tile
  const int hg = sub & 1;                              // head group: heads 32 hg .. +31
  const int head = 32 * hg + lane;
  const int slot = kh * 2 + ch;                        // which of the head's four threads
  const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(sub * 32) << 16);
  const uint32_t p_row = c.base + kSmemP + kh * kChunk + head * 128;
  const int psw = head & 7;
  float m_seen = -INFINITY;  // the head's reference max (identical in its four threads)
  float l_run = 0.f;         // this thread's share of the row sum
  bool ok = true;
  const bool first_warp = warp == kPairSoftmaxWarp0;
  uint32_t nwait = 0;
  auto meet = [&]() {  // the four warps of a head group: orders their mt writes before the reads (named barriers 4, 5)
    if (hg == 0) asm volatile("bar.sync 4, 128;" ::: "memory");
    else asm volatile("bar.sync 5, 128;" ::: "memory");
  };
  for (int j = 0; j < ntiles; ++j) {
    const int b = j & 1;
    ok = pair_group_wait<1, 256>(ctl, nwait, smem_u32(&ctl->sfull[b]), (j >> 1) & 1, first_warp);
    if (!ok) break;
    tc_fence_after();
    float s[32];
    {
      uint32_t v[32];
      tmem_ld_32x32b_x32(lane_addr + kPairColS + 64 * b + 32 * ch, v);
      tc_wait_ld();
#pragma unroll
      for (int i = 0; i < 32; ++i) s[i] = __uint_as_float(v[i]);
    }
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&ctl->sread[b]));  // the score buffer may be overwritten
    // ---- mask rows past the token's selected count (last tile only) --------------------------------
    const int key0 = c.begin + j * kPT + 64 * kh + 32 * ch;
    if (key0 + 32 > c.end) {
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        if (key0 + i >= c.end) s[i] = -INFINITY;
      }
    }
    float mt2[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int i = 0; i < 32; ++i) mt2[i & 1] = fmaxf(mt2[i & 1], s[i]);
    const float mt_part = fmaxf(mt2[0], mt2[1]) * p.scale_log2;  // scale > 0
    ctl->mt[b][slot][head] = mt_part;
    // ---- exponentials against a speculative reference (corrected by one factor once the head's max is known) --
    float m_spec = (m_seen == -INFINITY || mt_part > m_seen + kPairRescale) ? mt_part : m_seen;
    if (m_spec == -INFINITY) m_spec = 0.f;
    const float neg_spec = -m_spec;
    float ls2[2] = {0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      s[i] = ex2f(fmaf(s[i], p.scale_log2, neg_spec));
      ls2[i & 1] += s[i];
    }
    const float lsum = ls2[0] + ls2[1];
    meet();
    const float mt = fmaxf(fmaxf(ctl->mt[b][0][head], ctl->mt[b][1][head]), fmaxf(ctl->mt[b][2][head], ctl->mt[b][3][head]));
    const float m_new = fmaxf(m_seen, mt);
    const bool need = (m_new > m_seen + kPairRescale) || (m_seen == -INFINITY && m_new > -INFINITY);
    float alpha = 1.f;
    if (need) {
      alpha = (m_seen == -INFINITY) ? 0.f : ex2f(m_seen - m_new);
      m_seen = m_new;
    }
    const float m_ref = (m_seen == -INFINITY) ? 0.f : m_seen;
    const float factor = ex2f(m_spec - m_ref);
    l_run = l_run * alpha + lsum * factor;
    // ---- the previous tile's P.V is complete: P may be overwritten, O is at rest ----------------------
    if (j > 0) {
      ok = pair_group_wait<1, 256>(ctl, nwait, smem_u32(&ctl->pvdone), (j - 1) & 1, first_warp);
      if (!ok) break;
      tc_fence_after();
    }
    if (j > 0 && __any_sync(0xffffffffu, need)) {  // rare: rescale this thread's 128 output columns
#pragma unroll 1
      for (int cc = 0; cc < 8; ++cc) {
        uint32_t o[16];
        tmem_ld_32x32b_x16(lane_addr + kPairColO + ch * 128 + cc * 16, o);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
        tmem_st_32x32b_x16(lane_addr + kPairColO + ch * 128 + cc * 16, o);
      }
      tc_wait_st();
    }
    // ---- P row piece into shared memory (A operand of P.V): 32 keys = four 16-byte units 4 ch .. 4 ch + 3 ----
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      uint4 w;
      w.x = pack_bf16x2(s[8 * u] * factor, s[8 * u + 1] * factor);
      w.y = pack_bf16x2(s[8 * u + 2] * factor, s[8 * u + 3] * factor);
      w.z = pack_bf16x2(s[8 * u + 4] * factor, s[8 * u + 5] * factor);
      w.w = pack_bf16x2(s[8 * u + 6] * factor, s[8 * u + 7] * factor);
      sts_v4u(p_row + (((4 * ch + u) ^ psw) << 4), w);
    }
    fence_proxy_async();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&ctl->pfull));
  }
  // ---- output ---------------------------------------------------------------------------------------
  if (ok) ok = pair_group_wait<1, 256>(ctl, nwait, smem_u32(&ctl->pvdone), (ntiles - 1) & 1, first_warp);
  float l_tot = 0.f;
  if (ok) {
    ctl->mt[ntiles & 1][slot][head] = l_run;
    meet();
    const int b = ntiles & 1;
    l_tot = (ctl->mt[b][0][head] + ctl->mt[b][1][head]) + (ctl->mt[b][2][head] + ctl->mt[b][3][head]);
  }
  // The rows go out through shared memory: a thread holds 128 values of ONE row, so direct stores put every lane of
  // a warp on its own 128-byte line (4096 lines per CTA, about 4 k cycles); staged, a warp writes 512 contiguous
  // bytes. Staging area: the tile buffers (all products of this cluster are complete once the last P.V is), rows of
  // 1 KB + 16 B (the pad keeps the lanes of a warp, which write different rows, on different banks); a row holds
  // the 256-byte pieces of the head's four threads. bf16 rows take one pass, fp32 partial rows two.
  {
    const uint32_t stage = c.base + kSmemT;
    constexpr uint32_t kStageRow = 1024 + 16;
    static_assert(64 * kStageRow <= 2 * kTileBytes, "output staging exceeds the tile buffers");
    const int stid = threadIdx.x - 32 * kPairSoftmaxWarp0;       // 0..255
    const uint32_t my_piece = stage + head * kStageRow + slot * 256;
    const bool direct = c.pt < 0;
    const float inv = l_tot > 0.f ? 1.f / l_tot : 0.f;
    const int npass = direct ? 1 : 2;
    if (ok) tc_fence_after();
#pragma unroll 1
    for (int ps = 0; ps < npass; ++ps) {
      if (ok) {
#pragma unroll 1
        for (int cc = 0; cc < (direct ? 4 : 2); ++cc) {
          uint32_t o[32];
          tmem_ld_32x32b_x32(lane_addr + kPairColO + ch * 128 + (direct ? cc : 2 * ps + cc) * 32, o);
          tc_wait_ld();
          if (direct) {  // 32 values -> 64 bytes
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              uint4 w;
              w.x = pack_bf16x2(__uint_as_float(o[i]) * inv, __uint_as_float(o[i + 1]) * inv);
              w.y = pack_bf16x2(__uint_as_float(o[i + 2]) * inv, __uint_as_float(o[i + 3]) * inv);
              w.z = pack_bf16x2(__uint_as_float(o[i + 4]) * inv, __uint_as_float(o[i + 5]) * inv);
              w.w = pack_bf16x2(__uint_as_float(o[i + 6]) * inv, __uint_as_float(o[i + 7]) * inv);
              sts_v4u(my_piece + cc * 64 + i * 2, w);
            }
          } else {       // 32 values -> 128 bytes
#pragma unroll
            for (int i = 0; i < 32; i += 4) sts_v4u(my_piece + cc * 128 + i * 4, make_uint4(o[i], o[i + 1], o[i + 2], o[i + 3]));
          }
        }
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");  // (every softmax thread reaches it, also after an expired wait)
      if (ok) {
        // 64 rows x 64 units of 16 bytes; consecutive threads take consecutive units of a row
        uint8_t* gbase;
        int64_t grow_bytes;  // bytes between rows in global memory
        if (direct) {
          gbase = reinterpret_cast<uint8_t*>(p.out + (c.q_row0 + 64 * static_cast<int>(c.crank)) * 512);
          grow_bytes = 1024;
        } else {
          const int64_t prow0 = (static_cast<int64_t>(c.pt) * p.n_split + c.sp) * p.nq + 64 * static_cast<int>(c.crank);
          gbase = reinterpret_cast<uint8_t*>(p.part_o + prow0 * 512);
          grow_bytes = 2048;
        }
#pragma unroll 4
        for (int it = 0; it < 16; ++it) {
          const int e = it * 256 + stid;
          const int r = e >> 6, unit = e & 63;        // unit: 16 bytes of the staged row; piece = unit / 16
          const uint4 w = lds_v4u(stage + r * kStageRow + unit * 16);
          // bf16: the row's bytes in order. fp32: piece q of pass ps holds floats 128 q + 64 ps .. + 63 of the row
          const int64_t off = direct ? unit * 16 : ((unit >> 4) * 512 + ps * 256 + (unit & 15) * 16);
          *reinterpret_cast<uint4*>(gbase + r * grow_bytes + off) = w;
        }
      }
      if (ps + 1 < npass) asm volatile("bar.sync 1, 256;" ::: "memory");  // staging area reused by the next pass
    }
    if (ok && !direct && slot == 0) {
      const int64_t prow = (static_cast<int64_t>(c.pt) * p.n_split + c.sp) * p.nq + 64 * static_cast<int>(c.crank) + head;
      p.part_ml[prow * 2] = m_seen;
      p.part_ml[prow * 2 + 1] = l_tot;
    }
  }
  if (!ok && lane == 0) {
    ctl->abort = 1;
    set_status(p.status, PTO_ST_WAIT_EXPIRED, blockIdx.x, 51);
  }
}

// ================================ K producers ===================================================
// Eight warps, four per half of the K chunks: warp (half, g) converts the half (256 bytes of latent: two lines of 128
// dims, each with its scale) of the CTA's rows 16g .. 16g+15. Every warp
// waits for its own half, so the load of a half, its conversion, the notice and the MMAs that read it overlap those of
// the other, and each warp pays the hand-over (wait, fence, arrive) once per tile. (All eight warps walking through
// quarters together paid it four times: 7.9 k cycles per tile instead of 6.5 k. Two warps per quarter, each one line of 32
// rows: as fast with separate arrays, slower with packed rows, whose 128-byte pieces straddle lines.)
// A gather instruction reads the line of FOUR rows, whole: lane l takes 16 bytes of row 4m + (l / 4) % 4. (Four threads
// per row, each reading its own 16 bytes of eight different lines, cost eight lines per instruction; with the V
// producers' gathers on top, the load/store unit's queue then delayed the tensor core's operand reads.)
// Lane l holds unit l % 4 of chunk 2 line + l / 16 of the half (16 int8 -> 16 bf16 = the store units 2 (l % 4) and 2 (l % 4) + 1 of the
// row's 128 bytes). The eight lanes of a quarter-warp are four units of two neighbouring rows, whose swizzle terms
// differ in the lowest bit: eight different bank groups.
// Lane r % 16 also walks the look-ahead chain of row 16g + r: the selected index four tiles ahead, its block-table entry three
// tiles ahead, an L2 prefetch of the half row two tiles ahead, the half row itself (by all lanes) one tile ahead.
// kFmt: 0 = int8 latent, bf16 rope and fp32 scales in three arrays, 1 = packed 656-byte rows, 2 = bf16 latent and
// rope arrays (the non-quantised cache), 3 = as 0 in 32-byte loads, half as many (kWide, see sfa_pair_wide_loads. Eight lanes of a store
// instruction are then both halves of four rows: eight different bank groups again). With a bf16 cache nothing passes through registers: when the half is free
// every lane issues its 16-byte `cp.async` copies from L2 (the rows were prefetched there two tiles ago) straight to
// the swizzled places the dequantised units would go, waits for them, fences and arrives.
// A padding or rejected row reads row 0 with scale 0, which dequantises to zeros.
template <int kFmt>
__device__ __forceinline__ void pair_role_kproducer(const SfaParams& p, const PairCtx c) {
  constexpr bool kPacked = kFmt == 1, kBf = kFmt == 2, kWide = kFmt == 3;
  PairCtl* ctl = c.ctl;
  const int ntiles = c.ntiles, bi = c.bi;
  const int lane = threadIdx.x & 31;
  const int ptid = threadIdx.x - kPairKWarp0 * 32;
  const int half = ptid >> 7, g = (ptid >> 5) & 3;
  const int u = lane & 3, r4 = (lane >> 2) & 3, cp = lane >> 4;
  const int line_off = cp * 64 + u * 16;  // this lane's 16 bytes of a line
  const int my_row = 64 * static_cast<int>(c.crank) + 16 * g + (lane & 15);  // key of the tile this lane looks ahead for
  const int32_t* idx_ptr = c.idx_row + c.begin + my_row;
  const int n_mine = c.end - (c.begin + my_row);  // entry j * 128 of idx_ptr is valid iff j * 128 < n_mine
  constexpr int stride_n = kPacked ? 656 : (kBf ? 1024 : 512), stride_s = kPacked ? 656 : 16;
  // (the base pointers are read from the parameter block where they are used: they would otherwise occupy six
  // registers across the whole tile loop)
#define PAIR_KN reinterpret_cast<const uint8_t*>(p.kn)
#define PAIR_ROPE (kPacked ? PAIR_KN + 512 : reinterpret_cast<const uint8_t*>(p.kr))
#define PAIR_SCL (kPacked ? PAIR_KN + 640 : reinterpret_cast<const uint8_t*>(p.kn_scales))
  uint4 d[4][2];   // [m][line]: this lane's 16 bytes of the line of row 4m + r4 (kWide: [2m, 2m + 1][line]: its 32 bytes of row 8m + r8)
  const int part = lane & 1, r8 = 4 * (lane >> 4) + ((lane >> 1) & 3), cpw = (lane >> 3) & 1;  // kWide
  float sc = 0.f;  // scale lane / 16 (of the half's two) of row lane % 16
  auto load_idx = [&](int j) -> int { return (j < ntiles && j * kPT < n_mine) ? ldg_pinned_i32(idx_ptr + j * kPT) : -1; };
  // `phys`: this lane's look-ahead row of the tile
  auto issue_loads = [&](int phys) {
    if (kBf) return;  // (copied from L2 when the buffer is free)
    if constexpr (kWide) {
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int pm = max(__shfl_sync(0xffffffffu, phys, 8 * m + r8), 0);
        const uint8_t* src = PAIR_KN + static_cast<int64_t>(pm) * stride_n + half * 256 + (2 * cpw + part) * 32;
        ldg_pinned_v8(src, d[2 * m][0], d[2 * m + 1][0]);
        ldg_pinned_v8(src + 128, d[2 * m][1], d[2 * m + 1][1]);
      }
    } else {
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int pm = max(__shfl_sync(0xffffffffu, phys, 4 * m + r4), 0);
      const uint8_t* src = PAIR_KN + static_cast<int64_t>(pm) * stride_n + half * 256 + line_off;
      d[m][0] = ldg_pinned_v4(src);
      d[m][1] = ldg_pinned_v4(src + 128);
    }
    }
    sc = 0.f;
    if (phys >= 0) asm volatile("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(sc) : "l"(PAIR_SCL + static_cast<int64_t>(phys) * stride_s + half * 8 + (lane >> 4) * 4));
  };
  auto prefetch_row = [&](int phys) {  // lanes r and r + 16: a line each of the half row; half 0 also the rope part, half 1 the scales
    if (phys < 0) return;
    const int l = lane >> 4;
    if (kBf) {
      const uint8_t* a = PAIR_KN + static_cast<int64_t>(phys) * 1024 + half * 512 + l * 256;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(a + 128));
      if (half == 0 && l == 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(PAIR_ROPE + static_cast<int64_t>(phys) * 128));
    } else if (kPacked) {
      if (half == 0 && lane < 16) bulk_prefetch_l2(PAIR_KN + static_cast<int64_t>(phys) * 656, 656);
    } else {
      asm volatile("prefetch.global.L2 [%0];" ::"l"(PAIR_KN + static_cast<int64_t>(phys) * 512 + half * 256 + l * 128));
      if (l == half) asm volatile("prefetch.global.L2 [%0];" ::"l"(half == 0 ? PAIR_ROPE + static_cast<int64_t>(phys) * 128 : PAIR_SCL + static_cast<int64_t>(phys) * 16));
    }
  };
  const uint32_t k_rows0 = c.base + kSmemT + (4 * half + cp) * kChunk + (16 * g + r4) * 128;  // row r4 of this lane's chunk of line 0
  bool ok = true;
  pair_setup_arrive();
  pdl_wait();          // the selected indices come from the kernel before this one, which may still be running
  int row_cur;         // this lane's row of tile j
  int row_n;           // this lane's row of tile j+1
  int idx_a, entry_a;  // tile j+2
  int idx_b;           // tile j+3
  {
    const int idx0 = load_idx(0), idx1 = load_idx(1);
    idx_a = load_idx(2);
    idx_b = load_idx(3);
    const int e0 = tc_table_entry(p, bi, idx0);
    const int e1 = tc_table_entry(p, bi, idx1);
    entry_a = tc_table_entry(p, bi, idx_a);
    row_cur = tc_row_from_entry(p, idx0, e0);
    issue_loads(row_cur);
    if (kBf) prefetch_row(row_cur);
    row_n = tc_row_from_entry(p, idx1, e1);
    prefetch_row(row_n);
  }
  for (int j = 0; j < ntiles; ++j) {
    const uint32_t b2 = j & 1;
    if (j >= 2) {  // the P.V MMAs that read this half of the buffer are complete
      ok = pair_wait(smem_u32(&ctl->bfree[b2][half]), ((j >> 1) - 1) & 1);
      if (!ok) break;
    }
    const uint32_t k_rows = k_rows0 + b2 * kTileBytes;
    if constexpr (kWide) {
      const uint32_t rows = c.base + kSmemT + b2 * kTileBytes + (4 * half + cpw) * kChunk + (16 * g + r8) * 128;
#pragma unroll
      for (int m = 0; m < 2; ++m) {
#pragma unroll
        for (int l = 0; l < 2; ++l) {
          const float scale = __shfl_sync(0xffffffffu, sc, 16 * l + 8 * m + r8);
          pair_store_wide(rows + 8 * m * 128 + l * 2 * kChunk, part, r8, d[2 * m][l], d[2 * m + 1][l], scale);
        }
      }
    } else {
#pragma unroll
    for (int m = 0; m < 4; ++m) {  // row 4m + r4: swizzle term 4 (m % 2) + r4
      const int x = 4 * (m & 1) + r4;
      const uint32_t a = ((2 * u) ^ x) << 4, b = ((2 * u + 1) ^ x) << 4;
#pragma unroll
      for (int l = 0; l < 2; ++l) {
        const uint32_t row_addr = k_rows + 4 * m * 128 + l * 2 * kChunk;
        if (kBf) {  // the unit's 16 values are 32 bytes of the bf16 row: two copies
          const int pm = __shfl_sync(0xffffffffu, row_cur, 4 * m + r4);
          const uint8_t* src = PAIR_KN + (pm >= 0 ? static_cast<int64_t>(pm) * 1024 + half * 512 + l * 256 + 2 * line_off : 0);
          cp_async_16(row_addr + a, src, pm >= 0 ? 16u : 0u);
          cp_async_16(row_addr + b, src + (pm >= 0 ? 16 : 0), pm >= 0 ? 16u : 0u);
        } else {
          const float scale = __shfl_sync(0xffffffffu, sc, 16 * l + 4 * m + r4);
          const uint4 v = d[m][l];
          sts_v4u(row_addr + a, pair_dequant8(v.x, v.y, scale));
          sts_v4u(row_addr + b, pair_dequant8(v.z, v.w, scale));
        }
      }
    }
    }
    if (kBf) asm volatile("cp.async.wait_all;" ::: "memory");
    fence_proxy_async();
    if (j == 0) pair_setup_wait();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&ctl->kfull[b2][half]));
    // The look-ahead comes before the row loads: what it waits for was requested a tile ago, but a wait behind the row loads
    // is a wait for these too (loads share the few scoreboards of a warp), 1.5-2 k cycles of a tile: 4096 tokens x 2048 rows 3.35 -> 3.19 ms.
    row_cur = row_n;
    row_n = tc_row_from_entry(p, idx_a, entry_a);  // tile j+2: into L2
    prefetch_row(row_n);
    idx_a = idx_b;
    entry_a = tc_table_entry(p, bi, idx_a);  // block-table entries of tile j+3
    idx_b = load_idx(j + 4);
    if (j + 1 < ntiles) issue_loads(row_cur);  // the half rows of tile j+1 (in L2: prefetched a tile ago)
  }
  if (!ok && lane == 0) {
    ctl->abort = 1;
    set_status(p.status, PTO_ST_WAIT_EXPIRED, blockIdx.x, 52);
  }
}

// ================================ V producers ===================================================
// Eight warps; warp v converts this CTA's half of the value columns (256 of the 512 latent bytes: two lines) of the peer's
// rows 8v .. 8v+7, lanes arranged as in the K producers (the other CTA's K producers have fetched or are fetching the same
// lines: L2 hits), and copies the rope parts of the CTA's own rows 8v .. 8v+7 of the next tile. Lane r < 8 walks the look-ahead
// chain of the peer's row 8v + r, lane 8 + r that of its own row 8v + r one tile later (no L2 prefetch: the row's owner issues it).
// What it may overwrite: V goes where q.K^T of the same tile has read K (CTA 1: half 0, early; CTA 0: half 1), the rope part
// where q.K^T has read the tile's own.
template <int kFmt>
__device__ __forceinline__ void pair_role_vproducer(const SfaParams& p, const PairCtx c) {
  constexpr bool kPacked = kFmt == 1, kBf = kFmt == 2, kWide = kFmt == 3;
  PairCtl* ctl = c.ctl;
  const int ntiles = c.ntiles;
  const int lane = threadIdx.x & 31;
  const int v = (threadIdx.x >> 5) - kPairVWarp0;
  const int crank = static_cast<int>(c.crank);
  const int u = lane & 3, r4 = (lane >> 2) & 3, cp = lane >> 4;
  const int line_off = cp * 64 + u * 16;  // this lane's 16 bytes of a line
  const bool for_rope = (lane & 8) != 0;
  const int my_row = 8 * v + (lane & 7) + (for_rope ? 64 * crank + kPT : 64 * (1 - crank));  // key this lane looks ahead for, from tile j's first on
  const int32_t* idx_ptr = c.idx_row + c.begin + my_row;
  const int n_mine = c.end - (c.begin + my_row);
  const int col0 = 256 * crank;  // first latent byte of this CTA's value columns
  constexpr int stride_n = kPacked ? 656 : (kBf ? 1024 : 512), stride_r = kPacked ? 656 : 128, stride_s = kPacked ? 656 : 16;
  uint4 d[2][2];   // [m][line]: this lane's 16 bytes of the line of row 4m + r4 (kWide: [0, 1][line]: its 32 bytes of row r8)
  const int part = lane & 1, r8 = 4 * (lane >> 4) + ((lane >> 1) & 3), cpw = (lane >> 3) & 1;  // kWide
  float sc = 0.f;  // scale lane / 16 (of this CTA's two) of row lane % 8
  auto load_idx = [&](int j) -> int { return (j < ntiles && j * kPT < n_mine) ? ldg_pinned_i32(idx_ptr + j * kPT) : -1; };
  auto issue_loads = [&](int phys) {
    if (kBf) return;
    if constexpr (kWide) {
      const int pm = max(__shfl_sync(0xffffffffu, phys, r8), 0);
      const uint8_t* src = PAIR_KN + static_cast<int64_t>(pm) * stride_n + col0 + (2 * cpw + part) * 32;
      ldg_pinned_v8(src, d[0][0], d[1][0]);
      ldg_pinned_v8(src + 128, d[0][1], d[1][1]);
    } else {
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int pm = max(__shfl_sync(0xffffffffu, phys, 4 * m + r4), 0);
        const uint8_t* src = PAIR_KN + static_cast<int64_t>(pm) * stride_n + col0 + line_off;
        d[m][0] = ldg_pinned_v4(src);
        d[m][1] = ldg_pinned_v4(src + 128);
      }
    }
    const int ps = __shfl_sync(0xffffffffu, phys, lane & 7);
    sc = 0.f;
    if (ps >= 0) asm volatile("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(sc) : "l"(PAIR_SCL + static_cast<int64_t>(ps) * stride_s + (col0 >> 5) + (lane >> 4) * 4));
  };
  auto copy_rope = [&](int phys) {  // rows in lanes 8 .. 15; a padding or rejected row becomes zeros
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int r = 4 * m + (lane >> 3);
      const int pr = __shfl_sync(0xffffffffu, phys, 8 + r);
      cp_async_16(c.base + kSmemRope + (8 * v + r) * 128 + (((lane & 7) ^ r) << 4),
                  PAIR_ROPE + (pr >= 0 ? static_cast<int64_t>(pr) * stride_r + (lane & 7) * 16 : 0), pr >= 0 ? 16u : 0u);
    }
  };
  // row r4 of this warp's 8 in this lane's chunk of line 0; line 1 lies two chunks further
  const uint32_t v_rows0 = c.base + kSmemT + (1 - crank) * kVHalfBytes + cp * kChunk + (8 * v + r4) * 128;
  bool ok = true;
  pair_setup_arrive();
  pdl_wait();
  int row_cur, row_n, idx_a, entry_a, idx_b;  // this lane's row of tiles j, j+1; index and block-table entry of j+2; index of j+3
  {
    const int first = for_rope && n_mine > -kPT ? ldg_pinned_i32(idx_ptr - kPT) : -1;  // rope of tile 0
    const int idx0 = load_idx(0), idx1 = load_idx(1);
    idx_a = load_idx(2);
    idx_b = load_idx(3);
    const int ef = tc_table_entry(p, c.bi, first);
    const int e0 = tc_table_entry(p, c.bi, idx0);
    const int e1 = tc_table_entry(p, c.bi, idx1);
    entry_a = tc_table_entry(p, c.bi, idx_a);
    copy_rope(tc_row_from_entry(p, first, ef));
    row_cur = tc_row_from_entry(p, idx0, e0);
    issue_loads(row_cur);
    row_n = tc_row_from_entry(p, idx1, e1);
    asm volatile("cp.async.wait_all;" ::: "memory");
    fence_proxy_async();
    pair_setup_wait();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&ctl->vfull[0]));
  }
  for (int j = 0; j < ntiles; ++j) {
    const uint32_t b2 = j & 1, ph = (j >> 1) & 1;
    ok = pair_wait(smem_u32(crank == 0 ? &ctl->sfull[b2] : &ctl->kread[b2]), ph);
    if (!ok) break;
    if (crank == 0 && j + 1 < ntiles) copy_rope(row_cur);
    const uint32_t v_rows = v_rows0 + b2 * kTileBytes;
    if constexpr (kWide) {
      const uint32_t rows = c.base + kSmemT + b2 * kTileBytes + (1 - crank) * kVHalfBytes + cpw * kChunk + (8 * v + r8) * 128;
#pragma unroll
      for (int l = 0; l < 2; ++l) {
        const float scale = __shfl_sync(0xffffffffu, sc, 16 * l + r8);
        pair_store_wide(rows + l * 2 * kChunk, part, r8, d[0][l], d[1][l], scale);
      }
    } else {
#pragma unroll
    for (int m = 0; m < 2; ++m) {  // row 4m + r4
      const int x = 4 * m + r4;
      const uint32_t a = ((2 * u) ^ x) << 4, b = ((2 * u + 1) ^ x) << 4;
#pragma unroll
      for (int l = 0; l < 2; ++l) {
        const uint32_t row_addr = v_rows + 4 * m * 128 + l * 2 * kChunk;
        if (kBf) {
          const int pm = __shfl_sync(0xffffffffu, row_cur, 4 * m + r4);
          const uint8_t* src = PAIR_KN + (pm >= 0 ? static_cast<int64_t>(pm) * 1024 + 2 * (col0 + l * 128 + line_off) : 0);
          cp_async_16(row_addr + a, src, pm >= 0 ? 16u : 0u);
          cp_async_16(row_addr + b, src + (pm >= 0 ? 16 : 0), pm >= 0 ? 16u : 0u);
        } else {
          const float scale = __shfl_sync(0xffffffffu, sc, 16 * l + 4 * m + r4);
          const uint4 w = d[m][l];
          sts_v4u(row_addr + a, pair_dequant8(w.x, w.y, scale));
          sts_v4u(row_addr + b, pair_dequant8(w.z, w.w, scale));
        }
      }
    }
    }
    if (crank == 1 && j + 1 < ntiles) {
      ok = pair_wait(smem_u32(&ctl->sfull[b2]), ph);
      if (!ok) break;
      copy_rope(row_cur);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&ctl->vfull[b2 ^ 1]));  // event j + 1
    row_cur = row_n;  // (look-ahead before the row loads, as in the K producers)
    row_n = tc_row_from_entry(p, idx_a, entry_a);
    idx_a = idx_b;
    entry_a = tc_table_entry(p, c.bi, idx_a);
    idx_b = load_idx(j + 4);
    if (j + 1 < ntiles) issue_loads(row_cur);
  }
  if (!ok && lane == 0) {
    ctl->abort = 1;
    set_status(p.status, PTO_ST_WAIT_EXPIRED, blockIdx.x, 53);
  }
}

__global__ void __launch_bounds__(kPairThreads, 1)
sfa_pair_kernel(const __grid_constant__ SfaParams p) {
  extern __shared__ __align__(1024) uint8_t sfa_pair_smem[];
  const uint32_t base = smem_u32(sfa_pair_smem);
  if ((base & 1023u) != 0) {  // the swizzled operand tiles need a 1024-byte aligned base
    if (threadIdx.x == 0) set_status(p.status, PTO_ST_WAIT_EXPIRED, static_cast<int>(base), 55);
    return;
  }
  PairCtx c;
  c.base = base;
  c.ctl = reinterpret_cast<PairCtl*>(sfa_pair_smem + kSmemCtl);
  PairCtl* ctl = c.ctl;
  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  c.crank = pair_ctarank();
  const uint32_t crank = c.crank;
  const int bid = blockIdx.x >> 1;  // cluster index
  c.sp = 0;
  c.pt = -1;
  int ti = bid, n_split = 1;
  if (p.n_split > 1 && bid >= p.split_begin) {
    n_split = p.n_split;
    c.sp = (bid - p.split_begin) % n_split;
    c.pt = (bid - p.split_begin) / n_split;
    ti = p.split_begin + c.pt;
  }
  c.bi = ti / p.s1;
  const int si = ti % p.s1;
  c.q_row0 = static_cast<int64_t>(ti) * p.nq_total + p.head_begin;

  // This CTA's 64 query rows for shared memory, nine swizzled chunks of 64 dims (A operand of q.K^T): 64 x 72 16-byte
  // units, twelve per thread of the twelve warps that are not producers. Requested before the sequence length is there (it
  // takes as long as they do), stored below.
  constexpr int kLoaders = 32 * kPairKWarp0;
  uint4 w[12];
  if (warp < kPairKWarp0) {
    const int64_t row0 = c.q_row0 + 64 * crank;
#pragma unroll
    for (int i = 0; i < 12; ++i) {
      const int e = tid + i * kLoaders;
      const int r = e / 72, u = e % 72;
      w[i] = (u < 64) ? ldg_pinned_v4(reinterpret_cast<const uint8_t*>(p.q_nope + (row0 + r) * 512) + 16 * u)
                      : ldg_pinned_v4(reinterpret_cast<const uint8_t*>(p.q_rope + (row0 + r) * 64) + 16 * (u - 64));
    }
  }

  int n = p.act_seq[c.bi] - p.s1 + 1 + si;
  n = max(0, min(n, p.topk_k));
  const int tiles_total = (n + kPT - 1) / kPT;
  const int tiles_per_split = (tiles_total + n_split - 1) / n_split;
  c.begin = min(n, c.sp * tiles_per_split * kPT);
  c.end = min(n, (c.sp + 1) * tiles_per_split * kPT);
  c.ntiles = (c.end - c.begin + kPT - 1) / kPT;
  c.idx_row = p.topk + static_cast<int64_t>(ti) * p.topk_k;

  if (c.ntiles == 0) {  // same decision in both CTAs of the pair
    if (c.pt < 0) {
      for (int e = tid; e < 64 * 64; e += kPairThreads) {
        const int r = e >> 6, cc = e & 63;
        *reinterpret_cast<uint4*>(p.out + (c.q_row0 + 64 * crank + r) * 512 + cc * 8) = make_uint4(0, 0, 0, 0);
      }
    } else {
      for (int r = tid; r < 64; r += kPairThreads) {
        float* ml = p.part_ml + ((static_cast<int64_t>(c.pt) * p.n_split + c.sp) * p.nq + 64 * crank + r) * 2;
        ml[0] = -INFINITY;
        ml[1] = 0.f;
      }
    }
    return;
  }

  // ---- setup ------------------------------------------------------------------------------------
  if (tid == 0) {
    mbar_init(smem_u32(&ctl->pvdone), 1);
    mbar_init(smem_u32(&ctl->pfull), kPairSoftmaxWarps);
    mbar_init(smem_u32(&ctl->ppeer), 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&ctl->sfull[b]), 1);
      mbar_init(smem_u32(&ctl->sread[b]), kPairSoftmaxWarps);
      mbar_init(smem_u32(&ctl->speer[b]), 1);
      mbar_init(smem_u32(&ctl->kread[b]), 1);
      mbar_init(smem_u32(&ctl->vfull[b]), kPairVWarps);
      mbar_init(smem_u32(&ctl->vpeer[b]), 1);
      for (int h = 0; h < 2; ++h) {
        mbar_init(smem_u32(&ctl->kfull[b][h]), kPairKWarps / 2);
        mbar_init(smem_u32(&ctl->kpeer[b][h]), 1);
        mbar_init(smem_u32(&ctl->bfree[b][h]), 1);
      }
    }
    ctl->abort = 0;
    fence_mbar_init();
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)),
                 "r"(kPairTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  // (the producers go straight to their first rows)
  if (warp < kPairKWarp0) {
#pragma unroll
    for (int i = 0; i < 12; ++i) {
      const int e = tid + i * kLoaders;
      const int r = e / 72, u = e % 72;
      sts_v4u(base + kSmemQ + (u >> 3) * kChunk + r * 128 + (((u & 7) ^ (r & 7)) << 4), w[i]);
    }
    fence_proxy_async();
  }
  static_assert(12 * 32 * kPairKWarp0 == 64 * 72, "Q units per loader thread");

#define PAIR_SETREG(x) asm volatile(x)
  if (warp < kPairSoftmaxWarp0) {
    PAIR_SETREG("setmaxnreg.dec.sync.aligned.u32 24;");
    const bool usual = base == kPairUsualBase;
    if (warp == 0 && crank == 0 && usual) pair_role_issue_qk<kPairUsualBase>(p, c);
    else if (warp == 0 && crank == 0) pair_role_issue_qk<0>(p, c);
    else if (warp == 2 && crank == 0 && usual) pair_role_issue_pv<kPairUsualBase>(p, c);
    else if (warp == 2 && crank == 0) pair_role_issue_pv<0>(p, c);
    else if (warp == 0) pair_role_relay<kRelayK>(p, c);
    else if (warp == 2) pair_role_relay<kRelayV>(p, c);
    else if (warp == 1 && crank == 1) pair_role_relay<kRelayP>(p, c);
    else pair_setup_sync(ctl);
  } else if (warp < kPairKWarp0) {
    PAIR_SETREG("setmaxnreg.inc.sync.aligned.u32 104;");
    pair_role_softmax(p, c);
  } else if (warp < kPairVWarp0) {
    PAIR_SETREG("setmaxnreg.inc.sync.aligned.u32 72;");  // (no change of the count; without it ptxas spills in this role)
    if (p.kn_bf16) pair_role_kproducer<2>(p, c);
    else if (p.packed) pair_role_kproducer<1>(p, c);
    else if (p.kn_wide) pair_role_kproducer<3>(p, c);
    else pair_role_kproducer<0>(p, c);
  } else {
    PAIR_SETREG("setmaxnreg.dec.sync.aligned.u32 64;");
    if (p.kn_bf16) pair_role_vproducer<2>(p, c);
    else if (p.packed) pair_role_vproducer<1>(p, c);
    else if (p.kn_wide) pair_role_vproducer<3>(p, c);
    else pair_role_vproducer<0>(p, c);
  }

  // ---- teardown: neither CTA may leave while the peer's MMAs can still read its shared memory --------
  // (nothing is kept in registers across the roles: what the teardown needs is read again)
  tc_fence_before();
  __syncthreads();
  pair_cluster_sync();
  if ((threadIdx.x >> 5) == 0) {
    tc_fence_after();
    const uint32_t tmem = reinterpret_cast<const PairCtl*>(sfa_pair_smem + kSmemCtl)->tmem_base;
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kPairTmemCols) : "memory");
  }
}

}  // namespace

// Split of the tokens' selected rows over clusters: fewer tokens than SM pairs fill the pairs once; of more tokens, those that are
// left over by whole rounds of pairs share the last round, if they leave half of it or more idle (256 tokens x 2048 rows, three
// rounds and 34 tokens: 318 -> 300 us). Behind many rounds half a round is no gain that could be measured.
constexpr int kPairSplitRounds = 8;
SfaSplit sfa_pair_split(int t, int num_sms) {
  const int pairs = num_sms / 2, rest = t % pairs;
  const int begin = t - rest, n = rest > 0 && begin <= kPairSplitRounds * pairs ? pairs / rest : 1;
  return n >= 2 ? SfaSplit{begin, n < 16 ? n : 16} : SfaSplit{0, 1};
}

// 32-byte row loads, but 16-byte ones in a single round of pairs, in which all of them go through their tiles in step, if the selected rows
// may lie apart (more than two positions for every one selected) and a pair has more than four tiles. Attention alone, tokens x 2048 rows
// in L2, 16 -> 32 bytes, us: 256 217.8 -> 210.6, 1024 879 -> 829, 4096 3314 -> 3130; 64 59.6 -> 62.9. Whole steps, called one by one with inputs
// that are not in L2: of up to 30000 keys 17 tokens 55.4 -> 56.9, 24 66.4 -> 69.3, 31 74.5 -> 81.1, 44 93.1 -> 100.1, 64 110.5 -> 115.8, 74 116.0 ->
// 120.3, but 76 130.5 -> 130.9, 111 184.4 -> 181.5, 148 200.7 -> 194.4, 256 295 -> 289; 5 42.3 -> 41.3, 12 50.4 -> 51.0, 16 51.7 -> 51.8. 64 tokens of 8200
// keys 91.9 -> 97.0, 5000 82.1 -> 84.8, 1200 51.8 -> 50.8, 900 44.9 -> 43.7 (60 tokens); 40 of 8200 82.3 -> 86.1, 5000 74.0 -> 75.0, 4000 72.9 -> 74.1,
// 2500 70.6 -> 70.9, 1700 59.7 -> 58.5, 900 41.0 -> 40.9; 20 of 6500 55.2 -> 57.3, 4000 49.0 -> 48.9, 900 32.7 -> 31.7.
constexpr int kPairWideFew = 16;
bool sfa_pair_wide_loads(int t, int topk, int64_t positions, int num_sms) {
  return t > num_sms / 2 || t <= kPairWideFew || positions <= 2 * static_cast<int64_t>(topk);
}

cudaError_t launch_sfa_pair(const SfaParams& p, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(sfa_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(kPairSmemBytes));
  if (e != cudaSuccess) return e;
  const int t = p.b * p.s1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((static_cast<unsigned>(p.split_begin) + static_cast<unsigned>(t - p.split_begin) * p.n_split) * 2, 1, 1);
  cfg.blockDim = dim3(kPairThreads, 1, 1);
  cfg.dynamicSmemBytes = kPairSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.pdl ? 2 : 1;
  count_launch();
  return cudaLaunchKernelEx(&cfg, sfa_pair_kernel, p);
}

}  // namespace pto
