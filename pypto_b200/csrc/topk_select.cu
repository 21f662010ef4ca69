// Exact per-row top-k over the fp32 score rows of the lightning indexer.
//
// Semantics (reference: examples/models/deepseek_v32_exp/lightning_indexer_quant_impl.py:196-312,
// golden deepseekv32_lightning_indexer_quant.py:244-262): row (b, i) selects over positions
// [0, eff), eff = S_b - (s1 - 1 - i); output is value-descending; when eff < k the first eff entries
// are valid and the rest is -1; eff <= 0 gives all -1. Ties are broken toward the smaller position,
// which makes the result deterministic (torch.topk leaves tie order unspecified).
//
// Every element is mapped to a unique 64-bit key (order-preserving image of the float in the high word, ~position in the
// low word), so "the k largest keys" is well defined.
//   1. Lower bound. A sample of the row (4096 values or more, groups of four spread over it) gives a value that about k +
//      4.5 standard deviations elements exceed. Rows no longer than the list skip this: all of them are the list.
//   2. One scan of the row, which bulk copies bring into shared memory meanwhile, collects the keys at or above the bound
//      into a list of up to 6144 (5120 where two rows share an SM). It is split over a cluster of 1, 2, 4 or 8 CTAs (as many as keep the grid within one
//      wave of SMs), each of which finds the bound for itself; the lists travel to rank 0 through distributed shared
//      memory.
//   3. Rank 0 distributes the list over 2048 bins that divide its value range, a prefix sum over the bins gives every bin
//      its place in the order, and a key's place within its bin is the number of larger keys there (a bin holds a
//      few keys). The first k places are the result; a caller that asked for no order gets the whole bins as they are.
// Where one of either histogram's bins holds too much, the values are distributed once more, by their images (see OrderMap). A
// list that is too long or too short all the same, or a bin of more than 512 keys then (massive ties), sends the row to
// an MSB-first radix select over the 64-bit keys on rank 0.
// What bounds it: one trip of the row from L2 (the first version scanned it three times, for its extremes, a histogram
// and the collection, with a cluster barrier behind each, and ordered its result with a bitonic sort) and about a dozen
// block barriers. Before -> after, alone: one row of 4096 12.4 -> 6.4 us (in order 18.5 -> 7.2), 8 x 32768 in order
// 26.7 -> 11.9, 64 x 65536 16.5 -> 13.9, 256 x 131072 86 -> 43, 1024 x 131072 295 -> 152 us.
// When the score kernel has left a histogram of the row (4096 bins over the top 12 bits of the order-preserving
// image of the float, counted over the positions below the row's causal end), the bound comes from it instead of the sample,
// if its total equals the row's length and the list it leads to is not too long.
#include "common.cuh"

namespace pto {

namespace {

constexpr int kTopkThreads = 512;  // (1024 threads wait longer at each of the dozen barriers than they save between them)
constexpr int kTopkWarps = kTopkThreads / 32;
constexpr int kBins = 2048;
constexpr int kMaxK = 2048;
constexpr int kBinCap = 512;               // keys of a bin that are still ranked by counting

constexpr int kVals = 16;                  // of a chunk per thread
// A chunk of the row is one bulk copy. kMany: two CTAs share an SM, each with a whole row (see launch_li_topk): fewer copies in flight, a
// shorter list, and none besides the row's own. A chunk is read by four of the sixteen warps; the four groups take the chunks in turn,
// each through places of its own. (What a warp spends per chunk besides the comparisons, about 100 instructions and a chain of
// shared-memory round trips, is what the scan costs there; with all warps in each chunk and eight values a thread a row of 131072 took
// 64 k cycles beside another, 2 k per chunk.) A CTA alone on its SM waits for the copies: all warps take each chunk, larger ones and
// fewer (one row to a CTA or cluster, four groups / one, us: 128 x 131072 23.7 / 23.0, 64 x 131072 18.4 / 17.8, 1 x 5000000 95.1 / 91.0).
template <bool kMany>
struct TopkSmem {
  static constexpr int kGroups = kMany ? 4 : 1, kGroupWarps = kTopkWarps / kGroups;
  static constexpr int kChunk = 32 * kGroupWarps * kVals;  // positions
  static constexpr int kPlaces = kMany ? 2 : 3;            // chunks of a group in flight
  static constexpr int kRing = kGroups * kPlaces;          // 64 / 96 KB
  static constexpr int kListCap = kMany ? 5120 : 6144;
  static_assert(kMaxK <= kListCap, "a row of at most k positions is handled as a list");
  union {
    float ring[kRing][kChunk];             // the row on its way through (until the list is complete)
    struct {
      unsigned long long sorted[kMaxK + kBinCap];
      unsigned int base[kBins];            // place of a bin's first key
    };
  };
  unsigned long long list[kListCap];       // rank 0: the candidates of the row
  unsigned long long mine[kMany ? 1 : kListCap];  // the keys this CTA collected, where they have to go elsewhere
  unsigned int hist[!kMany && kLiHistBins > kBins ? kLiHistBins : kBins];
  unsigned int warp_tot[32];
  unsigned int red_min[32], red_max[32];   // order-preserving images
  uint64_t full[kRing];                    // bytes of a chunk landed
  uint64_t empty[kRing];                   // the group's warps have read it
  unsigned int n_mine;                     // keys this CTA collected (more than kListCap: some are missing)
  unsigned int n_list;                     // rank 0: keys in `list` (more than kListCap: some are missing)
  unsigned int offset;                     // of this CTA's keys in the list
  unsigned int hist_total;
  unsigned int n_sel;
  int thr_bin;
  unsigned int thr_above;
  unsigned int thr_count;
};

__device__ __forceinline__ unsigned int cluster_rank() {
  unsigned int r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned int cluster_size() {
  unsigned int r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t peer_addr(const void* local, unsigned int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(local)), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_peer_u64(uint32_t a, unsigned long long v) {
  asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}
__device__ __forceinline__ void st_peer_u32(uint32_t a, unsigned int v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned int atom_peer_add_u32(uint32_t a, unsigned int v) {
  unsigned int old;
  asm volatile("atom.relaxed.cluster.shared::cluster.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(a), "r"(v) : "memory");
  return old;
}

__device__ __forceinline__ unsigned int float_order(float f) { return li_float_order(f); }
__device__ __forceinline__ unsigned long long make_key(float f, int pos) {
  return (static_cast<unsigned long long>(float_order(f)) << 32) | static_cast<unsigned int>(~static_cast<unsigned int>(pos));
}
__device__ __forceinline__ int key_pos(unsigned long long key) {
  return static_cast<int>(~static_cast<unsigned int>(key & 0xffffffffull));
}

__device__ __forceinline__ float order_float(unsigned int o) {  // inverse of float_order
  return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}
__device__ __forceinline__ unsigned int key_order(unsigned long long key) { return static_cast<unsigned int>(key >> 32); }

__device__ __forceinline__ unsigned int at_least(float v, float bound) {  // all ones or none (NaN: none)
  unsigned int r;
  asm("set.ge.u32.f32 %0, %1, %2;" : "=r"(r) : "f"(v), "f"(bound));
  return r;
}

// Descending bitonic sort of n (power of two) keys in shared memory; all threads of the CTA call it.
// Shared-memory version: pair t of a stage is handled by thread t (and t + blockDim, ...), so for strides
// below 64 warp w only touches the 64-key blocks w, w + 32, ...: those stages need a warp barrier only,
// unless the previous stage had a larger stride and other warps wrote into the block.
__device__ void bitonic_sort_desc_smem(unsigned long long* buf, int n) {
  __syncthreads();
  int prev_stride = 64;
  for (int size = 2; size <= n; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      if (stride >= 64 || prev_stride >= 64) __syncthreads(); else __syncwarp();
      prev_stride = stride;
      for (int t = threadIdx.x; t < (n >> 1); t += blockDim.x) {
        const int lo = 2 * t - (t & (stride - 1));  // index with the `stride` bit clear
        const int hi = lo + stride;
        const bool desc = (lo & size) == 0;
        const unsigned long long a = buf[lo], b = buf[hi];
        if ((a < b) == desc) {
          buf[lo] = b;
          buf[hi] = a;
        }
      }
    }
  }
  __syncthreads();
}

// Register version for n <= 2 * blockDim: thread t keeps keys 2t and 2t+1. Stride 1 is a compare inside
// the thread, strides 2..32 exchange with lane (t ^ stride/2) by shuffle (a warp holds 64 consecutive
// keys), and only strides >= 64 (15 of the 66 stages at n = 2048) go through shared memory and a block
// barrier. Lanes beyond n/2 carry zeros and are never paired with a real key (i ^ stride < n).
__device__ void bitonic_sort_desc(unsigned long long* buf, int n) {
  if (n > 2 * static_cast<int>(blockDim.x) || n < 2) {
    bitonic_sort_desc_smem(buf, n);
    return;
  }
  __syncthreads();
  const int t = threadIdx.x;
  const int i0 = 2 * t;
  const bool live = i0 < n;
  unsigned long long e0 = live ? buf[i0] : 0ull, e1 = live ? buf[i0 + 1] : 0ull;
  for (int size = 2; size <= n; size <<= 1) {
    int stride = size >> 1;
    if (stride >= 64) {
      if (live) {
        buf[i0] = e0;
        buf[i0 + 1] = e1;
      }
      for (; stride >= 64; stride >>= 1) {
        __syncthreads();
        if (t < (n >> 1)) {
          const int lo = 2 * t - (t & (stride - 1));
          const int hi = lo + stride;
          const bool desc = (lo & size) == 0;
          const unsigned long long a = buf[lo], b = buf[hi];
          if ((a < b) == desc) {
            buf[lo] = b;
            buf[hi] = a;
          }
        }
      }
      __syncthreads();
      if (live) {
        e0 = buf[i0];
        e1 = buf[i0 + 1];
      }
    }
    const bool desc = (i0 & size) == 0;  // the same for both keys of the thread (size >= 2)
    for (; stride >= 2; stride >>= 1) {
      const unsigned long long o0 = __shfl_xor_sync(0xffffffffu, e0, stride >> 1);
      const unsigned long long o1 = __shfl_xor_sync(0xffffffffu, e1, stride >> 1);
      const bool keep_max = ((i0 & stride) == 0) == desc;
      e0 = keep_max ? (e0 > o0 ? e0 : o0) : (e0 < o0 ? e0 : o0);
      e1 = keep_max ? (e1 > o1 ? e1 : o1) : (e1 < o1 ? e1 : o1);
    }
    {
      const unsigned long long hi = e0 > e1 ? e0 : e1, lo = e0 > e1 ? e1 : e0;
      e0 = desc ? hi : lo;
      e1 = desc ? lo : hi;
    }
  }
  if (live) {
    buf[i0] = e0;
    buf[i0 + 1] = e1;
  }
  __syncthreads();
}

// Finds, scanning the histogram of kPer * kTopkThreads bins from the top bin down, the bin where the running count reaches
// `need`. Results in sm->thr_bin (bin), thr_above (count in bins above it), thr_count (its count), hist_total.
// kBase: every bin's count of the bins above it goes to sm->base.
template <int kPer, bool kBase = false, typename Smem>
__device__ void find_threshold_bin(Smem* sm, unsigned int need) {
  constexpr int kN = kPer * kTopkThreads;
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  // thread t owns bins kN-1-kPer*t down to kN-kPer-kPer*t: a descending walk is a prefix scan over t
  unsigned int c[kPer];
  unsigned int s = 0;
#pragma unroll
  for (int e = 0; e < kPer; ++e) {
    c[e] = sm->hist[kN - 1 - kPer * tid - e];
    s += c[e];
  }
  unsigned int incl = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    unsigned int n = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += n;
  }
  if (lane == 31) sm->warp_tot[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    unsigned int w = lane < kTopkWarps ? sm->warp_tot[lane] : 0u;
    unsigned int wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      unsigned int n = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += n;
    }
    sm->warp_tot[lane] = wi - w;  // exclusive
    if (lane == 31) sm->hist_total = wi;
  }
  __syncthreads();
  unsigned int run = sm->warp_tot[warp] + incl - s;  // count in the bins above this thread's first
#pragma unroll
  for (int e = 0; e < kPer; ++e) {
    if (run < need && need <= run + c[e]) {
      sm->thr_bin = kN - 1 - kPer * tid - e;
      sm->thr_above = run;
      sm->thr_count = c[e];
    }
    if constexpr (kBase) sm->base[kN - 1 - kPer * tid - e] = run;
    run += c[e];
  }
  __syncthreads();
}

// Monotone map of a value range to the bins, equal widths. A range that is not finite, or
// empty: everything in bin 0.
struct BinMap {
  float lo, inv;
  __device__ __forceinline__ void set(float vmin, float vmax) {
    lo = vmin;
    inv = 0.f;
    const float range = vmax - vmin;
    if (range > 0.f && range < INFINITY) inv = static_cast<float>(kBins - 1) / range;
    if (!(inv < INFINITY)) inv = 0.f;
  }
  __device__ __forceinline__ int bin(float v) const { return max(0, min(kBins - 1, static_cast<int>((v - lo) * inv))); }
};

// The same over the order-preserving images: equal widths within a power of two, and as many bins for each power of two of the
// range. A few values far from the others (an outlier, a long tail, masked positions) leave the others spread over many bins,
// where equal widths put all of them into one: 256 rows of 131072 with one value at 300 standard deviations 293 us, all of them
// in the radix select, now 75. What lies outside goes to the ends; images above `top` (NaN) to bin 0.
struct OrderMap {
  unsigned int lo, top;
  float scale;
  __device__ __forceinline__ void set(unsigned int omin, unsigned int omax) {
    lo = omin;
    top = 0xffffffffu;
    scale = omax > omin ? __fdividef(static_cast<float>(kBins - 1), static_cast<float>(omax - omin)) : 0.f;
  }
  __device__ __forceinline__ int bin(unsigned int o) const {
    const int b = min(kBins - 1, static_cast<int>(__uint2float_rz(o > lo ? o - lo : 0u) * scale));
    return o > top ? 0 : b;
  }
};

// block-wide minimum and maximum of order-preserving images, returned to every thread (one barrier)
template <typename Smem>
__device__ __forceinline__ void block_range(Smem* sm, unsigned int& omin, unsigned int& omax) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned int lo = __reduce_min_sync(0xffffffffu, omin), hi = __reduce_max_sync(0xffffffffu, omax);
  if (lane == 0) {
    sm->red_min[warp] = lo;
    sm->red_max[warp] = hi;
  }
  __syncthreads();
  omin = __reduce_min_sync(0xffffffffu, sm->red_min[lane & (kTopkWarps - 1)]);
  omax = __reduce_max_sync(0xffffffffu, sm->red_max[lane & (kTopkWarps - 1)]);
}

// The sample of a row: groups of four, evenly spread, `per` of them for every thread.
__device__ __forceinline__ float4 sample_group(const float* row, int eff, int per, int u) {
  const int g = static_cast<int>(static_cast<long long>(threadIdx.x + u * kTopkThreads) * (eff >> 2) / (static_cast<long long>(kTopkThreads) * per));
  return __ldg(reinterpret_cast<const float4*>(row) + g);
}
// How many samples are to lie above the bound: about k + 4.5 standard deviations elements of the row exceed it. At most `most` of
// them let expect a list of three quarters of its capacity.
template <typename Smem>
__device__ __forceinline__ unsigned int sample_need(int eff, int k, int per, float* most) {
  const float samples = static_cast<float>(4 * kTopkThreads) * static_cast<float>(per);
  const float mean = static_cast<float>(k) * samples / static_cast<float>(eff);
  *most = 0.75f * static_cast<float>(Smem::kListCap) * samples / static_cast<float>(eff);
  return static_cast<unsigned int>(mean + 4.5f * sqrtf(mean) + 4.0f);
}

// The bound where the first histogram does not give it: the bin that holds the threshold over again, by the images of its values
// [zlo, zhi], until it is fine enough. zlo > zhi: all of the row. The sample is read again for every pass.
template <typename Smem>
__device__ __noinline__ float sample_bound_fine(Smem* sm, const float* row, int eff, int k, int per, unsigned int zlo, unsigned int zhi) {
  float most;
  const unsigned int need = sample_need<Smem>(eff, k, per, &most);
  auto each = [&](auto&& f) {
    for (int u = 0; u < per; ++u) {
      const float4 v = sample_group(row, eff, per, u);
      f(v.x);
      f(v.y);
      f(v.z);
      f(v.w);
    }
  };
  if (zlo > zhi) {
    float vmin = INFINITY, vmax = -INFINITY;
    each([&](float x) {
      vmin = fminf(vmin, x);
      vmax = fmaxf(vmax, x);
    });
    zlo = float_order(vmin);
    zhi = float_order(vmax);
    block_range(sm, zlo, zhi);
  }
  for (int pass = 0; pass < 3 && zhi > zlo; ++pass) {
    OrderMap zoom;
    zoom.set(zlo, zhi);
    for (int j = threadIdx.x; j < kBins; j += kTopkThreads) sm->hist[j] = 0;
    __syncthreads();
    each([&](float x) { atomicAdd(&sm->hist[zoom.bin(float_order(x))], 1u); });
    __syncthreads();
    find_threshold_bin<kBins / kTopkThreads>(sm, need);
    const unsigned int b = static_cast<unsigned int>(sm->thr_bin);
    zlo = zoom.lo + __float2uint_rz(__fdividef(static_cast<float>(b), zoom.scale));
    if (b + 1 < static_cast<unsigned int>(kBins)) zhi = min(zhi, zoom.lo + __float2uint_ru(__fdividef(static_cast<float>(b + 1), zoom.scale)));
    if (static_cast<float>(sm->thr_above + sm->thr_count) <= most) return order_float(zlo);
  }
  return -INFINITY;
}

// Lower bound of the k largest of row[0, eff) from a sample: 1024 groups of four, or a multiple of that: long rows need a larger
// sample for a list of the same length (beyond 2^20 positions one that meets 32 or more of 2048 selected ones, which is enough for a
// list of 6144; rows as long as that do not come here with the list of 5120). -inf: no useful bound.
template <typename Smem>
__device__ float sample_bound(Smem* sm, const float* row, int eff, int k) {
  const int tid = threadIdx.x;
  if (eff > (1 << 20)) return sample_bound_fine(sm, row, eff, k, (eff + (1 << 17) - 1) >> 17, 1u, 0u);
  constexpr int kMaxPer = 4096 / kTopkThreads;
  const int per = (eff <= (1 << 16) ? 1024 : (eff <= (1 << 18) ? 2048 : 4096)) / kTopkThreads;
  float4 v[kMaxPer];
  float vmin = INFINITY, vmax = -INFINITY;
#pragma unroll
  for (int u = 0; u < kMaxPer; ++u) {
    if (u < per) v[u] = sample_group(row, eff, per, u);
  }
#pragma unroll
  for (int u = 0; u < kMaxPer; ++u) {
    if (u < per) {
      vmin = fminf(vmin, fminf(fminf(v[u].x, v[u].y), fminf(v[u].z, v[u].w)));
      vmax = fmaxf(vmax, fmaxf(fmaxf(v[u].x, v[u].y), fmaxf(v[u].z, v[u].w)));
    }
  }
  for (int j = tid; j < kBins; j += kTopkThreads) sm->hist[j] = 0;
  unsigned int olo = float_order(vmin), ohi = float_order(vmax);
  block_range(sm, olo, ohi);
  BinMap map;
  map.set(order_float(olo), order_float(ohi));
#pragma unroll
  for (int u = 0; u < kMaxPer; ++u) {
    if (u < per) {
      atomicAdd(&sm->hist[map.bin(v[u].x)], 1u);
      atomicAdd(&sm->hist[map.bin(v[u].y)], 1u);
      atomicAdd(&sm->hist[map.bin(v[u].z)], 1u);
      atomicAdd(&sm->hist[map.bin(v[u].w)], 1u);
    }
  }
  __syncthreads();
  float most;
  const unsigned int need = sample_need<Smem>(eff, k, per, &most);
  find_threshold_bin<kBins / kTopkThreads>(sm, need);
  const int b = sm->thr_bin;
  const float bound = map.lo + static_cast<float>(b) / map.inv;
  if (map.inv != 0.f) {
    if (static_cast<float>(sm->thr_above + sm->thr_count) <= most) return bound;
    olo = float_order(bound);
    if (b + 1 < kBins) ohi = float_order(map.lo + static_cast<float>(b + 1) / map.inv);
  }
  return sample_bound_fine(sm, row, eff, k, per, olo, ohi);
}

// Applies f(value, position) to every element of row[0, eff). Sixteen values are requested before the first body runs, so the
// latency of one batch is paid once (the bodies contain shared-memory atomics the compiler will not move loads across). A row is
// a multiple of four long in memory.
template <typename F>
__device__ __forceinline__ void for_each_element(const float* row, int eff, F&& f) {
  constexpr int kStep = 4 * kTopkThreads;
  for (int j0 = 4 * threadIdx.x; j0 < eff; j0 += 4 * kStep) {
    float4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (j0 + u * kStep < eff) v[u] = __ldg(reinterpret_cast<const float4*>(row + j0 + u * kStep));
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float x[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int pos = j0 + u * kStep + e;
        if (pos < eff) f(x[e], pos);
      }
    }
  }
}

template <bool kMany>
__global__ void __launch_bounds__(kTopkThreads, kMany ? 2 : 1)
li_topk_kernel(TopkParams p) {
  using Smem = TopkSmem<kMany>;
  constexpr int kRing = Smem::kRing, kPlaces = Smem::kPlaces, kListCap = Smem::kListCap;
  constexpr int kGroups = Smem::kGroups, kGroupWarps = Smem::kGroupWarps, kChunk = Smem::kChunk;
  extern __shared__ __align__(16) uint8_t topk_smem_raw[];
  Smem* sm = reinterpret_cast<Smem*>(topk_smem_raw);
  // with programmatic serialization the score kernel before it may still be running
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const unsigned int csize = kMany ? 1u : cluster_size();
  const unsigned int rank = kMany ? 0u : cluster_rank();
  const int row_id = blockIdx.x / csize;
  const int bi = row_id / p.s1;
  const int i = row_id % p.s1;
  int32_t* out = p.out + static_cast<int64_t>(row_id) * p.k;
  const float* row = p.scores + static_cast<int64_t>(row_id) * p.row_stride;
  // the row's length is an input of the call, not a result of the score kernel: its trip to memory runs while
  // this grid still waits for that kernel
  int eff = p.act_seq[bi] - (p.s1 - 1 - i);
  if (eff > p.row_stride) eff = static_cast<int>(p.row_stride);
  const int k = min(p.k, eff);  // entries of the result
  if (tid < kRing) {  // (a thread each: one that set them all took a thousand cycles)
    mbar_init(smem_u32(&sm->full[tid]), 1);
    mbar_init(smem_u32(&sm->empty[tid]), kGroupWarps);
    fence_mbar_init();
    fence_proxy_async();
  }
  __syncwarp();
  if (tid == 0) {
    sm->n_mine = 0;
    sm->n_list = 0;
    sm->n_sel = 0;
    sm->thr_bin = 0;
  }
  const bool whole = eff <= kListCap;         // the list is the row: rank 0 alone, no cluster barrier on this path
  if (!whole && csize > 1) cluster_arrive();  // (rank 0's counter is set before anyone adds to it)
  pdl_wait();
  pdl_trigger();
  if (rank == 0) {
    for (int j = max(k, 0) + tid; j < p.k; j += kTopkThreads) out[j] = -1;
  }
  if (eff <= 0 || (whole && rank != 0)) return;
  if (eff <= p.k && (p.flags & PTO_LI_UNSORTED) != 0) {  // everything is selected and the order is free
    for (int j = tid; j < eff; j += kTopkThreads) out[j] = j;  // (k <= kListCap: `whole`, so this is rank 0)
    return;
  }

  unsigned int omin = 0xffffffffu, omax = 0u;  // range of the list, as order-preserving images
  float bound = -INFINITY;                     // no smaller value is among the k largest, if the list has k keys or more
  unsigned int n_list, n_front = kListCap;  // the first n_front keys at the front, the others from the end backwards
  auto key_at = [&](unsigned int j) { return sm->list[j < n_front ? j : kListCap - 1 - (j - n_front)]; };
  if (whole) {
    __syncthreads();
#pragma unroll
    for (int u = 0; u < (kListCap / 4 + kTopkThreads - 1) / kTopkThreads; ++u) {
      const int j = 4 * (tid + u * kTopkThreads);
      if (j < eff) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(row + j));  // (rows are a multiple of 4 long)
        const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (j + e < eff) {
            sm->list[j + e] = make_key(x[e], j + e);
            if (x[e] == x[e] || eff <= p.k) {  // (see OrderMap's use below: NaN)
              omin = min(omin, float_order(x[e]));
              omax = max(omax, float_order(x[e]));
            }
          }
        }
      }
    }
    n_list = static_cast<unsigned int>(eff);
  } else {
    // this rank's share of the row: the first chunks are on their way while the bound is found
    const int share = (((eff + static_cast<int>(csize) - 1) / static_cast<int>(csize)) + 3) & ~3;
    const int begin = min(eff, static_cast<int>(rank) * share);
    const int end = min(eff, begin + share);
    const int chunks = (end - begin + kChunk - 1) / kChunk;
    auto fetch = [&](int c) {  // one thread
      const uint32_t bytes = static_cast<uint32_t>((min(kChunk, end - begin - c * kChunk) + 3) & ~3) * 4u;
      const int place = (c % kGroups) * kPlaces + (c / kGroups) % kPlaces;
      const uint32_t bar = smem_u32(&sm->full[place]);
      mbar_arrive_expect_tx(bar, bytes);
      bulk_load_1d(smem_u32(sm->ring[place]), row + begin + c * kChunk, bytes, bar);
    };
    if (tid == 0) {
      for (int c = 0; c < min(chunks, kRing); ++c) fetch(c);
    }
    // ---- 1. lower bound -------------------------------------------------------------------------
    bool known = false;
    if (!kMany && p.hist != nullptr) {
      const uint4* h4 = reinterpret_cast<const uint4*>(p.hist + static_cast<int64_t>(row_id) * kLiHistBins);
      for (int j = tid; j < kLiHistBins / 4; j += kTopkThreads) reinterpret_cast<uint4*>(sm->hist)[j] = __ldg(h4 + j);
      __syncthreads();
      find_threshold_bin<kLiHistBins / kTopkThreads>(sm, static_cast<unsigned int>(k));
      known = sm->hist_total == static_cast<unsigned int>(eff) && sm->thr_above + sm->thr_count <= static_cast<unsigned int>(kListCap);
      bound = order_float(static_cast<unsigned int>(sm->thr_bin) << kLiHistShift);
      __syncthreads();  // every thread has read the outcome before the histogram area is reused
    }
    if (!known) bound = sample_bound(sm, row, eff, k);
    // ---- 2. this rank's keys at or above the bound ------------------------------------------------
    // One list for the CTA, in which a warp reserves its places chunk by chunk: however the selected positions lie in the row,
    // nothing but their number limits it. (With a list of its own for each warp, 384 places, a run of 385 neighbouring
    // selected positions could fill one, and sent the row to the radix select: 64 rows of 65536 whose last 2048 positions are
    // selected 62 -> 27 us, scattered selections 26 either way.) It is the row's list at once where this rank's
    // keys are the first in that: where it is the only rank, and rank 0 of two.
    unsigned long long* const mine = rank == 0 && csize <= 2 ? sm->list : sm->mine;
    bool ok = true;
    const int member = warp % kGroupWarps;
    for (int c = warp / kGroupWarps, visit = 0; c < chunks; c += kGroups, ++visit) {
      // the group's chunk before this one: when its warps have read it, its place is refilled
      if (member == 0 && lane == 0 && visit > 0 && c + (kPlaces - 1) * kGroups < chunks) {
        const int place = (c % kGroups) * kPlaces + (visit - 1) % kPlaces;
        if (mbar_wait_spin(smem_u32(&sm->empty[place]), ((visit - 1) / kPlaces) & 1)) fetch(c + (kPlaces - 1) * kGroups);
      }
      __syncwarp();
      const int place = (c % kGroups) * kPlaces + visit % kPlaces;
      ok = mbar_wait_warp(smem_u32(&sm->full[place]), (visit / kPlaces) & 1) && ok;
      const float* chunk = sm->ring[place];
      const int p0 = begin + c * kChunk;
      // Few elements pass. Sixteen comparisons a thread give a mask; its count behind the counts of the lanes below is the
      // thread's place in the warp's part of the list (a ballot per element needs two population counts each, which run at an
      // eighth of the rate); the few set bits are walked and their values read again. A warp takes neighbouring positions.
      auto offset = [&](int e) { return member * 32 * kVals + (e >> 2) * 128 + lane * 4 + (e & 3); };
      unsigned int mask = 0u;
#pragma unroll
      for (int u = 0; u < kVals / 4; ++u) {
        const float4 v = *reinterpret_cast<const float4*>(chunk + offset(4 * u));
        if constexpr (kMany) {
          mask |= (at_least(v.x, bound) & (1u << (4 * u))) | (at_least(v.y, bound) & (2u << (4 * u)));
          mask |= (at_least(v.z, bound) & (4u << (4 * u))) | (at_least(v.w, bound) & (8u << (4 * u)));
        } else {  // (the masks of the other form, us: 1 x 5000000 91.0 -> 91.9, 200 x 2^20 222.7 -> 225.6)
          mask |= (v.x >= bound ? 1u << (4 * u) : 0u) | (v.y >= bound ? 2u << (4 * u) : 0u) | (v.z >= bound ? 4u << (4 * u) : 0u) |
                  (v.w >= bound ? 8u << (4 * u) : 0u);
        }
      }
      if (p0 + kChunk > end) {  // the last chunk: what lies behind the end is not part of the row
#pragma unroll
        for (int e = 0; e < kVals; ++e) {
          if (p0 + offset(e) >= end) mask &= ~(1u << e);
        }
      }
      const unsigned int cnt = __popc(mask);
      const unsigned int n = __reduce_add_sync(0xffffffffu, cnt);
      if (n != 0u) {  // (uniform)
        unsigned int at = 0;
        if (lane == 0) at = atomicAdd(&sm->n_mine, n);
        unsigned int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const unsigned int up = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += up;
        }
        at = __shfl_sync(0xffffffffu, at, 0);
        if (at + n <= static_cast<unsigned int>(kListCap)) {  // (else the list is spoilt, its length says so below)
          at += incl - cnt;
          while (mask != 0u) {
            const int e = 31 - __clz(mask);
            mask ^= 1u << e;
            const int off = offset(e);
            mine[at++] = make_key(chunk[off], p0 + off);
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sm->empty[place]));
    }
    if (!ok && lane == 0) {
      set_status(p.status, PTO_ST_WAIT_EXPIRED, row_id, 30);
      atomicAdd(&sm->n_mine, static_cast<unsigned int>(kListCap + 1));
    }
    __syncthreads();
    // ---- the lists of all ranks, one behind the other, into rank 0's --------------------------------
    const unsigned int total = min(sm->n_mine, static_cast<unsigned int>(kListCap + 1));  // (what is spoilt stays spoilt)
    if (csize == 2) {
      // two ranks: rank 0's keys from the front of the list, rank 1's from its end, with their number: nobody waits for a count
      cluster_wait();
      if (rank == 1) {
        if (total <= static_cast<unsigned int>(kListCap)) {
          for (unsigned int j = tid; j < total; j += kTopkThreads) st_peer_u64(peer_addr(&sm->list[kListCap - 1 - j], 0), sm->mine[j]);
        }
        if (tid == 0) st_peer_u32(peer_addr(&sm->n_list, 0), total);
      }
      cluster_arrive();
      cluster_wait();
      if (rank != 0) return;
      n_front = total;
      n_list = total + sm->n_list;  // (where the two would overlap the list is too long and not read)
    } else if (csize > 1) {
      cluster_wait();
      if (tid == 0) sm->offset = atom_peer_add_u32(peer_addr(&sm->n_list, 0), total);
      __syncthreads();
      const unsigned int off = sm->offset;
      if (total <= static_cast<unsigned int>(kListCap)) {
        for (unsigned int j = tid; j < total; j += kTopkThreads) {
          if (off + j < static_cast<unsigned int>(kListCap)) st_peer_u64(peer_addr(&sm->list[off + j], 0), sm->mine[j]);
        }
      }
      cluster_arrive();
      cluster_wait();
      if (rank != 0) return;
      n_list = sm->n_list;
    } else {
      n_list = total;
    }
    if (n_list <= static_cast<unsigned int>(kListCap)) {
      for (unsigned int j = tid; j < n_list; j += kTopkThreads) {
        const unsigned int o = key_order(key_at(j));
        omin = min(omin, o);
        omax = max(omax, o);
      }
    }
  }

  // ---- 3. order ------------------------------------------------------------------------------------
  const bool good = n_list <= static_cast<unsigned int>(kListCap) && n_list >= static_cast<unsigned int>(k);  // (uniform)
  if (good) {
    for (int j = tid; j < kBins; j += kTopkThreads) sm->hist[j] = 0;
    block_range(sm, omin, omax);
    auto order = [&](auto&& bin, unsigned int cap) {  // true: the result is written. cap: keys of a bin that are ranked by counting
      constexpr int kPer = kListCap / kTopkThreads;
      unsigned int where[kPer];  // bin, and which of its keys
#pragma unroll
      for (int u = 0; u < kPer; ++u) {
        const unsigned int j = tid + u * kTopkThreads;
        if (j < n_list) {
          const unsigned int b = bin(key_at(j));
          where[u] = (b << 16) | atomicAdd(&sm->hist[b], 1u);
        }
      }
      __syncthreads();
      find_threshold_bin<kBins / kTopkThreads, true>(sm, static_cast<unsigned int>(k));
      // Bins that lie in the result whole need no order when the caller asked for none: only the keys of the others go to their
      // bin's place in `sorted`, to be ranked there.
      const bool unsorted = (p.flags & PTO_LI_UNSORTED) != 0;
      const unsigned int uk = static_cast<unsigned int>(k);
      bool crowded = false;
      unsigned int chosen[kPer], n_chosen = 0;  // per run of 32 keys of the list: which go out as they are (unordered)
#pragma unroll
      for (int u = 0; u < kPer; ++u) {
        const unsigned int j = tid + u * kTopkThreads;
        bool go = false;
        if (j < n_list) {
          const unsigned int b = where[u] >> 16, first = sm->base[b], slot = where[u] & 0xffffu;
          if (first < uk) {
            if (unsorted && first + sm->hist[b] <= uk) go = true;
            else if (slot < cap) sm->sorted[first + slot] = key_at(j);
            else crowded = true;
          }
        }
        chosen[u] = __ballot_sync(0xffffffffu, go);
        n_chosen += __popc(chosen[u]);
      }
      if (unsorted) {
        // In runs as they lie in the list, i.e. of neighbouring positions: the attention kernel gathers the selected rows in this
        // order, and in the order of the bins (a random walk over the cache) its gathers cost 64 sequences 3 us more than the
        // selection had gained.
        unsigned int at = 0;
        if (lane == 0) at = atomicAdd(&sm->n_sel, n_chosen);
        at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
          if ((chosen[u] >> lane) & 1u) out[at + __popc(chosen[u] & ((1u << lane) - 1u))] = key_pos(key_at(tid + u * kTopkThreads));
          at += __popc(chosen[u]);
        }
      }
      if (__syncthreads_or(crowded ? 1 : 0) != 0) return false;
      // keys of the bins that reach into the result; without order, of the one bin that lies across its end
      const unsigned int n_sorted = sm->thr_above + sm->thr_count;
      if (!(unsorted && n_sorted == uk)) {
        for (unsigned int j = (unsorted ? sm->thr_above : 0u) + tid; j < n_sorted; j += kTopkThreads) {
          const unsigned long long key = sm->sorted[j];
          const unsigned int b = bin(key);
          const unsigned int first = sm->base[b], last = first + sm->hist[b];
          unsigned int at = first;
          for (unsigned int x = first; x < last; ++x) at += sm->sorted[x] > key ? 1u : 0u;
          if (at < uk) out[at] = key_pos(key);
        }
      }
      return true;
    };
    BinMap even;
    even.set(order_float(omin), order_float(omax));
    // Equal widths first: the images give the values near zero many bins and the others few, and their conversion costs more (64 x
    // 65536 in a whole step 139.1 us, with the images at once 141.3).
    if (even.inv != 0.f) {
      if (order([&](unsigned long long key) { return static_cast<unsigned int>(even.bin(order_float(key_order(key)))); }, kBinCap / 4)) return;
      for (int j = tid; j < kBins; j += kTopkThreads) sm->hist[j] = 0;
      if (tid == 0) sm->n_sel = 0;
      __syncthreads();
    }
    OrderMap map;
    map.set(omin, omax);
    if (eff > p.k) map.top = 0xff800000u;  // (NaN is not selected before numbers, but in a row that is selected whole it comes first)
    if (order([&](unsigned long long key) { return static_cast<unsigned int>(map.bin(key_order(key))); }, kBinCap)) return;
  }

  // ---- 3'. MSB-first radix select on the 64-bit keys of the whole row (rank 0) ----------------------------
  if (tid == 0) {
    sm->n_sel = 0;
    if (p.status != nullptr) atomicAdd(p.status + PTO_STATUS_RADIX_ROWS, 1);
  }
  // (of a list that is too long, i.e. of many equal values, at least the bound is good: what lies below it needs no counting)
  const float floor = n_list >= static_cast<unsigned int>(k) ? bound : -INFINITY;
  // digits: 11/11/10 bits of the value word, then 11/11/10 bits of the inverted position.
  // invariant: keys with (key >> shift) > prefix are selected; `remaining` more are needed among those with
  // (key >> shift) == prefix.
  __syncthreads();
  unsigned long long prefix = 0ull;
  int shift = 64;
  unsigned int remaining = static_cast<unsigned int>(k);
  const int widths[6] = {11, 11, 10, 11, 11, 10};
  bool exact = false;
  for (int pass = 0; pass < 6 && !exact; ++pass) {
    const int w = widths[pass];
    const int new_shift = shift - w;
    for (int j = tid; j < kBins; j += kTopkThreads) sm->hist[j] = 0;
    __syncthreads();
    for_each_element(row, eff, [&](float v, int pos) {
      if (v < floor) return;
      const unsigned long long key = make_key(v, pos);
      if (shift < 64 && (key >> shift) != prefix) return;
      atomicAdd(&sm->hist[static_cast<unsigned int>(key >> new_shift) & ((1u << w) - 1u)], 1u);
    });
    __syncthreads();
    find_threshold_bin<kBins / kTopkThreads>(sm, remaining);
    remaining -= sm->thr_above;
    exact = (sm->thr_count == remaining);
    prefix = (prefix << w) | static_cast<unsigned long long>(sm->thr_bin);
    shift = new_shift;
    __syncthreads();
  }
  for_each_element(row, eff, [&](float v, int pos) {
    if (v < floor) return;
    const unsigned long long key = make_key(v, pos);
    if ((key >> shift) >= prefix) {
      const unsigned int slot = atomicAdd(&sm->n_sel, 1u);
      if (slot < static_cast<unsigned int>(kMaxK)) sm->sorted[slot] = key;
    }
  });
  __syncthreads();
  int kpow2 = 2;
  while (kpow2 < k) kpow2 <<= 1;
  for (int j = k + tid; j < kpow2; j += kTopkThreads) sm->sorted[j] = 0ull;
  bitonic_sort_desc(sm->sorted, kpow2);
  for (int j = tid; j < k; j += kTopkThreads) out[j] = key_pos(sm->sorted[j]);
}

}  // namespace

cudaError_t launch_li_topk(const TopkParams& p, int num_sms, cudaStream_t stream, bool pdl) {
  // as many CTAs per row as keep the grid within one wave, each with 8192 positions or more to scan (a row
  // that fits the list is one CTA's work)
  const int rows = p.b * p.s1;
  int csize = 1;
  while (csize < 8 && rows * csize * 2 <= num_sms && p.row_stride > static_cast<int64_t>(csize) * 8192) csize *= 2;
  // More rows than SMs: two to an SM, so that one streams while the other finds its bound or orders its list (behind their score
  // kernel, with the scan by groups of warps: 4096 rows of 131072 990 -> 780 us, 256 rows 88 -> 78; 4096 rows of 4096, which are lists,
  // 106 -> 79, 1000 rows of 3000 42 -> 27). Not where only the longer list of a CTA alone takes whole rows, and not rows so long that
  // the sample's bound leaves the shorter list no room: what it collects, about 2048 (1 + 4.5 / sqrt(m) + 4 / m) keys where the sample
  // meets m of 2048 selected ones, is 4.4 standard deviations below 5120 at m = 51, i.e. 655360 positions, and from 960 thousand on too
  // many to be expected at all, so that such rows went to the radix select (200 rows, us, one to an SM / two: 600000 positions 153 / 132,
  // 983040 226 / 481, 2^20 223 / 1286; two with twice the sample 326, 342).
  constexpr int64_t kManyMaxRow = 5 << 17;
  const bool many = rows > num_sms && p.hist == nullptr && p.row_stride <= kManyMaxRow &&
                    (p.row_stride <= TopkSmem<true>::kListCap || p.row_stride > TopkSmem<false>::kListCap);
  auto kernel = many ? li_topk_kernel<true> : li_topk_kernel<false>;
  static_assert(sizeof(TopkSmem<true>) <= 113 * 1024, "two CTAs to an SM");
  const size_t smem = many ? sizeof(TopkSmem<true>) : sizeof(TopkSmem<false>);
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(rows * csize), 1, 1);
  cfg.blockDim = dim3(kTopkThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(csize);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  // behind the score kernel of the same call: may be scheduled while that drains, and reads only the row's length, which is no
  // result of it, before it waits. Behind a kernel of somebody else's, which may have written the lengths: the ordinary way
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 2 : 1;
  count_launch();
  return cudaLaunchKernelEx(&cfg, kernel, p);
}

int topk_max_k() { return kMaxK; }

}  // namespace pto
