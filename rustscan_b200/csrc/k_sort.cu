// k_sort.cu — segmented LSD radix sort of (u32 key, u32 value) pairs and
// decoupled-look-back scans.
//
// The reference sorts with a bitonic network (radix_sort.wgsl, 2 +
// log2(P)(log2(P)+1)/2 launches of P = next_pow2(n) threads) and scans with
// Hillis-Steele steps (prefix_sum.wgsl, 1 + log2(n) launches). Here:
//  - one histogram pass over the keys computes the digit counts of every
//    radix pass at once;
//  - each radix pass is one persistent launch: blocks take 4096-key
//    partitions by ticket, rank keys stably inside the block (the peer lanes
//    of a digit from a word per digit that they set their bit in; warps in
//    order), publish per-digit counts and look back across partitions for
//    their global offsets, then scatter through shared memory so that every
//    digit's run is written contiguously. A block whose segment has no
//    partition left takes those of the other segments;
//  - scans are single-pass with the same look-back.
// Keys are u32; `bits` (from bit shift0) set the passes: ceil(bits / 8)
// passes of equal digits of at most 8 bits (12 bits: two 6-bit passes, whose
// 64 digit runs per partition are written in longer stretches than 256). Stability (ties in input order) is what the reference's index
// tie-break provides (radix_sort.wgsl:21-26). Without values, the keys are
// sorted alone (the binning packs tile id and compact index into one key
// when both fit in 32 bits).
#include <algorithm>
#include <atomic>

#include <cooperative_groups.h>

#include "gsr_kernels.h"

namespace gsr {

namespace {

constexpr int kSortThreads = 256;
constexpr int kSortItems = 16;
constexpr int kSortTile = kSortThreads * kSortItems;  // 4096
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kWarpKeys = kSortItems * 32;  // 512 keys per warp
constexpr uint64_t kSortManyParts = 2048;

__device__ __forceinline__ uint32_t seg_count(const uint32_t* counts, uint32_t stride, uint32_t seg, uint32_t n_host,
                                              uint64_t cap) {
  if (!counts) return n_host;
  const uint64_t c = counts[(size_t)seg * stride];
  return (uint32_t)(c < cap ? c : cap);
}

__global__ void __launch_bounds__(256) sort_hist_kernel(const uint32_t* keys, uint64_t seg_stride,
                                                        const uint32_t* counts, uint32_t count_stride,
                                                        uint32_t n_host, uint64_t cap, int passes, uint32_t shift0,
                                                        uint32_t dbits, uint32_t* hist) {
  __shared__ uint32_t h[4][256];
  for (int i = threadIdx.x; i < 4 * 256; i += blockDim.x) (&h[0][0])[i] = 0;
  __syncthreads();
  const uint32_t seg = blockIdx.y;
  const uint32_t n = seg_count(counts, count_stride, seg, n_host, cap);
  const uint32_t* k = keys + (size_t)seg * seg_stride;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t key = k[i];
    for (int p = 0; p < passes; ++p) atomicAdd(&h[p][(key >> (shift0 + dbits * p)) & ((1u << dbits) - 1u)], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * 256; i += blockDim.x) {
    const uint32_t c = (&h[0][0])[i];
    if (c) atomicAdd(hist + (size_t)seg * 1024 + i, c);
  }
}

__global__ void __launch_bounds__(256) sort_hist_scan_kernel(const uint32_t* hist, uint32_t* base) {
  __shared__ uint32_t s_scan[32];
  const uint32_t p = blockIdx.x, seg = blockIdx.y;
  const size_t o = (size_t)seg * 1024 + p * 256 + threadIdx.x;
  uint32_t tot;
  base[o] = block_exclusive_scan(hist[o], s_scan, &tot);
}

struct SortPassArgs {
  const uint32_t* keys_in;
  const uint32_t* vals_in;  // null: values are the input positions
  uint32_t* keys_out;
  uint32_t* vals_out;
  uint64_t seg_stride;
  const uint32_t* counts;
  uint32_t count_stride;
  uint32_t n_host;
  uint64_t cap;
  uint32_t shift;
  uint32_t dmask;  // digit mask: (1 << digit bits) - 1, at most 255
  uint32_t pass;
  const uint32_t* base;  // [seg][4][256]
  uint32_t drop;         // 1: keys equal to 0xffffffff take digit dmask + 1 and are not written (dmask < 255)
  unsigned long long* states;
  uint32_t parts_cap;
  LookbackCtl* ctl;
  DevStatus* status;
};

// KV: values travel with the keys; otherwise the keys are sorted alone. What
// bounds it is the latency of the ranking's rounds and, in the first
// partitions, of the look-back. Ranking by a shared-memory word per digit
// (about 12 ALU instructions a round, where a ballot per digit bit takes 40 and
// match_any slows with the distinct digits) took the tile sort of 8 views of
// 1M Gaussians from 0.986 to 0.754 ms and their depth sort from 0.302 to
// 0.285; blocks that help other segments then took the tile sort to 0.628 and
// the depth sort to 0.249, and the tile sort of 16 uneven views of 2M from 5.50
// to 2.52 ms.
// RES: blocks resident per SM (the register bound).
template <bool KV, int RES>
__global__ void __launch_bounds__(kSortThreads, RES) sort_pass_kernel(SortPassArgs a) {
  __shared__ uint32_t s_keys[kSortTile];
  __shared__ uint32_t s_vals[KV ? kSortTile : 1];
  __shared__ uint32_t s_whist[kSortWarps][256];
  __shared__ uint32_t s_dstart[256];
  __shared__ uint32_t s_gbase[256];
  __shared__ uint32_t s_scan[32];
  __shared__ uint32_t s_ticket;
  __shared__ uint32_t s_dropped;
  const uint32_t epoch = epoch_begin(a.ctl);
  const unsigned long long tag = (unsigned long long)(epoch & 0x3fffffffu) << 34;
  const uint32_t kDropDigit = a.dmask + 1u;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt_mask = (1u << lane) - 1u;
  // A block starts on its own segment and helps the others when that one has
  // no partition left: segments are of uneven length.
  for (uint32_t turn = 0; turn < gridDim.y; ++turn) {
    const uint32_t seg = blockIdx.y + turn < gridDim.y ? blockIdx.y + turn : blockIdx.y + turn - gridDim.y;
    const uint32_t n = seg_count(a.counts, a.count_stride, seg, a.n_host, a.cap);
    const uint32_t* kin = a.keys_in + (size_t)seg * a.seg_stride;
    const uint32_t* vin = a.vals_in ? a.vals_in + (size_t)seg * a.seg_stride : nullptr;
    uint32_t* kout = a.keys_out + (size_t)seg * a.seg_stride;
    uint32_t* vout = a.vals_out + (size_t)seg * a.seg_stride;
    unsigned long long* states = a.states + (size_t)seg * a.parts_cap * 256;
    const uint32_t* gbase = a.base + (size_t)seg * 1024 + a.pass * 256;
    for (;;) {
      const uint32_t part = next_ticket(a.ctl, seg, &s_ticket);
      if ((uint64_t)part * kSortTile >= n) break;
      const uint32_t tile0 = part * kSortTile;
      uint32_t key[kSortItems];
#pragma unroll
      for (int i = 0; i < kSortItems; ++i) {
        const uint32_t idx = tile0 + warp * kWarpKeys + i * 32 + lane;
        key[i] = idx < n ? kin[idx] : 0xffffffffu;
      }
      uint32_t* peer = s_keys + warp * 256;  // per digit, the lanes of a round that hold it
      for (int j = lane; j < 256; j += 32) s_whist[warp][j] = peer[j] = 0;
      __syncwarp();
      // Stable rank within the warp: rounds in order, lanes in order.
      uint32_t lrank[kSortItems / 2];  // two 16-bit ranks a word
#pragma unroll
      for (int i = 0; i < kSortItems; ++i) {
        const bool ok = tile0 + warp * kWarpKeys + i * 32 + lane < n;
        const uint32_t d = (a.drop && key[i] == 0xffffffffu) ? kDropDigit : (key[i] >> a.shift) & a.dmask;
        if (ok) atomicOr(peer + d, 1u << lane);
        __syncwarp();
        uint32_t peers = 0, b = 0;
        if (ok) {
          peers = peer[d];
          b = s_whist[warp][d];
        }
        const uint32_t below = peers & lt_mask;
        __syncwarp();
        if (ok && below == 0) {
          s_whist[warp][d] = b + __popc(peers);
          peer[d] = 0;
        }
        __syncwarp();
        const uint32_t r = b + __popc(below);
        if (i & 1)
          lrank[i / 2] |= r << 16;
        else
          lrank[i / 2] = r;
      }
      uint32_t val[KV ? kSortItems : 1];  // loaded late: the ranking needs the registers
      if (KV) {
#pragma unroll
        for (int i = 0; i < kSortItems; ++i) {
          const uint32_t idx = tile0 + warp * kWarpKeys + i * 32 + lane;
          val[i] = idx < n ? (vin ? vin[idx] : idx) : 0u;
        }
      }
      __syncthreads();
      // Per digit (one per thread): warp offsets and the block count.
      const uint32_t d = threadIdx.x;
      uint32_t sum = 0;
#pragma unroll
      for (int w = 0; w < kSortWarps; ++w) {
        const uint32_t t = s_whist[w][d];
        s_whist[w][d] = sum;
        sum += t;
      }
      // The digit counts are published before the block scan, so that later
      // partitions can sum past this one as early as possible; only the
      // pass's digits look back.
      if (d <= a.dmask) st_volatile64(states + (size_t)part * 256 + d, tag | (part == 0 ? kFlagPre : kFlagAgg) | sum);
      uint32_t tot;
      const uint32_t dstart = block_exclusive_scan(sum, s_scan, &tot);
      const uint32_t excl = d <= a.dmask ? lookback(states + d, 256, part, sum, epoch, a.status, kWaitSort) : 0u;
      s_dstart[d] = dstart;
      s_gbase[d] = gbase[d] + excl - dstart;
      // The dropped keys are placed last in the block and never written (one
      // thread sets the count: the drop digit's, or thread 0 when nothing drops).
      if (d == (a.drop ? kDropDigit : 0u)) s_dropped = a.drop ? sum : 0u;
      // This partition writes digit d's keys to gbase[d] + excl onwards; a
      // position past the segment would mean the digit histogram did not
      // describe these keys. Such a partition writes nothing and is reported
      // through the status words.
      const bool outside = d <= a.dmask && sum != 0u && s_gbase[d] + dstart + sum > n;  // each term is below 2^30
      if (__syncthreads_or(outside)) {
        if (threadIdx.x == 0) atomicOr(&a.status->internal, 1u);
        continue;
      }
#pragma unroll
      for (int i = 0; i < kSortItems; ++i) {
        const uint32_t idx = tile0 + warp * kWarpKeys + i * 32 + lane;
        if (idx < n) {
          const uint32_t dd = (a.drop && key[i] == 0xffffffffu) ? kDropDigit : (key[i] >> a.shift) & a.dmask;
          const uint32_t pos = s_dstart[dd] + s_whist[warp][dd] + ((lrank[i / 2] >> (16 * (i & 1))) & 0xffffu);
          s_keys[pos] = key[i];
          if (KV) s_vals[pos] = val[KV ? i : 0];
        }
      }
      __syncthreads();
      const uint32_t nvalid = min((uint32_t)kSortTile, n - tile0) - s_dropped;
      for (uint32_t j = threadIdx.x; j < nvalid; j += kSortThreads) {
        const uint32_t k = s_keys[j];
        const uint32_t dst = s_gbase[(k >> a.shift) & a.dmask] + j;
        kout[dst] = k;
        if (KV) vout[dst] = s_vals[j];
      }
    }
  }
  epoch_end(a.ctl, epoch);
}

// ---------------------------------------------------------------------------
// Decoupled look-back scan: 2048 elements per partition, thread-striped
// rounds. in[gather[i]] when gather is set. Exclusive or inclusive output.
// Per segment totals: totals[seg * tstride + 0] = min(total, cap_total),
// totals[seg * tstride + 1] = total; overflow is flagged when total exceeds
// cap_total.
// ---------------------------------------------------------------------------
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

struct ScanArgs {
  const uint32_t* in;
  const uint32_t* gather;
  uint32_t* out;
  uint64_t seg_stride;
  const uint32_t* counts;
  uint32_t count_stride;
  uint32_t n_host;
  uint64_t cap;
  int inclusive;
  uint32_t* totals;
  uint32_t totals_stride;
  uint64_t cap_total;
  unsigned long long* states;
  uint32_t parts_cap;
  LookbackCtl* ctl;
  DevStatus* status;
  uint32_t seg_base;  // segment of blockIdx.y == 0
};

__global__ void __launch_bounds__(kScanThreads) scan_kernel(ScanArgs a) {
  __shared__ uint32_t s_scan[32];
  __shared__ uint32_t s_ticket, s_excl;
  const uint32_t epoch = epoch_begin(a.ctl);
  const uint32_t seg = a.seg_base + blockIdx.y;
  const uint32_t n = seg_count(a.counts, a.count_stride, seg, a.n_host, a.cap);
  const uint32_t* in = a.in + (size_t)seg * a.seg_stride;
  const uint32_t* ga = a.gather ? a.gather + (size_t)seg * a.seg_stride : nullptr;
  uint32_t* out = a.out + (size_t)seg * a.seg_stride;
  unsigned long long* states = a.states + (size_t)seg * a.parts_cap;
  const uint32_t nparts = (n + kScanTile - 1) / kScanTile;
  if (n == 0 && a.totals && blockIdx.x == 0 && threadIdx.x == 0) {
    a.totals[(size_t)seg * a.totals_stride + 0] = 0;
    a.totals[(size_t)seg * a.totals_stride + 1] = 0;
  }
  for (;;) {
    const uint32_t part = next_ticket(a.ctl, seg, &s_ticket);
    if (part >= nparts) break;
    const uint32_t tile0 = part * kScanTile;
    uint32_t v[kScanItems];
    uint32_t local = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
      const uint32_t idx = tile0 + i * kScanThreads + threadIdx.x;
      v[i] = (idx < n) ? (ga ? in[ga[idx]] : in[idx]) : 0u;
    }
    // Rounds in order; within a round threads in order.
    uint32_t round_base[kScanItems];
    uint32_t carry = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
      uint32_t tot;
      const uint32_t e = block_exclusive_scan(v[i], s_scan, &tot);
      round_base[i] = carry + e;
      carry += tot;
    }
    local = carry;
    if (threadIdx.x == 0) s_excl = lookback(states, 1, part, local, epoch, a.status, kWaitScan);
    __syncthreads();
    const uint32_t excl = s_excl;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
      const uint32_t idx = tile0 + i * kScanThreads + threadIdx.x;
      if (idx < n) out[idx] = excl + round_base[i] + (a.inclusive ? v[i] : 0u);
    }
    if (part == nparts - 1 && threadIdx.x == 0 && a.totals) {
      const uint64_t total = (uint64_t)excl + local;
      a.totals[(size_t)seg * a.totals_stride + 0] = (uint32_t)(total < a.cap_total ? total : a.cap_total);
      a.totals[(size_t)seg * a.totals_stride + 1] = (uint32_t)total;
      if (total > a.cap_total) {
        atomicExch(&a.status->overflow, 1u);
        atomicMax(&a.status->required, (unsigned long long)total);
      }
    }
  }
  epoch_end(a.ctl, epoch);
}

// ---------------------------------------------------------------------------
// Depth order and intersection offsets of a small view in one launch: a
// cluster of 16 CTAs per view holds the view's (key, index) pairs in its
// shared memory, a chunk of consecutive positions per CTA, and runs every
// radix pass and the offset scan there. Per pass each warp ranks its pairs
// stably (as sort_pass_kernel does), the CTAs send their digit counts to one
// another, and every pair is stored straight to its place in the CTA that
// owns it. Two cluster barriers per pass take the place of a launch and a
// look-back (another, that every CTA has started, hides behind the key loads). What bounds it is latency: about 2000 cycles per barrier, and per
// 1024 pairs of a CTA 1300 to send them (single 8-byte stores) besides the
// ranking.
// ---------------------------------------------------------------------------
constexpr int kClusterThreads = 1024;
constexpr int kClusterWarps = kClusterThreads / 32;
constexpr int kClusterDigits = 512;  // of at most 9 bits
// Up to 13 pairs per thread of 16 CTAs, and for more than 4 views (the GPU
// holds about so many of these clusters at a time) few enough pairs that the
// later waves stay cheap. Depth order and offsets by the radix passes and by the
// cluster, in us, all Gaussians visible: one view of 20k 73 and 28, of 60k 81 and
// 40, of 120k 91 and 58, of 160k 93 and 73, of 213k 103 and 87; 4 views of 60k 95
// and 40, of 213k 115 and 87; 8 views of 60k 116 and 69, of 100k 120 and 97, of 140k
// 125 and 126 (of 200k, past the line, 156 and 157); 16 views of 60k 139 and 101.
constexpr uint32_t kClusterMaxKeys = 16u * kClusterThreads * 13u;
constexpr uint64_t kClusterMaxWaveKeys = 300000;

struct ClusterSortArgs {
  const uint32_t* key;    // [V] depth bits (31 of them order)
  const uint32_t* count;  // [V] intersections per compact index
  uint32_t* perm;         // [V] compact index per depth rank
  uint32_t* offset;       // [V] exclusive scan of count[perm]
  uint64_t stride;        // elements per view
  uint32_t* vcount;       // [view][4]: visible, intersections (clamped), intersections required, pad
  uint64_t cap_total;
  DevStatus* status;
};

template <int C, int IT> struct ClusterSortSmem {
  union {
    uint2 pair[IT * kClusterThreads];
    uint32_t peer[kClusterWarps][kClusterDigits];  // ranking, when the pairs are in registers
  };
  uint16_t whist[kClusterWarps][kClusterDigits];  // per warp: digit counts, then starts
  uint32_t counts[C][kClusterDigits];             // every CTA's digit counts of the pass
  uint32_t base[kClusterDigits];
  uint32_t scan[32];
  uint32_t red[2][32];
  uint2 range[C];                                 // every CTA's smallest and largest key
  uint32_t totals[C];
};

// C CTAs per cluster, at most IT pairs per thread.
template <int C, int IT>
__global__ void __launch_bounds__(kClusterThreads, 1) cluster_sort_kernel(ClusterSortArgs a) {
  namespace cg = cooperative_groups;
  extern __shared__ uint4 smem_cs[];
  ClusterSortSmem<C, IT>& S = *reinterpret_cast<ClusterSortSmem<C, IT>*>(smem_cs);
  cg::cluster_group cluster = cg::this_cluster();
  cluster.barrier_arrive();  // this CTA has started; the loads below hide the wait for the others
  const uint32_t rank = cluster.block_rank(), v = blockIdx.y;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t V = a.vcount[v * 4 + 0];
  // Pairs per thread (uniform over the cluster) and per CTA; the division of
  // a position by the chunk is exact for positions below 2^19.
  const uint32_t it = max((V + C * kClusterThreads - 1) / (C * kClusterThreads), 1u);
  const uint32_t chunk = it * kClusterThreads;
  const uint32_t magic = (65536u + it - 1u) / it;
  const uint32_t first = rank * chunk;
  const uint32_t mine = V > first ? min(V - first, chunk) : 0u;
  const uint32_t* key = a.key + a.stride * v;
  uint2 kv[IT];
  const uint32_t at0 = warp * 32u * it + lane;  // this thread's pairs: at0 + 32 i
  uint32_t lo = 0xffffffffu, hi = 0u;
#pragma unroll
  for (int i = 0; i < IT; ++i) {
    const uint32_t j = at0 + 32u * i;
    if ((uint32_t)i < it && j < mine) {
      kv[i] = make_uint2(key[first + j] & 0x7fffffffu, first + j);
      lo = min(lo, kv[i].x);
      hi = max(hi, kv[i].x);
    }
  }
  // The keys' range over the view: their distances from the smallest order
  // them as well and take fewer bits (27 hold depths of a ratio of 65536, in
  // three passes of 9).
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if (lane == 0) {
    S.red[0][warp] = lo;
    S.red[1][warp] = hi;
  }
  __syncthreads();
  lo = __reduce_min_sync(0xffffffffu, S.red[0][lane]);
  hi = __reduce_max_sync(0xffffffffu, S.red[1][lane]);
  cluster.barrier_wait();  // every CTA has started: its shared memory may be written
  if (tid < (uint32_t)C) *cluster.map_shared_rank(&S.range[rank], tid) = make_uint2(lo, hi);
  cluster.sync();
#pragma unroll
  for (int c = 0; c < C; ++c) {
    lo = min(lo, S.range[c].x);
    hi = max(hi, S.range[c].y);
  }
  const uint32_t bits = hi > lo ? 32u - (uint32_t)__clz(hi - lo) : 1u;
  const uint32_t passes = bits <= 27u ? 3u : 4u;
  const uint32_t dbits = (bits + passes - 1u) / passes;
  const uint32_t digits = 1u << dbits, dmask = digits - 1u;
#pragma unroll
  for (int i = 0; i < IT; ++i) kv[i].x -= lo;
  for (uint32_t shift = 0; shift < bits; shift += dbits) {
    uint32_t* peer = S.peer[warp];  // per digit, the lanes of a round that hold it
    for (uint32_t d = lane; d < digits; d += 32u) {
      S.whist[warp][d] = 0;
      peer[d] = 0;
    }
    __syncwarp();
    // Stable rank within the warp: rounds in order, lanes in order.
    uint32_t ranks[(IT + 1) / 2];  // two 16-bit ranks a word
#pragma unroll
    for (int i = 0; i < IT; ++i) {
      uint32_t r = 0;
      if ((uint32_t)i < it) {
        const bool ok = at0 + 32u * i < mine;
        const uint32_t d = (kv[i].x >> shift) & dmask;
        if (ok) atomicOr(peer + d, 1u << lane);
        __syncwarp();
        uint32_t peers = 0, b = 0;
        if (ok) {
          peers = peer[d];
          b = S.whist[warp][d];
        }
        const uint32_t below = peers & ((1u << lane) - 1u);
        __syncwarp();
        if (ok && below == 0) {
          S.whist[warp][d] = (uint16_t)(b + __popc(peers));
          peer[d] = 0;
        }
        __syncwarp();
        r = b + __popc(below);
      }
      if (i & 1)
        ranks[i / 2] |= r << 16;
      else
        ranks[i / 2] = r;
    }
    __syncthreads();
    // One thread per digit: warp starts, and the CTA's count to every CTA.
    uint32_t sum = 0;
    if (tid < digits) {
#pragma unroll 16
      for (int w = 0; w < kClusterWarps; ++w) {
        const uint32_t t = S.whist[w][tid];
        S.whist[w][tid] = (uint16_t)sum;
        sum += t;
      }
#pragma unroll
      for (int c = 0; c < C; ++c) *cluster.map_shared_rank(&S.counts[rank][tid], c) = sum;
    }
    cluster.sync();  // the counts have arrived, and every CTA's pairs are in registers
    uint32_t total = 0, before = 0;
    if (tid < digits) {
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const uint32_t t = S.counts[c][tid];
        before += (uint32_t)c < rank ? t : 0u;
        total += t;
      }
    }
    uint32_t all;
    const uint32_t start = block_exclusive_scan(total, S.scan, &all);
    if (tid < digits) S.base[tid] = start + before;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < IT; ++i) {
      if ((uint32_t)i < it && at0 + 32u * i < mine) {
        const uint32_t d = (kv[i].x >> shift) & dmask;
        const uint32_t pos = S.base[d] + S.whist[warp][d] + ((ranks[i / 2] >> (16 * (i & 1))) & 0xffffu);
        const uint32_t to = ((pos >> 10) * magic) >> 16;
        *cluster.map_shared_rank(&S.pair[pos - to * chunk], to) = kv[i];
      }
    }
    cluster.sync();  // the pairs have arrived
#pragma unroll
    for (int i = 0; i < IT; ++i) {
      const uint32_t j = at0 + 32u * i;
      if ((uint32_t)i < it && j < mine) kv[i] = S.pair[j];
    }
    __syncthreads();  // the next pass ranks in the pairs' memory
  }
  // Depth order out, and the exclusive scan of the counts along it: a warp's
  // pairs are consecutive, rounds in order.
  const uint32_t* count = a.count + a.stride * v;
  uint32_t* perm = a.perm + a.stride * v;
  uint32_t* offset = a.offset + a.stride * v;
#pragma unroll
  for (int i = 0; i < IT; ++i) {
    const uint32_t j = at0 + 32u * i;
    const bool ok = (uint32_t)i < it && j < mine;
    if (ok) perm[first + j] = kv[i].y;
    kv[i].x = ok ? count[kv[i].y] : 0u;
  }
  uint32_t run = 0;
#pragma unroll
  for (int i = 0; i < IT; ++i) {
    if ((uint32_t)i < it) {
      uint32_t x = kv[i].x;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
      }
      kv[i].x = run + x - kv[i].x;  // before this pair, within the warp
      run += __shfl_sync(0xffffffffu, x, 31);
    }
  }
  uint32_t all;
  const uint32_t incl = block_exclusive_scan(lane == 31u ? run : 0u, S.scan, &all);
  const uint32_t wstart = __shfl_sync(0xffffffffu, incl, 0);  // the warps before this one
  if (tid < (uint32_t)C) *cluster.map_shared_rank(&S.totals[rank], tid) = all;
  cluster.sync();  // also the last access to another CTA's memory
  uint64_t total = 0;
  uint32_t before = 0;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    if ((uint32_t)c < rank) before += S.totals[c];
    total += S.totals[c];
  }
#pragma unroll
  for (int i = 0; i < IT; ++i) {
    const uint32_t j = at0 + 32u * i;
    if ((uint32_t)i < it && j < mine) offset[first + j] = before + wstart + kv[i].x;
  }
  if (rank == 0 && tid == 0) {
    a.vcount[v * 4 + 1] = (uint32_t)(total < a.cap_total ? total : a.cap_total);
    a.vcount[v * 4 + 2] = (uint32_t)total;
    if (total > a.cap_total) {
      atomicExch(&a.status->overflow, 1u);
      atomicMax(&a.status->required, (unsigned long long)total);
    }
  }
}

// Launches the kernel or, with only_query, asks whether the device can hold
// such a cluster.
template <int C, int IT>
cudaError_t cluster_sort_launch(const ClusterSortArgs& a, uint32_t views, cudaStream_t st, bool only_query) {
  constexpr int bytes = (int)sizeof(ClusterSortSmem<C, IT>);
  auto* kernel = cluster_sort_kernel<C, IT>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && C > 8) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = C;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(C, views);
  cfg.blockDim = dim3(kClusterThreads);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (only_query) {
    int n = 0;
    e = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg);
    return e != cudaSuccess ? e : (n > 0 ? cudaSuccess : cudaErrorInvalidConfiguration);
  }
  return cudaLaunchKernelEx(&cfg, kernel, a);
}
cudaError_t cluster_sort_pick(uint32_t n, const ClusterSortArgs& a, uint32_t views, cudaStream_t st, bool only_query) {
  const uint32_t k = (n + kClusterThreads - 1) / kClusterThreads;
  if (k <= 16 * 2) return cluster_sort_launch<16, 2>(a, views, st, only_query);
  if (k <= 16 * 5) return cluster_sort_launch<16, 5>(a, views, st, only_query);
  if (k <= 16 * 8) return cluster_sort_launch<16, 8>(a, views, st, only_query);
  return cluster_sort_launch<16, 13>(a, views, st, only_query);
}

int persistent_blocks(int num_sms, uint32_t segments, int per_sm) {
  const int total = num_sms * per_sm;
  const int per = total / (int)(segments ? segments : 1);
  return per < 1 ? 1 : per;
}

}  // namespace

cudaError_t radix_sort_pairs(const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out, uint32_t* vals_out,
                             uint32_t* keys_tmp, uint32_t* vals_tmp, uint64_t seg_stride, uint32_t segments,
                             const uint32_t* counts, uint32_t count_stride, uint32_t n_host, uint64_t cap_per_segment,
                             int bits, const Scratch& s, cudaStream_t st, bool hist_ready, uint32_t shift0,
                             const uint32_t* counts_dropped, int first_bits) {
  if (segments == 0 || segments > (uint32_t)kMaxSegments) return cudaErrorInvalidValue;
  if (shift0 >= 32 || (keys_in == nullptr)) return cudaErrorInvalidValue;
  const bool kv = vals_out != nullptr;
  const int passes = sort_passes(bits);
  // Digit widths: uniform, or (with histograms from the caller and two
  // passes) first_bits for the first pass and the rest for the second.
  const bool split = first_bits > 0 && hist_ready && passes == 2 && first_bits < bits && bits - first_bits <= 8;
  const int dbits = split ? first_bits : sort_digit_bits(bits);
  auto pass_bits = [&](int p) { return split ? (p == 0 ? first_bits : bits - first_bits) : dbits; };
  // Dropping the all-ones keys in the first pass needs a spare digit value.
  const bool drop = counts_dropped != nullptr;
  if (drop && (dbits >= 8 || !hist_ready)) return cudaErrorInvalidValue;
  const uint32_t parts_cap = (uint32_t)((cap_per_segment + kSortTile - 1) / kSortTile);
  if ((uint64_t)parts_cap * 256 * segments > s.lb_states_words) return cudaErrorInvalidValue;
  if (!hist_ready) {
    cudaError_t e = cudaMemsetAsync(s.hist, 0, sizeof(uint32_t) * 1024 * segments, st);
    if (e != cudaSuccess) return e;
    dim3 grid(persistent_blocks(s.num_sms, segments, 4), segments);
    sort_hist_kernel<<<grid, 256, 0, st>>>(keys_in, seg_stride, counts, count_stride, n_host, cap_per_segment, passes,
                                           shift0, (uint32_t)dbits, s.hist);
  }
  sort_hist_scan_kernel<<<dim3(passes, segments), 256, 0, st>>>(s.hist, s.hist_base);
  // Ping-pong so that the last pass writes keys_out/vals_out.
  const uint32_t* ki = keys_in;
  const uint32_t* vi = vals_in;
  for (int p = 0; p < passes; ++p) {
    const bool to_out = ((passes - 1 - p) % 2) == 0;
    uint32_t* ko = to_out ? keys_out : keys_tmp;
    uint32_t* vo = to_out ? vals_out : vals_tmp;
    SortPassArgs a;
    a.keys_in = ki;
    a.vals_in = vi;
    a.keys_out = ko;
    a.vals_out = vo;
    a.seg_stride = seg_stride;
    a.counts = (drop && p > 0) ? counts_dropped : counts;
    a.count_stride = count_stride;
    a.drop = (drop && p == 0) ? 1u : 0u;
    a.n_host = n_host;
    a.cap = cap_per_segment;
    a.shift = shift0 + dbits * p;  // a split's second pass starts after the first's bits
    a.dmask = (1u << pass_bits(p)) - 1u;
    a.pass = p;
    a.base = s.hist_base;
    a.states = s.lb_states;
    a.parts_cap = parts_cap;
    a.ctl = s.ctl;
    a.status = s.status;
    // Three blocks of the pair kernel per SM spill a little; it pays once there
    // are partitions enough to fill them several times (16 uneven views of 2M
    // Gaussians: tile sort 2.78 -> 2.52 ms, depth sort 0.93 -> 0.90) and costs
    // where few partitions wait for one another (one view of 345k keys 82 -> 97
    // us). The keys-only kernel runs 4.
    const int res = !kv ? 4 : (uint64_t)parts_cap * segments > kSortManyParts ? 3 : 2;
    dim3 grid(persistent_blocks(s.num_sms, segments, res), segments);
    if (res == 4)
      sort_pass_kernel<false, 4><<<grid, kSortThreads, 0, st>>>(a);
    else if (res == 3)
      sort_pass_kernel<true, 3><<<grid, kSortThreads, 0, st>>>(a);
    else
      sort_pass_kernel<true, 2><<<grid, kSortThreads, 0, st>>>(a);
    ki = ko;
    vi = vo;
  }
  return cudaGetLastError();
}

cudaError_t inclusive_scan_u32(const uint32_t* in, uint32_t* out, uint32_t n_host, const Scratch& s,
                               cudaStream_t st) {
  if (n_host == 0) return cudaSuccess;
  ScanArgs a{};
  a.in = in;
  a.gather = nullptr;
  a.out = out;
  a.seg_stride = 0;
  a.counts = nullptr;
  a.n_host = n_host;
  a.cap = n_host;
  a.inclusive = 1;
  a.totals = nullptr;
  a.parts_cap = (n_host + kScanTile - 1) / kScanTile;
  if (a.parts_cap > s.lb_states_words) return cudaErrorInvalidValue;
  a.states = s.lb_states;
  a.ctl = s.ctl;
  a.status = s.status;
  scan_kernel<<<dim3(persistent_blocks(s.num_sms, 1, 4), 1), kScanThreads, 0, st>>>(a);
  return cudaGetLastError();
}

cudaError_t inclusive_scan_u32_scratch(const uint32_t* in, uint32_t* out, uint32_t n_host, unsigned long long* states,
                                       uint64_t states_words, LookbackCtl* ctl, DevStatus* status, int num_sms,
                                       cudaStream_t st) {
  if (n_host == 0) return cudaSuccess;
  ScanArgs a{};
  a.in = in;
  a.gather = nullptr;
  a.out = out;
  a.seg_stride = 0;
  a.counts = nullptr;
  a.n_host = n_host;
  a.cap = n_host;
  a.inclusive = 1;
  a.totals = nullptr;
  a.parts_cap = (n_host + kScanTile - 1) / kScanTile;
  if (a.parts_cap > states_words) return cudaErrorInvalidValue;
  a.states = states;
  a.ctl = ctl;
  a.status = status;
  scan_kernel<<<dim3(persistent_blocks(num_sms, 1, 4), 1), kScanThreads, 0, st>>>(a);
  return cudaGetLastError();
}

bool cluster_sort_available(int device) {
  // A property of the device (0: not asked yet, 1: yes, 2: no), asked once per
  // process: the occupancy query can take milliseconds.
  static std::atomic<int> known[64];
  const bool listed = device >= 0 && device < 64;
  if (listed && known[device].load() != 0) return known[device].load() == 1;
  bool ok = true;
  for (uint32_t it : {2u, 5u, 8u, 13u})
    ok = ok && cluster_sort_pick(it * 16u * kClusterThreads, ClusterSortArgs{}, 1, nullptr, true) == cudaSuccess;
  (void)cudaGetLastError();
  if (listed) known[device].store(ok ? 1 : 2);
  return ok;
}

bool order_fits_cluster(uint32_t n, uint32_t views, const Scratch& s) {
  return s.cluster_sort && n <= kClusterMaxKeys && (uint64_t)n * ((views + 3) / 4) <= kClusterMaxWaveKeys;
}

cudaError_t launch_order_offsets(const ViewSet& vs, uint32_t n, FwdBufs& b, const Scratch& s, cudaStream_t st) {
  ClusterSortArgs a{};
  a.key = b.depth_key;
  a.count = b.count;
  a.perm = b.perm;
  a.offset = b.offset;
  a.stride = b.Vcap;
  a.vcount = b.vcount;
  a.cap_total = b.Icap;
  a.status = s.status;
  return cluster_sort_pick(n, a, vs.n_views, st, false);
}

cudaError_t launch_offsets(const ViewSet& vs, FwdBufs& b, const Scratch& s, cudaStream_t st) {
  ScanArgs a{};
  a.in = b.count;
  a.gather = b.perm;
  a.out = b.offset;
  a.seg_stride = b.Vcap;
  a.counts = b.vcount;
  a.count_stride = 4;
  a.cap = b.Vcap;
  a.inclusive = 0;
  a.totals = b.vcount + 1;
  a.totals_stride = 4;
  a.cap_total = b.Icap;
  a.parts_cap = (uint32_t)((b.Vcap + kScanTile - 1) / kScanTile);
  if ((uint64_t)a.parts_cap * vs.n_views > s.lb_states_words) return cudaErrorInvalidValue;
  a.states = s.lb_states;
  a.ctl = s.ctl;
  a.status = s.status;
  // The scan gathers the counts through the depth order, one 4-byte read
  // per random index. Views are scanned in groups whose count arrays fit in
  // about a third of L2 together, so each 32-byte sector is fetched from
  // DRAM once rather than once per element read from it.
  constexpr uint64_t kGatherBytes = 40ull << 20;
  const uint32_t per = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(vs.n_views, kGatherBytes / (4 * b.Vcap)));
  for (uint32_t v0 = 0; v0 < vs.n_views; v0 += per) {
    const uint32_t nv = std::min(per, vs.n_views - v0);
    a.seg_base = v0;
    scan_kernel<<<dim3(persistent_blocks(s.num_sms, nv, 4), nv), kScanThreads, 0, st>>>(a);
  }
  return cudaGetLastError();
}

}  // namespace gsr

// ---------------------------------------------------------------------------
// Self-test of the bounded wait: one thread plays partition 1 of a look-back
// whose partition 0 never publishes (its state word carries another epoch),
// so the wait must give up after max_polls polls, flag the status and return.
// ---------------------------------------------------------------------------
namespace gsr {
namespace {
__global__ void lookback_timeout_probe_kernel(unsigned long long* states, DevStatus* status, uint32_t max_polls,
                                              uint32_t* out) {
  if (threadIdx.x == 0) {
    states[0] = 0ull;  // epoch 0: never the probe's epoch below
    *out = lookback(states, 1, 1, 7u, 0x3fffffffu, status, kWaitSelfTest, max_polls);
  }
}
}  // namespace

cudaError_t launch_lookback_timeout_probe(unsigned long long* states, DevStatus* status, uint32_t max_polls,
                                          uint32_t* out, cudaStream_t st) {
  lookback_timeout_probe_kernel<<<1, 32, 0, st>>>(states, status, max_polls, out);
  return cudaGetLastError();
}
}  // namespace gsr
