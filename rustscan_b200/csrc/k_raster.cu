// k_raster.cu — front-to-back blending (rasterize.wgsl:21-99) and its
// reverse-walk adjoint.
//
// One CTA per (view, tile) work item across all views of the launch. Each
// warp owns an 8x8 pixel block of the tile (or strips and whole tiles, see the
// kernels); each lane owns pixels of one column (rows y, y+4, ...), so the
// per-Gaussian terms a*dx*dx and 2b*dx are formed once for all of them. The tile's depth-sorted list is staged in
// shared memory batch by batch; while staging, the smallest sigma over each
// warp block's rectangle gives a bit per block that the Gaussian's
// {sigma <= log(255*opacity) + 1e-3} ellipse can reach (reached_blocks).
// Each warp then walks, in order, only the Gaussians whose bit it holds
// (ballot compaction into a per-warp list). The test is conservative and
// sigma is evaluated with the same expression tree as the oracle, so every
// contributor decision is unchanged: culled Gaussians could not pass the
// alpha >= 1/255 test (see kRejectMargin).
//
// The forward records per pixel the final transmittance and the list index
// of the last contributor, and per list entry a bit for each warp block in
// which some pixel took the Gaussian. The backward walks, per warp, only the
// entries whose forward bit covers its block (its contributor decisions
// repeat the forward's, so no other entry can contribute there), from
// the tile's largest last index down, recovers the transmittance before each
// contributor by division (T_i = T_{i+1} / (1 - alpha_i)), keeps the colour
// accumulated behind it, and forms per-pixel gradients (blend_step_grad).
// Per Gaussian the gradient sums over a warp's pixels come from a
// reduce-scatter butterfly (13 shuffles), over the CTA's warps from shared
// memory in warp order, and over tiles from float4 atomics (or, in
// deterministic mode, per-intersection records reduced later in a fixed
// order).
//
// Work items are the (view, tile) pairs of the launch. With the persistent
// schedule the raster kernels run as many CTAs as the SMs hold at once, each
// taking the next item from an atomic ticket, in decreasing order of an
// estimated cost, so the longest tiles start first and the launch does not
// end in a tail of long tiles on a few SMs; views of different sizes and
// visible counts share one queue. The backward's cost is the number of list
// entries up to the tile's last contributor: the forward appends each item
// to the list of its cost's bit length (32 lists), and a backward ticket
// walks the lists from the longest costs down. A launch of few 16x16 tiles
// cuts every tile's list into segments, each a backward item of its own, from
// checkpoints that the forward leaves. A persistent forward orders
// its items by list length with a single-block counting sort first.
// Otherwise one CTA per item runs in item order.
#include <algorithm>

#include <type_traits>

#include "gsr_kernels.h"

namespace gsr {

namespace {

// Pixels per lane: the forward gains nothing from more than 2. The
// backward of 16x16 tiles runs one warp per tile, or per segment of a tile's
// list, with 8 pixels per lane (raster_bwd_tile_kernel), so that each
// Gaussian's warp reduction serves the whole tile; the other tile shapes run
// raster_bwd_kernel with 2.

// The one-warp backward's batch (entries staged per round, double-buffered)
// and its resident CTAs per SM: 64 entries take 13 KB of shared memory, so
// that 16 CTAs fit an SM, the register bound of 16 (at most 128 a thread).
constexpr int kTileBwdBatch = 64;
constexpr int kTileBwdBlocks = 16;

struct RasterArgs {
  ViewSet vs;
  FwdBufs b;
  float bg[3];
  float* out_rgba;
  const float* v_rgba;
  int ref_mode;
  int long_tiles;  // forward: tiles of long lists are listed as an item per 8x8 block (see kLongTile)
  int split;    // forward: a CTA per 8x8 block of a 16x16 tile
  int persist;  // 0: one CTA per item; 1: persistent, items from sched_order; 2: persistent, items from the cost lists
};

__device__ __forceinline__ uint32_t find_view(const ViewSet& vs, uint32_t item) {
  uint32_t v = 0;
  for (uint32_t i = 1; i < vs.n_views; ++i)
    if (vs.views[i].tile_base <= item) v = i;
  return v;
}

constexpr uint32_t kNoItem = 0xffffffffu;

// Backward items of 16x16 tiles: the tile, and above kBlockShift which of its 8x8
// blocks the item takes (0: all). A launch has fewer than 2^28 tiles, each with
// 8 KB of pixel state.
constexpr uint32_t kBlockShift = 28;
constexpr int kCostLists = 32;  // bit lengths 0..31 of a cost (a list is shorter than 2^30); one per lane

__device__ __forceinline__ uint32_t cost_bucket(uint32_t cost) { return cost ? 32u - (uint32_t)__clz(cost) : 0u; }

// Per CTA, for the cost lists, entry l the list of the l-th largest costs:
// its length and its first place in the order. Read once per launch, one load
// per lane of warp 0 and a warp scan, because a small launch's first items
// wait for it.
struct CostListView {
  uint32_t count[kCostLists];
  uint32_t first[kCostLists];
};
__device__ __forceinline__ void load_cost_lists(const RasterArgs& a, CostListView* s) {
  if (!a.persist || threadIdx.x >= 32) return;
  const uint32_t lane = threadIdx.x;
  const uint32_t n = a.b.sched_lcount[kCostLists - 1 - lane];
  uint32_t incl = n;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= (uint32_t)d) incl += t;
  }
  s->count[lane] = n;
  s->first[lane] = incl - n;
}

// The next work item of this CTA (block-uniform; kNoItem when done). In
// the grid schedule a CTA runs item blockIdx.x once; in the persistent one
// thread 0 takes a ticket and reads the item at that place of the order: the
// forward's sched_order, or the backward's cost lists. The leading barrier
// keeps the previous item's shared state intact until every thread is done
// with it (and publishes load_cost_lists).
template <class At>
__device__ __forceinline__ uint32_t take_item(const RasterArgs& a, uint32_t round, uint32_t* s_item, At at) {
  if (!a.persist) return round == 0 ? blockIdx.x : kNoItem;
  __syncthreads();
  if (threadIdx.x == 0) *s_item = at(atomicAdd(a.b.sched_ticket, 1u));
  __syncthreads();
  return *s_item;
}
// PARTS: items per tile, in its place of the order.
template <int PARTS>
__device__ __forceinline__ uint32_t next_item(const RasterArgs& a, uint32_t round, uint32_t* s_item) {
  return take_item(a, round, s_item, [&](uint32_t slot) {
    const uint32_t at = slot / PARTS;
    return at < a.vs.total_tiles ? a.b.sched_order[at] * PARTS + slot % PARTS : kNoItem;
  });
}
// FIRST (launches whose items fit the resident CTAs a few times over, and tiles
// of several warps or few pixels): a CTA's first place is its own index, without a
// ticket, and warp 0's lanes look through the lists at once, because there an
// item's start is a good part of its time. Backward of 8x8 tiles, one view of
// 639x479 over 200k Gaussians, 164 us without and 146 with it, of 32x8 tiles 242
// and 195, 4 views of 1280x720 over 300k in 32x8 tiles 957 and 930.
template <bool FIRST>
__device__ __forceinline__ uint32_t next_item(const RasterArgs& a, uint32_t round, uint32_t* s_item,
                                              const CostListView* lists) {
  if constexpr (!FIRST) {
    return take_item(a, round, s_item, [&](uint32_t slot) {
#pragma unroll 1
      for (int k = 0; k < kCostLists; ++k)
        if (slot - lists->first[k] < lists->count[k])
          return a.b.sched_lists[(size_t)(kCostLists - 1 - k) * a.b.sched_items_cap + (slot - lists->first[k])];
      return kNoItem;
    });
  }
  if (!a.persist) return round == 0 ? blockIdx.x : kNoItem;
  __syncthreads();
  if (threadIdx.x == 0) *s_item = kNoItem;
  __syncthreads();
  if (threadIdx.x < 32) {
    uint32_t slot = blockIdx.x;
    if (round > 0) {
      if (threadIdx.x == 0) slot = gridDim.x + atomicAdd(a.b.sched_ticket, 1u);
      slot = __shfl_sync(0xffffffffu, slot, 0);
    }
    const uint32_t at = slot - lists->first[threadIdx.x];  // wraps past every count below the list's first place
    if (at < lists->count[threadIdx.x])
      *s_item = a.b.sched_lists[(size_t)(kCostLists - 1 - threadIdx.x) * a.b.sched_items_cap + at];
  }
  __syncthreads();
  return *s_item;
}

// One block: the work items of a persistent forward in decreasing order of
// cost bucket (bit length of the list length; order within a bucket is
// arbitrary), and the ticket reset.
constexpr int kOrderThreads = 1024;
__global__ void __launch_bounds__(kOrderThreads) sched_order_kernel(ViewSet vs, FwdBufs b) {
  __shared__ uint32_t s_hist[kCostLists];
  __shared__ uint32_t s_start[kCostLists];
  if (threadIdx.x < kCostLists) s_hist[threadIdx.x] = 0;
  __syncthreads();
  const uint32_t total = vs.total_tiles;
  auto cost_of = [&](uint32_t item) -> uint32_t {
    const uint32_t v = find_view(vs, item);
    const uint32_t t = item - vs.views[v].tile_base;
    const uint32_t* r = slice(b.ranges, 2 * b.Tcap, v);
    return r[2 * t + 1] - r[2 * t];
  };
  for (uint32_t i = threadIdx.x; i < total; i += kOrderThreads) atomicAdd(&s_hist[cost_bucket(cost_of(i))], 1u);
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t run = 0;
    for (int k = kCostLists - 1; k >= 0; --k) {
      s_start[k] = run;
      run += s_hist[k];
    }
    *b.sched_ticket = 0u;
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < total; i += kOrderThreads)
    b.sched_order[atomicAdd(&s_start[cost_bucket(cost_of(i))], 1u)] = i;
}

// Block w of a TW-wide tile is the 8x8 pixels at (x0, y0); a warp's lane l owns
// its column x0 + (l & 7) and rows y0 + (l >> 3) + {0, 4}.
template <int TW> struct WarpBlock {
  static_assert(TW % 8 == 0, "tile width is a multiple of the 8-pixel warp block");
  static constexpr int kWarpsX = TW / 8;
  __device__ static int x0(int w) { return (w % kWarpsX) * 8; }
  __device__ static int y0(int w) { return (w / kWarpsX) * 8; }
};

// The warp blocks (8 columns, ROWS rows) of a tile at (tx0, ty0) that a
// Gaussian can reach: bit w set unless sigma exceeds the cut over the whole
// rectangle of block w's pixel centres. The smallest value of a positive-definite quadratic over a
// rectangle that does not hold its centre lies on an edge facing the centre,
// so two clamped edge minima give it. The test errs on the side of keeping:
// sigma as the pixels evaluate it (and this minimum) is within 10 units of
// 2^-24 of (a dx^2 + c dy^2), which the last term covers threefold, and the
// cut itself lies kRejectMargin above any sigma that can contribute. A conic
// that float arithmetic cannot tell from an indefinite one, or a value that is
// not a number, keeps every block.
template <int TW, int NW, int ROWS>
__device__ __forceinline__ uint32_t reached_blocks(float x, float y, float a, float b, float c, float cut, float tx0,
                                                   float ty0) {
  uint32_t mask = (1u << NW) - 1u;
  if (!(a > 0.f && c > 0.f && a * c > b * b * (1.f + 5e-7f))) return mask;
  const float ka = __fdividef(-b, a), kc = __fdividef(-b, c), b2 = 2.f * b;
#pragma unroll
  for (int w = 0; w < NW; ++w) {
    // Offsets mean - centre over the block's columns and rows.
    constexpr int S = 8 / ROWS;  // warps per 8x8 block
    const float x1 = x - (tx0 + (float)(8 * (w / S % (TW / 8))) + 0.5f), x0 = x1 - 7.f;
    const float y1 = y - (ty0 + (float)(8 * (w / S / (TW / 8)) + ROWS * (w % S)) + 0.5f), y0 = y1 - (float)(ROWS - 1);
    const float nx = fminf(fmaxf(0.f, x0), x1), ny = fminf(fmaxf(0.f, y0), y1);
    const float ey = fminf(fmaxf(kc * nx, y0), y1), ex = fminf(fmaxf(ka * ny, x0), x1);
    const float q1 = fmaf(fmaf(a, nx, b2 * ey), nx, c * ey * ey);
    const float q2 = fmaf(fmaf(c, ny, b2 * ex), ny, a * ex * ex);
    const float fx = fmaxf(fabsf(x0), fabsf(x1)), fy = fmaxf(fabsf(y0), fabsf(y1));
    if (0.5f * fminf(q1, q2) - 2e-6f * (a * fx * fx + c * fy * fy) > cut) mask &= ~(1u << w);
  }
  return mask;
}

// Order-preserving compaction of the batch entries whose mask has a bit of
// wsel.
__device__ __forceinline__ int build_list(const uint8_t* s_mask, uint32_t nb, uint32_t wsel, int lane,
                                          uint16_t* list) {
  int cnt = 0;
  for (uint32_t base = 0; base < nb; base += 32) {
    const uint32_t j = base + lane;
    const bool bit = j < nb && (s_mask[j] & wsel) != 0u;
    const uint32_t bal = __ballot_sync(0xffffffffu, bit);
    if (bit) list[cnt + __popc(bal & ((1u << lane) - 1u))] = (uint16_t)j;
    cnt += __popc(bal);
  }
  __syncwarp();
  return cnt;
}

// Paired FP32 arithmetic: every lane owns its pixels in pairs (rows y + 8k and
// y + 8k + 4 of one column), and the per-pixel arithmetic of a pair runs as
// two-wide operations (fma2 is a fused multiply-add per half, add2 and mul2
// round per half like the scalar operations).
//
// The compiler contracts a paired multiply feeding a paired add into one
// fused multiply-add, even when written as PTX with .rn and with contraction
// switched off (--fmad=false; measured: the paired and the fused results
// agree bit for bit, the separately rounded scalar chain does not). The
// decision arithmetic is therefore defined with its multiply-adds fused
// (sigma and the range reduction of the exponential, gsr_math.h), and the
// kernels spell those as fma2, which is then exact by construction; no
// decision depends on a paired multiply feeding a paired add. The file is
// built without contraction, like the CPU oracle, so that the remaining
// scalar expressions keep their written rounding.
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
// The same operations for a lane with one pixel.
__device__ __forceinline__ float add2(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float mul2(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fma2(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float neg2(float a) { return -a; }

// blend_sigma_shared for the two pixels of a pair (same column: same t1,
// t2): the same operations in the same order, each half rounded on its own.
__device__ __forceinline__ float2 sigma2(float t1, float t2, float2 dy, float cc) {
  return mul2(f2(0.5f), fma2(mul2(f2(cc), dy), dy, fma2(f2(t2), dy, f2(t1))));
}

// blend_expf(-sigma) for both pixels, without its range clamps: for every
// sigma the contribution test can accept (0 <= sigma <= log(255) + margin)
// they change nothing, so there the result is bit-identical to blend_expf.
// For a pixel outside that range the value is meaningless (possibly not
// finite); every use of it is selected away by the pixel's contribution
// flags, never multiplied in.
__device__ __forceinline__ float2 blend_exp2(float2 sigma) {
  const float2 x = make_float2(-sigma.x, -sigma.y);
  const float2 t = fma2(x, f2(bexp::kLog2e), f2(bexp::kMagic));
  const float2 n = add2(t, f2(-bexp::kMagic));
  // 2^n by exponent-field addition, as blend_expf: t's bits are those of
  // 1.5 * 2^23 plus n, and a left shift by 23 drops the constant (its low 22
  // bits are zero), leaving n << 23 modulo 2^32.
  static_assert((bexp::kMagicBits << 23) == 0u, "the constant part shifts out");
  const uint32_t ex = __float_as_uint(t.x) << 23;
  const uint32_t ey = __float_as_uint(t.y) << 23;
  float2 r = fma2(neg2(n), f2(bexp::kLn2Hi), x);
  r = fma2(neg2(n), f2(bexp::kLn2Lo), r);
  float2 p = f2(bexp::kC6);
  p = fma2(p, r, f2(bexp::kC5));
  p = fma2(p, r, f2(bexp::kC4));
  p = fma2(p, r, f2(bexp::kC3));
  p = fma2(p, r, f2(bexp::kC2));
  p = fma2(p, r, f2(1.0f));
  p = fma2(p, r, f2(1.0f));
  return make_float2(__uint_as_float(__float_as_uint(p.x) + ex), __uint_as_float(__float_as_uint(p.y) + ey));
}
__device__ __forceinline__ float blend_exp2(float sigma) {
  const float x = -sigma;
  const float t = __fmaf_rn(x, bexp::kLog2e, bexp::kMagic);
  const float n = __fadd_rn(t, -bexp::kMagic);
  float r = __fmaf_rn(-n, bexp::kLn2Hi, x);
  r = __fmaf_rn(-n, bexp::kLn2Lo, r);
  float p = bexp::kC6;
  p = __fmaf_rn(p, r, bexp::kC5);
  p = __fmaf_rn(p, r, bexp::kC4);
  p = __fmaf_rn(p, r, bexp::kC3);
  p = __fmaf_rn(p, r, bexp::kC2);
  p = __fmaf_rn(p, r, 1.0f);
  p = __fmaf_rn(p, r, 1.0f);
  return __uint_as_float(__float_as_uint(p) + (__float_as_uint(t) << 23));
}

// The pixels of a forward lane: a pair in one register pair, or one.
template <int PX> struct Lane;
template <> struct Lane<2> {
  using V = float2;
  __device__ static V all(float x) { return make_float2(x, x); }
  __device__ static V of(float2 twice) { return twice; }
  __device__ static V make(const float (&x)[2]) { return make_float2(x[0], x[1]); }
  __device__ static V pick(const bool (&c)[2], V a, V b) { return make_float2(c[0] ? a.x : b.x, c[1] ? a.y : b.y); }
  __device__ static float get(V v, int h) { return h ? v.y : v.x; }
};
template <> struct Lane<1> {
  using V = float;
  __device__ static V all(float x) { return x; }
  __device__ static V of(float2 twice) { return twice.x; }
  __device__ static V make(const float (&x)[1]) { return x[0]; }
  __device__ static V pick(const bool (&c)[1], V a, V b) { return c[0] ? a : b; }
  __device__ static float get(V v, int) { return v; }
};

// The segments of a list of `len` entries: segment k begins at len (k / K)^2,
// rounded up to the 32 entries the forward steps by, or at 32 k (64 k where that
// does not cover the list) if that is further on, and the last one is open-ended.
// An item of a latency-bound launch takes about 1000 cycles an entry, so short
// segments end it sooner; most lists saturate within a fraction of their length,
// so the early ones are short, and a list that does not ends in segments of at
// most 2 / K of it. Every segment begins at least 32 entries after the one before.
// With equal segments of 64 and the rest in the last one, the backward of 2 uneven
// views up to 260x146 over 141k Gaussians (a list of 48894) took 15.7 ms and takes
// 0.61, of 5 up to 640x400 over 500k 7.0 and 1.5, of 8 of 400x300 over 100k 0.66
// and 0.39; of one of 639x479 over 200k 0.118 and 0.121.
struct Segments {
  uint32_t len;  // shortest segment
  float grow;
  // First entry of segment k.
  __device__ __forceinline__ uint32_t begin(uint32_t k) const {
    return max(k * len, ((uint32_t)(grow * (float)(k * k)) + 31u) & ~31u);
  }
};
__device__ __forceinline__ Segments segments_of(uint32_t len, uint32_t k) {
  return Segments{len <= 32u * k ? 32u : 64u, (float)len / (float)(k * k)};
}

// A list entry as the forward stages it. Values that both pixels of a pair
// take lie twice side by side, so that a load brings them as the register
// pair a two-wide operation wants.
struct __align__(16) FwdEntry {
  float x, a, b2, cut;    // mean x, conic a, 2 conic b (exact), reject cut
  float2 y, c;            // mean y, conic c
  float2 opac, r;         // opacity, max(red, 0)
  float2 g, b;            // max(green, 0), max(blue, 0)
  uint32_t last;          // list index + 1
  uint8_t hit[4];         // warp block w took the entry
  uint32_t cidx, pad;
};
// Entries a warp evaluates together. Two cost nothing on large launches but
// 2% on a launch of 300 tiles, where few warps hide each other's latency.
constexpr int kFwdUnroll = 4;
template <int BATCH, int NW> struct FwdSmem {
  FwdEntry e[BATCH + 1];  // the last one is never taken: it pads the lists
  uint8_t mask[BATCH];
  alignas(8) uint16_t list[NW][BATCH + kFwdUnroll];  // byte offsets into e
  uint32_t item;
  uint32_t work;  // the item's largest last contributor
  uint32_t top;   // the tile's, in the last of a split tile's CTAs
};
// Resident threads per SM the register bound allows (768: 80 registers): 8
// views of 1280x720 blend in 0.832 ms, in 0.844 at 640 and 0.830 with more
// spills at 896.
constexpr int kFwdThreadsPerSm = 768;

// One CTA per tile, a warp per 8x8 block, a lane per pixel pair (rows y and
// y + 4 of one column). Per batch every entry is staged once with the blocks
// it can reach; each warp walks the entries of its block in list order, four
// at a time. The four sigmas, exponentials and contribution tests are
// independent of the pixel state and run as one straight-line block, so their
// latencies overlap; the four blends then follow in order. No branch depends
// on a pixel: a pixel that does not take an entry blends with alpha 0, which
// leaves its transmittance and, where all colours are finite, its colour bit for
// bit unchanged, and a saturated pixel (transmittance below 1e-4) takes nothing. What bounds it is
// instruction issue and, on launches of few tiles, the latency of the
// longest tile. Against a walk of two entries with a vote and
// a branch each, over blocks culled by the footprint's bounding box: 8 views
// of 1280x720 over 1M Gaussians 1.10 -> 0.83 ms (135M -> 90M warp instructions
// a view), one view of 320x240 over 74k 0.193 -> 0.104 ms.
// CKPT: at the end of every segment of the list (see Segments) the
// tile's pixels leave a checkpoint for the segmented backward (see
// raster_bwd_tile_kernel): the transmittance there and the colour the segment
// added, turned into the colour of all later segments once the tile is done.
// The colour is summed per segment on its own, not taken as a difference of
// running totals, so that what lies far behind keeps its relative accuracy.
// The next batch's records are then also loaded while the current one is
// walked, since few warps are there to hide the loads.
// SPLIT (16x16 tiles, with CKPT): a CTA per 8x8 block of a tile, two warps with
// one pixel per lane, each walking the entries that reach its 8x4 strip (see
// kFwdSplitTiles). The four CTAs of a tile set their hit bits one by one, and
// the last of them lists the tile for the backward.
// FINITE: no colour is infinite. 0 times infinity is not 0, so otherwise a pixel
// that does not take an entry keeps its sums by selection. That costs a split
// tile's lanes, of one pixel each, up to 2 us (300 tiles over 74k Gaussians 80.5 ->
// 82.4), but 14% with two pixels and checkpoints (1200 tiles over 200k 93 -> 106);
// so the launches that are not split take it only if the projection reports an
// infinite colour. The report's load takes 0.6% of a large launch (8 views of
// 1280x720 0.822 -> 0.827 ms).
template <int TW, int TH, int BATCH, bool CKPT, bool SPLIT, bool FINITE>
__device__ __forceinline__ void blend_items(const RasterArgs& a, FwdSmem<BATCH, SPLIT ? 2 : TW * TH / 64>& S) {
  constexpr int PX = SPLIT ? 1 : 2;  // pixels per lane
  using L = Lane<PX>;
  using V = typename L::V;
  constexpr int NT = SPLIT ? 64 : TW * TH / 2;
  constexpr int NW = NT / 32;
  constexpr int WB = 2 / PX;                  // warps per 8x8 block
  constexpr int BW = SPLIT ? 8 : TW;          // width of the CTA's pixel area
  constexpr int kSI = (BATCH + NT - 1) / NT;  // entries a thread stages per batch
  static_assert(NW / WB <= 4 && TW % 8 == 0 && TH % 8 == 0, "hit bits of at most four 8x8 blocks");
  auto& s_e = S.e;
  auto& s_mask = S.mask;
  uint32_t& s_work = S.work;
  if (threadIdx.x == 0) {
    s_work = 0u;
    s_e[BATCH] = FwdEntry{};  // sigma 0, opacity 0: alpha 0
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int half = warp % WB;  // SPLIT: the block's rows y + 4 half
  uint16_t* list = S.list[warp];
  for (uint32_t round = 0;; ++round) {
    const uint32_t work = next_item<SPLIT ? 4 : 1>(a, round, &S.item);
    if (work == kNoItem) break;
    const uint32_t item = SPLIT ? work / 4 : work;
    const int block = SPLIT ? (int)(work % 4) : warp;  // 8x8 block of the tile
    const uint32_t v = find_view(a.vs, item);
    const ViewDesc& vd = a.vs.views[v];
    const uint32_t t = item - vd.tile_base;
    const uint32_t tx = t % vd.tiles_x, ty = t / vd.tiles_x;
    const uint32_t px = tx * TW + WarpBlock<TW>::x0(block) + (lane & 7);
    const uint32_t py = ty * TH + WarpBlock<TW>::y0(block) + (lane >> 3) + 4 * half;
    const float pcx = (float)px + 0.5f;
    float rows[PX], first[PX];
    bool inside[PX];
#pragma unroll
    for (int h = 0; h < PX; ++h) {
      rows[h] = -((float)(py + 4 * h) + 0.5f);
      inside[h] = px < vd.w && py + 4 * h < vd.h;
      first[h] = inside[h] ? 1.f : 0.f;  // a pixel outside the image starts saturated
    }
    const V npcy = L::make(rows);
    const uint32_t* ranges = slice(a.b.ranges, 2 * a.b.Tcap, v);
    const uint32_t s0 = ranges[2 * t], s1 = ranges[2 * t + 1];
    const uint32_t* vals = isect_index_src(a.b, v);
    const uint32_t vmask = isect_index_mask(a.b);
    const float4* rec = slice(a.b.rec, a.b.Vcap * 3, v);
    uint8_t* vis = slice(a.b.visible_c, a.b.Vcap, v);
    uint8_t* hitw = slice(a.b.hitw, a.b.Icap, v);
    // Corner of the CTA's pixel area.
    const float tx0 = (float)(tx * TW + (SPLIT ? WarpBlock<TW>::x0(block) : 0));
    const float ty0 = (float)(ty * TH + (SPLIT ? WarpBlock<TW>::y0(block) : 0));
    V T = L::make(first), C0 = L::all(0.f), C1 = C0, C2 = C0;
    uint32_t last[PX] = {}, nc[PX] = {};
    auto saturated = [&] {
      bool all = true;
#pragma unroll
      for (int h = 0; h < PX; ++h) all = all && L::get(T, h) < 1e-4f;
      return all;
    };
    // Checkpoints of this tile, segment by segment: half h of lane l's pair in
    // block q at ck[segment * pixels + h * pixels / 2 + 32 q + l].
    constexpr int kHalf = TW * TH / 2;
    float4* ck = CKPT ? a.b.ckpt + (size_t)item * a.b.seg_k * (TW * TH) + half * kHalf + block * 32 + lane : nullptr;
    V S0 = C0, S1 = C0, S2 = C0;  // colour added since the last checkpoint
    uint32_t stored = 0;                              // checkpoints written
    const Segments segs = segments_of(s1 - s0, CKPT ? a.b.seg_k : 1u);
    uint32_t seg_end = s0 + segs.begin(1);
    struct Raw {
      uint32_t c;
      float4 r0, r1, r2;
    };
    auto load = [&](uint32_t i) {
      Raw r;
      r.c = vals[i] & vmask;
      r.r0 = rec[(size_t)r.c * 3 + 0];
      r.r1 = rec[(size_t)r.c * 3 + 1];
      r.r2 = rec[(size_t)r.c * 3 + 2];
      return r;
    };
    auto stage = [&](uint32_t j, uint32_t i, const Raw& r) {
      const float cut = r.r2.y + kRejectMargin;
      FwdEntry& E = s_e[j];
      E.x = r.r0.x;
      E.a = r.r0.z;
      E.b2 = 2.f * r.r0.w;
      E.cut = cut;
      E.y = f2(r.r0.y);
      E.c = f2(r.r1.x);
      E.opac = f2(r.r1.y);
      E.r = f2(fmaxf(r.r1.z, 0.f));
      E.g = f2(fmaxf(r.r1.w, 0.f));
      E.b = f2(fmaxf(r.r2.x, 0.f));
      E.last = i + 1;
      *reinterpret_cast<uint32_t*>(E.hit) = 0u;
      E.cidx = r.c;
      s_mask[j] = (uint8_t)reached_blocks<BW, NW, 8 / WB>(r.r0.x, r.r0.y, r.r0.z, r.r0.w, r.r1.x, cut, tx0, ty0);
    };
    Raw next[CKPT ? kSI : 1];  // CKPT: this thread's entries of the next batch
    auto fetch = [&](uint32_t b0) {
#pragma unroll
      for (int i = 0; i < kSI; ++i) {
        const uint32_t j = threadIdx.x + i * NT;
        if (j < (uint32_t)BATCH && b0 + j < s1) next[CKPT ? i : 0] = load(b0 + j);
      }
    };
    if (CKPT) fetch(s0);
    for (uint32_t b0 = s0; b0 < s1; b0 += BATCH) {
      const uint32_t nb = min((uint32_t)BATCH, s1 - b0);
      if (CKPT) {
#pragma unroll
        for (int i = 0; i < kSI; ++i) {
          const uint32_t j = threadIdx.x + i * NT;
          if (j < nb) stage(j, b0 + j, next[CKPT ? i : 0]);
        }
      } else {
        for (uint32_t j = threadIdx.x; j < nb; j += NT) stage(j, b0 + j, load(b0 + j));
      }
      __syncthreads();
      if (CKPT && b0 + BATCH < s1) fetch(b0 + BATCH);
      // The walk over cnt listed entries, padded to a multiple of the unroll.
      auto walk = [&](uint32_t cnt) {
        if (lane < kFwdUnroll) list[cnt + lane] = (uint16_t)(BATCH * sizeof(FwdEntry));
        __syncwarp();
        for (uint32_t e = 0; e < cnt; e += kFwdUnroll) {
          const uint2 off2 = *reinterpret_cast<const uint2*>(list + e);
          const uint32_t off[kFwdUnroll] = {off2.x & 0xffffu, off2.x >> 16, off2.y & 0xffffu, off2.y >> 16};
          V al[kFwdUnroll];
          bool take[kFwdUnroll][PX];
#pragma unroll
          for (int u = 0; u < kFwdUnroll; ++u) {
            const FwdEntry& E = *reinterpret_cast<const FwdEntry*>(reinterpret_cast<const char*>(s_e) + off[u]);
            const float dx = esub(E.x, pcx);
            const float t1 = emul(emul(E.a, dx), dx);
            const float t2 = emul(E.b2, dx);
            const V dy = add2(L::of(E.y), npcy);
            float in[PX], cl[PX];
#pragma unroll
            for (int h = 0; h < PX; ++h) in[h] = fmaf(t2, L::get(dy, h), t1);
            // Sigma, as blend_sigma_shared.
            const V sg = mul2(L::all(0.5f), fma2(mul2(L::of(E.c), dy), dy, L::make(in)));
            const V og = mul2(L::of(E.opac), blend_exp2(sg));
            // 0 <= sigma <= cut in one unsigned comparison of the bits (sigma is
            // never -0; a negative one has the sign bit set) and alpha >= 1/255,
            // as blend_alpha_of decides.
            const uint32_t cut = __float_as_uint(E.cut);
#pragma unroll
            for (int h = 0; h < PX; ++h) {
              cl[h] = fminf(0.999f, L::get(og, h));
              take[u][h] = __float_as_uint(L::get(sg, h)) <= cut && cl[h] >= (float)(1.0 / 255.0);
            }
            al[u] = L::make(cl);
          }
#pragma unroll
          for (int u = 0; u < kFwdUnroll; ++u) {
            FwdEntry& E = *reinterpret_cast<FwdEntry*>(reinterpret_cast<char*>(s_e) + off[u]);
            float am[PX];
            bool any = false;
#pragma unroll
            for (int h = 0; h < PX; ++h) {
              take[u][h] = take[u][h] && !(L::get(T, h) < 1e-4f);
              am[h] = take[u][h] ? L::get(al[u], h) : 0.f;
              any = any || take[u][h];
            }
            const V alpha = L::make(am);
            const V w = mul2(alpha, T);
            auto add = [&](V& sum, float2 c) {  // blend_accum; the colours were clamped at staging
              const V more = fma2(L::of(c), w, sum);
              sum = FINITE ? more : L::pick(take[u], more, sum);
            };
            add(C0, E.r);
            add(C1, E.g);
            add(C2, E.b);
            if constexpr (CKPT) {
              add(S0, E.r);
              add(S1, E.g);
              add(S2, E.b);
            }
            T = mul2(T, add2(L::all(1.f), neg2(alpha)));
            if (any) E.hit[SPLIT ? 0 : warp] = 1;
#pragma unroll
            for (int h = 0; h < PX; ++h)
              if (take[u][h]) {
                last[h] = E.last;
                ++nc[h];
              }
          }
          if (__all_sync(0xffffffffu, saturated())) break;
        }
      };
      // The entries of this warp's block in list order: the whole batch, or
      // (CKPT) 32 at a time, the shortest segment.
      uint32_t cnt = 0;
      const bool live = !__all_sync(0xffffffffu, saturated());
      for (uint32_t base = 0; (CKPT || live) && base < nb; base += 32) {
        const uint32_t j = base + lane;
        const bool bit = j < nb && ((s_mask[j] >> warp) & 1u);
        const uint32_t bal = __ballot_sync(0xffffffffu, bit);
        if (bit) list[cnt + __popc(bal & ((1u << lane) - 1u))] = (uint16_t)(j * sizeof(FwdEntry));
        cnt += __popc(bal);
        if constexpr (CKPT) {
          if (cnt && !__all_sync(0xffffffffu, saturated())) walk(cnt);
          cnt = 0;
          __syncwarp();  // the list is free again
          if (b0 + base + 32 == seg_end) {
            float4* c = ck + (size_t)stored * (TW * TH);
#pragma unroll
            for (int h = 0; h < PX; ++h)
              c[h * kHalf] = make_float4(L::get(T, h), L::get(S0, h), L::get(S1, h), L::get(S2, h));
            S0 = S1 = S2 = L::all(0.f);
            ++stored;
            seg_end = stored + 1 < a.b.seg_k ? s0 + segs.begin(stored + 1) : 0u;  // the last one is open-ended
          }
        }
      }
      if (!CKPT && live) walk(cnt);
      __syncthreads();
      for (uint32_t j = threadIdx.x; j < nb; j += NT) {
        const uint32_t h = *reinterpret_cast<const uint32_t*>(s_e[j].hit);
        if (SPLIT) {
          // The other blocks' CTAs set their bits in the same byte.
          const uintptr_t at = reinterpret_cast<uintptr_t>(hitw + b0 + j);
          if (h) atomicOr(reinterpret_cast<uint32_t*>(at & ~uintptr_t(3)), (1u << block) << (8 * (at & 3)));
        } else {
          hitw[b0 + j] = (uint8_t)((h | (h >> 7) | (h >> 14) | (h >> 21)) & 0xfu);  // bit w: the 8x8 block of warp w
        }
        if (h) vis[s_e[j].cidx] = 1;
      }
      if (__syncthreads_and(saturated())) break;
    }
    if constexpr (CKPT) {
      // A split tile's CTA may stop, saturated, before the tile does: its pixels'
      // last entries then lie in a segment that other CTAs see the end of, and the
      // state there is the present one.
      if (SPLIT && stored + 1 < a.b.seg_k) {
        float4* c = ck + (size_t)stored * (TW * TH);
#pragma unroll
        for (int h = 0; h < PX; ++h)
          c[h * kHalf] = make_float4(L::get(T, h), L::get(S0, h), L::get(S1, h), L::get(S2, h));
        S0 = S1 = S2 = L::all(0.f);
        ++stored;
      }
      // Each thread turns its own checkpoints' colours into the sum over the
      // later segments, from the last one forward.
      for (int k = (int)stored - 1; k >= 0; --k) {
        float4* c = ck + (size_t)k * (TW * TH);
        float c0[PX], c1[PX], c2[PX];
#pragma unroll
        for (int h = 0; h < PX; ++h) {
          const float4 u = c[h * kHalf];
          c[h * kHalf] = make_float4(u.x, L::get(S0, h), L::get(S1, h), L::get(S2, h));
          c0[h] = u.y;
          c1[h] = u.z;
          c2[h] = u.w;
        }
        S0 = add2(S0, L::make(c0));
        S1 = add2(S1, L::make(c1));
        S2 = add2(S2, L::make(c2));
      }
    }
    float4* out = reinterpret_cast<float4*>(a.out_rgba) + vd.pix_base;
    uint32_t ml = 0;
#pragma unroll
    for (int h = 0; h < PX; ++h) {
      ml = max(ml, last[h]);
      if (!inside[h]) continue;
      const size_t pix = (size_t)(py + 4 * h) * vd.w + px;
      const float Tq = L::get(T, h);
      out[pix] = make_float4(L::get(C0, h) + Tq * a.bg[0], L::get(C1, h) + Tq * a.bg[1], L::get(C2, h) + Tq * a.bg[2],
                             1.f - Tq);
      slice(a.b.tfinal, a.b.Pcap, v)[pix] = Tq;
      slice(a.b.last, a.b.Pcap, v)[pix] = last[h];
      slice(a.b.ncontrib, a.b.Pcap, v)[pix] = nc[h];
      slice(a.b.nvisit, a.b.Pcap, v)[pix] = (Tq < 1e-4f ? last[h] : s1) - s0;  // a saturated pixel stopped there
    }
    // The backward's cost of this item: list entries up to the tile's
    // largest last contributor.
    ml = __reduce_max_sync(0xffffffffu, ml);
    if (lane == 0 && ml) atomicMax(&s_work, ml);
    __syncthreads();
    uint32_t top = s_work;
    if (SPLIT) {
      // The last of the tile's four CTAs knows the tile's.
      if (threadIdx.x == 0) {
        uint32_t* sync = a.b.tile_sync + 2 * (size_t)item;
        atomicMax(sync, top);
        __threadfence();
        S.top = atomicAdd(sync + 1, 1u) == 3u ? atomicMax(sync, 0u) : 0xffffffffu;
      }
      __syncthreads();
      top = S.top;
    }
    if (!SPLIT || top != 0xffffffffu) {
      const uint32_t cost = top > s0 ? top - s0 : 0u;
      for (uint32_t g = threadIdx.x; g < (CKPT ? a.b.seg_k : 1u); g += NT) {  // the tile's backward items
        const uint32_t lo = CKPT ? segs.begin(g) : 0u;
        if (g > 0 && lo >= cost) break;
        const uint32_t n = (CKPT && g + 1 < a.b.seg_k ? min(segs.begin(g + 1), cost) : cost) - lo;
        const uint32_t work = item * a.b.seg_k + g;
        if (TW == 16 && TH == 16 && a.long_tiles && n > kLongTile && atomicAdd(a.b.long_count, 1u) < kLongTiles) {
          // A long walk: an item per 8x8 block.
          const uint32_t c = cost_bucket(n / 2);
          const uint32_t at = atomicAdd(a.b.sched_lcount + c, 4u);
          for (uint32_t q = 0; q < 4; ++q)
            a.b.sched_lists[(size_t)c * a.b.sched_items_cap + at + q] = work | (q + 1) << kBlockShift;
        } else {
          const uint32_t c = cost_bucket(n);
          a.b.sched_lists[(size_t)c * a.b.sched_items_cap + atomicAdd(a.b.sched_lcount + c, 1u)] = work;
        }
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) s_work = 0u;
  }
}

template <int TW, int TH, int BATCH, bool CKPT, bool SPLIT>
__global__ void __launch_bounds__(SPLIT ? 64 : TW * TH / 2, SPLIT ? 8 : CKPT ? 4 : kFwdThreadsPerSm / (TW * TH / 2))
    raster_fwd_kernel(RasterArgs a) {
  __shared__ FwdSmem<BATCH, SPLIT ? 2 : TW * TH / 64> S;
  if (!SPLIT && *a.b.inf_colour == 0u)
    blend_items<TW, TH, BATCH, CKPT, SPLIT, true>(a, S);
  else
    blend_items<TW, TH, BATCH, CKPT, SPLIT, false>(a, S);
}

// Reduce-scatter of 12 per-lane values over the warp in 13 shuffles. Lane
// l ends with the warp total of value reduce12_slot(l) (lanes whose bit 1 is
// set and bit 2 differs hold the same value; the fixed summation order makes
// them equal). Stages: xor 16 halves 12 -> 6, xor 8 halves 6 -> 3, xor 4
// splits values 0 and 2 and sums value 1 in both lanes, xor 2 splits the two
// left, xor 1 completes the sum.
__device__ __forceinline__ int reduce12_slot(int lane) {
  const int g16 = (lane >> 4) & 1, g8 = (lane >> 3) & 1, g4 = (lane >> 2) & 1, g2 = (lane >> 1) & 1;
  return (g2 ? 1 : (g4 ? 2 : 0)) + 3 * g8 + 6 * g16;
}
__device__ __forceinline__ float warp_reduce_scatter12(float (&x)[12], int lane) {
  const uint32_t full = 0xffffffffu;
  {
    const bool hi = lane & 16;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const float send = hi ? x[i] : x[i + 6];
      const float keep = hi ? x[i + 6] : x[i];
      x[i] = keep + __shfl_xor_sync(full, send, 16);
    }
  }
  {
    const bool hi = lane & 8;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const float send = hi ? x[i] : x[i + 3];
      const float keep = hi ? x[i + 3] : x[i];
      x[i] = keep + __shfl_xor_sync(full, send, 8);
    }
  }
  float w0, w1;
  {
    const bool hi = lane & 4;
    const float send = hi ? x[0] : x[2];
    const float keep = hi ? x[2] : x[0];
    w0 = keep + __shfl_xor_sync(full, send, 4);
    w1 = x[1] + __shfl_xor_sync(full, x[1], 4);
  }
  float u;
  {
    const bool hi = lane & 2;
    const float send = hi ? w0 : w1;
    const float keep = hi ? w1 : w0;
    u = keep + __shfl_xor_sync(full, send, 2);
  }
  return u + __shfl_xor_sync(full, u, 1);
}

// Per-pair state of the reverse walk (pixel q = 2k + h is half h of pair k).
struct BwdPair {
  uint32_t last0, last1;
  float2 T;             // transmittance
  float2 SK;            // the background term plus dot(colour accumulated behind the current Gaussian,
                        // upstream colour gradient)
  float2 vr, vg, vb;    // upstream colour gradient
};

__device__ __forceinline__ void load_bwd_pair(const RasterArgs& a, const ViewDesc& vd, uint32_t v, uint32_t px,
                                              uint32_t py0, BwdPair& p) {
  float T[2] = {1.f, 1.f}, K[2] = {0.f, 0.f}, g[2][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
  uint32_t last[2] = {0u, 0u};
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t py = py0 + 4 * h;
    if (!(px < vd.w && py < vd.h)) continue;
    const size_t pix = (size_t)py * vd.w + px;
    last[h] = slice(a.b.last, a.b.Pcap, v)[pix];
    T[h] = slice(a.b.tfinal, a.b.Pcap, v)[pix];
    const float4 u = reinterpret_cast<const float4*>(a.v_rgba)[vd.pix_base + pix];
    g[h][0] = u.x;
    g[h][1] = u.y;
    g[h][2] = u.z;
    K[h] = (u.x * a.bg[0] + u.y * a.bg[1] + u.z * a.bg[2] - u.w) * T[h];
  }
  p.last0 = last[0];
  p.last1 = last[1];
  p.T = make_float2(T[0], T[1]);
  p.SK = make_float2(K[0], K[1]);
  p.vr = make_float2(g[0][0], g[1][0]);
  p.vg = make_float2(g[0][1], g[1][1]);
  p.vb = make_float2(g[0][2], g[1][2]);
}

__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// A lane's sums over its pixels for the current Gaussian. With dx shared
// by the lane's column and vs the gradient with respect to sigma at each
// pixel, the mean and conic gradient sums factor through three moments,
// M0 = sum vs, M1 = sum vs dy, M2 = sum vs dy^2:
//   sum vs (a dx + b dy) = a S1 + b S2,   sum vs (b dx + c dy) = b S1 + c S2,
//   sum vs dx^2 / 2 = S3 / 2,   sum vs dx dy = S4,   sum vs dy^2 / 2 = S5 / 2,
// with S1 = dx M0, S2 = M1, S3 = dx^2 M0, S4 = dx M1 and S5 = M2 per lane.
// The S sums are what the warp reduces; the conic combination runs once per
// tile, on the CTA's totals. Where the pixel's alpha is not clamped, alpha =
// opacity * G, so the opacity-path gradient sum va * G over those pixels is
// -(sum vs) / opacity: M0 serves for both. The absolute mean-gradient sums
// (densification statistics) stay per pixel.
struct BwdMom {
  float2 m0, m1, m2;
};
struct BwdAcc {
  float2 cr, cg, cb;  // colour gradients
  float2 ax, ay;      // sums of |d/dx| and |d/dy| of the per-pixel mean gradients
  uint32_t n;         // contributing pixels
};

// The first part of a reverse-walk step for both pixels of a pair: the
// offsets and sigma, and whether each pixel can take the Gaussian at all
// (it is before its last contributor and sigma is in [0, cut]).
struct PairPre {
  float2 dy, sg;
  bool l0, l1;
};
__device__ __forceinline__ PairPre bwd_pair_pre(const BwdPair& p, float2 npcy, uint32_t s, float t1, float t2,
                                                const float4& A, const float4& B) {
  PairPre q;
  const bool in0 = s < p.last0, in1 = s < p.last1;
  q.dy = add2(f2(A.y), npcy);
  q.sg = sigma2(t1, t2, q.dy, B.x);
  // 0 <= sigma <= cut in one unsigned comparison, as in the forward.
  const uint32_t cut = __float_as_uint(B.y);
  q.l0 = in0 && __float_as_uint(q.sg.x) <= cut;
  q.l1 = in1 && __float_as_uint(q.sg.y) <= cut;
  return q;
}

// The rest of the step: the contribution decisions repeat the forward's bit
// for bit; the gradient follows blend_step_grad (rasterize_backwards, exact
// adjoint), with the transmittance recovered with a Newton-refined hardware
// reciprocal. Adds the pair's terms into mom and acc (FIRST_MOM, FIRST_ACC:
// sets them to the terms). Straight-line code: a pixel that does not take
// the Gaussian contributes zeros and keeps its state. With REF (the
// reference semantics) a pixel whose transmittance fell to 1e-4 no longer
// counts as a contributor and gets no gradient.
template <bool REF, bool FIRST_MOM, bool FIRST_ACC>
__device__ __forceinline__ void bwd_pair_rest(BwdPair& p, const PairPre& q, float adx, float bdx, float cb,
                                              const float4& B, const float2 cpv, const float2 vr, const float2 vg,
                                              const float2 vb, BwdMom& mom, BwdAcc& acc) {
  const float2 dy = q.dy;
  const float2 gs = blend_exp2(q.sg);
  const float2 og = mul2(f2(B.z), gs);
  const float ax = fminf(0.999f, og.x), ay = fminf(0.999f, og.y);
  const bool c0 = q.l0 && ax >= (float)(1.0 / 255.0);
  const bool c1 = q.l1 && ay >= (float)(1.0 / 255.0);
  const bool sk0 = REF && p.T.x <= 1e-4f, sk1 = REF && p.T.y <= 1e-4f;
  const float2 al = make_float2(ax, ay);
  const float2 am = make_float2(c0 ? ax : 0.f, c1 ? ay : 0.f);
  const float2 om = add2(f2(1.f), neg2(am));
  // Hardware reciprocal refined by one Newton step (r + r(1 - om r)); a
  // pixel that does not take this Gaussian keeps its transmittance exactly.
#ifdef GSR_EXACT_RCP
  float2 ra = make_float2(__frcp_rn(om.x), __frcp_rn(om.y));
#else
  float2 ra = make_float2(rcp_approx(om.x), rcp_approx(om.y));
  ra = fma2(ra, fma2(neg2(om), ra, f2(1.f)), ra);
#endif
  // A pixel that does not take the Gaussian has om = 1 exactly, so ra = 1
  // exactly (the refined reciprocal of 1 is 1) and its state is unchanged.
  const float2 Ti = mul2(p.T, ra);
  const float2 vis = mul2(am, Ti);
  // The colour behind only enters through its dot product with the
  // upstream gradient, which accumulates directly: sum vis_i * dot(c_i, v).
  const float2 va = fma2(Ti, cpv, neg2(mul2(p.SK, ra)));
  p.SK = fma2(vis, cpv, p.SK);
  p.T = Ti;
  const bool gm0 = c0 && !sk0, gm1 = c1 && !sk1;
  const bool gg0 = gm0 && og.x <= 0.999f, gg1 = gm1 && og.y <= 0.999f;
  // vis is zero where the pixel does not take the Gaussian; only the
  // reference semantics drop contributors beyond that.
  const float2 visg = REF ? make_float2(gm0 ? vis.x : 0.f, gm1 ? vis.y : 0.f) : vis;
  const float2 av = mul2(al, va);
  const float2 vs = make_float2(gg0 ? -av.x : 0.f, gg1 ? -av.y : 0.f);
  const float2 vsdy = mul2(vs, dy);
  // |vs (a dx + b dy)| and |vs (b dx + c dy)| per pixel.
  const float2 avs = make_float2(fabsf(vs.x), fabsf(vs.y));
  const float2 g0 = fma2(f2(cb), dy, f2(adx)), g1 = fma2(f2(B.x), dy, f2(bdx));
  const float2 ag0 = make_float2(fabsf(g0.x), fabsf(g0.y)), ag1 = make_float2(fabsf(g1.x), fabsf(g1.y));
  const uint32_t nc = (gm0 ? 1u : 0u) + (gm1 ? 1u : 0u);
  if constexpr (FIRST_MOM) {
    mom.m0 = vs;
    mom.m1 = vsdy;
    mom.m2 = mul2(vsdy, dy);
  } else {
    mom.m0 = add2(mom.m0, vs);
    mom.m1 = add2(mom.m1, vsdy);
    mom.m2 = fma2(vsdy, dy, mom.m2);
  }
  if constexpr (FIRST_ACC) {
    acc.ax = mul2(avs, ag0);
    acc.ay = mul2(avs, ag1);
    acc.cr = mul2(visg, vr);
    acc.cg = mul2(visg, vg);
    acc.cb = mul2(visg, vb);
    acc.n = nc;
  } else {
    acc.ax = fma2(avs, ag0, acc.ax);
    acc.ay = fma2(avs, ag1, acc.ay);
    acc.cr = fma2(visg, vr, acc.cr);
    acc.cg = fma2(visg, vg, acc.cg);
    acc.cb = fma2(visg, vb, acc.cb);
    acc.n += nc;
  }
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// Deterministic mode: the partial sums of list entries [lo, hi), which no pixel
// got to, are zero.
__device__ __forceinline__ void zero_parts(float* part, uint32_t lo, uint32_t hi) {
  float4* p = reinterpret_cast<float4*>(part);
  for (size_t i = (size_t)lo * 3 + threadIdx.x; i < (size_t)hi * 3; i += blockDim.x)
    p[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// The backward walks the tile's list from its largest last-contributor
// index down in batches. Batches are double-buffered: while batch k is
// evaluated, the raw records of batch k + 1 are in flight (asynchronous
// copies into the other buffer) and the list entries of batch k + 2 (hit
// bits and compact indices) are loaded into registers. A warp owns one of the
// forward's 8x8 blocks, a lane a pixel pair of it.
template <int TW, int TH, int BATCH, bool REF, bool DET>
__global__ void __launch_bounds__(TW* TH / 2) raster_bwd_kernel(RasterArgs a) {
  static_assert(TW % 8 == 0 && TH % 8 == 0, "warp blocks tile the tile");
  constexpr int NT = TW * TH / 2;
  constexpr int NW = NT / 32;
  constexpr int kSI = (BATCH + NT - 1) / NT;  // entries a thread stages per batch
  __shared__ float4 s_rec[2][BATCH][3];        // raw records
  __shared__ uint32_t s_cidx[2][BATCH];
  __shared__ uint8_t s_mask[2][BATCH];         // blocks, and so warps, that take the entry
  __shared__ uint16_t s_list[NW][BATCH];
  __shared__ float4 s_part[NW][BATCH][3];      // written by the warps whose bit is set
  __shared__ uint32_t s_max;
  __shared__ uint32_t s_item;
  __shared__ CostListView s_lists;
  load_cost_lists(a, &s_lists);
  for (uint32_t round = 0;; ++round) {
    const uint32_t item = next_item<true>(a, round, &s_item, &s_lists);
    if (item == kNoItem) break;
    const uint32_t v = find_view(a.vs, item);
    const ViewDesc& vd = a.vs.views[v];
    const uint32_t t = item - vd.tile_base;
    const uint32_t tx = t % vd.tiles_x, ty = t / vd.tiles_x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t px = tx * TW + WarpBlock<TW>::x0(warp) + (lane & 7);
    const uint32_t pyb = ty * TH + WarpBlock<TW>::y0(warp) + (lane >> 3);
    const float pcx = (float)px + 0.5f;
    const uint32_t* ranges = slice(a.b.ranges, 2 * a.b.Tcap, v);
    const uint32_t s0 = ranges[2 * t];
    const uint32_t* vals = isect_index_src(a.b, v);
    const uint32_t vmask = isect_index_mask(a.b);
    const float4* rec = slice(a.b.rec, a.b.Vcap * 3, v);
    const uint8_t* hitw = slice(a.b.hitw, a.b.Icap, v);
    float4* sgrad = slice(a.b.sgrad, a.b.Vcap * 3, v);
    float* part = a.b.sgrad_part + (size_t)a.b.Icap * 12 * v;
    BwdPair pp;
    load_bwd_pair(a, vd, v, px, pyb, pp);
    const uint32_t mylast = max(pp.last0, pp.last1);
    if (threadIdx.x == 0) s_max = 0;
    __syncthreads();
    const uint32_t wmax = __reduce_max_sync(0xffffffffu, mylast);
    if (lane == 0) atomicMax(&s_max, wmax);
    __syncthreads();
    const uint32_t smax = s_max;
    const int slot = reduce12_slot(lane);                          // the gradient value this lane ends with
    const bool writer = (lane & 1) == 0 && !((lane & 2) && (lane & 4));  // one lane per value
    auto batch_lo = [&](uint32_t e) { return (e - s0 > (uint32_t)BATCH) ? e - BATCH : s0; };
    // List entries [lo, hi) of a batch into registers.
    uint32_t pc[kSI], ph[kSI];
    auto fetch = [&](uint32_t lo, uint32_t hi) {
  #pragma unroll
      for (int it = 0; it < kSI; ++it) {
        const uint32_t s = lo + threadIdx.x + it * NT;
        const bool ok = threadIdx.x + it * NT < (uint32_t)BATCH && s < hi;
        ph[it] = ok ? hitw[s] : 0u;
        pc[it] = ok ? (vals[s] & vmask) : 0u;
      }
    };
    // Masks, indices and record copies of the fetched batch [lo, hi) into
    // buffer `buf`; one commit group per call.
    auto issue = [&](uint32_t lo, uint32_t hi, int buf) {
  #pragma unroll
      for (int it = 0; it < kSI; ++it) {
        const uint32_t j = threadIdx.x + it * NT;
        if (j < (uint32_t)BATCH && lo + j < hi) {
          s_mask[buf][j] = (uint8_t)ph[it];  // the forward's 8x8 block bits
          if (ph[it]) {
            s_cidx[buf][j] = pc[it];
            const float4* r = rec + (size_t)pc[it] * 3;
            cp_async16(&s_rec[buf][j][0], r);
            cp_async16(&s_rec[buf][j][1], r + 1);
            cp_async16(&s_rec[buf][j][2], r + 2);
          }
        }
      }
      cp_async_commit();
    };
    uint32_t be = smax, bs = be > s0 ? batch_lo(be) : s0;
    if (be > s0) {
      fetch(bs, be);
      issue(bs, be, 0);
    }
    uint32_t nbe = bs, nbs = nbe > s0 ? batch_lo(nbe) : s0;
    if (nbe > s0) fetch(nbs, nbe);
    int buf = 0;
    while (be > s0) {
      const uint32_t nb = be - bs;
      if (nbe > s0)
        issue(nbs, nbe, buf ^ 1);
      else
        cp_async_commit();
      const uint32_t n2e = nbs, n2s = n2e > s0 ? batch_lo(n2e) : s0;
      if (n2e > s0) fetch(n2s, n2e);
      cp_async_wait1();  // this thread's copies of the current batch have landed
      __syncthreads();
      if (bs < wmax) {
        const int cnt = build_list(s_mask[buf], nb, 1u << warp, lane, s_list[warp]);
        for (int e = cnt - 1; e >= 0; --e) {
          const uint32_t j = s_list[warp][e];
          const uint32_t s = bs + j;
          const float4 r0 = s_rec[buf][j][0], r1 = s_rec[buf][j][1], r2 = s_rec[buf][j][2];
          const float4 A = make_float4(r0.x, r0.y, r0.z, 2.f * r0.w);  // 2b is exact
          const float4 B = make_float4(r1.x, r2.y + kRejectMargin, r1.y, 0.f);
          const float4 Cc = make_float4(r1.z, r1.w, r2.x, 0.f);
          const float dx = esub(A.x, pcx);
          const float t1 = emul(emul(A.z, dx), dx);
          const float t2 = emul(A.w, dx);
          const float cb = r0.w;  // the conic's b
          const float adx = A.z * dx, bdx = cb * dx;
          BwdMom mom;
          BwdAcc acc;
          const float cp0 = fmaxf(Cc.x, 0.f), cp1 = fmaxf(Cc.y, 0.f), cp2 = fmaxf(Cc.z, 0.f);
          const float2 npcy = make_float2(-((float)pyb + 0.5f), -((float)(pyb + 4) + 0.5f));
          const PairPre pre = bwd_pair_pre(pp, npcy, s, t1, t2, A, B);
          const float2 cpv = fma2(f2(cp2), pp.vb, fma2(f2(cp1), pp.vg, mul2(f2(cp0), pp.vr)));
          bwd_pair_rest<REF, true, true>(pp, pre, adx, bdx, cb, B, cpv, pp.vr, pp.vg, pp.vb, mom, acc);
          const float M0 = mom.m0.x + mom.m0.y, M1 = mom.m1.x + mom.m1.y, M2 = mom.m2.x + mom.m2.y;
          float x[12];
          x[0] = dx * M0;  // S1..S5 (the conic combination follows the CTA sum)
          x[1] = M1;
          x[2] = dx * x[0];
          x[3] = dx * M1;
          x[4] = M2;
          x[5] = acc.cr.x + acc.cr.y;
          x[6] = acc.cg.x + acc.cg.y;
          x[7] = acc.cb.x + acc.cb.y;
          x[8] = M0;
          x[9] = acc.ax.x + acc.ax.y;
          x[10] = acc.ay.x + acc.ay.y;
          x[11] = (float)acc.n;
          const float r = warp_reduce_scatter12(x, lane);
          float* sp = reinterpret_cast<float*>(&s_part[warp][j][0]);
          if (writer) sp[slot] = r;
        }
      }
      __syncthreads();
      for (uint32_t q = threadIdx.x; q < nb * 3; q += NT) {
        const uint32_t j = q / 3, k = q % 3;
        const uint32_t m = s_mask[buf][j];  // warps that wrote a slot
        float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
        bool any = false;
  #pragma unroll
        for (int w = 0; w < NW; ++w) {
          if (!((m >> w) & 1u)) continue;
          const float4 g = s_part[w][j][k];
          if (!any) {
            f = g;
            any = true;
          } else {
            f.x = f.x + g.x;
            f.y = f.y + g.y;
            f.z = f.z + g.z;
            f.w = f.w + g.w;
          }
        }
        if (any) {
          // The tile's S sums and sum vs into the screen-space gradients.
          if (k == 0) {
            const float4 r0 = s_rec[buf][j][0];
            const float cc = s_rec[buf][j][1].x;
            f = make_float4(r0.z * f.x + r0.w * f.y, r0.w * f.x + cc * f.y, 0.5f * f.z, f.w);
          } else if (k == 1) {
            // v_rgb is zero for a channel whose raw colour is negative.
            const float4 r1 = s_rec[buf][j][1];
            const float rb = s_rec[buf][j][2].x;
            f = make_float4(0.5f * f.x, r1.z < 0.f ? 0.f : f.y, r1.w < 0.f ? 0.f : f.z, rb < 0.f ? 0.f : f.w);
          } else {
            f.x = f.x != 0.f ? -f.x / s_rec[buf][j][1].y : 0.f;
          }
        }
        if (DET) {
          reinterpret_cast<float4*>(part + (size_t)(bs + j) * 12)[k] = f;
        } else if (f.x != 0.f || f.y != 0.f || f.z != 0.f || f.w != 0.f) {
          atomicAdd(sgrad + (size_t)s_cidx[buf][j] * 3 + k, f);
        }
      }
      __syncthreads();  // the next batch's copies reuse this buffer
      be = bs;
      bs = nbs;
      nbe = n2e;
      nbs = n2s;
      buf ^= 1;
    }
    if (DET) zero_parts(part, max(smax, s0), ranges[2 * t + 1]);
    asm volatile("cp.async.wait_all;" ::: "memory");  // no copy may outlive the block
  }
}

// The backward of 16x16 tiles with one warp per tile. Lane l owns, in each
// of the tile's four 8x8 blocks q (block column q & 1, block row q >> 1), the
// pixel pair (8 (q & 1) + (l & 7), 8 (q >> 1) + (l >> 3) + {0, 4}), so that
// pair q lies in the forward's warp block q and an entry's block bits say
// which pairs need it. Against two warps per tile, each list entry is staged,
// set up and reduced once per tile rather than once per warp whose block it
// reaches, and the tile's sum needs no second warp. The pairs of a block
// column share dx and the terms that depend on it; the sigma-gradient
// moments are kept per column (S1 = dx0 M0_0 + dx1 M0_1 and so on).
// SEG: an item is one segment of a tile's list (launches of few tiles, see
// pick_segments). Its pixels start from the forward's checkpoint at the
// segment's end: the transmittance there, and the colour behind it, which
// enters as its dot product with the upstream gradient. The segment's entries
// are then walked as a whole tile's are.
template <int BATCH, bool REF, bool SEG, bool DET>
__global__ void __launch_bounds__(32, kTileBwdBlocks) raster_bwd_tile_kernel(RasterArgs a) {
  constexpr int NT = 32;
  constexpr int kSI = BATCH / NT;  // entries a lane stages per batch
  static_assert(BATCH % NT == 0, "whole batches per lane");
  __shared__ float4 s_rec[2][BATCH][3];  // raw records
  __shared__ uint32_t s_cidx[2][BATCH];
  __shared__ uint8_t s_mask[2][BATCH];  // forward blocks that take the entry
  __shared__ uint16_t s_list[BATCH];
  __shared__ float4 s_part[BATCH][3];   // the tile's reduced sums of listed entries
  __shared__ float2 s_v[4][3][32];      // upstream colour gradient of each lane's pairs (read only)
  __shared__ uint32_t s_item;
  __shared__ CostListView s_lists;
  load_cost_lists(a, &s_lists);
  const int lane = threadIdx.x;
  const int slot = reduce12_slot(lane);                          // the gradient value this lane ends with
  const bool writer = (lane & 1) == 0 && !((lane & 2) && (lane & 4));  // one lane per value
  for (uint32_t round = 0;; ++round) {
    const uint32_t work = next_item<SEG>(a, round, &s_item, &s_lists);
    if (work == kNoItem) break;
    // The 8x8 blocks this item takes: all, or one of a long walk.
    const uint32_t blocks = work < (1u << kBlockShift) ? 0xfu : 1u << ((work >> kBlockShift) - 1u);
    const uint32_t id = work & ((1u << kBlockShift) - 1u);
    const uint32_t item = SEG ? id / a.b.seg_k : id, seg = SEG ? id % a.b.seg_k : 0u;
    const uint32_t v = find_view(a.vs, item);
    const ViewDesc& vd = a.vs.views[v];
    const uint32_t t = item - vd.tile_base;
    const uint32_t tx = t % vd.tiles_x, ty = t / vd.tiles_x;
    const uint32_t px0 = tx * 16 + (lane & 7), py0 = ty * 16 + (lane >> 3);
    const float pcx0 = (float)px0 + 0.5f, pcx1 = (float)(px0 + 8) + 0.5f;
    // Negated pixel-centre rows of the lane's pairs: block row h, half u at
    // row py0 + 8 h + 4 u (small integers plus 0.5: exact).
    const float npy[4] = {-((float)py0 + 0.5f), -((float)(py0 + 4) + 0.5f), -((float)(py0 + 8) + 0.5f),
                          -((float)(py0 + 12) + 0.5f)};
    const uint32_t* ranges = slice(a.b.ranges, 2 * a.b.Tcap, v);
    const uint32_t s0 = ranges[2 * t];
    const Segments segs = segments_of(ranges[2 * t + 1] - s0, SEG ? a.b.seg_k : 1u);
    const uint32_t* vals = isect_index_src(a.b, v);
    const uint32_t vmask = isect_index_mask(a.b);
    const float4* rec = slice(a.b.rec, a.b.Vcap * 3, v);
    const uint8_t* hitw = slice(a.b.hitw, a.b.Icap, v);
    float4* sgrad = slice(a.b.sgrad, a.b.Vcap * 3, v);
    float* part = a.b.sgrad_part + (size_t)a.b.Icap * 12 * v;
    BwdPair pp[4];
    uint32_t mylast = 0;
  #pragma unroll
    for (int q = 0; q < 4; ++q) {
      load_bwd_pair(a, vd, v, px0 + 8 * (q & 1), py0 + 8 * (q >> 1), pp[q]);
      if ((blocks >> q) & 1u) mylast = max(mylast, max(pp[q].last0, pp[q].last1));
      s_v[q][0][lane] = pp[q].vr;  // kept in shared memory, not registers
      s_v[q][1][lane] = pp[q].vg;
      s_v[q][2][lane] = pp[q].vb;
    }
    const uint32_t smax = __reduce_max_sync(0xffffffffu, mylast);
    // This segment's entries [lo, hi); the last segment ends at the tile's
    // last contributor and starts from the pixels' final state, the others
    // from their checkpoint.
    const uint32_t lo = SEG ? s0 + segs.begin(seg) : s0;
    if (SEG && seg > 0 && lo >= smax) continue;  // grid schedule: past the tile's segments
    const uint32_t end = SEG ? s0 + segs.begin(seg + 1) : 0u;
    const bool final_seg = !SEG || seg + 1 == a.b.seg_k || smax <= end;
    const uint32_t hi = final_seg ? smax : end;
    if (!final_seg) {
      const float4* ck = a.b.ckpt + (size_t)id * 256 + lane;
  #pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 u = ck[q * 32], w = ck[128 + q * 32];
        pp[q].T = make_float2(u.x, w.x);
        pp[q].SK = add2(pp[q].SK, fma2(make_float2(u.w, w.w), pp[q].vb,
                                       fma2(make_float2(u.z, w.z), pp[q].vg, mul2(make_float2(u.y, w.y), pp[q].vr))));
      }
    }
    auto batch_lo = [&](uint32_t e) { return (e - lo > (uint32_t)BATCH) ? e - BATCH : lo; };
    uint32_t pc[kSI], ph[kSI];
    auto fetch = [&](uint32_t lo, uint32_t hi) {
  #pragma unroll
      for (int it = 0; it < kSI; ++it) {
        const uint32_t s = lo + lane + it * NT;
        const bool ok = s < hi;
        ph[it] = ok ? hitw[s] & blocks : 0u;
        pc[it] = ok ? (vals[s] & vmask) : 0u;
      }
    };
    auto issue = [&](uint32_t lo, uint32_t hi, int buf) {
  #pragma unroll
      for (int it = 0; it < kSI; ++it) {
        const uint32_t j = lane + it * NT;
        if (lo + j < hi) {
          s_mask[buf][j] = (uint8_t)ph[it];
          if (ph[it]) {
            s_cidx[buf][j] = pc[it];
            const float4* r = rec + (size_t)pc[it] * 3;
            cp_async16(&s_rec[buf][j][0], r);
            cp_async16(&s_rec[buf][j][1], r + 1);
            cp_async16(&s_rec[buf][j][2], r + 2);
          }
        }
      }
      cp_async_commit();
    };
    uint32_t be = hi, bs = be > lo ? batch_lo(be) : lo;
    if (be > lo) {
      fetch(bs, be);
      issue(bs, be, 0);
    }
    uint32_t nbe = bs, nbs = nbe > lo ? batch_lo(nbe) : lo;
    if (nbe > lo) fetch(nbs, nbe);
    int buf = 0;
    while (be > lo) {
      const uint32_t nb = be - bs;
      if (nbe > lo)
        issue(nbs, nbe, buf ^ 1);
      else
        cp_async_commit();
      const uint32_t n2e = nbs, n2s = n2e > lo ? batch_lo(n2e) : lo;
      if (n2e > lo) fetch(n2s, n2e);
      cp_async_wait1();  // this lane's copies of the current batch have landed
      __syncthreads();   // and every lane's
      const int cnt = build_list(s_mask[buf], nb, 0xfu, lane, s_list);
      for (int e = cnt - 1; e >= 0; --e) {
        const uint32_t j = s_list[e];
        const uint32_t s = bs + j;
        const float4 r0 = s_rec[buf][j][0], r1 = s_rec[buf][j][1], r2 = s_rec[buf][j][2];
        const float4 A = make_float4(r0.x, r0.y, r0.z, 2.f * r0.w);  // 2b is exact
        const float4 B = make_float4(r1.x, r2.y + kRejectMargin, r1.y, 0.f);
        const float cb = r0.w;  // the conic's b
        const float cp0 = fmaxf(r1.z, 0.f), cp1 = fmaxf(r1.w, 0.f), cp2 = fmaxf(r2.x, 0.f);
        const uint32_t need = s_mask[buf][j];  // bit q: pair q takes part
        const float dx0 = esub(A.x, pcx0), dx1 = esub(A.x, pcx1);
        BwdMom mom0, mom1;
        BwdAcc acc;
        constexpr std::integral_constant<bool, true> kT{};
        constexpr std::integral_constant<bool, false> kF{};
        // The pairs of block column c (q = c upper, q = c + 2 lower) as one
        // straight-line block; FM: the column's first pair sets its moments,
        // FA: the entry's first pair sets the shared sums.
        auto column = [&](auto cc, auto fa, BwdMom& mom) {
          constexpr int c = decltype(cc)::value;
          constexpr bool FA = decltype(fa)::value;
          const float dx = c ? dx1 : dx0;
          const float t1 = emul(emul(A.z, dx), dx);
          const float t2 = emul(A.w, dx);
          const float adx = A.z * dx, bdx = cb * dx;
          auto rest = [&](auto qq, auto fm, auto fa2) {
            constexpr int q = decltype(qq)::value;
            const float2 npcy = make_float2(npy[2 * (q >> 1)], npy[2 * (q >> 1) + 1]);
            const PairPre pre = bwd_pair_pre(pp[q], npcy, s, t1, t2, A, B);
            const float2 vr = s_v[q][0][lane], vg = s_v[q][1][lane], vb = s_v[q][2][lane];
            const float2 cpv = fma2(f2(cp2), vb, fma2(f2(cp1), vg, mul2(f2(cp0), vr)));
            bwd_pair_rest<REF, decltype(fm)::value, decltype(fa2)::value>(pp[q], pre, adx, bdx, cb, B, cpv, vr, vg,
                                                                          vb, mom, acc);
          };
          const uint32_t nc = (need >> c) & 5u;  // bit 0: upper pair, bit 2: lower pair
          if (nc == 5u) {
            rest(std::integral_constant<int, c>{}, kT, std::integral_constant<bool, FA>{});
            rest(std::integral_constant<int, c + 2>{}, kF, kF);
          } else if (nc == 1u) {
            rest(std::integral_constant<int, c>{}, kT, std::integral_constant<bool, FA>{});
          } else {
            rest(std::integral_constant<int, c + 2>{}, kT, std::integral_constant<bool, FA>{});
          }
        };
        if (need & 5u) {
          column(std::integral_constant<int, 0>{}, kT, mom0);
        } else {
          mom0.m0 = mom0.m1 = mom0.m2 = acc.cr = acc.cg = acc.cb = acc.ax = acc.ay = f2(0.f);
          acc.n = 0u;
        }
        if (need & 10u)
          column(std::integral_constant<int, 1>{}, kF, mom1);
        else
          mom1.m0 = mom1.m1 = mom1.m2 = f2(0.f);
        const float M00 = mom0.m0.x + mom0.m0.y, M01 = mom1.m0.x + mom1.m0.y;
        const float M10 = mom0.m1.x + mom0.m1.y, M11 = mom1.m1.x + mom1.m1.y;
        const float e0 = dx0 * M00, e1 = dx1 * M01;
        float x[12];
        x[0] = e0 + e1;  // S1..S5 (the conic combination follows the reduction)
        x[1] = M10 + M11;
        x[2] = dx0 * e0 + dx1 * e1;
        x[3] = dx0 * M10 + dx1 * M11;
        x[4] = (mom0.m2.x + mom0.m2.y) + (mom1.m2.x + mom1.m2.y);
        x[5] = acc.cr.x + acc.cr.y;
        x[6] = acc.cg.x + acc.cg.y;
        x[7] = acc.cb.x + acc.cb.y;
        x[8] = M00 + M01;
        x[9] = acc.ax.x + acc.ax.y;
        x[10] = acc.ay.x + acc.ay.y;
        x[11] = (float)acc.n;
        const float r = warp_reduce_scatter12(x, lane);
        if (writer) reinterpret_cast<float*>(&s_part[j][0])[slot] = r;
      }
      __syncwarp();
      for (uint32_t qi = lane; qi < nb * 3; qi += NT) {
        const uint32_t j = qi / 3, k = qi % 3;
        float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
        if (s_mask[buf][j]) {
          f = s_part[j][k];
          if (k == 0) {
            const float4 r0 = s_rec[buf][j][0];
            const float cc = s_rec[buf][j][1].x;
            f = make_float4(r0.z * f.x + r0.w * f.y, r0.w * f.x + cc * f.y, 0.5f * f.z, f.w);
          } else if (k == 1) {
            // v_rgb is zero for a channel whose raw colour is negative.
            const float4 r1 = s_rec[buf][j][1];
            const float rb = s_rec[buf][j][2].x;
            f = make_float4(0.5f * f.x, r1.z < 0.f ? 0.f : f.y, r1.w < 0.f ? 0.f : f.z, rb < 0.f ? 0.f : f.w);
          } else {
            f.x = f.x != 0.f ? -f.x / s_rec[buf][j][1].y : 0.f;
          }
        }
        if (DET) {
          if (!SEG || s_mask[buf][j]) reinterpret_cast<float4*>(part + (size_t)(bs + j) * 12)[k] = f;
        } else if (f.x != 0.f || f.y != 0.f || f.z != 0.f || f.w != 0.f) {
          atomicAdd(sgrad + (size_t)s_cidx[buf][j] * 3 + k, f);
        }
      }
      __syncthreads();  // the next batch's copies reuse this buffer
      be = bs;
      bs = nbs;
      nbe = n2e;
      nbs = n2s;
      buf ^= 1;
    }
    if (DET && !SEG) zero_parts(part, max(smax, s0), ranges[2 * t + 1]);
    asm volatile("cp.async.wait_all;" ::: "memory");  // no copy may outlive the block
  }
}

// A split forward's CTAs set the hit bits of their blocks one by one.
__global__ void __launch_bounds__(256) zero_hits_kernel(FwdBufs b) {
  const uint32_t v = blockIdx.y, n = b.vcount[v * 4 + 1];
  uint8_t* hitw = slice(b.hitw, b.Icap, v);
  // Whole 16-byte words and the ragged ends.
  const uint32_t head = min(n, (uint32_t)(-reinterpret_cast<uintptr_t>(hitw) & 15)), words = (n - head) / 16;
  const uint32_t i0 = blockIdx.x * 256 + threadIdx.x;
  uint4* mid = reinterpret_cast<uint4*>(hitw + head);
  for (uint32_t i = i0; i < words; i += gridDim.x * 256) mid[i] = make_uint4(0, 0, 0, 0);
  if (i0 < head) hitw[i0] = 0;
  if (i0 < n - head - words * 16) hitw[head + words * 16 + i0] = 0;
}

// Deterministic mode of a segmented backward: zero partial sums for every
// intersection; the backward then writes those of the entries that some pixel
// took. Most list entries lie behind saturated pixels, and a plain sweep at HBM
// rate clears them faster than a warp per tile would. With more tiles, or smaller
// ones, the stores hide behind other items' arithmetic and the backward clears its
// own lists' rest: 4 views of 1280x720 over 300k Gaussians 0.80 ms with the sweep,
// 0.73 so, in 8x8 tiles 1.22 and 0.96.
__global__ void __launch_bounds__(256) zero_parts_kernel(FwdBufs b) {
  const uint32_t v = blockIdx.y;
  const uint64_t n = (uint64_t)b.vcount[v * 4 + 1] * 3;
  float4* part = reinterpret_cast<float4*>(b.sgrad_part + (size_t)b.Icap * 12 * v);
  for (uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (uint64_t)gridDim.x * 256)
    part[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// Gaussians per shared-memory batch: 0 selects the tuned defaults (128 in
// the forward, 64 in the backward); other values round up to 64, 128 or 256.
// The backward of shapes with two or more warps per tile caps at 128 (its
// double-buffered records and per-warp partial sums would not fit the 48 KB
// of static shared memory).
inline int pick_batch(uint32_t want, int dflt) {
  if (want == 0) return dflt;
  return want <= 64 ? 64 : (want <= 128 ? 128 : 256);
}

// Launches kernel over the launch's work items: one CTA per item (grid
// schedule), or as many CTAs as the SMs hold at once (persistent schedule;
// the residency of each instantiation is looked up once).
// Resident CTAs per SM of a raster kernel instantiation, looked up once
// (context creation warms it up, so that a first launch inside a stream
// capture needs no lookup).
template <void (*Kernel)(RasterArgs)> int resident_per_sm(int threads) {
  static int per_sm = 0;  // one per kernel instantiation
  if (per_sm <= 0) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, Kernel, threads, 0) != cudaSuccess || n < 1) {
      (void)cudaGetLastError();
      n = 1;
    }
    per_sm = n;
  }
  return per_sm;
}

template <void (*Kernel)(RasterArgs)>
cudaError_t launch_items(int threads, const RasterArgs& a, uint32_t items, int num_sms, cudaStream_t st) {
  uint32_t grid = items;
  if (a.persist)
    grid = std::min<uint32_t>(grid, (uint32_t)resident_per_sm<Kernel>(threads) * (uint32_t)std::max(num_sms, 1));
  if (grid == 0) return cudaSuccess;  // a warm-up call (no items)
  Kernel<<<grid, threads, 0, st>>>(a);
  return cudaGetLastError();
}

template <int TW, int TH, int BATCH, bool CKPT, bool SPLIT>
cudaError_t launch_fwd_batch(const RasterArgs& a, int num_sms, cudaStream_t st) {
  return launch_items<raster_fwd_kernel<TW, TH, BATCH, CKPT, SPLIT>>(SPLIT ? 64 : TW * TH / 2, a,
                                                                     a.vs.total_tiles * (SPLIT ? 4 : 1), num_sms, st);
}
template <int TW, int TH>
cudaError_t launch_fwd_shape(const RasterArgs& a, uint32_t batch, int num_sms, cudaStream_t st) {
  switch (pick_batch(batch, 128)) {
    case 64: return launch_fwd_batch<TW, TH, 64, false, false>(a, num_sms, st);
    case 128: return launch_fwd_batch<TW, TH, 128, false, false>(a, num_sms, st);
    default: return launch_fwd_batch<TW, TH, 256, false, false>(a, num_sms, st);
  }
}
// 16x16 tiles: with checkpoints when the backward is segmented.
cudaError_t launch_fwd_16(const RasterArgs& a, uint32_t batch, int num_sms, cudaStream_t st) {
  if (a.b.seg_k == 1) return launch_fwd_shape<16, 16>(a, batch, num_sms, st);
  if (a.split) return launch_fwd_batch<16, 16, 64, true, true>(a, num_sms, st);
  switch (pick_batch(batch, 64)) {
    case 64: return launch_fwd_batch<16, 16, 64, true, false>(a, num_sms, st);
    case 128: return launch_fwd_batch<16, 16, 128, true, false>(a, num_sms, st);
    default: return launch_fwd_batch<16, 16, 256, true, false>(a, num_sms, st);
  }
}
template <int TW, int TH, bool REF, bool DET>
cudaError_t launch_bwd_mode(const RasterArgs& a, uint32_t batch, int num_sms, cudaStream_t st) {
  constexpr int NT = TW * TH / 2;
  constexpr int kMaxBatch = NT / 32 >= 2 ? 128 : 256;
  const uint32_t items = a.vs.total_tiles;
  int b = pick_batch(batch, 64);
  if (b > kMaxBatch) b = kMaxBatch;
  switch (b) {
    case 64: return launch_items<raster_bwd_kernel<TW, TH, 64, REF, DET>>(NT, a, items, num_sms, st);
    case 128: return launch_items<raster_bwd_kernel<TW, TH, 128, REF, DET>>(NT, a, items, num_sms, st);
    default:
      return launch_items<raster_bwd_kernel<TW, TH, (kMaxBatch > 128 ? 256 : 128), REF, DET>>(NT, a, items,
                                                                                               num_sms, st);
  }
}
template <int TW, int TH>
cudaError_t launch_bwd_shape(const RasterArgs& a, uint32_t batch, bool det, int num_sms, cudaStream_t st) {
  if (det)
    return a.ref_mode ? launch_bwd_mode<TW, TH, true, true>(a, batch, num_sms, st)
                      : launch_bwd_mode<TW, TH, false, true>(a, batch, num_sms, st);
  return a.ref_mode ? launch_bwd_mode<TW, TH, true, false>(a, batch, num_sms, st)
                    : launch_bwd_mode<TW, TH, false, false>(a, batch, num_sms, st);
}
// 16x16 tiles: one warp per (tile, segment). It stages 64 entries per batch
// whatever the forward's batch: 13 KB of shared memory and at most 128
// registers per one-warp CTA let 16 CTAs share an SM (a 128-entry batch would
// fit 9).
template <bool REF, bool DET>
cudaError_t launch_bwd_tile16(const RasterArgs& a, int num_sms, cudaStream_t st) {
  const uint32_t items = a.vs.total_tiles * a.b.seg_k;
  return a.b.seg_k > 1 ? launch_items<raster_bwd_tile_kernel<kTileBwdBatch, REF, true, DET>>(32, a, items, num_sms, st)
                       : launch_items<raster_bwd_tile_kernel<kTileBwdBatch, REF, false, DET>>(32, a, items, num_sms, st);
}
cudaError_t launch_bwd_16(const RasterArgs& a, bool det, int num_sms, cudaStream_t st) {
  if (det) return a.ref_mode ? launch_bwd_tile16<true, true>(a, num_sms, st) : launch_bwd_tile16<false, true>(a, num_sms, st);
  return a.ref_mode ? launch_bwd_tile16<true, false>(a, num_sms, st) : launch_bwd_tile16<false, false>(a, num_sms, st);
}

// Segments a tile's list is cut into for the backward of this launch (1: none).
// A launch of few tiles waits for its longest list, one entry after another;
// segments spread it over the idle SMs, for a forward that writes a checkpoint
// per segment. Forward plus backward, without and with: 256 tiles (16k
// Gaussians) 0.295 -> 0.105 ms, 300 tiles (74k) 0.465 -> 0.181, 1200 tiles
// (200k) 0.303 -> 0.218, 3600 tiles (500k, 4 segments) 0.377 -> 0.373. With 2
// segments each it costs more than it gives: 5800 tiles 0.650 -> 0.661, 8160
// tiles 0.702 -> 0.733. So at least 4, that is at most 4096 tiles.
uint32_t pick_segments(const ViewSet& vs) {
  if (vs.tile_w != 16 || vs.tile_h != 16 || vs.total_tiles == 0) return 1;
  const uint32_t k = std::min(kSegMax, kSegItems / vs.total_tiles);
  return k < 4 ? 1 : k;
}

}  // namespace

void raster_warm_up(uint32_t tile_w, uint32_t tile_h, uint32_t batch, int deterministic, int num_sms) {
  const bool det = deterministic != 0;
  RasterArgs a{};
  a.persist = 1;  // total_tiles 0: the launchers only look up the residency
  a.vs.batch = batch;
  for (int ref = 0; ref < 2; ++ref) {
    a.ref_mode = ref;
    if (tile_w == 16 && tile_h == 16) {
      a.b.seg_k = 1;
      (void)launch_fwd_16(a, batch, num_sms, nullptr);
      (void)launch_bwd_16(a, det, num_sms, nullptr);
      a.b.seg_k = 2;
      for (a.split = 0; a.split < 2; ++a.split) (void)launch_fwd_16(a, batch, num_sms, nullptr);
      (void)launch_bwd_16(a, det, num_sms, nullptr);
    } else if (tile_w == 8 && tile_h == 8) {
      (void)launch_fwd_shape<8, 8>(a, batch, num_sms, nullptr);
      (void)launch_bwd_shape<8, 8>(a, batch, det, num_sms, nullptr);
    } else if (tile_w == 32 && tile_h == 8) {
      (void)launch_fwd_shape<32, 8>(a, batch, num_sms, nullptr);
      (void)launch_bwd_shape<32, 8>(a, batch, det, num_sms, nullptr);
    }
  }
}

cudaError_t launch_raster_fwd(const ViewSet& vs, FwdBufs& b, const float* bg, float* out_rgba, int deterministic,
                              const Scratch& s, cudaStream_t st) {
  b.seg_k = pick_segments(vs);
  RasterArgs a{};
  a.vs = vs;
  a.b = b;
  a.bg[0] = bg[0];
  a.bg[1] = bg[1];
  a.bg[2] = bg[2];
  a.out_rgba = out_rgba;
  a.long_tiles = !deterministic;  // the blocks' sums of an entry meet in an atomic add
  cudaError_t e;
  if (vs.total_tiles == 0) return cudaSuccess;
  a.split = vs.tile_w == 16 && vs.tile_h == 16 && vs.total_tiles <= kFwdSplitTiles &&
            (uint64_t)vs.n_splats >= (uint64_t)kFwdSplitSplats * vs.total_tiles;
  // The CTAs of a split tile leave checkpoints and meet in tile_sync, which the
  // projection cleared, as it did the cost lists' counts.
  static_assert(kFwdSplitTiles <= kSegItems / 4, "split tiles leave checkpoints");
  if (a.split) {
    zero_hits_kernel<<<dim3(std::max(1, s.num_sms * 2 / (int)vs.n_views), vs.n_views), 256, 0, st>>>(b);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  a.persist = (vs.persistent & kPersistFwd) != 0 ? 1 : 0;
  if (a.persist) {
    sched_order_kernel<<<1, kOrderThreads, 0, st>>>(vs, b);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  if (vs.tile_w == 16 && vs.tile_h == 16) return launch_fwd_16(a, vs.batch, s.num_sms, st);
  if (vs.tile_w == 8 && vs.tile_h == 8) return launch_fwd_shape<8, 8>(a, vs.batch, s.num_sms, st);
  if (vs.tile_w == 32 && vs.tile_h == 8) return launch_fwd_shape<32, 8>(a, vs.batch, s.num_sms, st);
  return cudaErrorInvalidValue;
}

cudaError_t launch_raster_bwd(const ViewSet& vs, FwdBufs& b, const float* bg, const float* v_rgba, int ref_mode,
                              int deterministic, const Scratch& s, cudaStream_t st) {
  RasterArgs a{};
  a.vs = vs;
  a.b = b;
  a.bg[0] = bg[0];
  a.bg[1] = bg[1];
  a.bg[2] = bg[2];
  a.v_rgba = v_rgba;
  a.ref_mode = ref_mode;
  const bool det = deterministic != 0;
  cudaError_t e = cudaSuccess;
  if (!det) {
    e = cudaMemsetAsync(b.sgrad, 0, sizeof(float4) * 3 * b.Vcap * vs.n_views, st);
  } else if (b.seg_k > 1) {
    zero_parts_kernel<<<dim3(std::max(1, s.num_sms * 8 / (int)vs.n_views), vs.n_views), 256, 0, st>>>(b);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) return e;
  if (vs.total_tiles == 0) return cudaSuccess;
  a.persist = (vs.persistent & kPersistBwd) != 0 ? 2 : 0;
  if (a.persist) {
    e = cudaMemsetAsync(b.sched_ticket, 0, sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
  }
  if (vs.tile_w == 16 && vs.tile_h == 16) return launch_bwd_16(a, det, s.num_sms, st);
  if (vs.tile_w == 8 && vs.tile_h == 8) return launch_bwd_shape<8, 8>(a, vs.batch, det, s.num_sms, st);
  if (vs.tile_w == 32 && vs.tile_h == 8) return launch_bwd_shape<32, 8>(a, vs.batch, det, s.num_sms, st);
  return cudaErrorInvalidValue;
}

}  // namespace gsr
