// k_project.cu — projection, SH colour, tile counting and compaction.
//
// Three passes over every Gaussian and every view of the launch
// (project_forward.wgsl:19-96, project_visible.wgsl:130-214):
//  1. visibility: one thread per Gaussian projects it in every view and
//     records warp ballot words and per-block visible counts;
//  2. one block per view scans the block counts;
//  3. records: the visible Gaussians' compact indices follow in global-id
//     order from the block base, the earlier warps' and lanes' bits; the
//     projection is recomputed and the SH colour evaluated from the block's
//     SH rows, staged in shared memory with coalesced asynchronous copies.
// What bounds it: instruction issue with many views (0.7 to 0.8 of the slots in
// passes 1 and 3), loads in flight with one. So what depends on the view alone
// is computed once per block (the Jacobian's limits, the tile sides'
// reciprocals), the cameras are launch arguments, and shared memory holds the SH
// rows alone, in their storage type, for more blocks per SM; each thread reads
// its own transform row (40 bytes; the lines are used up by the warp). Together:
// 3M BF16 Gaussians in one view 359 -> 200 us, 500k FP32 82 -> 64, 1M FP32 in
// 8 views 371 -> 308, 2M BF16 in 16 views 1282 -> 1064.
// The first pass also puts the view descriptors into device memory, and the two
// clear what the later stages count in: a launch and three memsets less, 2 to
// 3 us each (train step of 74k Gaussians, 320x240, 276.6 -> 268.3 us; forward of
// 16k, 256x256, 141 -> 136 us).
// No block waits on another: one pass that took its compact base from the blocks
// before it by look-back was as fast with 8 and 16 views but slower with one (3M
// Gaussians 354 -> 403 us, 500k 76 -> 88), for its blocks mostly waited.
// The tiles each visible Gaussian touches are
// counted afterwards by the warp-cooperative walk over the compact records.
// This replaces the atomic compaction of project_forward.wgsl:94-96
// (nondeterministic order) and fuses the separate project_visible pass.
//
// Projected record, three float4 per visible Gaussian:
//   r0 = (x, y, conic_a, conic_b)
//   r1 = (conic_c, opacity, red, green)
//   r2 = (blue, log(255*opacity), tile box x0 | x1 << 16, tile box y0 | y1 << 16)
#include <cuda_bf16.h>

#include <cstring>
#include <type_traits>

#include "gsr_kernels.h"

namespace gsr {

namespace {

constexpr int kProjThreads = (int)kProjBlock;

struct ProjectArgs {
  SplatsDev sp;
  ViewSet vs;
  float cov_blur;
  int hp;
  FwdBufs b;
  uint32_t parts;       // blocks of kProjThreads Gaussians
  uint32_t words;       // visibility words per view (parts * warps per block)
  uint32_t* vis_bits;   // [views][words]
  uint32_t* blk_count;  // [views][parts]
  uint32_t* blk_base;   // [views][parts]
  ViewDesc* views;      // device copy of the descriptors
};

// The block's SH rows live in shared memory. Rows of whole 16- or 8-byte units
// (degrees 1 and 3) keep their storage type, have an odd stride in units and are
// moved and read a unit at a time; the others are FP32 with an odd stride in
// words. Either way a warp reading its 32 rows meets no bank conflict.
template <class SHT, int DEG> struct ShRows {
  static constexpr int kN = 3 * (DEG + 1) * (DEG + 1);
  static constexpr int kRowBytes = kN * (int)sizeof(SHT);
  static constexpr int kUnit = kRowBytes % 16 == 0 ? 16 : kRowBytes % 8 == 0 ? 8 : 0;
  static constexpr int kPer = kUnit ? kUnit / (int)sizeof(SHT) : 1;  // elements per unit
  using Store = typename std::conditional<kUnit != 0, SHT, float>::type;
  static constexpr int kStride = kPer * ((kN / kPer) | 1);
  static constexpr size_t kBytes = sizeof(Store) * kProjThreads * kStride;
  __device__ static uint32_t place(uint32_t e) { return (e / kN) * kStride + e % kN; }
};

__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// Stages the SH rows of Gaussians g0 .. g0 + rows - 1 (global element order,
// coalesced, by units where the array allows it), asynchronously where the copy
// is of whole words (completed by sh_rows_wait).
template <class SHT, int DEG>
__device__ __forceinline__ void sh_rows_issue(const SHT* sh, uint32_t g0, uint32_t rows,
                                              typename ShRows<SHT, DEG>::Store* s_sh) {
  using L = ShRows<SHT, DEG>;
  const SHT* src = sh + (size_t)g0 * L::kN;
  if (L::kUnit && (reinterpret_cast<uintptr_t>(sh) & (L::kUnit - 1)) == 0) {
    for (uint32_t q = threadIdx.x; q < rows * (L::kN / L::kPer); q += kProjThreads) {
      if (L::kUnit == 16) cp_async16(s_sh + L::place(L::kPer * q), src + L::kPer * q);
      else cp_async8(s_sh + L::place(L::kPer * q), src + L::kPer * q);
    }
  } else {
    for (uint32_t e = threadIdx.x; e < rows * L::kN; e += kProjThreads) {
      if constexpr (sizeof(SHT) == 4) {
        cp_async4(s_sh + L::place(e), src + e);
      } else {
        s_sh[L::place(e)] = src[e];
      }
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void sh_rows_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Element e of a staged row (e known at compile time).
template <class SHT, int DEG>
__device__ __forceinline__ float sh_at(const typename ShRows<SHT, DEG>::Store* row, int e) {
  using L = ShRows<SHT, DEG>;
  if constexpr (L::kUnit == 0) {
    return row[e];
  } else {
    using Unit = typename std::conditional<L::kUnit == 16, uint4, uint2>::type;
    const Unit x = *reinterpret_cast<const Unit*>(row + e / L::kPer * L::kPer);
    const int word = e % L::kPer * (int)sizeof(SHT) / 4;
    uint32_t w = word == 0 ? x.x : x.y;
    if constexpr (L::kUnit == 16) w = word == 2 ? x.z : word == 3 ? x.w : w;
    if constexpr (sizeof(SHT) == 4) return __uint_as_float(w);
    else return __uint_as_float((e & 1) ? w & 0xffff0000u : w << 16);  // BF16 is the upper half of FP32
  }
}

struct GaussParams {
  V3<float> mean{0.f, 0.f, 0.f};
  V4<float> quat{1.f, 0.f, 0.f, 0.f};
  V3<float> ls{0.f, 0.f, 0.f};
  float raw = 0.f;
};
// The thread's own row: 40 bytes, 8-byte aligned (the array is 16-byte aligned).
__device__ __forceinline__ GaussParams load_params(const SplatsDev& sp, uint32_t g, bool valid) {
  GaussParams q;
  if (valid) {
    const float2* t = reinterpret_cast<const float2*>(sp.transforms + (size_t)g * 10);
    const float2 t0 = __ldg(t), t1 = __ldg(t + 1), t2 = __ldg(t + 2), t3 = __ldg(t + 3), t4 = __ldg(t + 4);
    q.mean = V3<float>{t0.x, t0.y, t1.x};
    q.quat = V4<float>{t1.y, t2.x, t2.y, t3.x};
    q.ls = V3<float>{t3.y, t4.x, t4.y};
    q.raw = __ldg(sp.raw_opac + g);
  }
  return q;
}
// The view descriptors travel as launch arguments (constant memory: the per-view
// camera is an operand, not a load). One view has instances of its own: the full
// block is 6.6 KB, which costs a launch 1 to 2 us (forward of 16k Gaussians,
// 256x256: 140 us with it, 134 so, the loop over views gone too).
template <int NV> struct ViewArgs {
  ViewDesc v[NV];
};

// Pass 1: visibility of every Gaussian in every view. Each warp's ballot
// word goes to vis_bits[view][warp], each block's count to
// blk_count[view][block].
template <int NV>
__global__ void __launch_bounds__(kProjThreads)
    visibility_kernel(const ProjectArgs a, const __grid_constant__ ViewArgs<NV> blk) {
  constexpr int kWarps = kProjThreads / 32;
  __shared__ uint32_t s_cnt[NV][kWarps];
  __shared__ CamLimits<float> s_lim[NV];
  const uint32_t n = a.sp.n, nv = NV == 1 ? 1u : a.vs.n_views;
  const uint32_t part = blockIdx.x;
  const uint32_t g0 = part * kProjThreads;
  const uint32_t rows = min(n - g0, (uint32_t)kProjThreads);
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  if (part == 0)
    for (uint32_t v = threadIdx.x; v < nv; v += kProjThreads) a.views[v] = blk.v[v];
  // Counters of the later stages: tile counts, and the cost lists' counts with
  // the split tiles' meeting places and the flag of pass 3 behind them.
  for (uint32_t v = 0; v < nv; ++v)
    for (uint32_t t = g0 + threadIdx.x; t < blk.v[v].tiles_x * blk.v[v].tiles_y; t += a.parts * kProjThreads)
      slice(a.b.tile_hist, a.b.Tcap, v)[t] = 0u;
  for (uint32_t t = g0 + threadIdx.x; t < kSchedWords; t += a.parts * kProjThreads) a.b.sched_lcount[t] = 0u;
  if (threadIdx.x < nv) s_lim[threadIdx.x] = cam_limits(cam_from_desc<float>(blk.v[threadIdx.x]));
  const GaussParams q = load_params(a.sp, g0 + threadIdx.x, threadIdx.x < rows);
  __syncthreads();
  const bool valid = threadIdx.x < rows;
  const V2<float> inv_tile{1.f / (float)a.vs.tile_w, 1.f / (float)a.vs.tile_h};
  const GaussWorld<float> gw = gauss_world(q.quat, q.ls, q.raw);  // once for all views
  for (uint32_t v = 0; v < nv; ++v) {
    const ViewDesc& vd = blk.v[v];
    const Cam<float> cam = cam_from_desc<float>(vd);
    bool vis = false;
    if (valid)
      vis = project_gaussian_w(cam, s_lim[v], q.mean, gw, a.cov_blur, inv_tile, vd.tiles_x, vd.tiles_y, a.hp != 0)
                .visible;
    const uint32_t m = __ballot_sync(0xffffffffu, vis);
    if (lane == 0) {
      a.vis_bits[(size_t)v * a.words + part * kWarps + warp] = m;
      s_cnt[v][warp] = (uint32_t)__popc(m);
    }
  }
  __syncthreads();
  if (threadIdx.x < nv) {
    uint32_t tot = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) tot += s_cnt[threadIdx.x][w];
    a.blk_count[(size_t)threadIdx.x * a.parts + part] = tot;
  }
}

// Pass 2: per view (one block each), the exclusive scan of the block counts
// in block order and the view's visible count.
constexpr int kBlkScanThreads = 1024;
__global__ void __launch_bounds__(kBlkScanThreads) block_scan_kernel(ProjectArgs a) {
  __shared__ uint32_t s_scan[32];
  __shared__ uint32_t s_carry;
  const uint32_t v = blockIdx.x;
  const uint32_t* cnt = a.blk_count + (size_t)v * a.parts;
  uint32_t* base = a.blk_base + (size_t)v * a.parts;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (uint32_t p0 = 0; p0 < a.parts; p0 += kBlkScanThreads) {
    const uint32_t p = p0 + threadIdx.x;
    const uint32_t x = p < a.parts ? cnt[p] : 0u;
    uint32_t tot;
    const uint32_t e = block_exclusive_scan(x, s_scan, &tot);
    const uint32_t carry = s_carry;
    if (p < a.parts) base[p] = carry + e;
    __syncthreads();
    if (threadIdx.x == 0) s_carry = carry + tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) a.b.vcount[v * 4 + 0] = s_carry;
}

// Pass 3: the visible Gaussians' records at their compact indices in
// global-id order (block base + warps before + lanes before); the
// projection is recomputed (the same expression on the same inputs), the SH
// colour is evaluated from the block's staged SH rows.
template <class SHT, int DEG, int NV>
__global__ void __launch_bounds__(kProjThreads)
    records_kernel(const ProjectArgs a, const __grid_constant__ ViewArgs<NV> blk) {
  constexpr int kWarps = kProjThreads / 32;
  extern __shared__ float4 s_sh4[];  // rows of kStride elements
  using Rows = ShRows<SHT, DEG>;
  auto* s_sh = reinterpret_cast<typename Rows::Store*>(s_sh4);
  __shared__ uint32_t s_mask[NV][kWarps];
  __shared__ uint32_t s_wpre[NV][kWarps];
  __shared__ uint32_t s_base[NV];
  __shared__ CamLimits<float> s_lim[NV];
  const uint32_t n = a.sp.n, nv = NV == 1 ? 1u : a.vs.n_views;
  const uint32_t part = blockIdx.x;
  const uint32_t g0 = part * kProjThreads;
  const uint32_t g = g0 + threadIdx.x;
  const uint32_t rows = min(n - g0, (uint32_t)kProjThreads);
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  sh_rows_issue<SHT, DEG>(reinterpret_cast<const SHT*>(a.sp.sh), g0, rows, s_sh);
  for (uint32_t i = threadIdx.x; i < nv * kWarps; i += kProjThreads) {
    const uint32_t v = i / kWarps, w = i % kWarps;
    s_mask[v][w] = a.vis_bits[(size_t)v * a.words + part * kWarps + w];
  }
  if (threadIdx.x < nv) {
    s_base[threadIdx.x] = a.blk_base[(size_t)threadIdx.x * a.parts + part];
    s_lim[threadIdx.x] = cam_limits(cam_from_desc<float>(blk.v[threadIdx.x]));
  }
  const GaussParams q = load_params(a.sp, g, threadIdx.x < rows);
  __syncthreads();
  if (threadIdx.x < nv) {
    uint32_t tot = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      s_wpre[threadIdx.x][w] = tot;
      tot += (uint32_t)__popc(s_mask[threadIdx.x][w]);
    }
  }
  sh_rows_wait();
  __syncthreads();
  const bool valid = threadIdx.x < rows;
  const V2<float> inv_tile{1.f / (float)a.vs.tile_w, 1.f / (float)a.vs.tile_h};
  const GaussWorld<float> gw = gauss_world(q.quat, q.ls, q.raw);  // once for all views
  const auto* shg = s_sh + threadIdx.x * Rows::kStride;
  for (uint32_t v = 0; v < nv; ++v) {
    const uint32_t m = s_mask[v][warp];
    const bool vis = (m >> lane) & 1u;
    const uint32_t c = s_base[v] + s_wpre[v][warp] + (uint32_t)__popc(m & ((1u << lane) - 1u));
    if (valid) slice(a.b.c_of_gid, a.b.Ncap, v)[g] = vis ? (int32_t)c : -1;
    if (vis) {
      const ViewDesc& vd = blk.v[v];
      const Cam<float> cam = cam_from_desc<float>(vd);
      const Projected<float> p =
          project_gaussian_w(cam, s_lim[v], q.mean, gw, a.cov_blur, inv_tile, vd.tiles_x, vd.tiles_y, a.hp != 0);
      auto coeff = [&](int k, int ch) { return sh_at<SHT, DEG>(shg, k * 3 + ch); };
      const V3<float> rgb = sh_to_color<float>(DEG, view_dir(cam, q.mean), coeff);
      float4* r = slice(a.b.rec, a.b.Vcap * 3, v) + (size_t)c * 3;
      r[0] = make_float4(p.mean2d.x, p.mean2d.y, p.conic.x, p.conic.y);
      r[1] = make_float4(p.conic.z, p.opacity, rgb.x, rgb.y);
      r[2] = make_float4(rgb.z, p.thr, __uint_as_float(p.box.x0 | (p.box.x1 << 16)),
                         __uint_as_float(p.box.y0 | (p.box.y1 << 16)));
      if (fmaxf(fmaxf(rgb.x, rgb.y), rgb.z) == INFINITY) *a.b.inf_colour = 1u;
      slice(a.b.gid_of_c, a.b.Vcap, v)[c] = g;
      slice(a.b.depth_key, a.b.Vcap, v)[c] = __float_as_uint(p.depth);
      slice(a.b.visible_c, a.b.Vcap, v)[c] = 0;
      // Tiles of the box: the intersection slots of the slot layout (the
      // counting walk replaces them by passing-tile counts otherwise).
      const uint32_t bw = p.box.x1 > p.box.x0 ? p.box.x1 - p.box.x0 : 0u;
      slice(a.b.count, a.b.Vcap, v)[c] = bw * (p.box.y1 > p.box.y0 ? p.box.y1 - p.box.y0 : 0u);
    }
  }
}

template <class SHT, int DEG, int NV>
cudaError_t launch_deg(dim3 grid, cudaStream_t st, const ProjectArgs& a, const ViewArgs<NV>& blk) {
  const size_t bytes = ShRows<SHT, DEG>::kBytes;
  cudaError_t e =
      cudaFuncSetAttribute(records_kernel<SHT, DEG, NV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) return e;
  records_kernel<SHT, DEG, NV><<<grid, kProjThreads, bytes, st>>>(a, blk);
  return cudaGetLastError();
}

template <class SHT, int NV>
cudaError_t dispatch(int degree, dim3 grid, cudaStream_t st, const ProjectArgs& a, const ViewArgs<NV>& blk) {
  switch (degree) {
    case 0: return launch_deg<SHT, 0>(grid, st, a, blk);
    case 1: return launch_deg<SHT, 1>(grid, st, a, blk);
    case 2: return launch_deg<SHT, 2>(grid, st, a, blk);
    case 3: return launch_deg<SHT, 3>(grid, st, a, blk);
    default: return launch_deg<SHT, 4>(grid, st, a, blk);
  }
}

template <int NV> cudaError_t launch_passes(const ProjectArgs& a, const ViewDesc* host_views, cudaStream_t st) {
  ViewArgs<NV> blk;
  memset(&blk, 0, sizeof(blk));
  for (uint32_t i = 0; i < a.vs.n_views; ++i) blk.v[i] = host_views[i];
  visibility_kernel<NV><<<a.parts, kProjThreads, 0, st>>>(a, blk);
  block_scan_kernel<<<a.vs.n_views, kBlkScanThreads, 0, st>>>(a);
  const dim3 grid(a.parts);
  return a.sp.sh_bf16 ? dispatch<__nv_bfloat16>(a.sp.degree, grid, st, a, blk)
                      : dispatch<float>(a.sp.degree, grid, st, a, blk);
}

}  // namespace

cudaError_t launch_project(const SplatsDev& sp, const ViewSet& vs, const ViewDesc* host_views, ViewDesc* dev_views,
                           float cov_blur, int fp64_conic, FwdBufs& b, cudaStream_t st) {
  if (sp.n == 0) {
    // No Gaussians: every view has zero visible.
    cudaError_t e = launch_set_views(dev_views, host_views, vs.n_views, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(b.vcount, 0, sizeof(uint32_t) * 4 * vs.n_views, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(b.tile_hist, 0, sizeof(uint32_t) * b.Tcap * vs.n_views, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(b.sched_lcount, 0, sizeof(uint32_t) * kSchedWords, st);
    return e;
  }
  if (vs.n_views > (uint32_t)kMaxViews) return cudaErrorInvalidValue;
  ProjectArgs a;
  a.sp = sp;
  a.vs = vs;
  a.cov_blur = cov_blur;
  a.hp = fp64_conic;
  a.b = b;
  a.parts = (sp.n + kProjThreads - 1) / kProjThreads;
  a.words = a.parts * (kProjThreads / 32);
  if (a.parts > b.proj_parts_cap) return cudaErrorInvalidValue;
  a.vis_bits = b.vis_bits;
  a.blk_count = b.blk_count;
  a.blk_base = b.blk_base;
  a.views = dev_views;
  return vs.n_views == 1 ? launch_passes<1>(a, host_views, st) : launch_passes<kMaxViews>(a, host_views, st);
}

}  // namespace gsr
