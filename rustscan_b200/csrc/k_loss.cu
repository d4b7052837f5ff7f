// k_loss.cu — 0.8 * L1 + 0.2 * (1 - SSIM) and its gradient
// (engine/loss.rs:42-76, 112-142, 233-276, default settings).
//
// SSIM uses an 11-tap sigma-1.5 normalised Gaussian window applied
// separably (horizontal, then vertical) with replicate padding, C1 = 1e-4,
// C2 = 9e-4 and denominators clamped at 1e-8. The reference builds it from
// ~10 burn ops and differentiates through burn autodiff; here two tiled
// kernels do the work:
//  pass 1: per 32x32 output tile and channel, the four blurred moments in
//          shared memory, the SSIM map, its partial derivatives with respect
//          to (mu_x, E[x^2], E[xy]) and per-tile partial sums of SSIM and L1;
//  pass 2: the adjoint of the padded separable blur applied to the three
//          partial maps, combined with the L1 sign into d loss / d pred.
// A last kernel reduces the per-tile sums in a fixed order (double).
#include "gsr_kernels.h"

namespace gsr {

namespace {

constexpr int LTX = 32, LTY = 32, R = 5, WIN = 11;
constexpr int HX = LTX + 2 * R, HY = LTY + 2 * R;
constexpr int kLT = 256;                          // threads per loss block
// Halo elements per thread: the first LTX columns of every kRowStep-th row, a
// warp per row (addresses step by whole rows), then the other 2 R columns.
constexpr int kRowStep = kLT / LTX;
constexpr int kHaloMain = (HY + kRowStep - 1) / kRowStep;
constexpr int kHaloIt = kHaloMain + (HY * 2 * R + kLT - 1) / kLT;

struct LossArgs {
  const ViewDesc* views;
  const float* pred;    // RGBA per view (pix_base)
  const float* target;  // RGB per view (pix_base)
  float* v_pred;
  float* maps;          // [view][3 ch][3 maps][Pcap]
  float* partial;       // [view][3 ch][tiles][2]
  uint64_t Pcap;
  uint32_t tiles_cap;
  float2 kk[WIN];      // (k[t], k[t]): operands of the paired arithmetic
  float2 kw[WIN + 1];  // (k[t], k[t - 1]), zero past the ends
  float k_pre[WIN], k_suf[WIN];  // sums of k[0 .. t] and k[t .. WIN - 1], in ascending order
  float l1_w, ssim_w;
};

// Halo row and column of a thread's it-th element; false past the halo.
__device__ __forceinline__ bool halo_pos(int it, int& hy, int& hx) {
  if (it < kHaloMain) {
    hy = threadIdx.x / LTX + it * kRowStep;
    hx = threadIdx.x % LTX;
  } else {
    const int i = threadIdx.x + (it - kHaloMain) * kLT;
    hy = i / (2 * R);
    hx = LTX + i % (2 * R);
  }
  return hy < HY;
}

__device__ __forceinline__ int clampi(int x, int lo, int hi) { return x < lo ? lo : (x > hi ? hi : x); }
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// Pass 1. Shared memory holds the replicate-padded halo as pairs (x, y), then the
// horizontally blurred moments as quads (x, y, x^2 + y^2, xy; the products are
// formed as the row is read). SSIM needs E[x^2] and E[y^2] only through their
// sum (in sigma_x^2 + sigma_y^2), and its derivatives with respect to both are
// equal, so one blurred plane carries the sum. The paired FP32 arithmetic takes
// two moments at once, so no register pair has to be put together.
// What bounds it: wavefronts of shared memory and L1. So every thread blurs
// four outputs from 14 inputs, read 16 bytes at a time: along a row with the
// lanes in different rows (odd strides of 16-byte units in both arrays), down a
// column with the lanes in different columns. Halo rows are loaded a warp to a
// row, so that addresses step by whole rows instead of being divided out. With
// the like in pass 2, both passes on 8 views of 1280x720: 541 -> 463 us (225 and
// 238; instruction issue at 0.7 in pass 1, wavefronts at 0.9 of L1's rate in
// pass 2), on 16 of up to 1920x1080: 1208 -> 1056, on one of 320x240: 27 -> 22.
struct SsimFwdSmem {
  float2 p[HY][HX];
  float4 h[HY][LTX + 1];
  float red[2][8];
};

__global__ void __launch_bounds__(kLT, 5) ssim_fwd_kernel(LossArgs a) {
  extern __shared__ float4 smem_raw[];
  SsimFwdSmem& S = *reinterpret_cast<SsimFwdSmem*>(smem_raw);
  const uint32_t v = blockIdx.z, ch = blockIdx.y;
  const ViewDesc& vd = a.views[v];
  const int W = (int)vd.w, H = (int)vd.h;
  const int tiles_x = (W + LTX - 1) / LTX, tiles_y = (H + LTY - 1) / LTY;
  const int tile = blockIdx.x;
  if (tile >= tiles_x * tiles_y) return;
  const int x0 = (tile % tiles_x) * LTX, y0 = (tile / tiles_x) * LTY;
  const float* pred = a.pred + vd.pix_base * 4;
  const float* tgt = a.target + vd.pix_base * 3;
  {
    // All of a thread's halo loads are issued before the first store.
    float xs[kHaloIt], ys[kHaloIt];
#pragma unroll
    for (int it = 0; it < kHaloIt; ++it) {
      int hy, hx;
      if (halo_pos(it, hy, hx)) {
        const int gx = clampi(x0 + hx - R, 0, W - 1), gy = clampi(y0 + hy - R, 0, H - 1);
        const size_t p = (size_t)gy * W + gx;
        xs[it] = pred[p * 4 + ch];
        ys[it] = tgt[p * 3 + ch];
      }
    }
#pragma unroll
    for (int it = 0; it < kHaloIt; ++it) {
      int hy, hx;
      if (halo_pos(it, hy, hx)) {
        S.p[hy][hx] = make_float2(xs[it], ys[it]);
      }
    }
  }
  __syncthreads();
  // Horizontal pass: every halo row, four output columns per task.
  for (int i = threadIdx.x; i < HY * (LTX / 4); i += kLT) {
    const int hy = i % HY, ox = 4 * (i / HY);
    const float4* row = reinterpret_cast<const float4*>(&S.p[hy][ox]);
    float2 m01[4], m23[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) m01[j] = m23[j] = f2(0.f);
#pragma unroll
    for (int u = 0; u < (WIN + 3) / 2; ++u) {
      const float4 q = row[u];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float2 xy = c ? make_float2(q.z, q.w) : make_float2(q.x, q.y);
        const float2 pr = make_float2(xy.x * xy.x + xy.y * xy.y, xy.x * xy.y);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int t = 2 * u + c - j;
          if (t < 0 || t >= WIN) continue;
          m01[j] = fma2(a.kk[t], xy, m01[j]);
          m23[j] = fma2(a.kk[t], pr, m23[j]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) S.h[hy][ox + j] = make_float4(m01[j].x, m01[j].y, m23[j].x, m23[j].y);
  }
  __syncthreads();
  // Vertical pass and the SSIM map: a column and four rows per thread.
  const float C1 = 1e-4f, C2 = 9e-4f;
  float ssum = 0.f, lsum = 0.f;
  float* maps = a.maps + ((size_t)v * 3 + ch) * 3 * a.Pcap;
  {
    static_assert(kLT == LTX * (LTY / 4), "a column and four rows per thread");
    const int ox = threadIdx.x % LTX, oy = 4 * (threadIdx.x / LTX);
    float2 m01[4], m23[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) m01[j] = m23[j] = f2(0.f);
#pragma unroll
    for (int u = 0; u < WIN + 3; ++u) {
      const float4 q = S.h[oy + u][ox];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int t = u - j;
        if (t < 0 || t >= WIN) continue;
        m01[j] = fma2(a.kk[t], make_float2(q.x, q.y), m01[j]);
        m23[j] = fma2(a.kk[t], make_float2(q.z, q.w), m23[j]);
      }
    }
#pragma unroll
    for (int ry = 0; ry < 4; ++ry) {
      const int gx = x0 + ox, gy = y0 + oy + ry;
      if (gx >= W || gy >= H) continue;
      const float mx = m01[ry].x, my = m01[ry].y;
      const float ess = m23[ry].x;  // E[x^2] + E[y^2]
      const float exy = m23[ry].y;
      const float sxy = exy - mx * my;
      const float A = 2.f * mx * my + C1, B = 2.f * sxy + C2;
      const float Cr = mx * mx + my * my + C1, Dr = ((ess - mx * mx) - my * my) + C2;
      const float Cc = fmaxf(Cr, 1e-8f), Dc = fmaxf(Dr, 1e-8f);
      const float inv = 1.f / (Cc * Dc);
      const float s = (A * B) * inv;
      const float dC = Cr > 1e-8f ? 1.f : 0.f, dD = Dr > 1e-8f ? 1.f : 0.f;
      const float gmx = 2.f * (my * (B - A) - (s * mx) * (dC * Dc - dD * Cc)) * inv;
      const size_t p = (size_t)gy * W + gx;
      maps[p] = gmx;
      maps[a.Pcap + p] = -s * dD / Dc;
      maps[2 * a.Pcap + p] = 2.f * A * inv;
      ssum += s;
      const float2 xy = S.p[oy + ry + R][ox + R];
      lsum += fabsf(xy.x - xy.y);
    }
  }
  // Fixed-order block reduction.
  for (int o = 16; o > 0; o >>= 1) {
    ssum += __shfl_xor_sync(0xffffffffu, ssum, o);
    lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
  }
  if ((threadIdx.x & 31) == 0) {
    S.red[0][threadIdx.x >> 5] = ssum;
    S.red[1][threadIdx.x >> 5] = lsum;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float a0 = 0.f, a1 = 0.f;
    for (int w = 0; w < 8; ++w) {
      a0 += S.red[0][w];
      a1 += S.red[1][w];
    }
    float* pp = a.partial + (((size_t)v * 3 + ch) * a.tiles_cap + tile) * 2;
    pp[0] = a0;
    pp[1] = a1;
  }
}

// Weight of output q, |q - p| <= R, in the adjoint of a replicate-padded 11-tap
// correlation at the border input p (0 or n - 1) of an axis of length n: it
// collects the clamped taps. (At an interior input it is k[R + q - p].)
__device__ __forceinline__ float adj_weight(const LossArgs& a, int p, int q, int n) {
  if (n == 1) return a.k_pre[WIN - 1];
  return p == 0 ? a.k_pre[R - q] : a.k_suf[n - 1 - q + R];
}

// Pass 2: the adjoint of the padded separable blur on the three partial
// maps (vertical, then horizontal), combined with the L1 sign. Every row and
// column is summed with the symmetric kernel in paired arithmetic over a halo
// that is zero outside the image (the zeros add exact +0); the first and last of
// the image are then summed again with the border's weights. As in
// pass 1 wavefronts bound it: the horizontal pass reads 16 bytes at a time and
// hands its sums over in shared memory (in place of the maps, which it no longer
// needs), so that the lanes write neighbouring pixels.
constexpr int VX = HX + 2;  // whole 16-byte units
struct SsimBwdSmem {
  union {
    float g[3][HY][HX];
    float s[3][LTY][LTX];
  };
  float v[3][LTY][VX];
};

__global__ void __launch_bounds__(kLT, 5) ssim_bwd_kernel(LossArgs a) {
  extern __shared__ float4 smem_raw[];
  SsimBwdSmem& S = *reinterpret_cast<SsimBwdSmem*>(smem_raw);
  const uint32_t v = blockIdx.z, ch = blockIdx.y;
  const ViewDesc& vd = a.views[v];
  const int W = (int)vd.w, H = (int)vd.h;
  const int tiles_x = (W + LTX - 1) / LTX, tiles_y = (H + LTY - 1) / LTY;
  const int tile = blockIdx.x;
  if (tile >= tiles_x * tiles_y) return;
  const int x0 = (tile % tiles_x) * LTX, y0 = (tile / tiles_x) * LTY;
  const float* maps = a.maps + ((size_t)v * 3 + ch) * 3 * a.Pcap;
  const float* pred = a.pred + vd.pix_base * 4;
  const float* tgt = a.target + vd.pix_base * 3;
  // The prediction and target values of this thread's output pixels (read
  // at the end) are loaded now, with the halo of the three maps.
  constexpr int kOutIt = LTY * LTX / kLT;
  float px_x[kOutIt], px_y[kOutIt];
#pragma unroll
  for (int it = 0; it < kOutIt; ++it) {
    const int i = threadIdx.x + it * kLT;
    const int px = x0 + i % LTX, py = y0 + i / LTX;
    const bool ok = px < W && py < H;
    const size_t p = (size_t)py * W + px;
    px_x[it] = ok ? pred[p * 4 + ch] : 0.f;
    px_y[it] = ok ? tgt[p * 3 + ch] : 0.f;
  }
  {
    float gs[kHaloIt][3];
#pragma unroll
    for (int it = 0; it < kHaloIt; ++it) {
      int hy, hx;
      const bool in = halo_pos(it, hy, hx);
      const int gx = x0 + hx - R, gy = y0 + hy - R;
      const bool ok = in && gx >= 0 && gx < W && gy >= 0 && gy < H;
      const size_t p = (size_t)gy * W + gx;
#pragma unroll
      for (int m = 0; m < 3; ++m) gs[it][m] = ok ? maps[m * a.Pcap + p] : 0.f;
    }
#pragma unroll
    for (int it = 0; it < kHaloIt; ++it) {
      int hy, hx;
      if (halo_pos(it, hy, hx)) {
#pragma unroll
        for (int m = 0; m < 3; ++m) S.g[m][hy][hx] = gs[it][m];
      }
    }
  }
  __syncthreads();
  // Adjoint of the vertical pass: tile rows, all halo columns (in pairs). A
  // thread slides down a column pair over four output rows, adding each loaded
  // halo row into the rows it reaches (14 loads per plane for 4 rows instead of
  // 44), in tap order.
  {
    constexpr int kRows = 4;
    for (int i = threadIdx.x; i < (LTY / kRows) * (HX / 2); i += kLT) {
      const int oy = kRows * (i / (HX / 2)), hx = 2 * (i % (HX / 2));
      float2 acc[3][kRows];
#pragma unroll
      for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int j = 0; j < kRows; ++j) acc[m][j] = f2(0.f);
#pragma unroll
      for (int r = 0; r < WIN + kRows - 1; ++r) {
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          const float2 val = *reinterpret_cast<const float2*>(&S.g[m][oy + r][hx]);
#pragma unroll
          for (int j = 0; j < kRows; ++j)
            if (r - j >= 0 && r - j < WIN) acc[m][j] = fma2(a.kk[r - j], val, acc[m][j]);
        }
      }
#pragma unroll
      for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int j = 0; j < kRows; ++j) *reinterpret_cast<float2*>(&S.v[m][oy + j][hx]) = acc[m][j];
#pragma unroll 1
      for (int e = 0; e < 2; ++e) {
        const int py = e ? H - 1 : 0;
        if (py < y0 + oy || py >= y0 + oy + kRows) continue;
        float2 b[3] = {f2(0.f), f2(0.f), f2(0.f)};
#pragma unroll 1
        for (int qy = max(py - R, 0); qy <= min(py + R, H - 1); ++qy) {
          const float w = adj_weight(a, py, qy, H);
#pragma unroll
          for (int m = 0; m < 3; ++m)
            b[m] = fma2(f2(w), *reinterpret_cast<const float2*>(&S.g[m][qy - y0 + R][hx]), b[m]);
        }
#pragma unroll
        for (int m = 0; m < 3; ++m) *reinterpret_cast<float2*>(&S.v[m][py - y0][hx]) = b[m];
      }
    }
  }
  __syncthreads();
  {
    static_assert(kLT == LTY * (LTX / 4), "four columns per thread");
    const int oy = threadIdx.x / (LTX / 4), ox = 4 * (threadIdx.x % (LTX / 4));
    const int px = x0 + ox;
    // Two columns at once. Each loaded value serves both, weights
    // (k[j], k[j - 1]); a zero weight adds an exact +0, so each column sums its
    // taps in tap order.
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      float val[16];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        *reinterpret_cast<float4*>(val + 4 * u) = reinterpret_cast<const float4*>(&S.v[m][oy][ox])[u];
      float2 a0 = f2(0.f), a1 = f2(0.f);
#pragma unroll
      for (int j = 0; j <= 2 * R + 1; ++j) {
        a0 = fma2(a.kw[j], f2(val[j]), a0);
        a1 = fma2(a.kw[j], f2(val[j + 2]), a1);
      }
      *reinterpret_cast<float4*>(&S.s[m][oy][ox]) = make_float4(a0.x, a0.y, a1.x, a1.y);
    }
#pragma unroll 1
    for (int e = 0; e < 2; ++e) {
      const int pc = e ? W - 1 : 0;
      if (pc < px || pc >= px + 4) continue;
      float s3[3] = {0.f, 0.f, 0.f};
#pragma unroll 1
      for (int qx = max(pc - R, 0); qx <= min(pc + R, W - 1); ++qx) {
        const float w = adj_weight(a, pc, qx, W);
#pragma unroll
        for (int m = 0; m < 3; ++m) s3[m] = s3[m] + w * S.v[m][oy][qx - x0 + R];
      }
#pragma unroll
      for (int m = 0; m < 3; ++m) S.s[m][oy][pc - x0] = s3[m];
    }
  }
  __syncthreads();
  float* out = a.v_pred + vd.pix_base * 4;
  const float M = 3.f * (float)W * (float)H;
  const float kl = a.l1_w / M, ks = -a.ssim_w / M;
#pragma unroll
  for (int it = 0; it < kOutIt; ++it) {
    const int i = threadIdx.x + it * kLT;
    const int px = x0 + i % LTX, py = y0 + i / LTX;
    if (px >= W || py >= H) continue;
    const float a0 = (&S.s[0][0][0])[i], a1 = (&S.s[1][0][0])[i], a2 = (&S.s[2][0][0])[i];
    const size_t p = (size_t)py * W + px;
    const float x = px_x[it], y = px_y[it];
    const float dlt = x - y;
    const float sg = dlt > 0.f ? 1.f : (dlt < 0.f ? -1.f : 0.f);
    out[p * 4 + ch] = kl * sg + ks * (a0 + 2.f * x * a1 + y * a2);
    if (ch == 0) out[p * 4 + 3] = 0.f;
  }
}

// One block per view: strided partial sums in double, then a fixed-order
// tree over the block (deterministic).
__global__ void __launch_bounds__(256) loss_reduce_kernel(LossArgs a, uint32_t n_views, float* loss) {
  __shared__ double s_ss[256], s_l1[256];
  const uint32_t v = blockIdx.x;
  if (v >= n_views) return;
  const ViewDesc& vd = a.views[v];
  const int W = (int)vd.w, H = (int)vd.h;
  const int tiles = ((W + LTX - 1) / LTX) * ((H + LTY - 1) / LTY);
  double ss = 0.0, l1 = 0.0;
  for (int i = threadIdx.x; i < 3 * tiles; i += blockDim.x) {
    const int ch = i / tiles, t = i % tiles;
    const float* pp = a.partial + (((size_t)v * 3 + ch) * a.tiles_cap + t) * 2;
    ss += pp[0];
    l1 += pp[1];
  }
  s_ss[threadIdx.x] = ss;
  s_l1[threadIdx.x] = l1;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) {
      s_ss[threadIdx.x] += s_ss[threadIdx.x + o];
      s_l1[threadIdx.x] += s_l1[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double M = 3.0 * (double)W * (double)H;
    loss[v] = (float)((double)a.l1_w * (s_l1[0] / M) + (double)a.ssim_w * (1.0 - s_ss[0] / M));
  }
}

}  // namespace

void ssim_window(float* k) {
  // loss.rs:233-250: values in f64, stored as f32, normalised in f32.
  float vals[WIN], sum = 0.0f;
  for (int o = -R; o <= R; ++o) {
    vals[o + R] = (float)exp(-(double)(o * o) / (2.0 * 1.5 * 1.5));
    sum += vals[o + R];
  }
  for (int i = 0; i < WIN; ++i) k[i] = vals[i] / (sum > 1e-8f ? sum : 1e-8f);
}

uint32_t loss_tiles(uint32_t w, uint32_t h) { return ((w + LTX - 1) / LTX) * ((h + LTY - 1) / LTY); }

cudaError_t launch_loss(const ViewSet& vs, const ViewDesc* host_views, const float* pred, const float* target,
                        float l1_w, float ssim_w, float* loss, float* v_pred, float* work, uint64_t work_floats,
                        cudaStream_t st) {
  LossArgs a{};
  a.views = vs.views;
  a.pred = pred;
  a.target = target;
  a.v_pred = v_pred;
  uint64_t pmax = 0;
  uint32_t tmax = 0;
  for (uint32_t v = 0; v < vs.n_views; ++v) {
    const uint64_t p = (uint64_t)host_views[v].w * host_views[v].h;
    if (p > pmax) pmax = p;
    const uint32_t t = loss_tiles(host_views[v].w, host_views[v].h);
    if (t > tmax) tmax = t;
  }
  a.Pcap = pmax;
  a.tiles_cap = tmax;
  const uint64_t need = (uint64_t)vs.n_views * 9 * pmax + (uint64_t)vs.n_views * 3 * tmax * 2;
  if (need > work_floats) return cudaErrorInvalidValue;
  a.maps = work;
  a.partial = work + (uint64_t)vs.n_views * 9 * pmax;
  float k[WIN];
  ssim_window(k);
  for (int t = 0; t < WIN; ++t) a.kk[t] = make_float2(k[t], k[t]);
  for (int t = 0; t <= WIN; ++t) a.kw[t] = make_float2(t < WIN ? k[t] : 0.f, t > 0 ? k[t - 1] : 0.f);
  for (int i = 0; i < WIN; ++i) {
    float lo = 0.f, hi = 0.f;
    for (int t = 0; t <= i; ++t) lo += k[t];
    for (int t = i; t < WIN; ++t) hi += k[t];
    a.k_pre[i] = lo;
    a.k_suf[i] = hi;
  }
  a.l1_w = l1_w;
  a.ssim_w = ssim_w;
  if (tmax == 0) return cudaSuccess;
  dim3 grid(tmax, 3, vs.n_views);
  // More than the 48 KB default of dynamic shared memory (set for the current device).
  cudaFuncSetAttribute(ssim_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SsimFwdSmem));
  cudaFuncSetAttribute(ssim_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SsimBwdSmem));
  ssim_fwd_kernel<<<grid, kLT, sizeof(SsimFwdSmem), st>>>(a);
  ssim_bwd_kernel<<<grid, kLT, sizeof(SsimBwdSmem), st>>>(a);
  loss_reduce_kernel<<<vs.n_views, 256, 0, st>>>(a, vs.n_views, loss);
  return cudaGetLastError();
}

}  // namespace gsr
