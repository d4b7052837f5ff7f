// k_backward.cu — projection backward (project_backwards.wgsl:12-151) over
// all views of the last forward, the densification statistics
// (engine/trainer.rs:651-728) and the bias-corrected Adam update
// (engine/optimizer.rs:122-162).
//
// One thread per Gaussian sums its views in a fixed order: per view the
// projection adjoint down to the mean, the 3D covariance and the opacity, and
// the SH gradients; after the views, once, the covariance's gradient into
// quaternion and scales. A block then writes its Gaussians' gradients, or in a
// training step applies Adam to their parameters at once. Rows of Gaussians no
// view sees get zero gradients, as the reference zero-fills. Adam as a call of
// its own is an element-wise pass with 16-byte accesses.
#include <cuda_bf16.h>

#include "gsr_kernels.h"

namespace gsr {

namespace {

__device__ __forceinline__ float to_f(float x) { return x; }
__device__ __forceinline__ float to_f(__nv_bfloat16 x) { return __bfloat162float(x); }
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ld4(const __nv_bfloat16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
  const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
  return make_float4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ void st4(float* p, float4 x) { *reinterpret_cast<float4*>(p) = x; }
__device__ __forceinline__ void st4(__nv_bfloat16* p, float4 x) {
  __nv_bfloat162 lo, hi;
  lo.x = __float2bfloat16_rn(x.x);
  lo.y = __float2bfloat16_rn(x.y);
  hi.x = __float2bfloat16_rn(x.z);
  hi.y = __float2bfloat16_rn(x.w);
  uint2 u;
  u.x = *reinterpret_cast<uint32_t*>(&lo);
  u.y = *reinterpret_cast<uint32_t*>(&hi);
  *reinterpret_cast<uint2*>(p) = u;
}
__device__ __forceinline__ void store_sh(float* p, float x) { *p = x; }
__device__ __forceinline__ void store_sh(__nv_bfloat16* p, float x) { *p = __float2bfloat16_rn(x); }

// engine/optimizer.rs:141-161 with the bias corrections applied as
// multiplications by their f32 reciprocals; every operation rounded on its
// own (the file builds with multiply-add contraction; Adam must match the
// oracle bit for bit).
__device__ __forceinline__ float adam_one(float p, float g, float& m, float& v, float lr, const AdamScalars& a) {
  const float m1 = eadd(emul(m, a.beta1), emul(g, esub(1.0f, a.beta1)));
  const float m2 = eadd(emul(v, a.beta2), emul(emul(g, g), esub(1.0f, a.beta2)));
  m = m1;
  v = m2;
  const float mh = emul(m1, a.rbc1), vh = emul(m2, a.rbc2);
  const float upd = __fdiv_rn(mh, eadd(__fsqrt_rn(vh), a.eps));
  return esub(p, emul(upd, lr));
}

__device__ __forceinline__ float group_lr(const AdamScalars& a, int group, uint32_t col) {
  if (group == 0) return col < 3 ? a.lr_pos : (col < 7 ? a.lr_rot : a.lr_scale);
  return group == 1 ? a.lr_color : a.lr_opac;
}


// ---------------------------------------------------------------------------
// The gradient kernel.
// ---------------------------------------------------------------------------
// A view as the adjoint reads it, in shared memory.
struct BwdView {
  float rot[9];   // rot[3 * column + row]
  float trans[3];
  float fx, fy;
  float xlo, xhi, ylo, yhi;  // the Jacobian's clamp
  float campos[3];
};

__device__ __forceinline__ void load_view(const ViewDesc& d, BwdView& o) {
  for (int i = 0; i < 9; ++i) o.rot[i] = d.rot[i];
  for (int i = 0; i < 3; ++i) {
    o.trans[i] = d.trans[i];
    o.campos[i] = d.campos[i];
  }
  o.fx = d.fx;
  o.fy = d.fy;
  o.xhi = (1.15f * (float)d.w - d.cx) / d.fx;
  o.yhi = (1.15f * (float)d.h - d.cy) / d.fy;
  o.xlo = (-0.15f * (float)d.w - d.cx) / d.fx;
  o.ylo = (-0.15f * (float)d.h - d.cy) / d.fy;
}

// The projection adjoint of one view (project_backward without the SH terms):
// adds into the gradients of the mean and, as the symmetric matrix (xx, xy, xz,
// yy, yz, zz), of the 3D covariance, returns the opacity logit's. Written out
// for the symmetric matrices and the Jacobian's zeros, which the general
// functions multiply through; divisions and roots are correctly rounded, as there.
struct ViewAdjoint {
  V3<float> v_mean;
  float v_cov[6];
  float v_raw_opac, depth;
};
__device__ __forceinline__ ViewAdjoint view_adjoint(const BwdView& w, V3<float> p, const float (&c3)[6], float opac,
                                                    float blur, const float4& q0, const float4& q1, const float4& q2,
                                                    bool exact, bool hp) {
  ViewAdjoint o;
  const float* R = w.rot;  // R(i, k) = R[3 k + i]
  const float x = R[0] * p.x + R[3] * p.y + R[6] * p.z + w.trans[0];
  const float y = R[1] * p.x + R[4] * p.y + R[7] * p.z + w.trans[1];
  const float z = R[2] * p.x + R[5] * p.y + R[8] * p.z + w.trans[2];
  o.depth = z;
  // M = R C R^T.
  float A[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    A[i][0] = R[i] * c3[0] + R[3 + i] * c3[1] + R[6 + i] * c3[2];
    A[i][1] = R[i] * c3[1] + R[3 + i] * c3[3] + R[6 + i] * c3[4];
    A[i][2] = R[i] * c3[2] + R[3 + i] * c3[4] + R[6 + i] * c3[5];
  }
  auto m = [&](int i, int j) { return A[i][0] * R[j] + A[i][1] * R[3 + j] + A[i][2] * R[6 + j]; };
  const float M00 = m(0, 0), M01 = m(0, 1), M02 = m(0, 2), M11 = m(1, 1), M12 = m(1, 2), M22 = m(2, 2);
  // The Jacobian's rows (jx, 0, a) and (0, jy, b).
  const float rz = 1.f / fmaxf(z, 0.01f);
  const float xr = x * rz, yr = y * rz;
  const float uc = fminf(fmaxf(xr, w.xlo), w.xhi), vc = fminf(fmaxf(yr, w.ylo), w.yhi);
  const float jx = w.fx * rz, jy = w.fy * rz, a = -jx * uc, b = -jy * vc;
  // Row 0 and 1 of J M, then the 2D covariance.
  const float n00 = jx * M00 + a * M02, n01 = jx * M01 + a * M12, n02 = jx * M02 + a * M22;
  const float n11 = jy * M11 + b * M12, n12 = jy * M12 + b * M22;
  const float s00 = n00 * jx + n02 * a, s01 = n01 * jy + n02 * b, s11 = n11 * jy + n12 * b;
  // Compensation sqrt(det / det of the blurred), and the conic (inverse2x2_packed).
  const float d00 = s00 + blur, d11 = s11 + blur;
  const float det_raw = fmaxf(s00 * s11 - s01 * s01, 0.f), det_blur = d00 * d11 - s01 * s01;
  const float det_end = fmaxf(det_blur, 1e-12f);
  const float ratio = det_raw / det_end;  // a product of both overflows from a projection of 65,500 pixels on
  const float comp = sqrtf(ratio);
  float fc = comp;
  const float i00 = d00 + 1e-6f, i11 = d11 + 1e-6f, det = i00 * i11 - s01 * s01;
  const float inv = det > 1e-10f ? 1.f / det : 0.f;
  V3<float> ci{i11 * inv, -s01 * inv, i00 * inv};
  if (hp) {
    M2<float> cov;
    cov.m[0][0] = s00;
    cov.m[0][1] = cov.m[1][0] = s01;
    cov.m[1][1] = s11;
    fc = compensate_cov2d_hp(cov, blur);
    ci = inverse2x2_packed_hp(cov);
  }
  o.v_raw_opac = fc * q2.x * opac * (1.f - opac);
  // G: gradient of the 2D covariance, -C V C, and through the compensation
  // (compensate_vjp, whose factor 1 / det_end is ratio / det_raw).
  const float v0 = q0.z, vh = 0.5f * q0.w, v2 = q1.x;
  const float t00 = ci.x * v0 + ci.y * vh, t01 = ci.x * vh + ci.y * v2;
  const float t10 = ci.y * v0 + ci.z * vh, t11 = ci.y * vh + ci.z * v2;
  float g00 = -(t00 * ci.x + t01 * ci.y), g01 = -(t00 * ci.y + t01 * ci.z), g11 = -(t10 * ci.y + t11 * ci.z);
  if (exact) {
    const float k = det_raw > 0.f ? (0.5f * q2.x * opac * comp) / det_raw : 0.f;
    const float rk = det_blur > 1e-12f ? ratio : 0.f;
    g00 += k * (s11 - rk * d11);
    g01 += k * (rk - 1.f) * s01;
    g11 += k * (s00 - rk * d00);
  }
  // H = G J: rows (g00 jx, g01 jy, e0) and (g01 jx, g11 jy, e1).
  const float e0 = g00 * a + g01 * b, e1 = g01 * a + g11 * b;
  const float h00 = g00 * jx, h01 = g01 * jy, h10 = g01 * jx, h11 = g11 * jy;
  // Gradient of J, 2 H M, where it is not constant.
  const float vj00 = 2.f * (h00 * M00 + h01 * M01 + e0 * M02), vj02 = 2.f * (h00 * M02 + h01 * M12 + e0 * M22);
  const float vj11 = 2.f * (h10 * M01 + h11 * M11 + e1 * M12), vj12 = 2.f * (h10 * M02 + h11 * M12 + e1 * M22);
  const float rz2 = rz * rz;
  float cx = jx * q0.x, cy = jy * q0.y;
  float cz = -(w.fx * x * q0.x + w.fy * y * q0.y) * rz2;
  if (xr <= w.xhi && xr >= w.xlo) {
    cx -= w.fx * rz2 * vj02;
    cz += 2.f * w.fx * x * rz2 * rz * vj02;
  } else {
    cz += w.fx * uc * rz2 * vj02;
  }
  if (yr <= w.yhi && yr >= w.ylo) {
    cy -= w.fy * rz2 * vj12;
    cz += 2.f * w.fy * y * rz2 * rz * vj12;
  } else {
    cz += w.fy * vc * rz2 * vj12;
  }
  cz -= w.fx * rz2 * vj00 + w.fy * rz2 * vj11;
  o.v_mean = V3<float>{R[0] * cx + R[1] * cy + R[2] * cz, R[3] * cx + R[4] * cy + R[5] * cz,
                       R[6] * cx + R[7] * cy + R[8] * cz};
  // J^T G J in the camera, then R^T (.) R.
  const float W00 = jx * h00, W01 = jx * h01, W02 = jx * e0, W11 = jy * h11, W12 = jy * e1, W22 = a * e0 + b * e1;
  float B[3][3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    B[0][k] = W00 * R[3 * k] + W01 * R[3 * k + 1] + W02 * R[3 * k + 2];
    B[1][k] = W01 * R[3 * k] + W11 * R[3 * k + 1] + W12 * R[3 * k + 2];
    B[2][k] = W02 * R[3 * k] + W12 * R[3 * k + 1] + W22 * R[3 * k + 2];
  }
  auto c = [&](int l, int k) { return R[3 * l] * B[0][k] + R[3 * l + 1] * B[1][k] + R[3 * l + 2] * B[2][k]; };
  o.v_cov[0] = c(0, 0);
  o.v_cov[1] = c(0, 1);
  o.v_cov[2] = c(0, 2);
  o.v_cov[3] = c(1, 1);
  o.v_cov[4] = c(1, 2);
  o.v_cov[5] = c(2, 2);
  return o;
}

struct GatherArgs {
  SplatsDev sp;
  ViewSet vs;
  FwdBufs b;
  float cov_blur;
  float* v_tr;   // gradients out (null with adam)
  float* v_sh;
  float* v_op;
  float* stats;
  float* acc;
  int use_visible;
  float grad_scale;
  int exact, hp;
  int adam;      // 1: update the parameters in place instead
  int vec_sh, vec_tr;  // every SH (transform) array allows 16-byte accesses (8 for BF16)
  AdamArgs ad;
};

// A block owns kGT consecutive Gaussians. Shared memory holds, per Gaussian,
// one row of its SH values (read by the view-direction term) that is reused for
// its SH gradients on the way out, a row of transform and opacity gradients,
// the densification sums and two stages of screen-space gradient records (view
// v + 1's copies are in flight while view v is summed). SH rows of whole
// float4s have an odd stride in them, the others an odd stride in floats:
// either way a warp reading its rows meets no bank conflict.
constexpr int kGT = 128;

template <int K> struct GatherSmem {
  static constexpr bool kQuads = (3 * K) % 4 == 0;
  static constexpr int kSh = kQuads ? 4 * ((3 * K / 4) | 1) : ((3 * K) | 1);
  static constexpr int kTr = 11;
  alignas(16) float sh[kGT * kSh];
  float tr[kGT * kTr];
  float acc[7][kGT];
  float4 rec[2][3][kGT];
};

__device__ __forceinline__ void cp_async16(float4* dst, const float4* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// The place of SH element e of the block (global element order) in its rows.
template <int K> __device__ __forceinline__ uint32_t sh_place(uint32_t e) {
  return (e / (3 * K)) * GatherSmem<K>::kSh + e % (3 * K);
}

// Stages the block's SH rows as FP32 (16 bytes at a time where the array
// allows it; with every load of a thread in flight at once for FP32).
template <int K>
__device__ __forceinline__ void stage_sh_rows(const float* src, uint32_t total, bool vec, float* s_sh) {
  if (GatherSmem<K>::kQuads && vec) {
    for (uint32_t q = threadIdx.x; q < total / 4; q += kGT)
      cp_async16(reinterpret_cast<float4*>(s_sh + sh_place<K>(4 * q)), reinterpret_cast<const float4*>(src) + q);
  } else {
    for (uint32_t e = threadIdx.x; e < total; e += kGT) {
      const uint32_t d = (uint32_t)__cvta_generic_to_shared(s_sh + sh_place<K>(e));
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src + e) : "memory");
    }
  }
}
template <int K>
__device__ __forceinline__ void stage_sh_rows(const __nv_bfloat16* src, uint32_t total, bool vec, float* s_sh) {
  if (GatherSmem<K>::kQuads && vec) {
#pragma unroll 6
    for (uint32_t q = threadIdx.x; q < total / 4; q += kGT) st4(s_sh + sh_place<K>(4 * q), ld4(src + 4 * (size_t)q));
  } else {
    for (uint32_t e = threadIdx.x; e < total; e += kGT) s_sh[sh_place<K>(e)] = __bfloat162float(src[e]);
  }
}

// One thread per Gaussian. What bounds it: the latency of its loads at 16 warps
// per SM (128 registers, 48 of them the SH sums; degree 3 spills 124 bytes, fewer
// registers spill more, and a third record stage or a fourth of the blocks less
// costs more than it hides), at 0.4 of the DRAM rate and of the issue slots each. It replaces a pass per (view,
// Gaussian) that wrote 96-byte adjoint records, a pass that summed them and, in
// a training step, the Adam passes that read the gradient back: 8 views of 1M
// Gaussians 0.817 -> 0.626 ms, 16 uneven views of 2M (BF16 SH) 2.77 -> 1.82, one
// view of 3M (BF16, gradients out) 0.548 -> 0.406. Correctly rounded divisions
// and roots are 6% to 10% of that: with estimates and a Newton step each it took
// 0.573, 1.63 and 0.386.
// Degree 4 runs three blocks per SM at 168 registers with a few spills: gradient
// and Adam of 300k Gaussians at 640x480 225 us (the separate passes 220), 600k in
// 5 views 560 (604), 659k in 2 501 (514); with two blocks 263, 615 and 600, when
// three took 223, 534 and 492.
template <class SHT, int DEG>
__global__ void __launch_bounds__(kGT, DEG >= 4 ? 3 : 4) gather_kernel(GatherArgs a) {
  constexpr int K = (DEG + 1) * (DEG + 1);
  constexpr int NSH = 3 * K;
  using L = GatherSmem<K>;
  extern __shared__ float4 smem_g[];
  L& S = *reinterpret_cast<L*>(smem_g);
  BwdView* s_view = reinterpret_cast<BwdView*>(reinterpret_cast<char*>(smem_g) + sizeof(L));  // [n_views]
  const uint32_t n = a.sp.n;
  const uint32_t nv = a.vs.n_views;
  const float sc = a.grad_scale;
  const SHT* sh = reinterpret_cast<const SHT*>(a.sp.sh);
  const bool dir_term = a.exact != 0 && DEG > 0;
  const uint32_t r = threadIdx.x;
  for (uint32_t v = r; v < nv; v += kGT) load_view(a.vs.views[v], s_view[v]);
  // The copy of this thread's record of view v (compact index c, none if c <
  // 0); one commit group per view whether or not it copies anything.
  auto issue = [&](uint32_t v, int32_t c) {
    if (c >= 0) {
      const float4* q = slice(a.b.sgrad, a.b.Vcap * 3, v) + (size_t)c * 3;
#pragma unroll
      for (int i = 0; i < 3; ++i) cp_async16(&S.rec[v & 1][i][r], q + i);
    }
    cp_async_commit();
  };
  for (uint32_t g0 = blockIdx.x * kGT; g0 < n; g0 += gridDim.x * kGT) {
    const uint32_t rows = min((uint32_t)kGT, n - g0);
    const uint32_t g = g0 + r;
    const bool own = r < rows;
    __syncthreads();
    if (dir_term) stage_sh_rows<K>(sh + (size_t)g0 * NSH, rows * NSH, a.vec_sh != 0, S.sh);
    int32_t c_cur = own && nv > 0 ? a.b.c_of_gid[g] : -1;
    if (nv > 0) issue(0, c_cur);  // completes with the SH copies, which are older
    int32_t c_nxt = own && nv > 1 ? slice(a.b.c_of_gid, a.b.Ncap, 1)[g] : -1;
    V3<float> mean{0.f, 0.f, 0.f};
    float c3[6] = {}, opac = 0.f;
    const float2* t2 = reinterpret_cast<const float2*>(a.sp.transforms + (size_t)g * 10);
    if (own) {
      const float2 t01 = t2[0], t23 = t2[1], t45 = t2[2], t67 = t2[3], t89 = t2[4];
      mean = V3<float>{t01.x, t01.y, t23.x};
      const GaussWorld<float> w = gauss_world(V4<float>{t23.y, t45.x, t45.y, t67.x}, V3<float>{t67.y, t89.x, t89.y},
                                              a.sp.raw_opac[g]);
      c3[0] = w.cov3d.m[0][0];
      c3[1] = w.cov3d.m[0][1];
      c3[2] = w.cov3d.m[0][2];
      c3[3] = w.cov3d.m[1][1];
      c3[4] = w.cov3d.m[1][2];
      c3[5] = w.cov3d.m[2][2];
      opac = w.opacity;
      if (a.acc) {
#pragma unroll
        for (int k = 0; k < 7; ++k) S.acc[k][r] = a.acc[k * (size_t)n + g];
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const float* cf = S.sh + r * L::kSh;
    auto coeff = [&](int k, int ch) { return cf[k * 3 + ch]; };
    float sg[NSH];
#pragma unroll
    for (int i = 0; i < NSH; ++i) sg[i] = 0.f;
    float vm[3] = {}, vcov[6] = {}, vop = 0.f, seen = 0.f;
    for (uint32_t v = 0; v < nv; ++v) {
      const int32_t c = c_cur;
      if (v + 1 < nv)
        issue(v + 1, c_nxt);
      else
        cp_async_commit();
      c_cur = c_nxt;
      c_nxt = own && v + 2 < nv ? slice(a.b.c_of_gid, a.b.Ncap, v + 2)[g] : -1;
      cp_async_wait1();  // view v's record has landed
      float st[7] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (c >= 0) {
        const float4 q0 = S.rec[v & 1][0][r], q1 = S.rec[v & 1][1][r], q2 = S.rec[v & 1][2][r];
        const BwdView& w = s_view[v];
        ViewAdjoint o = view_adjoint(w, mean, c3, opac, a.cov_blur, q0, q1, q2, a.exact != 0, a.hp != 0);
        // View direction (view_dir) and the mean's gradient through it
        // (sh_viewdir_vjp).
        V3<float> dir{mean.x - w.campos[0], mean.y - w.campos[1], mean.z - w.campos[2]};
        const float n2 = dir.x * dir.x + dir.y * dir.y + dir.z * dir.z;
        const float rn = 1.f / sqrtf(fmaxf(n2, 1e-12f));
        dir = V3<float>{dir.x * rn, dir.y * rn, dir.z * rn};
        const float rgb[3] = {q1.y, q1.z, q1.w};
        if (dir_term) {
          float wk[25];
          wk[0] = 0.f;
#pragma unroll
          for (int k = 1; k < K; ++k) wk[k] = rgb[0] * coeff(k, 0) + rgb[1] * coeff(k, 1) + rgb[2] * coeff(k, 2);
          const V3<float> gd = sh_weighted_grad<float>(DEG, dir.x, dir.y, dir.z, wk);
          const float ug = n2 > 1e-12f ? dir.x * gd.x + dir.y * gd.y + dir.z * gd.z : 0.f;
          o.v_mean.x += (gd.x - dir.x * ug) * rn;
          o.v_mean.y += (gd.y - dir.y * ug) * rn;
          o.v_mean.z += (gd.z - dir.z * ug) * rn;
        }
        vm[0] += o.v_mean.x;
        vm[1] += o.v_mean.y;
        vm[2] += o.v_mean.z;
#pragma unroll
        for (int k = 0; k < 6; ++k) vcov[k] += o.v_cov[k];
        vop += o.v_raw_opac;
        float bas[25];
        sh_basis<float>(DEG, dir.x, dir.y, dir.z, bas);
        float bsum = 0.f;
#pragma unroll
        for (int k = 0; k < K; ++k) {
          bsum += fabsf(bas[k]);
#pragma unroll
          for (int ch = 0; ch < 3; ++ch) sg[k * 3 + ch] += bas[k] * rgb[ch];
        }
        // project_backwards.wgsl:33-36, 105-108.
        st[0] = q0.x;
        st[1] = q0.y;
        st[2] = q2.y;
        st[3] = q2.z;
        st[4] = q2.w * sqrtf(q2.y * q2.y + q2.z * q2.z);
        st[5] = q2.w;
        st[6] = q2.w * o.depth;
        if (a.acc) {
          // Densification quantities of this view (engine/trainer.rs:660-727),
          // one view at a time, in view order, as a per-view accumulation does.
          // A third, correctly rounded: a quotient by 3 lies too far from the middle
          // of two floats for the product in 64 bits to round otherwise.
          S.acc[0][r] += (float)((double)(fabsf(o.v_mean.x) + fabsf(o.v_mean.y) + fabsf(o.v_mean.z)) * (1.0 / 3.0));
          S.acc[1][r] += sqrtf(st[0] * st[0] + st[1] * st[1]);
          S.acc[2][r] += sqrtf(st[2] * st[2] + st[3] * st[3]);
          S.acc[3][r] += st[4];
          S.acc[4][r] += st[5];
          S.acc[5][r] += st[6];
          // Mean over coefficients of the channel mean of |basis * v_rgb|.
          S.acc[6][r] += bsum * (fabsf(rgb[0]) + fabsf(rgb[1]) + fabsf(rgb[2])) * (1.0f / (float)NSH);
          if (a.use_visible && slice(a.b.visible_c, a.b.Vcap, v)[c]) seen += 1.f;
        }
      }
      if (own && a.stats) {
        float* so = a.stats + ((size_t)v * n + g) * 7;
#pragma unroll
        for (int k = 0; k < 7; ++k) so[k] = st[k];
      }
    }
    if (own && a.acc) {
#pragma unroll
      for (int k = 0; k < 7; ++k) a.acc[k * (size_t)n + g] = S.acc[k][r];
      // Counts: whole numbers, so that adding them at once rounds no otherwise
      // than one by one (below 2^24).
      a.acc[7 * (size_t)n + g] += (float)nv;
      a.acc[8 * (size_t)n + g] += a.use_visible ? seen : (float)nv;
    }
    // The covariance's gradient into scales and quaternion.
    float gt[10];
    gt[0] = vm[0];
    gt[1] = vm[1];
    gt[2] = vm[2];
#pragma unroll
    for (int k = 3; k < 10; ++k) gt[k] = 0.f;
    bool any = false;
#pragma unroll
    for (int k = 0; k < 6; ++k) any = any || vcov[k] != 0.f;
    if (any) {
      // Read again rather than held through the views.
      const float2 t23 = t2[1], t45 = t2[2], t67 = t2[3], t89 = t2[4];
      const V4<float> quat{t23.y, t45.x, t45.y, t67.x};
      const V3<float> ls{t67.y, t89.x, t89.y};
      const float rs = 1.f / sqrtf(quat.x * quat.x + quat.y * quat.y + quat.z * quat.z + quat.w * quat.w);
      const V4<float> q{quat.x * rs, quat.y * rs, quat.z * rs, quat.w * rs};
      const V3<float> scale{gexp(ls.x), gexp(ls.y), gexp(ls.z)};
      const M3<float> rot = quat_to_mat3(q);
      M3<float> v2;
      v2.m[0][0] = 2.f * vcov[0];
      v2.m[0][1] = v2.m[1][0] = 2.f * vcov[1];
      v2.m[0][2] = v2.m[2][0] = 2.f * vcov[2];
      v2.m[1][1] = 2.f * vcov[3];
      v2.m[1][2] = v2.m[2][1] = 2.f * vcov[4];
      v2.m[2][2] = 2.f * vcov[5];
      const M3<float> v_m = mul(v2, rot_scale(rot, scale));
      const float sv[3] = {scale.x, scale.y, scale.z};
#pragma unroll
      for (int j = 0; j < 3; ++j)
        gt[7 + j] =
            (rot.m[j][0] * v_m.m[j][0] + rot.m[j][1] * v_m.m[j][1] + rot.m[j][2] * v_m.m[j][2]) * sv[j];
      const V4<float> vq = normalize_vjp_apply(quat, quat_to_mat3_vjp(q, rot_scale(v_m, scale)));
      gt[3] = vq.x;
      gt[4] = vq.y;
      gt[5] = vq.z;
      gt[6] = vq.w;
    }
    __syncthreads();  // every thread is done with the SH values
    float* tg = S.tr + r * L::kTr;
#pragma unroll
    for (int k = 0; k < 10; ++k) tg[k] = gt[k] * sc;
    tg[10] = vop * sc;
    float* sgr = S.sh + r * L::kSh;
    if constexpr (L::kQuads) {
#pragma unroll
      for (int i = 0; i < NSH; i += 4)
        st4(sgr + i, make_float4(sg[i] * sc, sg[i + 1] * sc, sg[i + 2] * sc, sg[i + 3] * sc));
    } else {
#pragma unroll
      for (int i = 0; i < NSH; ++i) sgr[i] = sg[i] * sc;
    }
    __syncthreads();
    const size_t s0 = (size_t)g0 * NSH, t0 = (size_t)g0 * 10;
    const uint32_t ns = rows * NSH, nt = rows * 10;
    const uint32_t qs = a.vec_sh ? ns / 4 : 0, qt = a.vec_tr ? nt / 4 : 0;
    auto sh4 = [&](uint32_t e) {
      if constexpr (L::kQuads) return ld4(S.sh + sh_place<K>(e));
      return make_float4(S.sh[sh_place<K>(e)], S.sh[sh_place<K>(e + 1)], S.sh[sh_place<K>(e + 2)],
                         S.sh[sh_place<K>(e + 3)]);
    };
    auto tr1 = [&](uint32_t e) { return S.tr[(e / 10) * L::kTr + e % 10]; };
    if (!a.adam) {
      for (uint32_t q = r; q < qs; q += kGT) st4(a.v_sh + s0 + 4 * q, sh4(4 * q));
      for (uint32_t e = 4 * qs + r; e < ns; e += kGT) a.v_sh[s0 + e] = S.sh[sh_place<K>(e)];
      for (uint32_t q = r; q < qt; q += kGT)
        st4(a.v_tr + t0 + 4 * q, make_float4(tr1(4 * q), tr1(4 * q + 1), tr1(4 * q + 2), tr1(4 * q + 3)));
      for (uint32_t e = 4 * qt + r; e < nt; e += kGT) a.v_tr[t0 + e] = tr1(e);
      if (own) a.v_op[g] = tg[10];
    } else {
      const AdamScalars ad = *a.ad.scal;
      SHT* psh = reinterpret_cast<SHT*>(a.ad.sh) + s0;
#pragma unroll 4
      for (uint32_t q = r; q < qs; q += kGT) {
        const uint32_t e = 4 * q;
        float4 P = ld4(psh + e), M = ld4(a.ad.m_sh + s0 + e), Q = ld4(a.ad.v_sh + s0 + e);
        const float4 G = sh4(e);
        P.x = adam_one(P.x, G.x, M.x, Q.x, ad.lr_color, ad);
        P.y = adam_one(P.y, G.y, M.y, Q.y, ad.lr_color, ad);
        P.z = adam_one(P.z, G.z, M.z, Q.z, ad.lr_color, ad);
        P.w = adam_one(P.w, G.w, M.w, Q.w, ad.lr_color, ad);
        st4(psh + e, P);
        st4(a.ad.m_sh + s0 + e, M);
        st4(a.ad.v_sh + s0 + e, Q);
      }
      for (uint32_t e = 4 * qs + r; e < ns; e += kGT)
        store_sh(psh + e, adam_one(to_f(psh[e]), S.sh[sh_place<K>(e)], a.ad.m_sh[s0 + e], a.ad.v_sh[s0 + e],
                                   ad.lr_color, ad));
      float* ptr = a.ad.transforms + t0;
      for (uint32_t q = r; q < qt; q += kGT) {
        const uint32_t e = 4 * q;
        float4 P = ld4(ptr + e), M = ld4(a.ad.m_tr + t0 + e), Q = ld4(a.ad.v_tr + t0 + e);
        P.x = adam_one(P.x, tr1(e), M.x, Q.x, group_lr(ad, 0, e % 10), ad);
        P.y = adam_one(P.y, tr1(e + 1), M.y, Q.y, group_lr(ad, 0, (e + 1) % 10), ad);
        P.z = adam_one(P.z, tr1(e + 2), M.z, Q.z, group_lr(ad, 0, (e + 2) % 10), ad);
        P.w = adam_one(P.w, tr1(e + 3), M.w, Q.w, group_lr(ad, 0, (e + 3) % 10), ad);
        st4(ptr + e, P);
        st4(a.ad.m_tr + t0 + e, M);
        st4(a.ad.v_tr + t0 + e, Q);
      }
      for (uint32_t e = 4 * qt + r; e < nt; e += kGT)
        ptr[e] = adam_one(ptr[e], tr1(e), a.ad.m_tr[t0 + e], a.ad.v_tr[t0 + e], group_lr(ad, 0, e % 10), ad);
      if (own) a.ad.raw_opac[g] = adam_one(a.ad.raw_opac[g], tg[10], a.ad.m_op[g], a.ad.v_op[g], ad.lr_opac, ad);
    }
  }
}

template <class SHT, int DEG> cudaError_t launch_gather(int blocks, cudaStream_t st, const GatherArgs& a) {
  constexpr int K = (DEG + 1) * (DEG + 1);
  constexpr size_t most = sizeof(GatherSmem<K>) + sizeof(BwdView) * kMaxViews;
  cudaError_t e = cudaFuncSetAttribute(gather_kernel<SHT, DEG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
  if (e != cudaSuccess) return e;
  gather_kernel<SHT, DEG><<<blocks, kGT, sizeof(GatherSmem<K>) + sizeof(BwdView) * a.vs.n_views, st>>>(a);
  return cudaGetLastError();
}

template <class SHT>
cudaError_t dispatch_gather(int degree, int blocks, cudaStream_t st, const GatherArgs& a) {
  switch (degree) {
    case 0: return launch_gather<SHT, 0>(blocks, st, a);
    case 1: return launch_gather<SHT, 1>(blocks, st, a);
    case 2: return launch_gather<SHT, 2>(blocks, st, a);
    case 3: return launch_gather<SHT, 3>(blocks, st, a);
    default: return launch_gather<SHT, 4>(blocks, st, a);
  }
}

// Element-wise Adam over one parameter group (0 transforms: columns 3
// position, 4 rotation, 3 scale; 1 SH coefficients; 2 opacities). Four
// elements per thread with 16-byte loads and stores when every array is
// aligned for them (vec), the remainder one by one.
template <class PT>
__global__ void __launch_bounds__(256) adam_kernel(PT* p, const float* g, float* m, float* v, uint64_t n, int group,
                                                   int vec, const AdamScalars* scal) {
  const AdamScalars a = *scal;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t t0 = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t nq = vec ? n / 4 : 0;
  for (uint64_t q = t0; q < nq; q += stride) {
    const uint64_t i = q * 4;
    float4 P = ld4(p + i);
    const float4 G = ld4(g + i);
    float4 M = ld4(m + i), Vv = ld4(v + i);
    uint32_t col = group == 0 ? (uint32_t)(i % 10u) : 0u;
    auto step = [&](float& pp, float gg, float& mm, float& vv) {
      pp = adam_one(pp, gg, mm, vv, group_lr(a, group, col), a);
      if (++col == 10u) col = 0u;
    };
    step(P.x, G.x, M.x, Vv.x);
    step(P.y, G.y, M.y, Vv.y);
    step(P.z, G.z, M.z, Vv.z);
    step(P.w, G.w, M.w, Vv.w);
    st4(p + i, P);
    st4(m + i, M);
    st4(v + i, Vv);
  }
  for (uint64_t i = nq * 4 + t0; i < n; i += stride) {
    const uint32_t col = group == 0 ? (uint32_t)(i % 10u) : 0u;
    store_sh(p + i, adam_one(to_f(p[i]), g[i], m[i], v[i], group_lr(a, group, col), a));
  }
}

__global__ void set_scalars_kernel(AdamScalars* dst, AdamScalars v) { *dst = v; }

__global__ void densify_kernel(const float* v_tr, const float* stats, const float* v_sh, const float* visible,
                               uint32_t n, int K, int use_visible, float* acc) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float* t = v_tr + (size_t)i * 10;
    const float* s = stats + (size_t)i * 7;
    const float g2 = (fabsf(t[0]) + fabsf(t[1]) + fabsf(t[2])) / 3.0f;
    float gc = 0.f;
    for (int k = 0; k < K; ++k) {
      const float* c = v_sh + ((size_t)i * K + k) * 3;
      gc = gc + (fabsf(c[0]) + fabsf(c[1]) + fabsf(c[2])) / 3.0f;
    }
    gc = gc / (float)K;
    acc[0 * (size_t)n + i] += g2;
    acc[1 * (size_t)n + i] += sqrtf(s[0] * s[0] + s[1] * s[1]);
    acc[2 * (size_t)n + i] += sqrtf(s[2] * s[2] + s[3] * s[3]);
    acc[3 * (size_t)n + i] += s[4];
    acc[4 * (size_t)n + i] += s[5];
    acc[5 * (size_t)n + i] += s[6];
    acc[6 * (size_t)n + i] += gc;
    acc[7 * (size_t)n + i] += 1.0f;
    acc[8 * (size_t)n + i] += use_visible ? visible[i] : 1.0f;
  }
}

}  // namespace

cudaError_t launch_set_scalars(AdamScalars* dst, const AdamScalars& v, cudaStream_t st) {
  set_scalars_kernel<<<1, 1, 0, st>>>(dst, v);
  return cudaGetLastError();
}

namespace {
bool aligned(const void* p, uintptr_t to) { return (reinterpret_cast<uintptr_t>(p) & (to - 1)) == 0; }
}  // namespace

cudaError_t launch_project_bwd(const SplatsDev& sp, const ViewSet& vs, float cov_blur, FwdBufs& b,
                               const ProjBwdArgs& pa, cudaStream_t st, int num_sms) {
  if (sp.n == 0) return cudaSuccess;
  GatherArgs a{};
  a.sp = sp;
  a.vs = vs;
  a.b = b;
  a.cov_blur = cov_blur;
  a.v_tr = pa.v_tr;
  a.v_sh = pa.v_sh;
  a.v_op = pa.v_op;
  a.stats = pa.stats;
  a.acc = pa.densify_acc;
  a.use_visible = pa.use_visible;
  a.grad_scale = pa.grad_scale;
  a.exact = pa.exact;
  a.hp = pa.hp;
  a.adam = pa.adam != nullptr;
  a.vec_sh = aligned(sp.sh, sp.sh_bf16 ? 8 : 16);
  if (pa.adam) {
    a.ad = *pa.adam;
    a.vec_sh = a.vec_sh && aligned(a.ad.m_sh, 16) && aligned(a.ad.v_sh, 16);
    a.vec_tr = aligned(a.ad.transforms, 16) && aligned(a.ad.m_tr, 16) && aligned(a.ad.v_tr, 16);
  } else {
    a.vec_sh = a.vec_sh && aligned(pa.v_sh, 16);
    a.vec_tr = aligned(pa.v_tr, 16);
  }
  int blocks = (int)((sp.n + kGT - 1) / kGT);
  const int cap = num_sms * 8;
  if (blocks > cap) blocks = cap;
  return sp.sh_bf16 ? dispatch_gather<__nv_bfloat16>(sp.degree, blocks, st, a)
                    : dispatch_gather<float>(sp.degree, blocks, st, a);
}

namespace {
template <class PT>
void adam_group(PT* p, const float* g, float* m, float* v, uint64_t n, int group, const AdamScalars* scal,
                cudaStream_t st, int num_sms) {
  if (n == 0) return;
  const int vec = aligned(p, 4 * sizeof(PT)) && aligned(g, 16) && aligned(m, 16) && aligned(v, 16);
  const uint64_t units = vec ? (n + 3) / 4 : n;
  uint64_t blocks = (units + 255) / 256;
  const uint64_t cap = (uint64_t)num_sms * 8;
  if (blocks > cap) blocks = cap;
  adam_kernel<PT><<<(unsigned)blocks, 256, 0, st>>>(p, g, m, v, n, group, vec, scal);
}
}  // namespace

cudaError_t launch_adam(const AdamArgs& a, const float* g_tr, const float* g_sh, const float* g_op, uint32_t n,
                        int degree, int sh_bf16, cudaStream_t st, int num_sms) {
  if (n == 0) return cudaSuccess;
  const uint64_t nsh = (uint64_t)n * (degree + 1) * (degree + 1) * 3;
  adam_group<float>(a.transforms, g_tr, a.m_tr, a.v_tr, (uint64_t)n * 10, 0, a.scal, st, num_sms);
  if (sh_bf16)
    adam_group<__nv_bfloat16>(reinterpret_cast<__nv_bfloat16*>(a.sh), g_sh, a.m_sh, a.v_sh, nsh, 1, a.scal, st,
                              num_sms);
  else
    adam_group<float>(reinterpret_cast<float*>(a.sh), g_sh, a.m_sh, a.v_sh, nsh, 1, a.scal, st, num_sms);
  adam_group<float>(a.raw_opac, g_op, a.m_op, a.v_op, n, 2, a.scal, st, num_sms);
  return cudaGetLastError();
}

cudaError_t launch_densify(const float* v_tr, const float* stats, const float* v_sh, const float* visible, uint32_t n,
                           int degree, int use_visible, float* acc, cudaStream_t st, int num_sms) {
  if (n == 0) return cudaSuccess;
  const int K = (degree + 1) * (degree + 1);
  densify_kernel<<<num_sms * 8, 256, 0, st>>>(v_tr, stats, v_sh, visible, n, K, use_visible, acc);
  return cudaGetLastError();
}

}  // namespace gsr
