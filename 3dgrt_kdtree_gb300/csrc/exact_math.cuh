// exact_math.cuh -- the reference's per-ray operations in the reference's
// order, in IEEE round-to-nearest FP32: every operation is an explicit
// __f*_rn intrinsic, which the compiler never contracts, so results do not
// depend on a unit's flags.
#pragma once
#include <cfloat>
#include <cstdint>
#include <cuda_runtime.h>

#include "device_common.cuh"
#include "kdgr_math.h"

namespace kdgr {
namespace {

struct F3 {
  float x, y, z;
};
__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fs(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fd(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ float fq(float a) { return __fsqrt_rn(a); }
__device__ __forceinline__ F3 mk(float x, float y, float z) { return F3{x, y, z}; }
__device__ __forceinline__ F3 add(F3 a, F3 b) { return mk(fa(a.x, b.x), fa(a.y, b.y), fa(a.z, b.z)); }
__device__ __forceinline__ F3 sub(F3 a, F3 b) { return mk(fs(a.x, b.x), fs(a.y, b.y), fs(a.z, b.z)); }
__device__ __forceinline__ F3 mulv(F3 a, F3 b) { return mk(fm(a.x, b.x), fm(a.y, b.y), fm(a.z, b.z)); }
__device__ __forceinline__ F3 muls(F3 a, float s) { return mk(fm(a.x, s), fm(a.y, s), fm(a.z, s)); }
__device__ __forceinline__ float dot(F3 a, F3 b) { return fa(fa(fm(a.x, b.x), fm(a.y, b.y)), fm(a.z, b.z)); }
__device__ __forceinline__ F3 cross(F3 a, F3 b) {
  return mk(fs(fm(a.y, b.z), fm(a.z, b.y)), fs(fm(a.z, b.x), fm(a.x, b.z)), fs(fm(a.x, b.y), fm(a.y, b.x)));
}

__device__ __forceinline__ F3 mat_mul(F3 p, const F3 m[3]) { return mk(dot(m[0], p), dot(m[1], p), dot(m[2], p)); }

// rayPrimIntersect with VOLUME_ISECT (cudaRenderer.cu:1070-1135).
__device__ __forceinline__ bool exact_test(F3 o, F3 d, const float4* __restrict__ rec, float t_near, float t_far,
                                           float* t_out, float* gray_out) {
  const float4 r0 = __ldg(rec), r1 = __ldg(rec + 1), r2 = __ldg(rec + 2), r3 = __ldg(rec + 3), r4 = __ldg(rec + 4);
  const F3 pos = mk(r0.x, r0.y, r0.z);
  const F3 giscl = mk(r1.x, r1.y, r1.z);
  const F3 pscale = mk(r1.w, r2.x, r2.y);
  const F3 rt[3] = {mk(r2.z, r2.w, r3.x), mk(r3.y, r3.z, r3.w), mk(r4.x, r4.y, r4.z)};
  const F3 gposc = sub(o, pos);
  const F3 gposcr = mat_mul(gposc, rt);
  const F3 gro = mulv(giscl, gposcr);
  const F3 ray_dir_r = mat_mul(d, rt);
  const F3 grdu = mulv(ray_dir_r, giscl);
  // safe_normalize with rsqrtf -> 1/sqrtf
  const float l = fa(fa(fm(grdu.x, grdu.x), fm(grdu.y, grdu.y)), fm(grdu.z, grdu.z));
  const F3 grd = l > 0.f ? muls(grdu, fd(1.f, fq(l))) : grdu;
  const float grp = -dot(grd, gro);
  const F3 grds = muls(mulv(pscale, grd), grp);
  const float t = fm(grp < 0.f ? -1.f : 1.f, fq(dot(grds, grds)));
  if (t < t_near || t > t_far) return false;
  const F3 gcrod = cross(grd, gro);
  const float gray = dot(gcrod, gcrod);
  *t_out = t;
  *gray_out = gray;
  return gray < 8.f;
}

// eval_sh_final(3, dir, g) (cudaRenderer.cu:487-558), constants
// cudaRenderer.h:33-48.
__device__ __forceinline__ F3 eval_sh(F3 d, const float4* __restrict__ shp) {
  float c[48];
#pragma unroll
  for (int i = 0; i < 12; ++i) {
    const float4 v = __ldg(shp + i);
    c[4 * i] = v.x;
    c[4 * i + 1] = v.y;
    c[4 * i + 2] = v.z;
    c[4 * i + 3] = v.w;
  }
#define SH(k) mk(c[3 * (k)], c[3 * (k) + 1], c[3 * (k) + 2])
  const float C0 = 0.28209479177387814f, C1 = 0.4886025119029199f;
  const float C20 = 1.0925484305920792f, C21 = -1.0925484305920792f, C22 = 0.31539156525252005f,
              C23 = -1.0925484305920792f, C24 = 0.5462742152960396f;
  const float C30 = -0.5900435899266435f, C31 = 2.890611442640554f, C32 = -0.4570457994644658f,
              C33 = 0.3731763325901154f, C34 = -0.4570457994644658f, C35 = 1.445305721320277f,
              C36 = -0.5900435899266435f;
  F3 rad = muls(SH(0), C0);
  const float x = d.x, y = d.y, z = d.z;
  rad = sub(add(sub(rad, muls(SH(1), fm(C1, y))), muls(SH(2), fm(C1, z))), muls(SH(3), fm(C1, x)));
  const float xx = fm(x, x), yy = fm(y, y), zz = fm(z, z);
  const float xy = fm(x, y), yz = fm(y, z), xz = fm(x, z);
  rad = add(rad, muls(SH(4), fm(C20, xy)));
  rad = add(rad, muls(SH(5), fm(C21, yz)));
  rad = add(rad, muls(SH(6), fm(C22, fs(fs(fm(2.f, zz), xx), yy))));
  rad = add(rad, muls(SH(7), fm(C23, xz)));
  rad = add(rad, muls(SH(8), fm(C24, fs(xx, yy))));
  rad = add(rad, muls(SH(9), fm(fm(C30, y), fs(fm(3.f, xx), yy))));
  rad = add(rad, muls(SH(10), fm(fm(C31, xy), z)));
  rad = add(rad, muls(SH(11), fm(fm(C32, y), fs(fs(fm(4.f, zz), xx), yy))));
  rad = add(rad, muls(SH(12), fm(fm(C33, z), fs(fs(fm(2.f, zz), fm(3.f, xx)), fm(3.f, yy)))));
  rad = add(rad, muls(SH(13), fm(fm(C34, x), fs(fs(fm(4.f, zz), xx), yy))));
  rad = add(rad, muls(SH(14), fm(fm(C35, z), fs(xx, yy))));
  rad = add(rad, muls(SH(15), fm(fm(C36, x), fs(xx, fm(3.f, yy)))));
#undef SH
  rad = add(rad, mk(0.5f, 0.5f, 0.5f));
  return mk(fmaxf(rad.x, 0.f), fmaxf(rad.y, 0.f), fmaxf(rad.z, 0.f));
}

// BoundsRayIntersect (cudaRenderer.cu:379-399) with IEEE division.
__device__ __forceinline__ bool exact_bounds(const float bmin[3], const float bmax[3], F3 o, F3 d, float* t0,
                                             float* t1) {
  float tmin = 1e-2f, tmax = FLT_MAX;
  const float oo[3] = {o.x, o.y, o.z}, dd[3] = {d.x, d.y, d.z};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float l1 = fd(fs(bmin[a], oo[a]), dd[a]);
    const float l2 = fd(fs(bmax[a], oo[a]), dd[a]);
    tmin = fmaxf(fminf(l1, l2), tmin);
    tmax = fminf(fmaxf(l1, l2), tmax);
  }
  *t0 = tmin;
  *t1 = tmax;
  return (tmax >= tmin) & (tmax >= 0.f);
}

// Composite one accepted hit (cudaRenderer.cu:1611-1687): false when it is
// skipped (response or alpha too small).
__device__ __forceinline__ bool exact_blend(const float4* __restrict__ rec, const float4* __restrict__ shp, F3 d,
                                            float t, float g, F3& acc, float& A, float& D) {
  const float opacity = __ldg(&rec->w);
  const float gres = kdgr_expf(fm(fm(-0.0555555555556f, g), g));
  const float alpha = fminf(0.99f, fm(opacity, gres));
  if (gres < 0.0113f || alpha < 1.0f / 255.0f) return false;
  const F3 c = eval_sh(d, shp);
  const float w = fm(alpha, fs(1.f, A));
  acc = add(acc, muls(muls(c, alpha), fs(1.f, A)));
  D = fa(D, fm(t, w));
  A = fa(A, fm(alpha, fs(1.f, A)));
  return true;
}

}  // namespace
}  // namespace kdgr
