// render_packet.cuh -- the ray walk of the render kernels: candidate pairs, the
// hit buffer, lane groups, warp packets and the per-ray walk, for the fast
// forms (render_fast.cu) and the plain form (render_exact.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cfloat>
#include <cstdint>
#include <cstring>
#include <type_traits>

#include "device_common.cuh"
#include "exact_math.cuh"

namespace kdgr {
namespace {

constexpr int kWarps = 4;
constexpr int kThreads = kWarps * 32;
constexpr int kTileW = 8, kTileH = 4;     // pixels per warp tile
constexpr int kBlockW = 16, kBlockH = 8;  // pixels per CTA block (4 warp tiles)
#ifndef KDGR_FAST_HITS
#define KDGR_FAST_HITS 4
#endif
#ifndef KDGR_FAST_STACK
#define KDGR_FAST_STACK 12
#endif
constexpr int kHits = KDGR_FAST_HITS;  // hit-buffer entries per leaf pass (a leaf averages <1 hit)

// Scene forms: the FP32 and the packed fast form (FastView), and the plain,
// oracle-matching form (PlainView).
constexpr int kFormFp32 = 0, kFormPacked = 1, kFormPlain = 2;
template <int FORM>
using SceneOf = std::conditional_t<FORM == kFormPlain, PlainView, FastView>;

__device__ __forceinline__ float dot3(F3 a, F3 b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, a.z * b.z)); }

__device__ __forceinline__ float bf16lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }
__device__ __forceinline__ float2 h2f(uint32_t w) {
  __half2 h;
  memcpy(&h, &w, 4);
  return __half22float2(h);
}

// ----------------------------------------------------------- candidate test
// Candidate records.  FP32 form: rows of M = diag(1/s) R^T with b = M mu
// (FP64 upload precompute), read as interleaved pairs (load_pair below).
// Storing Sigma^-1 = M^T M instead would square the condition number (a
// scale ratio of 2500 gives ~6e6, beyond FP32), so the factor is kept.
// ------------------------------------------------- paired FP32x2 candidate test
// Both forms store leaf entries in pairs: pair p holds entries 2p and 2p+1
// interleaved, so every quantity of the test is one 64-bit register with
// entry 2p in the low and entry 2p+1 in the high half, and one packed FP32x2
// instruction (fma/mul/add/sub.rn.f32x2) does the work of two.
// FP32 pair, 6 x 16 bytes, for rows i = 0..2 of M and b = M mu:
//   q[2i]   = (M_i0 lo, M_i0 hi, M_i1 lo, M_i1 hi)
//   q[2i+1] = (M_i2 lo, M_i2 hi, b_i lo, b_i hi)
// Packed pair, 4 x 16 bytes (FP32 means, FP16 M as half2 (lo, hi)):
//   w[0] = (mu.x lo, mu.x hi, mu.y lo, mu.y hi)
//   w[1] = (mu.z lo, mu.z hi, M00, M01)
//   w[2] = (M02, M10, M11, M12)
//   w[3] = (M20, M21, M22, flags)   flags bit k: entry k reads the FP32 factors
//                                   of the FP64 upload precompute instead; its
//                                   mean.x slot then holds the table index
typedef unsigned long long f2;

__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
  f2 d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 bcast2(float x) {
  f2 d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x));
  return d;
}
__device__ __forceinline__ void split2(f2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2 join2(float lo, float hi) {
  f2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ f2 h2f2(uint32_t w) {  // half2 -> (lo, hi) FP32 pair
  const float2 f = h2f(w);
  return join2(f.x, f.y);
}
__device__ __forceinline__ f2 u2f2(uint32_t lo, uint32_t hi) {
  return join2(__uint_as_float(lo), __uint_as_float(hi));
}

struct PairRec {
  ulonglong2 q[6];
};

template <typename SV>
__device__ __forceinline__ PairRec load_pair(const SV& S, uint32_t p) {
  const ulonglong2* a = reinterpret_cast<const ulonglong2*>(S.leaf_pairs) + 6ull * p;
  PairRec r;
#pragma unroll
  for (int k = 0; k < 6; ++k) r.q[k] = __ldg(a + k);
  return r;
}

// Ray constants of the pair test, broadcast to both halves once per leaf.
struct Ray2 {
  f2 nox, noy, noz, dx, dy, dz;
};
__device__ __forceinline__ Ray2 ray2(F3 o, F3 d) {
  return Ray2{bcast2(-o.x), bcast2(-o.y), bcast2(-o.z), bcast2(d.x), bcast2(d.y), bcast2(d.z)};
}

// The M-form test (grdu = M d, ng = M (mu - o), t* = (grdu . ng) / |grdu|^2,
// gray = |grdu x ng|^2 / |grdu|^2) for both entries of a pair, in two steps:
// pair_t decides t* in [t_near, t_far), pair_g the response bound, so a warp
// packet can skip the second step together when no lane's t* is in range.
struct PairT {
  f2 ng[3], gd[3];
  float q0, q1, a0, a1;
};
__device__ __forceinline__ unsigned pair_t(PairT& p, float t_near, float t_far) {
  const f2 q = fma2(p.gd[0], p.gd[0], fma2(p.gd[1], p.gd[1], mul2(p.gd[2], p.gd[2])));
  const f2 a = fma2(p.gd[0], p.ng[0], fma2(p.gd[1], p.ng[1], mul2(p.gd[2], p.ng[2])));
  // t* = a / q in [t_near, t_far)  <=>  a - t_near q >= 0 and a - t_far q < 0  (q > 0),
  // each difference formed by one fused multiply-add and read by its sign.
  // A leaf's t_far is the next leaf's t_near, so one rounded difference
  // decides both sides of a split plane: a Gaussian straddling it is
  // accepted in exactly one of the two leaves.  Padding entries (q = a = 0)
  // give +0 on both sides and are refused.
  const f2 lo = fma2(q, bcast2(-t_near), a), hi = fma2(q, bcast2(-t_far), a);
  float q0, q1, a0, a1, l0, l1, h0, h1;
  split2(q, q0, q1);
  split2(a, a0, a1);
  split2(lo, l0, l1);
  split2(hi, h0, h1);
  p.q0 = q0;
  p.q1 = q1;
  p.a0 = a0;
  p.a1 = a1;
  const uint32_t m0 = __float_as_uint(h0) & ~__float_as_uint(l0), m1 = __float_as_uint(h1) & ~__float_as_uint(l1);
  return (m0 >> 31) | ((m1 >> 31) << 1);
}
// FP32 pair: ng = b - M o.
template <typename P>
__device__ __forceinline__ void setup_pair(const PairRec& r, const Ray2& w, P& p) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const f2 m0 = r.q[2 * i].x, m1 = r.q[2 * i].y, m2 = r.q[2 * i + 1].x, b = r.q[2 * i + 1].y;
    p.ng[i] = fma2(m0, w.nox, fma2(m1, w.noy, fma2(m2, w.noz, b)));
    p.gd[i] = fma2(m0, w.dx, fma2(m1, w.dy, mul2(m2, w.dz)));
  }
}

struct PPairRec {
  uint4 w[4];
};

// Packed pair: FP16 rows of M, FP32 mean, ng = M (mu - o) (no M o - M mu
// cancellation, so the FP16 rounding stays a small consistent perturbation
// of the Gaussian).
__device__ __forceinline__ void setup_ppair(const PPairRec& r, const Ray2& w, PairT& p) {
  const f2 nqx = add2(u2f2(r.w[0].x, r.w[0].y), w.nox);
  const f2 nqy = add2(u2f2(r.w[0].z, r.w[0].w), w.noy);
  const f2 nqz = add2(u2f2(r.w[1].x, r.w[1].y), w.noz);
  const uint32_t mw[9] = {r.w[1].z, r.w[1].w, r.w[2].x, r.w[2].y, r.w[2].z, r.w[2].w, r.w[3].x, r.w[3].y, r.w[3].z};
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const f2 m0 = h2f2(mw[3 * i]), m1 = h2f2(mw[3 * i + 1]), m2 = h2f2(mw[3 * i + 2]);
    p.ng[i] = fma2(m0, nqx, fma2(m1, nqy, mul2(m2, nqz)));
    p.gd[i] = fma2(m0, w.dx, fma2(m1, w.dy, mul2(m2, w.dz)));
  }
}

__device__ __forceinline__ PPairRec load_ppair(const FastView& S, uint32_t p) {
  const uint4* a = S.leaf_packed + 4ull * p;
  PPairRec r;
#pragma unroll
  for (int k = 0; k < 4; ++k) r.w[k] = __ldg(a + k);
  return r;
}

// A leaf of either form: `np` pairs of the main stream from pair `pb`
// (FP32 pairs, or packed FP16 pairs), then in the packed form `nf` FP32
// pairs of its flagged entries from pair `fb` (leaf_pairs holds that stream).
struct LeafRef {
  uint32_t pb, np, fb, nf;
};

template <int FORM>
__device__ __forceinline__ LeafRef leaf_ref(const SceneOf<FORM>& S, uint32_t node, uint2 nd) {
  LeafRef L{nd.y, ((nd.x >> 3) + 1) >> 1, 0u, 0u};
  if constexpr (FORM == kFormPacked) {
    const uint2 a = __ldg(S.leaf_aux + node);
    L.fb = a.x;
    L.nf = (a.y + 1) >> 1;
  }
  return L;
}

template <int FORM>
__device__ __forceinline__ bool leaf_in_bounds(const SceneOf<FORM>& S, const LeafRef& L) {
  if constexpr (FORM == kFormPlain) return 2ull * ((uint64_t)L.pb + L.np) <= S.n_offsets;
  else return 2ull * ((uint64_t)L.pb + L.np) <= S.n_offsets && 2ull * ((uint64_t)L.fb + L.nf) <= S.n_flag;
}

// The t* step for pair j of leaf L.
template <int FORM>
__device__ __forceinline__ unsigned leaf_pair_t(const FastView& S, const LeafRef& L, uint32_t j, const Ray2& w,
                                                float t_near, float t_far, PairT& p) {
  if (FORM == kFormPacked && j < L.np) {
    setup_ppair(load_ppair(S, L.pb + j), w, p);
  } else {
    setup_pair(load_pair(S, FORM == kFormPacked ? L.fb + (j - L.np) : L.pb + j), w, p);
  }
  return pair_t(p, t_near, t_far);
}

// Gaussian of leaf entry ik.
template <int FORM>
__device__ __forceinline__ uint32_t leaf_gid(const SceneOf<FORM>& S, const LeafRef& L, uint32_t ik) {
  if constexpr (FORM == kFormPacked)
    if (ik >= 2 * L.np) return __ldg(S.flag_offsets + 2 * L.fb + (ik - 2 * L.np));
  return __ldg(S.offsets + 2 * L.pb + ik);
}

__device__ __forceinline__ unsigned test_pair_g(const PairT& p, unsigned m, float t[2], float g[2]) {
  const float r0 = __fdividef(1.f, p.q0), r1 = __fdividef(1.f, p.q1);
  t[0] = p.a0 * r0;
  t[1] = p.a1 * r1;
  const f2 c0 = sub2(mul2(p.gd[1], p.ng[2]), mul2(p.gd[2], p.ng[1]));
  const f2 c1 = sub2(mul2(p.gd[2], p.ng[0]), mul2(p.gd[0], p.ng[2]));
  const f2 c2 = sub2(mul2(p.gd[0], p.ng[1]), mul2(p.gd[1], p.ng[0]));
  const f2 cc = fma2(c0, c0, fma2(c1, c1, mul2(c2, c2)));
  float cc0, cc1;
  split2(cc, cc0, cc1);
  g[0] = cc0 * r0;
  g[1] = cc1 * r1;
  if (!(g[0] < 8.f)) m &= ~1u;
  if (!(g[1] < 8.f)) m &= ~2u;
  return m;
}

template <int FORM>
__device__ __forceinline__ float gauss_opacity(const FastView& S, uint32_t gid) {
  return __ldg(S.opacity + gid);
}

// eval_sh_final(3, dir, g) (cudaRenderer.cu:487-558), FMA form.
template <int FORM>
__device__ __forceinline__ F3 eval_sh_fast(const FastView& S, uint32_t gid, F3 d) {
  float c[48];
  if (FORM != kFormPacked) {
    const float4* p = S.sh + 12ull * gid;
#pragma unroll
    for (int i = 0; i < 12; ++i) {
      const float4 v = __ldg(p + i);
      c[4 * i] = v.x;
      c[4 * i + 1] = v.y;
      c[4 * i + 2] = v.z;
      c[4 * i + 3] = v.w;
    }
  } else {
    const uint4* p = S.sh_bf16 + 6ull * gid;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const uint4 v = __ldg(p + i);
      c[8 * i] = bf16lo(v.x);
      c[8 * i + 1] = bf16hi(v.x);
      c[8 * i + 2] = bf16lo(v.y);
      c[8 * i + 3] = bf16hi(v.y);
      c[8 * i + 4] = bf16lo(v.z);
      c[8 * i + 5] = bf16hi(v.z);
      c[8 * i + 6] = bf16lo(v.w);
      c[8 * i + 7] = bf16hi(v.w);
    }
  }
  const float x = d.x, y = d.y, z = d.z;
  const float xx = x * x, yy = y * y, zz = z * z, xy = x * y, yz = y * z, xz = x * z;
  float b[16];
  b[0] = 0.28209479177387814f;
  b[1] = -0.4886025119029199f * y;
  b[2] = 0.4886025119029199f * z;
  b[3] = -0.4886025119029199f * x;
  b[4] = 1.0925484305920792f * xy;
  b[5] = -1.0925484305920792f * yz;
  b[6] = 0.31539156525252005f * (2.f * zz - xx - yy);
  b[7] = -1.0925484305920792f * xz;
  b[8] = 0.5462742152960396f * (xx - yy);
  b[9] = -0.5900435899266435f * y * (3.f * xx - yy);
  b[10] = 2.890611442640554f * xy * z;
  b[11] = -0.4570457994644658f * y * (4.f * zz - xx - yy);
  b[12] = 0.3731763325901154f * z * (2.f * zz - 3.f * xx - 3.f * yy);
  b[13] = -0.4570457994644658f * x * (4.f * zz - xx - yy);
  b[14] = 1.445305721320277f * z * (xx - yy);
  b[15] = -0.5900435899266435f * x * (xx - 3.f * yy);
  float r = 0.5f, g = 0.5f, bl = 0.5f;
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    r = fmaf(b[k], c[3 * k], r);
    g = fmaf(b[k], c[3 * k + 1], g);
    bl = fmaf(b[k], c[3 * k + 2], bl);
  }
  return mk(fmaxf(r, 0.f), fmaxf(g, 0.f), fmaxf(bl, 0.f));
}

// K smallest (t, leaf position) keys of a leaf pass, ascending; equal t keep
// leaf order (the stable sortHits, cudaRenderer.cu:415-426).
template <int K>
struct HitBuf {
  float t[K], g[K];
  uint32_t i[K];
  // only t: g and i are read where t is finite, and insert moves them with t
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int k = 0; k < K; ++k) t[k] = __int_as_float(0x7f800000);
  }
  // returns true when an entry fell off the end (the leaf needs another pass)
  __device__ __forceinline__ bool insert(float ct, float cg, uint32_t ci) {
    // t is ascending, so c[k] = ct < t[k] is false up to the insertion point
    // and true after it: every slot takes its old value, the new key or its
    // left neighbour's old value, decided without a chain between slots
    bool c[K];
#pragma unroll
    for (int k = 0; k < K; ++k) c[k] = ct < t[k];
    const float out = c[K - 1] ? t[K - 1] : ct;  // the key that falls off
#pragma unroll
    for (int k = K - 1; k > 0; --k) {
      t[k] = c[k] ? (c[k - 1] ? t[k - 1] : ct) : t[k];
      g[k] = c[k] ? (c[k - 1] ? g[k - 1] : cg) : g[k];
      i[k] = c[k] ? (c[k - 1] ? i[k - 1] : ci) : i[k];
    }
    t[0] = c[0] ? ct : t[0];
    g[0] = c[0] ? cg : g[0];
    i[0] = c[0] ? ci : i[0];
    return out != __int_as_float(0x7f800000);
  }
};

// ------------------------------------------------------------------ one ray
constexpr int kStack = KDGR_FAST_STACK;  // short-stack ring entries (ring + root restart as the reference)

// Per-lane ray state; one leaf is processed per call of leaf_step.
// The colour and depth accumulators of this thread's ray (r, g, b, depth),
// in shared memory: they change only when a hit is blended and are read
// once when the pixel is stored, so keeping them out of registers through
// the candidate loop and the descent leaves those loops fewer spills
// (64-register cap).
__device__ __forceinline__ float4* acc_slot() {
  __shared__ float4 s_acc[kThreads];
  return &s_acc[threadIdx.x];
}

struct Ray {
  F3 o, d, inv;  // inv: fast forms only
  float t_near, t_far, t_scene_far;
  float oo;  // plain form: |o|^2, for the filter's tolerance
  float A;  // opacity; colour and depth accumulate in acc_slot()
  uint32_t cur, steps;
  unsigned top, quant;
};

__device__ __forceinline__ float sel3(const F3& v, uint32_t axis) { return axis == 0 ? v.x : axis == 1 ? v.y : v.z; }

// Where the ray meets a split plane: the plain form divides, as the reference
// (cudaRenderer.cu:1560); the fast forms multiply by the reciprocal.
template <int FORM>
__device__ __forceinline__ float split_t(const Ray& R, uint32_t axis, uint32_t bits) {
  if constexpr (FORM == kFormPlain) return fd(fs(__uint_as_float(bits), sel3(R.o, axis)), sel3(R.d, axis));
  else return (__uint_as_float(bits) - sel3(R.o, axis)) * sel3(R.inv, axis);
}

// Ray generation (cudaRenderer.cu:2336-2339) and the scene-box slab test
// (:379-399).  Returns false when the ray misses the box.
__device__ __forceinline__ bool ray_init(const FastView& S, const CamInfo& C, int x, int y, Ray& R) {
  const float sx = (float)x + 0.5f, sy = (float)y + 0.5f;
  R.o = mk(__ldg(&C.eye[0]), __ldg(&C.eye[1]), __ldg(&C.eye[2]));
  const float sxx = sx * __ldg(&C.step_x), syy = sy * __ldg(&C.step_y);
  F3 d;
  d.x = __ldg(&C.start[0]) + __ldg(&C.u[0]) * sxx - __ldg(&C.v[0]) * syy - R.o.x;
  d.y = __ldg(&C.start[1]) + __ldg(&C.u[1]) * sxx - __ldg(&C.v[1]) * syy - R.o.y;
  d.z = __ldg(&C.start[2]) + __ldg(&C.u[2]) * sxx - __ldg(&C.v[2]) * syy - R.o.z;
  const float il = rsqrtf(dot3(d, d));
  R.d = mk(d.x * il, d.y * il, d.z * il);
  R.inv = mk(1.f / R.d.x, 1.f / R.d.y, 1.f / R.d.z);
  R.A = 0.f;
  *acc_slot() = make_float4(0.f, 0.f, 0.f, 0.f);
  float tmin = 1e-2f, tmax = FLT_MAX;
  const float oo[3] = {R.o.x, R.o.y, R.o.z}, iv[3] = {R.inv.x, R.inv.y, R.inv.z};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float l1 = (S.bmin[a] - oo[a]) * iv[a];
    const float l2 = (S.bmax[a] - oo[a]) * iv[a];
    tmin = fmaxf(fminf(l1, l2), tmin);
    tmax = fminf(fmaxf(l1, l2), tmax);
  }
  R.t_near = tmin;
  R.t_far = tmax;
  R.t_scene_far = tmax;
  R.cur = 0;
  R.steps = 0;
  R.top = kStack - 1;
  R.quant = 0;
  return (tmax >= tmin) & (tmax >= 0.f);
}

// ------------------------------------------------------------ plain form
// The plain form's candidate loop first discards, two candidates at a time
// in the fast form's M-form arithmetic, those whose t* is certainly outside
// the leaf interval; exact_test then decides the rest in the reference's
// operations.  With a = gd . ng and q = |gd|^2 as there, every rounding of
// the reference's chain and of this one moves a - t q by at most
//   u G (|gd| (|o| + |mu| + t) + |ng|) c,   u = 2^-24, G = |1/s|, c = 128
// (the chain's rotation, scaling and normalisation contribute at most 104 u;
// a quaternion off unit length by more than 2e-6, or a scale outside
// [1e-8, 1e8], makes the record's constants infinite: never discarded).  The
// tolerance T used is at least that for a t* in the interval (t <= t_far):
//   T^2 = Ce (q (|o|^2 + t_far^2) + |ng|^2) + Cmu q,  Ce = 2^-31 G^2,  Cmu = Ce |mu|^2
// and random records, needles of ratio 4000 along the ray among them, stayed
// below 0.065 T.  A NaN anywhere keeps the candidate.
struct PlainFilter {
  f2 tn, tf, rr;  // -t_near and -t_far widened by 2^-16, |o|^2 + t_far^2
};
__device__ __forceinline__ PlainFilter plain_filter(float tn, float tf, float oo) {
  return PlainFilter{bcast2(-tn * (1.0f - 1.52587890625e-5f)), bcast2(-tf * (1.0f + 1.52587890625e-5f)),
                     bcast2(fmaf(tf, tf, oo))};
}
// Candidates with t* in the interval for some lane of a packet are many more
// than the accepted ones, so those are filtered once more by the response
// bound |gd x ng|^2 / q < 8: the cross product is off by at most 28 of the 128
// u above (unit length does not enter), and (a + b)^2 <= 17/16 a^2 + 17 b^2
// leaves |gd x ng|^2 <= 8.5 q + T^2.
struct PlainPair {
  f2 ng[3], gd[3], q, t2;  // t2: T^2
};
// Bit k: entry k of pair p may have its t* in the interval.
__device__ __forceinline__ unsigned plain_pair_t(const PlainView& S, uint32_t p, const Ray2& w, const PlainFilter& F,
                                                 PlainPair& x) {
  setup_pair(load_pair(S, p), w, x);
  const ulonglong2 tol = __ldg(reinterpret_cast<const ulonglong2*>(S.leaf_tol) + p);
  const f2 q = x.q = fma2(x.gd[0], x.gd[0], fma2(x.gd[1], x.gd[1], mul2(x.gd[2], x.gd[2])));
  const f2 a = fma2(x.gd[0], x.ng[0], fma2(x.gd[1], x.ng[1], mul2(x.gd[2], x.ng[2])));
  const f2 g = fma2(x.ng[0], x.ng[0], fma2(x.ng[1], x.ng[1], mul2(x.ng[2], x.ng[2])));
  const f2 lo = fma2(q, F.tn, a), hi = fma2(q, F.tf, a);
  const f2 t2 = x.t2 = fma2(tol.x, g, mul2(q, fma2(tol.x, F.rr, tol.y)));
  float l0, l1, h0, h1, m0, m1;
  split2(lo, l0, l1);
  split2(hi, h0, h1);
  split2(t2, m0, m1);
  // beyond the tolerance on either side: z > T, as z |z| > T^2
  const float z0 = fmaxf(-l0, h0), z1 = fmaxf(-l1, h1);
  return (z0 * fabsf(z0) > m0 ? 0u : 1u) | (z1 * fabsf(z1) > m1 ? 0u : 2u);
}
// Bit k: entry k may pass the response bound.
__device__ __forceinline__ unsigned plain_pair_g(const PlainPair& x) {
  const f2 c0 = sub2(mul2(x.gd[1], x.ng[2]), mul2(x.gd[2], x.ng[1]));
  const f2 c1 = sub2(mul2(x.gd[2], x.ng[0]), mul2(x.gd[0], x.ng[2]));
  const f2 c2 = sub2(mul2(x.gd[0], x.ng[1]), mul2(x.gd[1], x.ng[0]));
  const f2 cc = fma2(c0, c0, fma2(c1, c1, mul2(c2, c2)));
  const f2 lim = fma2(bcast2(8.5f), x.q, x.t2);
  float c[2], m[2];
  split2(cc, c[0], c[1]);
  split2(lim, m[0], m[1]);
  return (c[0] > m[0] ? 0u : 1u) | (c[1] > m[1] ? 0u : 2u);
}

// Ray generation and scene-box test of the plain form (render_exact.cu's
// primary rays): max_t clips the interval; false when there is nothing to walk.
__device__ __forceinline__ bool ray_init_plain(const PlainView& S, const F3 o, const F3 d, float max_t, Ray& R) {
  R.o = o;
  R.d = d;
  float tmin, tmax;
  const bool hit = exact_bounds(S.bmin, S.bmax, o, d, &tmin, &tmax);
  tmax = fminf(tmax, max_t);
  R.t_near = tmin;
  R.t_far = tmax;
  R.t_scene_far = tmax;
  R.oo = dot3(o, o);
  return hit && !(tmin > tmax);
}

// ------------------------------------------------------------ lane groups
// With fewer than 32 rays per warp, each ray is held by a group of LPR
// consecutive lanes (LPR = 2, 4 or 8).  The lanes of a group hold the same ray
// state and take the same decisions; lane `sub` of the group tests pairs
// sub, sub + LPR, ... of each leaf, and the group takes its hits in key
// order from the lanes' buffers.  `mask` names the lanes that make the
// collective calls together: the whole warp (packets) or the group
// (independent rays).

// Minimum over the group of the keys (t, i), carrying g.
template <int LPR>
__device__ __forceinline__ void group_min(float& t, uint32_t& i, float& g, unsigned mask) {
#pragma unroll
  for (int o = 1; o < LPR; o <<= 1) {
    const float ot = __shfl_xor_sync(mask, t, o);
    const uint32_t oi = __shfl_xor_sync(mask, i, o);
    const float og = __shfl_xor_sync(mask, g, o);
    if (ot < t || (ot == t && oi < i)) {
      t = ot;
      i = oi;
      g = og;
    }
  }
}

__device__ __forceinline__ unsigned group_mask(int LPR) {
  const unsigned lane = threadIdx.x & 31u;
  return ((1u << LPR) - 1u) << (lane & ~(unsigned)(LPR - 1));
}

// The plain form's candidate scan (see scan_share): both filter steps, then
// the reference's test for the entries that pass.
//   PACKET: the warp takes the entries one by one, in order, each for
//     whichever lanes need it: its ID and record are warp-uniform loads.
//   otherwise the filter marks the entries of up to kChunk pairs per lane and
//     every lane then takes its own marked entries in order: lanes on
//     different leaves mark different entries, so entry by entry the
//     reference's 110 instructions would run for few lanes at a time.
//     `mask` names the lanes that run this together (0: each on its own).
// Measured (GB300, 64 or 80 registers): a 1080p packet frame 2.39 ms entry by
// entry, 2.75 ms marked (spills, 32 different records per load); a 320x240
// frame of independent rays 391 us entry by entry, 378 us marked.
// COUNT: *found counts the accepted hits.
constexpr uint32_t kChunk = 16;
template <int K, int LPR, bool PACKET, bool COUNT = false>
__device__ __forceinline__ bool scan_plain(const PlainView& S, const LeafRef& L, const Ray& R, float tn, unsigned mask,
                                           bool have_last, float last_t, uint32_t last_i, HitBuf<K>& hb,
                                           uint32_t* found = nullptr) {
  const unsigned sub = threadIdx.x & (LPR - 1u);
  bool overflow = false;
  const Ray2 w = ray2(R.o, R.d);
  const PlainFilter F = plain_filter(tn, R.t_far, R.oo);
  auto test = [&](uint32_t ik) {
    float t, g;
    const uint32_t gid = __ldg(S.offsets + 2ull * L.pb + ik);
    if (gid >= S.n_gauss || !exact_test(R.o, R.d, S.test + kTestWords * (size_t)gid, tn, R.t_far, &t, &g)) return;
    if (COUNT) ++*found;
    if (!have_last || t > last_t || (t == last_t && ik > last_i)) overflow |= hb.insert(t, g, ik);
  };
  // pair p of the leaf; a lane past its end tests the last pair again and drops it
  auto filter_t = [&](uint32_t p, PlainPair& x) {
    const unsigned m = plain_pair_t(S, L.pb + (LPR == 1 ? p : min(p, L.np - 1u)), w, F, x);
    return LPR > 1 && p >= L.np ? 0u : m;
  };
  if constexpr (PACKET) {
    for (uint32_t pb = 0; pb < L.np; pb += LPR) {
      const uint32_t p = pb + sub;
      PlainPair x;
      unsigned m = filter_t(p, x);
      if (!__any_sync(mask, m != 0u)) continue;
      m &= plain_pair_g(x);
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (__any_sync(mask, (m >> k) & 1u))
          if ((m >> k) & 1u) test(2 * p + k);
    }
  } else {
    auto any = [&](bool c) { return LPR > 1 ? __any_sync(mask, c) != 0 : c; };
    for (uint32_t c0 = 0; c0 < L.np; c0 += kChunk * LPR) {
      uint32_t left = 0u;  // bit 2 j + k: entry k of pair c0 + j LPR + sub passed
      const uint32_t n = min(kChunk, (L.np - c0 + LPR - 1) / LPR);
      for (uint32_t j = 0; j < n; ++j) {
        PlainPair x;
        const unsigned m = filter_t(c0 + j * LPR + sub, x);
        if (any(m != 0u)) left |= (m & plain_pair_g(x)) << (2u * j);
      }
      while (any(left != 0u)) {
        if (left == 0u) continue;
        const uint32_t b = __ffs(left) - 1;
        test(2 * (c0 + (b >> 1) * LPR + sub) + (b & 1u));
        left &= left - 1u;
      }
    }
  }
  return overflow;
}

// The candidate scan of one leaf pass for this lane's share of the pairs:
// the K smallest (t, leaf position) keys above the last key taken, on
// [tn, t_far).  Returns true when the share had more accepted hits than K.
template <int K, int FORM, int LPR, bool PACKET>
__device__ __forceinline__ bool scan_share(const SceneOf<FORM>& S, const LeafRef& L, const Ray& R, float tn,
                                           unsigned mask, bool have_last, float last_t, uint32_t last_i,
                                           HitBuf<K>& hb) {
  const unsigned sub = threadIdx.x & (LPR - 1u);
  bool overflow = false;
  hb.clear();
  if constexpr (FORM == kFormPlain) {
    return scan_plain<K, LPR, PACKET>(S, L, R, tn, mask, have_last, last_t, last_i, hb);
  } else {
    const Ray2 w = ray2(R.o, R.d);
    const uint32_t np = L.np + L.nf;
    for (uint32_t pb = 0; pb < np; pb += LPR) {
      const uint32_t p = pb + sub;
      float t2[2], g2[2];
      PairT pt;
      // a lane past the end of the leaf tests its last pair again and drops it
      unsigned m = leaf_pair_t<FORM>(S, L, LPR == 1 || p < np ? p : np - 1u, w, tn, R.t_far, pt);
      if (LPR > 1 && p >= np) m = 0u;
      // uniform branches: most pairs have no lane with t* in range
      if (__any_sync(mask, m != 0u)) {
        m = test_pair_g(pt, m, t2, g2);
        if (__any_sync(mask, m != 0u)) {
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const uint32_t ik = 2 * p + k;
            if (((m >> k) & 1u) && (!have_last || t2[k] > last_t || (t2[k] == last_t && ik > last_i)))
              overflow |= hb.insert(t2[k], g2[k], ik);
          }
        }
      }
    }
  }
  return overflow;
}

// Composite one accepted hit (t, g) of Gaussian gid: response, alpha with
// the 0.99 cap, the 0.0113 / (1/255) skips, SH colour, front-to-back update.
template <int FORM>
__device__ __forceinline__ void blend_hit(const SceneOf<FORM>& S, Ray& R, float t, float g, uint32_t gid) {
  float4* const acc = acc_slot();
  if constexpr (FORM == kFormPlain) {
    const float4 v = *acc;
    F3 c = mk(v.x, v.y, v.z);
    float D = v.w;
    if (exact_blend(S.test + kTestWords * (size_t)gid, S.sh + 12ull * gid, R.d, t, g, c, R.A, D))
      *acc = make_float4(c.x, c.y, c.z, D);
  } else {
    const float gres = __expf(-0.0555555555556f * g * g);
    const float alpha = fminf(0.99f, gauss_opacity<FORM>(S, gid) * gres);
    if (gres < 0.0113f || alpha < 1.0f / 255.0f) return;
    const F3 c = eval_sh_fast<FORM>(S, gid, R.d);
    const float w = alpha * (1.f - R.A);
    float4 v = *acc;
    v.x = fmaf(c.x, w, v.x);
    v.y = fmaf(c.y, w, v.y);
    v.z = fmaf(c.z, w, v.z);
    v.w = fmaf(t, w, v.w);
    *acc = v;
    R.A += w;
  }
}

// The group takes its hits of one leaf pass in key order: the smallest
// head key of the lanes' buffers, popped from the lane that holds it, as
// long as no lane whose share overflowed has run out of buffered keys (its
// next key is not known).  Every lane of the group blends the same hits.
// Stops once A > 0.99.  Returns whether the group must re-scan the leaf
// above (last_t, last_i).
template <int K, int FORM, int LPR>
__device__ __forceinline__ bool take_group_hits(const SceneOf<FORM>& S, const LeafRef& L, Ray& R, const HitBuf<K>& hb,
                                                bool overflow, unsigned mask, bool active, bool& ok,
                                                float& last_t, uint32_t& last_i, uint32_t* status) {
  const float kInf = __int_as_float(0x7f800000);
  const unsigned gm = group_mask(LPR);
  uint32_t h = 0;  // next unconsumed entry of this lane's buffer
#pragma unroll 1
  for (int it = 0; it < K * LPR; ++it) {
    float kt = kInf, kg = 0.f;
    uint32_t ki = 0xFFFFFFFFu;
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (h == (uint32_t)k) {
        kt = hb.t[k];
        kg = hb.g[k];
        ki = hb.i[k];
      }
    const bool blocked = (__ballot_sync(mask, overflow && h == (uint32_t)K) & gm) != 0u;
    float mt = kt, mg = kg;
    uint32_t mi = ki;
    group_min<LPR>(mt, mi, mg, mask);
    const bool act = active && ok && !blocked && mt != kInf && !(R.A > 0.99f);
    if (!__any_sync(mask, act)) break;
    if (act) {
      if (kt == mt && ki == mi) ++h;
      last_t = mt;
      last_i = mi;
      const uint32_t gid = leaf_gid<FORM>(S, L, mi);
      if (gid >= S.n_gauss) {
        atomicOr(status, kStatusBadId);
        ok = false;
      } else {
        blend_hit<FORM>(S, R, mt, mg, gid);
      }
    }
  }
  return (__ballot_sync(mask, overflow) & gm) != 0u;
}

// Descend from R.cur to the next leaf, test and composite it, then pop or
// restart (singlePassIntersectGaussian_sortNode_onlyShortStack,
// cudaRenderer.cu:1552-1708).  Returns true when the ray is finished.  With
// LPR > 1 the lanes of a group walk the same ray together and split each
// leaf's candidates.
template <int K, int FORM, int LPR>
__device__ __forceinline__ bool leaf_step(const SceneOf<FORM>& S, uint32_t (*s_id)[kThreads], float (*s_t)[kThreads],
                                          int tid, Ray& R, uint32_t* status) {
  uint2 nd = __ldg(S.nodes + R.cur);
  if (++R.steps > kMaxRaySteps) {
    atomicOr(status, kStatusStepLimit);
    return true;
  }
  while ((nd.x & 7u) != 3u) {
    const uint32_t child = nd.x >> 3;
    const uint32_t axis = nd.x & 3u;
    const float t_split = split_t<FORM>(R, axis, nd.y);
    const unsigned sign = __float_as_uint(sel3(FORM == kFormPlain ? R.d : R.inv, axis)) >> 31;
    const uint32_t idx = child + (sign ^ (t_split <= R.t_near ? 1u : 0u));
    if (R.t_near < t_split && t_split < R.t_far) {
      if (++R.top == kStack) R.top = 0;
      R.quant = min(R.quant + 1, (unsigned)kStack);
      s_id[R.top][tid] = child + (sign ^ 1u);
      s_t[R.top][tid] = R.t_far;
      R.t_far = t_split;
    }
    R.cur = idx;
    nd = __ldg(S.nodes + R.cur);
  }
  const LeafRef L = leaf_ref<FORM>(S, R.cur, nd);
  if (!leaf_in_bounds<FORM>(S, L)) {
    atomicOr(status, kStatusBadLeaf);
    return true;
  }
  bool have_last = false;
  float last_t = 0.f;
  uint32_t last_i = 0;
  if constexpr (LPR > 1) {
    const unsigned gm = group_mask(LPR);
    bool ok = true;
    while (true) {
      HitBuf<K> hb;
      const bool overflow = scan_share<K, FORM, LPR, false>(S, L, R, R.t_near, gm, have_last, last_t, last_i, hb);
      const bool again = take_group_hits<K, FORM, LPR>(S, L, R, hb, overflow, gm, true, ok, last_t, last_i, status);
      if (!ok || R.A > 0.99f) return true;
      if (!again) break;
      have_last = true;
    }
  } else {
    while (true) {
      HitBuf<K> hb;
      hb.clear();
      bool overflow = false;
      if constexpr (FORM == kFormPlain) {
        overflow = scan_plain<K, 1, false>(S, L, R, R.t_near, 0u, have_last, last_t, last_i, hb);
      } else {
        const Ray2 w = ray2(R.o, R.d);
        for (uint32_t p = 0; p < L.np + L.nf; ++p) {
          float t2[2], g2[2];
          PairT pt;
          unsigned m = leaf_pair_t<FORM>(S, L, p, w, R.t_near, R.t_far, pt);  // padding never passes
          if (m) {
            m = test_pair_g(pt, m, t2, g2);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const uint32_t ik = 2 * p + k;
              if (((m >> k) & 1u) && (!have_last || t2[k] > last_t || (t2[k] == last_t && ik > last_i)))
                overflow |= hb.insert(t2[k], g2[k], ik);
            }
          }
        }
      }
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (hb.t[k] == __int_as_float(0x7f800000)) break;
        const uint32_t gid = leaf_gid<FORM>(S, L, hb.i[k]);
        if (gid >= S.n_gauss) {
          atomicOr(status, kStatusBadId);
          return true;
        }
        blend_hit<FORM>(S, R, hb.t[k], hb.g[k], gid);
        if (R.A > 0.99f) return true;
      }
      if (!overflow) break;
      have_last = true;
      last_t = hb.t[K - 1];
      last_i = hb.i[K - 1];
    }
  }
  if (R.t_far >= R.t_scene_far) return true;
  if (R.quant == 0) {
    R.cur = 0;
    R.t_near = R.t_far;
    R.t_far = R.t_scene_far;
  } else {
    const uint32_t id = s_id[R.top][tid];
    const float tm = s_t[R.top][tid];
    if (R.top == 0) R.top = kStack;
    --R.top;
    --R.quant;
    R.cur = id;
    R.t_near = R.t_far;
    R.t_far = tm;
  }
  return false;
}

// ------------------------------------------------------------ warp packets
// Packet traversal of one warp tile (32 rays): the warp walks the tree together.
// Primary rays of a tile share the eye point and, away from the image lines
// where a direction component changes sign, the sign of every direction
// component, so the front-to-back child order at a node is the same for all
// of them.  Each lane keeps its own interval and makes the per-ray decision
// of leaf_step (near child when t_split > t_near, far child when t_split <=
// t_near or t_split < t_far); the warp enters a child when any lane needs it
// and masks the others there.  A lane therefore meets exactly its own leaves,
// in its own order, with its own [t_near, t_far), and the leaf's records are
// warp-uniform loads.  Stack entries: (node, lane mask) per warp and
// (t_near, t_far) per lane, a ring of kStack entries; when the ring has lost
// entries the unfinished lanes restart at the root from the end of their
// last leaf, as the per-ray short stack does.
struct PktEnt {
  uint32_t node, mask;
};

// Leaf L for the lanes with part set; every lane runs the same candidate
// loop (lanes without part test against an empty interval).  With LPR > 1
// the lanes of each group split the leaf's candidates and take the group's
// hits in key order.  Inside the leaf a ray stops compositing once
// A > 0.99.  Returns false on a bad Gaussian ID (status set).
template <int K, int FORM, int LPR>
__device__ __forceinline__ bool pkt_leaf(const SceneOf<FORM>& S, const LeafRef& L, Ray& R, bool part,
                                         uint32_t* status) {
  const unsigned full = 0xFFFFFFFFu;
  const float kInf = __int_as_float(0x7f800000);
  bool have_last = false, ok = true;
  float last_t = 0.f;
  uint32_t last_i = 0;
  bool more = part;
  while (__any_sync(full, more)) {
    HitBuf<K> hb;
    const bool overflow =
        scan_share<K, FORM, LPR, true>(S, L, R, more ? R.t_near : kInf, full, have_last, last_t, last_i, hb);
    if constexpr (LPR > 1) {
      const bool again = take_group_hits<K, FORM, LPR>(S, L, R, hb, overflow, full, more, ok, last_t, last_i,
                                                         status);
      more = more && ok && again && !(R.A > 0.99f);
    } else {
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (hb.t[k] == kInf || R.A > 0.99f) break;
        const uint32_t gid = leaf_gid<FORM>(S, L, hb.i[k]);
        if (gid >= S.n_gauss) {
          atomicOr(status, kStatusBadId);
          ok = false;
          break;
        }
        blend_hit<FORM>(S, R, hb.t[k], hb.g[k], gid);
      }
      more = more && ok && overflow && !(R.A > 0.99f);
      last_t = hb.t[K - 1];
      last_i = hb.i[K - 1];
    }
    have_last = true;
  }
  return ok;
}

// Trace the warp's rays as one packet.  live: the lane's ray entered the
// scene box; sgn: bit a = sign of direction component a (warp-uniform).
template <int K, int FORM, int LPR>
__device__ __forceinline__ void pkt_trace(const SceneOf<FORM>& S, Ray& R, bool live, unsigned sgn,
                                          uint32_t (*s_tn)[kThreads], float (*s_tf)[kThreads],
                                          PktEnt (*s_ent)[kWarps], int tid, int warp, uint32_t* status) {
  const unsigned full = 0xFFFFFFFFu;
  bool act = live, done = !live;
  float t_done = R.t_near;  // end of the part of the ray already composited
  uint32_t cur = 0, steps = 0;
  unsigned top = kStack - 1, quant = 0;
  while (true) {
    if (++steps > kMaxRaySteps) {
      if ((tid & 31) == 0) atomicOr(status, kStatusStepLimit);
      break;
    }
    uint2 nd = __ldg(S.nodes + cur);
    bool leaf = true;
    while ((nd.x & 7u) != 3u) {
      const uint32_t child = nd.x >> 3, axis = nd.x & 3u;
      const unsigned sign = (sgn >> axis) & 1u;
      const float t_split = split_t<FORM>(R, axis, nd.y);
      const bool wn = act && !(t_split <= R.t_near);
      const bool wf = act && ((t_split <= R.t_near) || (t_split < R.t_far));
      const unsigned bn = __ballot_sync(full, wn), bf = __ballot_sync(full, wf);
      if (bn && bf) {
        if (++top == kStack) top = 0;
        quant = min(quant + 1, (unsigned)kStack);
        s_ent[top][warp] = PktEnt{child + (sign ^ 1u), bf};
        s_tn[top][tid] = __float_as_uint(wn ? t_split : R.t_near);
        s_tf[top][tid] = R.t_far;
        if (wn && wf) R.t_far = t_split;
        act = wn;
        cur = child + sign;
      } else if (bn) {
        cur = child + sign;
      } else if (bf) {
        cur = child + (sign ^ 1u);
      } else {
        leaf = false;
        break;
      }
      nd = __ldg(S.nodes + cur);
    }
    if (leaf) {
      const LeafRef L = leaf_ref<FORM>(S, cur, nd);
      if (!leaf_in_bounds<FORM>(S, L)) {
        if ((tid & 31) == 0) atomicOr(status, kStatusBadLeaf);
        break;
      }
      const bool part = act && !done;
      if (__any_sync(full, part)) {
        if (!pkt_leaf<K, FORM, LPR>(S, L, R, part, status)) done = true;
        if (part) {
          t_done = R.t_far;
          // inside a leaf only A > 0.99 stops a ray; at a leaf boundary the
          // walk goes on only while A < 0.99 (A == 0.99 stops here)
          if (!(R.A < 0.99f) || R.t_far >= R.t_scene_far) done = true;
        }
      }
    }
    // next subtree: pop entries until one holds an unfinished lane
    bool found = false;
    while (quant > 0) {
      const PktEnt e = s_ent[top][warp];
      const float tn = __uint_as_float(s_tn[top][tid]), tf = s_tf[top][tid];
      if (top == 0) top = kStack;
      --top;
      --quant;
      act = ((e.mask >> (tid & 31)) & 1u) && !done;
      if (act) {
        R.t_near = tn;
        R.t_far = tf;
      }
      if (__any_sync(full, act)) {
        cur = e.node;
        found = true;
        break;
      }
    }
    if (!found) {
      // the ring lost entries: unfinished lanes restart at the root
      act = !done;
      if (!__any_sync(full, act)) break;
      cur = 0;
      if (act) {
        R.t_near = t_done;
        R.t_far = R.t_scene_far;
      }
    }
  }
}

// Bit a: sign of component a (-0 counts as negative).
__device__ __forceinline__ unsigned sign_bits(const F3& v) {
  return (__float_as_uint(v.x) >> 31) | ((__float_as_uint(v.y) >> 31) << 1) | ((__float_as_uint(v.z) >> 31) << 2);
}

// The warp's rays, one packet per direction-sign pattern among them (almost
// always one; two or more only for tiles on a sign-change line).
template <int K, int FORM, int LPR>
__device__ __forceinline__ void trace_packets(const SceneOf<FORM>& S, Ray& R, bool live, unsigned my_sgn,
                                              uint32_t (*s_id)[kThreads], float (*s_t)[kThreads],
                                              PktEnt (*s_ent)[kWarps], int tid, uint32_t* status) {
  unsigned pending = __ballot_sync(0xFFFFFFFFu, live);
  while (pending) {
    const unsigned sgn = __shfl_sync(0xFFFFFFFFu, my_sgn, __ffs(pending) - 1);
    const bool in = live && my_sgn == sgn && ((pending >> (tid & 31)) & 1u);
    pending &= ~__ballot_sync(0xFFFFFFFFu, in);
    pkt_trace<K, FORM, LPR>(S, R, in, sgn, s_id, s_t, s_ent, tid, tid >> 5, status);
  }
}

constexpr int kSchedGroups = 4;  // the groups schedule (render_fast.cu); not a KDGR_SCHED_* value
__device__ __forceinline__ int find_view(const ViewDesc* views, int n_views, uint32_t item, int sched) {
  int lo = 0, hi = n_views - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    const uint32_t b = sched == kSchedGroups              ? __ldg(&views[mid].grp_base)
                       : sched == KDGR_SCHED_WARP_TILES ? __ldg(&views[mid].wt_base)
                                                        : __ldg(&views[mid].cb_base);
    if (b <= item) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Store the ray of pixel (x, y) of view V.
__device__ __forceinline__ void store_px(const ViewDesc& V, int x, int y, const Ray& R, float* rgb, float* alpha_out,
                                         float* depth_out) {
  const int W = __ldg(&V.W), H = __ldg(&V.H);
  const size_t idx = (size_t)__ldg(&V.out_off) + (size_t)(H - 1 - y) * W + x;  // rows flipped per view
  const float4 v = *acc_slot();
  rgb[3 * idx] = v.x;
  rgb[3 * idx + 1] = v.y;
  rgb[3 * idx + 2] = v.z;
  if (alpha_out) alpha_out[idx] = R.A;
  if (depth_out) depth_out[idx] = v.w;
}

// Render the ray of pixel (x, y) of view V to completion and store it.
// PKT: warp packets (every lane of the warp calls this together);
// otherwise one independent ray per lane.  With LPR > 1 each group of LPR
// consecutive lanes has the same pixel and its first lane stores it.
template <int K, int FORM, bool PKT, int LPR>
__device__ __forceinline__ void render_px(const FastView& S, const ViewDesc& V, int x, int y,
                                          uint32_t (*s_id)[kThreads], float (*s_t)[kThreads],
                                          PktEnt (*s_ent)[kWarps], int tid, float* rgb, float* alpha_out,
                                          float* depth_out, uint32_t* status) {
  const int W = __ldg(&V.W), H = __ldg(&V.H);
  if constexpr (PKT) {
    const bool inimg = x < W && y < H;
    Ray R;
    const bool live = ray_init(S, V.cam, inimg ? x : 0, inimg ? y : 0, R) && inimg;
    trace_packets<K, FORM, LPR>(S, R, live, sign_bits(R.inv), s_id, s_t, s_ent, tid, status);
    if (!inimg || (tid & (LPR - 1)) != 0) return;
    store_px(V, x, y, R, rgb, alpha_out, depth_out);
  } else {
    if (x >= W || y >= H) return;
    Ray R;
    if (ray_init(S, V.cam, x, y, R)) {
      while (R.A < 0.99f && !leaf_step<K, FORM, LPR>(S, s_id, s_t, tid, R, status)) {
      }
    }
    if ((tid & (LPR - 1)) != 0) return;
    store_px(V, x, y, R, rgb, alpha_out, depth_out);
  }
}

// i-th of n positions from the middle outwards: blocks are handed out in this
// order, so that a launch ends on the image border, where rays are short.
__device__ __forceinline__ uint32_t middle_out(uint32_t i, uint32_t n) {
  const uint32_t m = (n - 1) / 2;
  return (i & 1u) ? m + (i + 1) / 2 : m - i / 2;
}

// Pixel of lane `lane` in quarter q (0..3) of the 16x8 block whose top-left
// pixel is (bx, by), for the warp tile shape (KDGR_TILE_*): 8x4 tiles in a
// 2x2 arrangement, 4x8 tiles side by side, or 16x2 tiles stacked.
__device__ __forceinline__ void block_pixel(int tile, int bx, int by, int q, int lane, int& x, int& y) {
  if (tile == KDGR_TILE_4X8) {
    x = bx + 4 * q + (lane & 3);
    y = by + (lane >> 2);
  } else if (tile == KDGR_TILE_16X2) {
    x = bx + (lane & 15);
    y = by + 2 * q + (lane >> 4);
  } else {
    x = bx + (q & 1) * kTileW + (lane & 7);
    y = by + (q >> 1) * kTileH + (lane >> 3);
  }
}

// Pixel of lane `lane` in item q (0 .. 4 LPR - 1) of the 16x8 block at
// (bx, by) when LPR lanes share a ray: the block is cut into 4 x (8 / LPR)
// tiles of 32 / LPR rays, 4 across and LPR down.
template <int LPR>
__device__ __forceinline__ void group_pixel(int bx, int by, int q, int lane, int& x, int& y) {
  const int gi = lane / LPR;
  x = bx + 4 * (q & 3) + (gi & 3);
  y = by + (8 / LPR) * (q >> 2) + (gi >> 2);
}

}  // namespace
}  // namespace kdgr
