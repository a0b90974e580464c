// MZI transfer matrices for the coefficient tiles in float-float arithmetic on the FP32 pipe.
//
// The tiles hold float32 values, and a deep mesh accumulates any systematic rounding error linearly, so each
// entry must be the float32 nearest to the exact value (then the rounding errors are unbiased and grow only
// as sqrt(L)).  The double-precision path (mzi_T in mg_device.cuh) delivers that, but GB300's FP64 pipe is
// narrow: it bounds the coefficient pass of a training step.  Here the same closed form is evaluated in
// float-float ("double-single") arithmetic - Dekker's exact two-product and Knuth's exact two-sum, a value is
// the unevaluated sum hi + lo of two floats, about 48 significant bits - so the result is correct to ~1e-13
// before its single rounding to float32, far below the float32 half-unit (3e-8), and the FP32 pipe does the
// work at many times the FP64 rate.
//
// sin and cos: Cody-Waite reduction by pi/2 (pi/2 split into three floats, the first two of 16 significant
// bits so that k * P1 and k * P2 are exact for |k| < 256), then the Taylor series on |r| <= pi/4, its first
// terms in float-float and the small tail in float (truncation below 1e-14).  Arguments of 400 or more in
// magnitude take the double-precision path.
#pragma once
#include "mg_device.cuh"

namespace mg {

struct ff {
  float h, l;
};

// exact a*b as hi + lo (FMA)
__device__ __forceinline__ ff ff_two_prod(float a, float b) {
  const float p = a * b;
  return {p, __fmaf_rn(a, b, -p)};
}
// exact a+b as hi + lo (Knuth)
__device__ __forceinline__ ff ff_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
// renormalise hi + lo with |hi| >= |lo|
__device__ __forceinline__ ff ff_quick(float a, float b) {
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ ff ff_add(ff a, ff b) {
  const ff s = ff_two_sum(a.h, b.h);
  return ff_quick(s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l)));
}
__device__ __forceinline__ ff ff_sub(ff a, ff b) { return ff_add(a, ff{-b.h, -b.l}); }
__device__ __forceinline__ ff ff_mul(ff a, ff b) {
  const float p = a.h * b.h;
  float e = __fmaf_rn(a.h, b.h, -p);
  e = __fmaf_rn(a.h, b.l, e);
  e = __fmaf_rn(a.l, b.h, e);
  return ff_quick(p, e);
}
__device__ __forceinline__ ff ff_mulf(ff a, float b) {
  const float p = a.h * b;
  float e = __fmaf_rn(a.h, b, -p);
  e = __fmaf_rn(a.l, b, e);
  return ff_quick(p, e);
}
__device__ __forceinline__ ff ff_neg(ff a) { return {-a.h, -a.l}; }
// the float nearest to hi + lo
__device__ __forceinline__ float ff_round(ff a) { return __fadd_rn(a.h, a.l); }

struct ffz {
  ff x, y;
};
__device__ __forceinline__ ffz ffz_mul(ffz a, ffz b) {
  return {ff_sub(ff_mul(a.x, b.x), ff_mul(a.y, b.y)), ff_add(ff_mul(a.x, b.y), ff_mul(a.y, b.x))};
}
__device__ __forceinline__ float2 ffz_round(ffz a) { return make_float2(ff_round(a.x), ff_round(a.y)); }

// sin and cos of a float x with |x| < 400 in float-float; returns false (nothing written) beyond.  The cosine's tail in float
// is good to 2e-13; fine (uniform over the launch): one more of its terms in float-float, to 2e-15, which the derivative tiles take,
// whose former form in double precision was good to 2e-14 (N = 130, 130 layers: no time that can be measured).
__device__ __forceinline__ bool ff_sincos(float x, ff* s, ff* c, bool fine = false) {
  if (!(fabsf(x) < 400.f)) return false;
  // Cody-Waite: pi/2 = P1 + P2 + P3 (residual 1.2e-18); k * P1, k * P2 exact for |k| < 256
  constexpr float P1 = 1.57080078125f, P2 = -4.4543994590640068e-06f, P3 = -5.5644315544167711e-11f;
  const float k = rintf(x * 0.636619747f);
  ff r = ff_two_sum(x, -k * P1);
  r = ff_add(r, ff{-k * P2, 0.f});
  r = ff_add(r, ff_neg(ff_two_prod(k, P3)));
  const ff r2 = ff_mul(r, r);
  const float t = r2.h;
  // sin r = r + r^3 (-1/3! + r^2 (1/5! + r^2 (-1/7! + r^2 q))), q in float (|r^9 q| < 3e-7)
  const float qs = __fmaf_rn(t, __fmaf_rn(t, __fmaf_rn(t, 1.60590444e-10f, -2.50521079e-08f), 2.75573188e-06f), 0.f);
  ff ps = ff_add(ff{-0.000198412701f, 2.72559687e-12f}, ff{qs, 0.f});                 // -1/7! + r^2 q
  ps = ff_add(ff{0.00833333377f, -4.34617203e-10f}, ff_mul(r2, ps));                   // 1/5!
  ps = ff_add(ff{-0.166666672f, 4.96705388e-09f}, ff_mul(r2, ps));                     // -1/3!
  const ff sr = ff_add(r, ff_mul(ff_mul(r, r2), ps));
  // cos r = 1 + r^2 (-1/2 + r^2 (1/4! + r^2 (-1/6! + r^2 q)))
  const float q10 = __fmaf_rn(t, __fmaf_rn(t, -1.14707454e-11f, 2.08767559e-09f), -2.755732e-07f);
  ff pc;
  if (fine) pc = ff_mul(r2, ff_add(ff{2.48015876e-05f, -3.406996e-13f}, ff_mulf(r2, q10)));   // r^2 (1/8! + r^2 q)
  else pc = ff_mulf(r2, __fmaf_rn(t, q10, 2.48015876e-05f));
  pc = ff_add(ff{-0.00138888892f, 3.36310944e-11f}, pc);                               // -1/6! + r^2 q
  pc = ff_add(ff{0.0416666679f, -1.24176347e-09f}, ff_mul(r2, pc));                    // 1/4!
  pc = ff_add(ff{-0.5f, 0.f}, ff_mul(r2, pc));                                         // -1/2!
  const ff cr = ff_add(ff{1.f, 0.f}, ff_mul(r2, pc));
  switch (static_cast<int>(k) & 3) {
    case 0: *s = sr; *c = cr; break;
    case 1: *s = cr; *c = ff_neg(sr); break;
    case 2: *s = ff_neg(sr); *c = ff_neg(cr); break;
    default: *s = ff_neg(cr); *c = sr; break;
  }
  return true;
}

// T in float-float, entries 00, 01, 10, 11 (for the frame pass, which needs it before its rounding to float32)
struct Tff {
  ffz t[4];
};
__device__ __forceinline__ void tff_round(const Tff& f, C2x2* T) {
  T->t00 = ffz_round(f.t[0]);
  T->t01 = ffz_round(f.t[1]);
  T->t10 = ffz_round(f.t[2]);
  T->t11 = ffz_round(f.t[3]);
}
__device__ __forceinline__ void tff_from(const C2x2& T, Tff* f) {
  const float2 t[4] = {T.t00, T.t01, T.t10, T.t11};
#pragma unroll
  for (int k = 0; k < 4; ++k) f->t[k] = {ff{t[k].x, 0.f}, ff{t[k].y, 0.f}};
}

// The standard MZI T (mzi_T in mg_device.cuh, reference crossing.py:216-221) from the float-float sin/cos of
// th/2, ph, alpha and beta, and, when given, the (cos, sin)(pi/4 + beta) pair of the direct gradient.
__device__ __forceinline__ void mzi_T_ff_from(ff S, ff C, ff Sph, ff Cph, ff sa, ff ca, ff sb, ff cb, Tff* T,
                                              float2* csb) {
  const ff Cp = ff_sub(ff_mul(ca, cb), ff_mul(sa, sb)), Sp = ff_add(ff_mul(sa, cb), ff_mul(ca, sb));
  const ff Cm = ff_add(ff_mul(ca, cb), ff_mul(sa, sb)), Sm = ff_sub(ff_mul(sa, cb), ff_mul(ca, sb));
  if (csb) {
    const ff r2 = {0.707106769f, 1.21016175e-08f};                                    // 1/sqrt 2
    *csb = make_float2(ff_round(ff_mul(r2, ff_sub(cb, sb))), ff_round(ff_mul(r2, ff_add(cb, sb))));
  }
  const ffz E0 = {C, S};                                    // e^{i th/2}
  const ffz E1 = ffz_mul(E0, ffz{Cph, Sph});                // e^{i(th/2 + ph)}
  const ff CSp = ff_mul(C, Sp), SCm = ff_mul(S, Cm), SSm = ff_mul(S, Sm), CCp = ff_mul(C, Cp);
  const ffz A00 = {ff_neg(CSp), SCm}, A01 = {ff_neg(SSm), CCp};
  const ffz A10 = {SSm, CCp}, A11 = {ff_neg(CSp), ff_neg(SCm)};
  T->t[0] = ffz_mul(E1, A00);
  T->t[1] = ffz_mul(E0, A01);
  T->t[2] = ffz_mul(E1, A10);
  T->t[3] = ffz_mul(E0, A11);
}

// mzi_T_ff_from on the angles of one thread; false (nothing written) when an angle is outside the float-float
// range, and the caller takes the double path.
__device__ __forceinline__ bool mzi_T_ff(float th, float ph, float al, float be, Tff* T, float2* csb) {
  ff S, C, Sph, Cph, sa, ca, sb, cb;
  if (!ff_sincos(0.5f * th, &S, &C) || !ff_sincos(ph, &Sph, &Cph) || !ff_sincos(al, &sa, &ca) ||
      !ff_sincos(be, &sb, &cb))
    return false;
  mzi_T_ff_from(S, C, Sph, Cph, sa, ca, sb, cb, T, csb);
  return true;
}

// The same over the four lanes of a quad (lanes 4k..4k+3 of a warp, all given the same angles and all calling it): lane k
// takes the sin/cos of angle k (th/2, ph, alpha, beta), the quad exchanges them by shuffles, and lane k combines them into
// entry k (00, 01, 10, 11) of T, which it returns; csb on every lane.  The entries are those of mzi_T_ff_from,
// operation by operation.  (All four entries on every lane: 45.6 us for a 600-mode, 600-layer mesh, 11.8 us for 256; one each:
// 20.0 and 5.9 us, GB300; with the derivatives, for 130 modes and layers, 4.0 us, in double precision by one thread
// per slot 8.1.)  false on every lane of the quad when any angle is out of range.
// ideal (uniform over the launch): no splitter array, alpha = beta = 0 (cos = 1, sin = 0) without the splitter products; each entry
// is the value of the general form, its operations reduced to those that are not exact.
// dth: receives the entry of dT/dth.  With e = e^{i th/2}, E = e or e e^{i ph} (entries 01, 11 and 00, 10), a sum behind each:
//   00: i/2 (cos(alpha-beta) - sin(alpha+beta)) E e     01: -1/2 (cos(alpha+beta) + sin(alpha-beta)) E e
//   10: 1/2 (sin(alpha-beta) - cos(alpha+beta)) E e     11: -i/2 (cos(alpha-beta) + sin(alpha+beta)) E e
__device__ __forceinline__ ff ff_sel(bool p, ff a, ff b) { return ff{p ? a.h : b.h, p ? a.l : b.l}; }
__device__ __forceinline__ bool mzi_T_ff_quad(float th, float ph, float al, float be, bool ideal, ffz* entry, float2* csb, ffz* dth) {
  const int lane = threadIdx.x & 31, base = lane & ~3, sub = lane & 3;
  const unsigned qmask = 0xFu << base;
  const float x = sub == 0 ? 0.5f * th : (sub == 1 ? ph : (sub == 2 ? al : be));
  ff s = {0.f, 0.f}, c = {1.f, 0.f};
  int ok = ff_sincos(x, &s, &c, dth != nullptr) ? 1 : 0;
  ok &= __shfl_xor_sync(qmask, ok, 1);
  ok &= __shfl_xor_sync(qmask, ok, 2);
  if (!ok) return false;
  auto get = [&](ff v, int k) { return ff{__shfl_sync(qmask, v.h, base + k), __shfl_sync(qmask, v.l, base + k)}; };
  const ff S = get(s, 0), C = get(c, 0), Sph = get(s, 1), Cph = get(c, 1);
  const bool diag = sub == 0 || sub == 3;                  // entries 00, 11
  const ffz E0 = {C, S}, E1 = ffz_mul(E0, ffz{Cph, Sph});  // e^{i th/2} (entries 01, 11), e^{i(th/2 + ph)} (00, 10)
  const ffz E = {ff_sel(sub & 1, E0.x, E1.x), ff_sel(sub & 1, E0.y, E1.y)};
  // g (p sine, q cosine of the splitters' sum or difference) times E e, for dT/dth
  auto derivative = [&](ff p, ff q) {
    const ff a = ff_sel(sub == 2, p, q), b = ff_sel(sub == 2, q, p);
    const ff g = ff_add(a, ff_sel(sub == 0 || sub == 2, ff_neg(b), b));
    const float h = sub == 1 ? -0.5f : 0.5f;
    const ffz w = ffz_mul(E, E0);
    const ff x = ff_mul(ff{h * g.h, h * g.l}, w.x), y = ff_mul(ff{h * g.h, h * g.l}, w.y);
    *dth = sub == 0 ? ffz{ff_neg(y), x} : sub == 3 ? ffz{y, ff_neg(x)} : ffz{x, y};
  };
  if (ideal) {
    if (dth) derivative(ff{0.f, 0.f}, ff{1.f, 0.f});
    if (csb) {
      const float r = 0.707106769f;   // (1/sqrt 2)(cos 0 -+ sin 0), rounded
      *csb = make_float2(r, r);
    }
    const ff f = ff_sel(diag, S, C), u = ff_mul(E.y, f), v = ff_mul(E.x, f);
    *entry = {sub == 3 ? u : ff_neg(u), sub == 3 ? ff_neg(v) : v};
    return true;
  }
  const ff sa = get(s, 2), ca = get(c, 2), sb = get(s, 3), cb = get(c, 3);
  if (csb) {   // lane 1 of the quad the sine, the others the cosine of pi/4 + beta
    const ff r2 = {0.707106769f, 1.21016175e-08f};         // 1/sqrt 2
    const float v = ff_round(ff_mul(r2, ff_add(cb, ff_sel(sub == 1, sb, ff_neg(sb)))));
    *csb = make_float2(__shfl_sync(qmask, v, base), __shfl_sync(qmask, v, base + 1));
  }
  // 00, 11: sin(alpha + beta), cos(alpha - beta); 01, 10: sin(alpha - beta), cos(alpha + beta)
  const ff casb = ff_mul(ca, sb), sasb = ff_mul(sa, sb);
  const ff p = ff_add(ff_mul(sa, cb), ff_sel(diag, casb, ff_neg(casb)));
  const ff q = ff_add(ff_mul(ca, cb), ff_sel(diag, sasb, ff_neg(sasb)));
  if (dth) derivative(p, q);
  const ff u = ff_mul(ff_sel(diag, C, S), p), v = ff_mul(ff_sel(diag, S, C), q);
  const ffz A = {sub == 2 ? u : ff_neg(u), sub == 3 ? ff_neg(v) : v};
  *entry = ffz_mul(E, A);
  return true;
}

}  // namespace mg
