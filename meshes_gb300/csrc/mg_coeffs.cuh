// Coefficient precompute: (p, s[, dp]) -> per-layer tiles in the order the propagation kernel's
// lanes read them, plus the layer kinds and (back-propagation) the dT/dp tiles.
//
// The reference rebuilds T inside every propagation block for every chunk of layers with the
// fast-math __sincosf (gpu/gmem.cu:242-318, gpu/crossing.cu:36-148): redundant work that grows with
// the number of blocks.  Here T is built once per call (or once per programmed mesh) with the
// accurate sincosf, and inactive slots become identities so the hot loop never branches on the
// layout.  Layout of the parameter grid follows gpu/mesh.py:77-81: p[l*ldp + q*n_p + k] with
// q < N/2 the MZI slot of the layer; a nearest-neighbour slot q is active iff
// shift/2 <= q < shift/2 + len (gpu/gmem.cu:236-238); a butterfly layer with stride 2^e couples
// modes (2*2^e*(q/2^e) + q%2^e, +2^e) (gpu/fwdprop.cu:52-93).
#pragma once
#include "mg_ffcoef.cuh"
#include "mg_prop.cuh"

namespace mg {

enum { CR_MZI = 0, CR_SYM = 1, CR_ORTH = 2, CR_GENERIC = 3 };
enum { GEO_NN = 0, GEO_FFT = 1 };

struct CoefArgs {
  int N, L, crossing, geometry, op;
  int gr;                // back-propagation gradient mode (0: dJ/dT + dT/dp tiles, 1: MZI direct, 2: orth direct)
  int M, G;
  const int* lens;
  const int* shifts;
  const int* strides;
  const float* p;        // [L][ldp]
  int ldp;
  const float* s;        // [L][lds] or null
  int lds;
  const float* dp;       // FWDDIFF direction, layout of p (or null = 0)
  const float2* Tgen;    // CR_GENERIC: [L][N/2][4] (t00, t01, t10, t11)
  const float2* Dgen;    // CR_GENERIC back-propagation: [L][N/2][2][4] (dT/dp0, dT/dp1)
  unsigned char* tiles;  // [L][layer_bytes]
  unsigned layer_bytes;
  unsigned char* dtiles; // BWD: [L][dlayer_bytes]
  unsigned dlayer_bytes;
  int* kinds;            // [L] layer kinds, followed by [L][2] (shift, len) of the active slot range
  int* status;
  // for the frame pass (mg_frame.cuh; all null without one), [L][2*np2] in mode order, a slot's first and second
  // mode holding (t00, t01) and (t11, t10): diagonal and off-diagonal entries in float-float (x.h, x.l, y.h, y.l),
  // |diagonal|^2, and [L][np2] in slot order the splitter pair
  float4* tdiag;
  float4* toff;
  float* tmag;
  float2* tcs;
  int* fcount;           // set to 0
};

__host__ __device__ inline int crossing_np(int c) { return c == CR_ORTH ? 1 : 2; }
__host__ __device__ inline int crossing_ns(int c) { return c == CR_MZI ? 2 : (c == CR_SYM ? 1 : 0); }

// csb (MZI crossings): receives (cos, sin)(pi/4 + beta) of an active slot
__device__ __forceinline__ void slot_T(const CoefArgs& a, int l, int q, bool active, C2x2& T, C2x2& D0, C2x2& D1,
                                       float2* csb, Tff& F) {
  if (!active) {
    T = c2x2_identity(); D0 = c2x2_zero(); D1 = c2x2_zero();
    tff_from(T, &F);
    return;
  }
  if (a.crossing == CR_GENERIC) {
    const float2* t = a.Tgen + ((size_t)l * (a.N / 2) + q) * 4;
    T.t00 = t[0]; T.t01 = t[1]; T.t10 = t[2]; T.t11 = t[3];
    tff_from(T, &F);
    if (a.Dgen) {
      const float2* d = a.Dgen + ((size_t)l * (a.N / 2) + q) * 8;
      D0.t00 = d[0]; D0.t01 = d[1]; D0.t10 = d[2]; D0.t11 = d[3];
      D1.t00 = d[4]; D1.t01 = d[5]; D1.t10 = d[6]; D1.t11 = d[7];
    } else {
      D0 = c2x2_zero(); D1 = c2x2_zero();
    }
    return;
  }
  const int n_p = crossing_np(a.crossing), n_s = crossing_ns(a.crossing);
  const float* pp = a.p + (size_t)l * a.ldp + (size_t)q * n_p;
  const float* ss = a.s ? a.s + (size_t)l * a.lds + (size_t)q * n_s : nullptr;
  // dT/dp only where a tile needs it: forward-mode tiles and the dT/dp tiles of back-propagation
  // without a direct-gradient mode
  const bool need_d = a.op == OP_FWDDIFF || (a.op == OP_BWD && a.gr == 0);
  if (!need_d) {
    D0 = c2x2_zero();
    D1 = c2x2_zero();
  }
  if (a.crossing == CR_MZI) {
    // (stored activations; every other MZI tile takes the quad form) T in float-float on the FP32 pipe; for angles beyond its
    // range the double-precision form
    const float al = ss ? ss[0] : 0.f, be = ss ? ss[1] : 0.f;
    if (!mzi_T_ff(pp[0], pp[1], al, be, &F, csb)) {
      mzi_T(pp[0], pp[1], al, be, &T, nullptr, nullptr, csb);
      tff_from(T, &F);
    } else {
      tff_round(F, &T);
    }
  } else {   // CR_SYM
    sym_T(pp[0], pp[1], ss ? ss[0] : 0.f, &T, need_d ? &D0 : nullptr, need_d ? &D1 : nullptr);
    tff_from(T, &F);
  }
}

__device__ __forceinline__ void slot_R(const CoefArgs& a, int l, int q, bool active, R2x2& T, R2x2& D0) {
  if (!active) {
    T.t00 = 1.f; T.t01 = 0.f; T.t10 = 0.f; T.t11 = 1.f;
    D0.t00 = D0.t01 = D0.t10 = D0.t11 = 0.f;
    return;
  }
  const bool need_d = a.op == OP_FWDDIFF || (a.op == OP_BWD && a.gr == 0);
  if (!need_d) D0.t00 = D0.t01 = D0.t10 = D0.t11 = 0.f;
  orth_T(a.p[(size_t)l * a.ldp + q], &T, need_d ? &D0 : nullptr);
}

// kind of layer l and whether slot q is active; flags malformed geometry
__device__ __forceinline__ int layer_kind(const CoefArgs& a, int l, int q, bool* active) {
  if (a.geometry == GEO_NN) {
    const int sh = __ldg(a.shifts + l), ln = __ldg(a.lens + l);
    const bool ok = sh >= 0 && ln >= 0 && sh + 2 * ln <= a.N;
    if (!ok && q == 0) set_status(a.status, ST_BAD_GEOMETRY);
    *active = ok && q >= sh / 2 && q < sh / 2 + ln;
    return (sh & 1) ? KIND_MIS : 0;
  }
  const int e = __ldg(a.strides + l);
  const bool ok = e >= 0 && e < 30 && (2 << e) <= a.N && (a.N % (2 << e)) == 0;
  if (!ok && q == 0) set_status(a.status, ST_BAD_GEOMETRY);
  *active = ok && q < a.N / 2;
  const int st = 1 << (ok ? e : 0);
  return (2 * st <= a.M) ? (ok ? e : 0) : KIND_XL + e;
}

// The frame pass's input for entry k of slot q (layer kinds 0 and odd-shift)
__device__ __forceinline__ void frame_entry(const CoefArgs& a, int l, int q, int k, int sh, ffz z, float2 cs) {
  const int modes = a.G * a.M, m = sh + 2 * q + (k >> 1);   // row of the entry
  if (m >= modes) return;                                   // (the last odd-shift slot has no second mode)
  const size_t o = (size_t)l * modes + m;
  if (k == 0 || k == 3) {
    // the framed gradient divides by cos(pi/4 + beta): NaN marks a slot that all but lacks it
    const bool flat = a.tcs && !(fabsf(cs.x) >= 0x1p-6f * fabsf(cs.y));
    float w = z.x.h * z.x.h + z.y.h * z.y.h;
    if (w < 0x1p-60f) {                    // a diagonal entry below 2^-30 counts as 2^-30
      z = {ff{0x1p-30f, 0.f}, ff{0.f, 0.f}};
      w = 0x1p-60f;
    }
    a.tdiag[o] = make_float4(z.x.h, z.x.l, z.y.h, z.y.l);
    a.tmag[o] = flat ? __int_as_float(0x7fc00000) : w;
  } else {
    a.toff[o] = make_float4(z.x.h, z.x.l, z.y.h, z.y.l);
  }
}
// and what a slot has once
__device__ __forceinline__ void frame_slot(const CoefArgs& a, int l, int q, int t, int sh, float2 cs) {
  const int modes = a.G * a.M;
  if (t == 0) *a.fcount = 0;
  if (a.tcs) a.tcs[(size_t)l * (modes / 2) + q] = cs;
  if (sh && q == 0) {                      // mode 0 lies in no slot
    const size_t o = (size_t)l * modes;
    a.tdiag[o] = make_float4(1.f, 0.f, 0.f, 0.f);
    a.toff[o] = make_float4(0.f, 0.f, 0.f, 0.f);
    a.tmag[o] = 1.f;
  }
}

// The layer's kind and its active range (shift, len), once per layer
__device__ __forceinline__ void write_layer(const CoefArgs& a, int l, int kind) {
  a.kinds[l] = kind;
  int sh = 0, ln = 0;
  if (a.geometry == GEO_NN) {
    sh = __ldg(a.shifts + l);
    ln = __ldg(a.lens + l);
    if (sh < 0 || ln < 0 || sh + 2 * ln > a.N) sh = ln = 0;
  } else {
    bool any = false;
    layer_kind(a, l, 0, &any);
    ln = any ? a.N / 2 : 0;
  }
  a.kinds[a.L + 2 * l] = sh;
  a.kinds[a.L + 2 * l + 1] = ln;
}

// Lane t & 3 of the quad of lanes that does slot t / 4: MZI crossings.  Quads leave at the bounds
// check whole; lane k computes and writes entry k.
template <bool FRAME>
__device__ __forceinline__ void coef_quad(const CoefArgs& a, int t) {
  const int np2 = a.G * a.M / 2, idx = t >> 2, k = t & 3;
  if (idx >= a.L * np2) return;
  const int l = idx / np2, q = idx - l * np2;
  bool active = false;
  const int kind = layer_kind(a, l, q, &active);
  if (q == 0 && k == 0) write_layer(a, l, kind);
  const bool bwd = a.op == OP_BWD, diff = a.op == OP_FWDDIFF;   // bwd: direct gradients
  float2 cs = make_float2(0.f, 0.f);   // (cos, sin)(pi/4 + beta) for the direct gradient; 0 if inactive
  ffz z = {ff{k == 0 || k == 3 ? 1.f : 0.f, 0.f}, ff{0.f, 0.f}};
  float2 v = make_float2(z.x.h, 0.f), dv = make_float2(0.f, 0.f);
  if (active) {
    const float* pp = a.p + (size_t)l * a.ldp + 2 * (size_t)q;
    const float* ss = a.s ? a.s + (size_t)l * a.lds + 2 * (size_t)q : nullptr;
    const float al = ss ? ss[0] : 0.f, be = ss ? ss[1] : 0.f;
    float2 d0 = make_float2(0.f, 0.f);   // the entry of dT/dth; that of dT/dph is i times T's first column
    ffz dth;
    if (mzi_T_ff_quad(pp[0], pp[1], al, be, ss == nullptr, &z, bwd ? &cs : nullptr, diff ? &dth : nullptr)) {
      v = ffz_round(z);
      if (diff) d0 = ffz_round(dth);
    } else {   // angles beyond the float-float range
      C2x2 T, D0, D1;
      mzi_T(pp[0], pp[1], al, be, &T, diff ? &D0 : nullptr, diff ? &D1 : nullptr, bwd ? &cs : nullptr);
      auto entry = [&](const C2x2& c) { return k == 0 ? c.t00 : k == 1 ? c.t01 : k == 2 ? c.t10 : c.t11; };
      v = entry(T);
      if (diff) d0 = entry(D0);
      z = {ff{v.x, 0.f}, ff{v.y, 0.f}};
    }
    if (diff && a.dp) {
      const float* d = a.dp + (size_t)l * a.ldp + 2 * (size_t)q;
      dv = cadd(cscale(d[0], d0), cscale(d[1], k & 1 ? make_float2(0.f, 0.f) : make_float2(-v.y, v.x)));
    }
  }
  if constexpr (FRAME) {
    const int sh = kind == KIND_MIS ? 1 : 0;
    frame_entry(a, l, q, k, sh, z, cs);
    if (k == 0) frame_slot(a, l, q, t, sh, cs);
  }
  const int M = a.M, G = a.G;
  float2* tl = reinterpret_cast<float2*>(a.tiles + (size_t)l * a.layer_bytes);   // two entries of a row side by side
  if (kind < KIND_XL) {
    const int j = q / (M / 2), e = q % (M / 2);
    if (bwd && k == 0) tl[2 * M * G + e * G + j] = cs;
    const int at = 2 * ((2 * e + (k >> 1)) * G + j) + (k & 1);
    tl[at] = v;
    if (diff) tl[2 * M * G + at] = dv;
  } else {
    // butterfly over lanes: own rows of T, a -> (t00, t01), b -> (t11, t10); back-propagation: of T^H, a -> (conj t00,
    // conj t10), b -> (conj t11, conj t01)
    const int st = 1 << (kind - KIND_XL);
    const int A = 2 * st * (q / st) + (q % st), row = bwd ? k & 1 : k >> 1, m = row ? A + st : A;
    const int la = A / M, ma = A % M;
    if (bwd && k == 0) tl[2 * M * G + ma * (G / 2) + a_lane_index(la, st / M)] = cs;
    const int at = 2 * ((m % M) * G + m / M) + (k == 0 || k == 3 ? 0 : 1);
    tl[at] = bwd ? make_float2(v.x, -v.y) : v;
    if (diff) tl[2 * M * G + at] = dv;
  }
}

// Thread t of the coefficient pass, one per slot: every other crossing and tile
template <bool FRAME>
__device__ __forceinline__ void coef_body(const CoefArgs& a, int t) {
  const int np2 = a.G * a.M / 2, idx = t;
  if (idx >= a.L * np2) return;
  const int l = idx / np2, q = idx - l * np2;
  bool active = false;
  const int kind = layer_kind(a, l, q, &active);
  if (q == 0) write_layer(a, l, kind);
  const int M = a.M, G = a.G;
  const bool real = a.crossing == CR_ORTH;
  float4* tl = reinterpret_cast<float4*>(a.tiles + (size_t)l * a.layer_bytes);
  const bool xl = kind >= KIND_XL;
  int la = 0, ma = 0, lb = 0, mb = 0;
  if (xl) {
    const int st = 1 << (kind - KIND_XL);
    const int A = 2 * st * (q / st) + (q % st), Bm = A + st;
    la = A / M; ma = A % M; lb = Bm / M; mb = Bm % M;
  }
  const int j = q / (M / 2), e = q % (M / 2);
  if (!real) {
    C2x2 T, D0, D1;
    float2 csv = make_float2(0.f, 0.f);   // (cos, sin)(pi/4 + beta) for the direct MZI gradient; 0 if inactive
    Tff F;
    slot_T(a, l, q, active, T, D0, D1, (a.op == OP_BWD && a.gr == 1) ? &csv : nullptr, F);
    if constexpr (FRAME) {
      const int sh = kind == KIND_MIS ? 1 : 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) frame_entry(a, l, q, k, sh, F.t[k], csv);
      frame_slot(a, l, q, t, sh, csv);
    }
    if (a.op == OP_BWD && a.gr == 1) {
      float2* cs = reinterpret_cast<float2*>(tl + M * G);
      if (!xl) cs[e * G + j] = csv;
      else {
        const int d = (1 << (kind - KIND_XL)) / M;
        cs[ma * (G / 2) + a_lane_index(la, d)] = csv;
      }
    }
    if (a.op == OP_BWD && a.gr == 0) {   // planes [k][pos]: D0 row 0, D0 row 1, D1 row 0, D1 row 1
      float4* D = reinterpret_cast<float4*>(a.dtiles + (size_t)l * a.dlayer_bytes) + slot_pos(q, M, G);
      D[0] = make_float4(D0.t00.x, D0.t00.y, D0.t01.x, D0.t01.y);
      D[np2] = make_float4(D0.t10.x, D0.t10.y, D0.t11.x, D0.t11.y);
      D[2 * np2] = make_float4(D1.t00.x, D1.t00.y, D1.t01.x, D1.t01.y);
      D[3 * np2] = make_float4(D1.t10.x, D1.t10.y, D1.t11.x, D1.t11.y);
    }
    C2x2 dT = c2x2_zero();
    if (a.op == OP_FWDDIFF && active && a.dp) {
      const int n_p = crossing_np(a.crossing);
      const float* d = a.dp + (size_t)l * a.ldp + (size_t)q * n_p;
      const float d0 = d[0], d1 = (n_p > 1) ? d[1] : 0.f;
      dT.t00 = cadd(cscale(d0, D0.t00), cscale(d1, D1.t00));
      dT.t01 = cadd(cscale(d0, D0.t01), cscale(d1, D1.t01));
      dT.t10 = cadd(cscale(d0, D0.t10), cscale(d1, D1.t10));
      dT.t11 = cadd(cscale(d0, D0.t11), cscale(d1, D1.t11));
    }
    const int doff = M * G;
    if (!xl) {
      tl[(2 * e) * G + j] = make_float4(T.t00.x, T.t00.y, T.t01.x, T.t01.y);
      tl[(2 * e + 1) * G + j] = make_float4(T.t10.x, T.t10.y, T.t11.x, T.t11.y);
      if (a.op == OP_FWDDIFF) {
        tl[doff + (2 * e) * G + j] = make_float4(dT.t00.x, dT.t00.y, dT.t01.x, dT.t01.y);
        tl[doff + (2 * e + 1) * G + j] = make_float4(dT.t10.x, dT.t10.y, dT.t11.x, dT.t11.y);
      }
    } else if (a.op == OP_BWD) {   // own rows of T^H: a -> (conj t00, conj t10), b -> (conj t11, conj t01)
      tl[ma * G + la] = make_float4(T.t00.x, -T.t00.y, T.t10.x, -T.t10.y);
      tl[mb * G + lb] = make_float4(T.t11.x, -T.t11.y, T.t01.x, -T.t01.y);
    } else {                        // own rows of T: a -> (t00, t01), b -> (t11, t10)
      tl[ma * G + la] = make_float4(T.t00.x, T.t00.y, T.t01.x, T.t01.y);
      tl[mb * G + lb] = make_float4(T.t11.x, T.t11.y, T.t10.x, T.t10.y);
      if (a.op == OP_FWDDIFF) {
        tl[doff + ma * G + la] = make_float4(dT.t00.x, dT.t00.y, dT.t01.x, dT.t01.y);
        tl[doff + mb * G + lb] = make_float4(dT.t11.x, dT.t11.y, dT.t10.x, dT.t10.y);
      }
    }
  } else {
    R2x2 T, D0;
    slot_R(a, l, q, active, T, D0);
    if (a.op == OP_BWD && a.gr == 0) {
      float4* D = reinterpret_cast<float4*>(a.dtiles + (size_t)l * a.dlayer_bytes) + slot_pos(q, M, G);
      D[0] = make_float4(D0.t00, D0.t01, D0.t10, D0.t11);
    }
    R2x2 dT;
    dT.t00 = dT.t01 = dT.t10 = dT.t11 = 0.f;
    if (a.op == OP_FWDDIFF && active && a.dp) {
      const float d0 = a.dp[(size_t)l * a.ldp + q];
      dT.t00 = d0 * D0.t00; dT.t01 = d0 * D0.t01; dT.t10 = d0 * D0.t10; dT.t11 = d0 * D0.t11;
    }
    const int doff = (M / 2) * G;
    if (!xl) {
      tl[e * G + j] = make_float4(T.t00, T.t01, T.t10, T.t11);
      if (a.op == OP_FWDDIFF) tl[doff + e * G + j] = make_float4(dT.t00, dT.t01, dT.t10, dT.t11);
    } else {
      float2* ta = reinterpret_cast<float2*>(&tl[(ma >> 1) * G + la]) + (ma & 1);
      float2* tb = reinterpret_cast<float2*>(&tl[(mb >> 1) * G + lb]) + (mb & 1);
      if (a.op == OP_BWD) {        // rows of T^T
        *ta = make_float2(T.t00, T.t10);
        *tb = make_float2(T.t11, T.t01);
      } else {
        *ta = make_float2(T.t00, T.t01);
        *tb = make_float2(T.t11, T.t10);
        if (a.op == OP_FWDDIFF) {
          float2* da = reinterpret_cast<float2*>(&tl[doff + (ma >> 1) * G + la]) + (ma & 1);
          float2* db = reinterpret_cast<float2*>(&tl[doff + (mb >> 1) * G + lb]) + (mb & 1);
          *da = make_float2(dT.t00, dT.t01);
          *db = make_float2(dT.t11, dT.t10);
        }
      }
    }
  }
}

template <bool QUAD, bool FRAME>
__global__ void coef_kernel(const CoefArgs a) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if constexpr (QUAD) coef_quad<FRAME>(a, t);
  else coef_body<FRAME>(a, t);
}

}  // namespace mg
