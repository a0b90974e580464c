// Framed propagation of nearest-neighbour complex meshes (forward, and back-propagation with direct MZI
// gradients) on the tiles of the frame pass (mg_frame.cuh): crossings with a unit diagonal, 8 FMAs per vector
// forward instead of 16 and 28 instead of 44 in back-propagation.
//
// Fields enter in the frames of the first boundary they meet (forward: scaled by 2^-kFrameExp; back-propagation:
// times conj(D(L))) and leave by the inverse of the last one's; a RESCALE multiplies them by a factor per mode.
//
// Packing: one packed f32x2 FMA serves two vectors (the same crossing, its coefficients used twice) or, for the last
// vector of an odd number, the lane's modes m and m + M/2 (the crossings e and e + M/4, whose coefficients lie side by
// side in the tile).  By modes, the odd-shift layer's last pair mixes the halves, (M/2 - 1, M/2) and (M - 1, the next
// lane's 0), which costs moves: 640 instructions per pair of layers in back-propagation at M = 8, V = 4, against 568.
//
// What bounds it: the register operands of the packed FMAs.  One with three register pairs of its own takes 3 cycles of a
// scheduler, one that shares a pair with the FMA before it 2.3 to 2.5 (a loop of independent ones, GB300); at N = 256,
// B = 4096 back-propagation's 458 per layer and scheduler are 1050 to 1370 of its 1500 cycles.  Three or four warps per
// scheduler with fewer vectors each do not raise that (257 us for 12 warps of 3, 201 for 8 of 4).  Measured on GB300 at
// N = 256, L = 256, B = 4096 against the unframed kernels: forward 94 -> 63 us, back-propagation 249 -> 197 us; N = 600,
// L = 600, B = 2048: forward 314 -> 200 us, back-propagation 1412 -> 684 us.
//
// Work decomposition, pipeline, bounded waits and the gradient partials are those of mg_prop.cuh; a stage holds
// its layers' tiles and the factors of their first RESCALEs.
//
// Framed fields are 2^-22 to 2^48 of the fields' own (forward) or 2^-48 to 2^22 (back-propagation, the products of two of them
// 2^-96 to 2^44), so every vector comes in times a power of two that brings its largest part to 2^kFieldTop and leaves by
// its inverse: nothing overflows, or falls below the normal range, that does not without frames (but for products 2^35
// times smaller than the largest of their warp's).  The factors are exact; results do not depend on them.  They cost
// a launch and its reduction up to 2 us (N = 256, B = 4096 back-propagation 205.8 -> 207.3 us, forward 69.3 -> 67.7).
#pragma once
#include "mg_frame.cuh"

namespace mg {

// A layer's tile (main plane, gamma's behind it) and its gradient staging as seen by one lane: shared-memory addresses
struct FTile {
  uint32_t main, grad;
};
// 16 bytes of shared memory (volatile keeps them behind the barriers and waits)
__device__ __forceinline__ ulonglong2 lds16(uint32_t addr) {
  ulonglong2 v;
  asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(addr));
  return v;
}
__device__ __forceinline__ unsigned long long lds8(uint32_t addr) {
  unsigned long long v;
  asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ int lds4(uint32_t addr) {
  int v;
  asm volatile("ld.shared.s32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ ulonglong2 ld16(const ulonglong2* p) {
  ulonglong2 v;
  asm volatile("ld.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ void sts16(uint32_t addr, unsigned long long x, unsigned long long y) {
  asm volatile("st.shared.v2.u64 [%0], {%1, %2};" ::"r"(addr), "l"(x), "l"(y) : "memory");
}

// A packed pair of floats as one 64-bit register pair from load to store: held as two floats, the compiler splits and
// rebuilds the pairs with moves around loops and branches.
using p64 = unsigned long long;
__device__ __forceinline__ p64 p_pack(float x, float y) {
  p64 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ float2 p_split(p64 a) {
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(a));
  return d;
}
__device__ __forceinline__ p64 pfma(p64 a, p64 b, p64 c) {
  p64 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ p64 pmul(p64 a, p64 b) {
  p64 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ p64 psub(p64 a, p64 b) {
  p64 d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ p64 padd(p64 a, p64 b) {
  p64 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ p64 pneg(p64 a) { return a ^ 0x8000000080000000ull; }

// two modes of a vector, or two coefficients
struct P2 {
  p64 r, i;
};
struct PK {
  p64 r, i, n;   // n = -i
};
__device__ __forceinline__ PK pk(ulonglong2 q) { return PK{q.x, q.y, pneg(q.y)}; }

// a + c b, a + conj(c) b
__device__ __forceinline__ P2 p2_axpy(const PK& c, const P2& a, const P2& b) {
  return P2{pfma(c.r, b.r, pfma(c.n, b.i, a.r)), pfma(c.r, b.i, pfma(c.i, b.r, a.i))};
}
__device__ __forceinline__ P2 p2_caxpy(const PK& c, const P2& a, const P2& b) {
  return P2{pfma(c.r, b.r, pfma(c.i, b.i, a.r)), pfma(c.r, b.i, pfma(c.n, b.r, a.i))};
}
// The fields of one lane: its first 2 (V / 2) vectors in pairs v[p][mode], the last one of an odd V by modes
// m[0][k] = modes (k, k + M/2)
template <int M, int V>
struct Fields {
  static constexpr int kPairs = V / 2, kOdd = V & 1;
  P2 v[kPairs ? kPairs : 1][M];
  P2 m[1][M / 2];
};

__device__ __forceinline__ PK pk_dup(float re, float im) { return PK{p_pack(re, re), p_pack(im, im), p_pack(-im, -im)}; }

// ---- one crossing per packed half, NP register pairs (ua, ub: the fields' two modes; wa, wb: the gradients'): forward, or
// back-propagation, which returns the packed (dJ/dth, dJ/dph) sums
template <int OP, int NP, typename UA, typename UB, typename WA, typename WB>
__device__ __forceinline__ P2 f_crossing(const PK& al, const PK& be, const PK& ga, UA ua, UB ub, WA wa, WB wb) {
  if constexpr (OP == OP_FWD) {
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const P2 a = ua(p), b = ub(p);
      ua(p) = p2_axpy(al, a, b);
      ub(p) = p2_axpy(be, b, a);
    }
    return P2{0, 0};
  } else {
    // dJ/dth = Im(h conj(m)) with m, h = y, g behind S(beta)^H (mode a), dJ/dph = Im(g conj(x)) of mode a at the input;
    // each difference's two products are summed apart
    p64 thp = 0, thq = 0, php = 0, phq = 0;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const P2 a = ua(p), b = ub(p), g = wa(p), h = wb(p);
      const P2 m = p2_axpy(ga, a, b), mg = p2_axpy(ga, g, h);
      thp = pfma(mg.i, m.r, thp);
      thq = pfma(mg.r, m.i, thq);
      const P2 x = p2_caxpy(be, a, b), gx = p2_caxpy(be, g, h);
      ub(p) = p2_caxpy(al, b, a);
      wb(p) = p2_caxpy(al, h, g);
      ua(p) = x;
      wa(p) = gx;
      php = pfma(gx.i, x.r, php);
      phq = pfma(gx.r, x.i, phq);
    }
    return P2{psub(thp, thq), psub(php, phq)};
  }
}

// ---- one layer on the lane's vectors: KIND 0 (pairs (2e, 2e+1) in the lane) or KIND_MIS (pairs (2e+1, 2e+2), the last
// one with the next lane's first mode, computed by this lane)
template <int OP, int M, int V, int KIND>
__device__ __forceinline__ void f_layer(const FTile& t, int G, int j, int r, Fields<M, V>& u, Fields<M, V>& w) {
  constexpr int H = M / 2, sh = KIND == 0 ? 0 : 1, NV = V / 2;
  constexpr bool odd = V & 1;
  P2 nu[NV + 1], nw[NV + 1];   // second modes of the boundary pairs (last: of the vector packed by modes)
  auto next_v = [&](const P2& p) {
    const float2 x = shfl_down(p_split(p.r), 1, G), y = shfl_down(p_split(p.i), 1, G);
    return P2{p_pack(x.x, x.y), p_pack(y.x, y.y)};
  };
  auto back_v = [&](P2& p, const P2& q) {
    const float2 x = shfl_up(p_split(q.r), 1, G), y = shfl_up(p_split(q.i), 1, G), pr = p_split(p.r), pi = p_split(p.i);
    p.r = p_pack(j != 0 ? x.x : pr.x, j != 0 ? x.y : pr.y);
    p.i = p_pack(j != 0 ? y.x : pi.x, j != 0 ? y.y : pi.y);
  };
  auto next_m = [&](const P2& p) {   // modes M/2 and the next lane's 0
    const float2 pr = p_split(p.r), pi = p_split(p.i);
    const float2 s = shfl_down(make_float2(pr.x, pi.x), 1, G);
    return P2{p_pack(pr.y, s.x), p_pack(pi.y, s.y)};
  };
  auto back_m = [&](P2& p, const P2& q) {
    const float2 pr = p_split(p.r), pi = p_split(p.i), qr = p_split(q.r), qi = p_split(q.i);
    const float2 s = shfl_up(make_float2(qr.y, qi.y), 1, G);
    p.r = p_pack(j != 0 ? s.x : pr.x, qr.x);
    p.i = p_pack(j != 0 ? s.y : pi.x, qi.x);
  };
  if constexpr (KIND != 0) {
#pragma unroll
    for (int p = 0; p < NV; ++p) {
      nu[p] = next_v(u.v[p][0]);
      if constexpr (OP != OP_FWD) nw[p] = next_v(w.v[p][0]);
    }
    if constexpr (odd) {
      nu[NV] = next_m(u.m[0][0]);
      if constexpr (OP != OP_FWD) nw[NV] = next_m(w.m[0][0]);
    }
  }
#pragma unroll
  for (int e = H / 2 - 1; e >= 0; --e) {   // (the boundary pair first: its results travel back while the others run)
    const uint32_t o = (uint32_t)(2 * e * G) * 16u;
    const ulonglong2 qa = lds16(t.main + o), qb = lds16(t.main + o + (uint32_t)G * 16u);
    const ulonglong2 qg = OP == OP_BWD ? lds16(t.main + (uint32_t)(G * M) * 8u + o / 2) : make_ulonglong2(0, 0);
    float2 dth = make_float2(0.f, 0.f), dph = dth;
    const bool last = KIND != 0 && e == H / 2 - 1;
    if constexpr (NV > 0) {
      const float2 ar = p_split(qa.x), ai = p_split(qa.y), br = p_split(qb.x), bi = p_split(qb.y);
      const float2 gr = p_split(qg.x), gi = p_split(qg.y);
#pragma unroll
      for (int c = 1; c >= 0; --c) {
        const int ma = 2 * (e + c * (M / 4)) + sh;
        const bool edge = last && c == 1;
        const P2 d = f_crossing<OP, NV>(
            c ? pk_dup(ar.y, ai.y) : pk_dup(ar.x, ai.x), c ? pk_dup(br.y, bi.y) : pk_dup(br.x, bi.x),
            c ? pk_dup(gr.y, gi.y) : pk_dup(gr.x, gi.x), [&](int p) -> P2& { return u.v[p][ma]; },
            [&](int p) -> P2& { return edge ? nu[p] : u.v[p][edge ? 0 : ma + 1]; }, [&](int p) -> P2& { return w.v[p][ma]; },
            [&](int p) -> P2& { return edge ? nw[p] : w.v[p][edge ? 0 : ma + 1]; });
        if constexpr (OP == OP_BWD) {
          const float2 th = p_split(d.r), ph = p_split(d.i);
          (c ? dth.y : dth.x) = th.x + th.y;
          (c ? dph.y : dph.x) = ph.x + ph.y;
        }
        if (edge) {
#pragma unroll
          for (int p = 0; p < NV; ++p) {
            back_v(u.v[p][0], nu[p]);
            if constexpr (OP != OP_FWD) back_v(w.v[p][0], nw[p]);
          }
        }
      }
    }
    p64 th = p_pack(dth.x, dth.y), ph = p_pack(dph.x, dph.y);
    if constexpr (odd) {
      const int k = 2 * e + sh;
      const P2 d = f_crossing<OP, 1>(
          pk(qa), pk(qb), pk(qg), [&](int) -> P2& { return u.m[0][k]; },
          [&](int) -> P2& { return last ? nu[NV] : u.m[0][last ? 0 : k + 1]; }, [&](int) -> P2& { return w.m[0][k]; },
          [&](int) -> P2& { return last ? nw[NV] : w.m[0][last ? 0 : k + 1]; });
      if constexpr (OP == OP_BWD) {
        th = NV ? padd(th, d.r) : d.r;
        ph = NV ? padd(ph, d.i) : d.i;
      }
      if (last) {
        back_m(u.m[0][0], nu[NV]);
        if constexpr (OP != OP_FWD) back_m(w.m[0][0], nw[NV]);
      }
    }
    if constexpr (OP == OP_BWD) {
      if (G < 32) {
        float2 t2 = p_split(th), p2 = p_split(ph);
        for (int off = G; off < 32; off <<= 1) {
          t2 = cadd(t2, shfl_xor(t2, off, 32));
          p2 = cadd(p2, shfl_xor(p2, off, 32));
        }
        th = p_pack(t2.x, t2.y);
        ph = p_pack(p2.x, p2.y);
      }
      if (r == 0) sts16(t.grad + o / 2, th, ph);
    }
  }
}

// u <- d u (CONJ: conj(d) u) with a factor for each of the lane's modes: d(k) is that of modes k and k + M/2
template <int M, int V, bool CONJ, typename D>
__device__ __forceinline__ void f_diag(D d, Fields<M, V>& u) {
  auto times = [](const PK& c0, P2& p) {
    const P2 a = p;
    const PK c = CONJ ? PK{c0.r, c0.n, c0.i} : c0;
    p = P2{pfma(c.r, a.r, pmul(c.n, a.i)), pfma(c.r, a.i, pmul(c.i, a.r))};
  };
#pragma unroll
  for (int k = 0; k < M / 2; ++k) {
    const ulonglong2 q = d(k);
    if constexpr (V > 1) {
      const float2 re = p_split(q.x), im = p_split(q.y);
      const PK lo = pk_dup(re.x, im.x), hi = pk_dup(re.y, im.y);
#pragma unroll
      for (int p = 0; p < V / 2; ++p) {
        times(lo, u.v[p][k]);
        times(hi, u.v[p][k + M / 2]);
      }
    }
    if constexpr (V & 1) times(pk(q), u.m[0][k]);
  }
}
// f(a, b) on the register pairs of two lanes' fields
template <int M, int V, typename F>
__device__ __forceinline__ void f_each(Fields<M, V>& u, Fields<M, V>& w, F f) {
#pragma unroll
  for (int p = 0; p < V / 2; ++p)
#pragma unroll
    for (int k = 0; k < M; ++k) f(u.v[p][k], w.v[p][k]);
  if constexpr (V & 1)
#pragma unroll
    for (int k = 0; k < M / 2; ++k) f(u.m[0][k], w.m[0][k]);
}
// 2^k, -126 <= k <= 127
__device__ __forceinline__ float pow2f(int k) { return __int_as_float((k + 127) << 23); }
// vector v of the lane times 2^k(v), |k| <= 252, in two steps
template <int M, int V, typename K>
__device__ __forceinline__ void f_scale(K k, Fields<M, V>& u) {
  auto times = [](p64 a, p64 b, P2& x) { x = P2{pmul(pmul(x.r, a), b), pmul(pmul(x.i, a), b)}; };
#pragma unroll
  for (int p = 0; p < V / 2; ++p) {
    const int k0 = k(2 * p), k1 = k(2 * p + 1);
    const p64 a = p_pack(pow2f(k0 >> 1), pow2f(k1 >> 1)), b = p_pack(pow2f(k0 - (k0 >> 1)), pow2f(k1 - (k1 >> 1)));
#pragma unroll
    for (int m = 0; m < M; ++m) times(a, b, u.v[p][m]);
  }
  if constexpr (V & 1) {
    const int k0 = k(V - 1);
    const float a = pow2f(k0 >> 1), b = pow2f(k0 - (k0 >> 1));
#pragma unroll
    for (int m = 0; m < M / 2; ++m) times(p_pack(a, a), p_pack(b, b), u.m[0][m]);
  }
}
// The k that brings the largest part of each of the warp's vectors to [2^kFieldTop, 2^(kFieldTop + 1)); kNoScale for one that is
// 0 or holds infinity
constexpr int kNoScale = 1 << 20;
template <int M, int V>
__device__ __forceinline__ void f_wanted(const Fields<M, V>& u, int (&k)[V]) {
  auto of = [](float m) {   // (fmaxf passes NaN by)
    const unsigned b = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
    if (b == 0 || b >= 0x7f800000u) return kNoScale;
    return kFieldTop - (b >= 0x00800000u ? (int)(b >> 23) - 127 : -118 - __clz(b));
  };
#pragma unroll
  for (int p = 0; p < V / 2; ++p) {
    float a = 0.f, b = 0.f;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const float2 re = p_split(u.v[p][m].r), im = p_split(u.v[p][m].i);
      a = fmaxf(a, fmaxf(fabsf(re.x), fabsf(im.x)));
      b = fmaxf(b, fmaxf(fabsf(re.y), fabsf(im.y)));
    }
    k[2 * p] = of(a);
    k[2 * p + 1] = of(b);
  }
  if constexpr (V & 1) {
    float a = 0.f;
#pragma unroll
    for (int m = 0; m < M / 2; ++m) {
      const float2 re = p_split(u.m[0][m].r), im = p_split(u.m[0][m].i);
      a = fmaxf(a, fmaxf(fmaxf(fabsf(re.x), fabsf(re.y)), fmaxf(fabsf(im.x), fabsf(im.y))));
    }
    k[V - 1] = of(a);
  }
}

// Steps: the walk goes by pairs of layers, (aligned, odd-shift) forward and (odd-shift, aligned) in back-propagation, as
// one straight-line body; a layer whose partner is not there goes with a layer of zeros (alpha = beta = 0: identity)
// in its place.  One body for everything: with a second one in the kernel's loop the compiler moves every field register
// where they join (300 moves per pair of layers in back-propagation, half again its arithmetic).
// The code of the step that starts at a layer: which of the two positions are layers of the mesh, and whether a RESCALE
// follows (back-propagation: goes before).
constexpr int STEP_0 = 1, STEP_1 = 2, STEP_RESCALE = 4;
constexpr int kCodePad = 4;   // codes readable before and after the layers
template <int OP>
__device__ __forceinline__ int step_code(const int* kinds, int L, int l) {
  auto at = [&](int i) { return i >= 0 && i < L ? __ldg(kinds + i) : -1; };
  const int k = at(l);
  if (k < 0) return 0;
  const bool mis = k & KIND_MIS, resc = k & KIND_RESCALE;
  const int c = resc ? STEP_RESCALE : 0;
  if (OP == OP_FWD) {
    if (mis || resc) return c | (mis ? STEP_1 : STEP_0);
    const int n = at(l + 1);
    return n < 0 || !(n & KIND_MIS) ? STEP_0 : STEP_0 | STEP_1 | (n & KIND_RESCALE ? STEP_RESCALE : 0);
  }
  return mis ? c | STEP_0 | (at(l - 1) == 0 ? STEP_1 : 0) : c | STEP_1;
}

// bytes of a layer's tile: forward launches read back-propagation's tiles too
template <int OP>
__device__ __forceinline__ uint32_t framed_layer(const FramedArgs& a, int np2) {
  return OP == OP_BWD ? (uint32_t)np2 * 24u : a.flb;
}

// Layers [lo, hi) of a chunk in the stage at st; resc: the factors of its first framed_resc_rows RESCALE (more are
// read from global memory); codes: layer 0's step code
template <int OP, int M, int V>
__device__ __forceinline__ void f_chunk(const FramedArgs& a, uint32_t codes, const FTile& st, uint32_t resc, const FTile& none,
                                        int np2, int lo, int hi, int G, int j, int r, Fields<M, V>& u, Fields<M, V>& w) {
  constexpr int kDir = OP == OP_BWD ? -1 : 1;
  const uint32_t layer = framed_layer<OP>(a, np2), grad = (uint32_t)np2 * 8u;
  int l = OP == OP_BWD ? hi - 1 : lo, left = hi - lo;
  int rows = framed_resc_rows(a.fcl);
  auto tile = [&](bool there, int at) {
    const uint32_t i = (uint32_t)(at - lo);
    return there ? FTile{st.main + i * layer, st.grad + i * grad} : none;
  };
  auto rescale = [&](int at) {
    const ulonglong2* p = rows > 0 ? static_cast<const ulonglong2*>(__cvta_shared_to_generic(resc))
                                   : reinterpret_cast<const ulonglong2*>(a.resc + (size_t)at * np2) + j;
    --rows;
    resc += (uint32_t)np2 * 16u;
    f_diag<M, V, OP == OP_BWD>([&](int k) { return ld16(p + k * G); }, u);
    if constexpr (OP == OP_BWD) f_diag<M, V, true>([&](int k) { return ld16(p + k * G); }, w);
  };
  int c = lds4(codes + 4 * l);
#pragma unroll 1
  while (left > 0) {
    if (OP == OP_BWD && (c & STEP_RESCALE)) rescale(l);
    bool due;
#pragma unroll 1
    do {
      if (left == 1 && (c & STEP_0) && (c & STEP_1)) c &= OP == OP_BWD ? ~STEP_1 : ~(STEP_1 | STEP_RESCALE);
      const int n = (c & 1) + ((c >> 1) & 1);
      const FTile t0 = tile(c & STEP_0, l), t1 = tile(c & STEP_1, l + (c & STEP_0 ? kDir : 0));
      due = OP == OP_FWD && (c & STEP_RESCALE);
      l += n * kDir;
      left -= n;
      c = lds4(codes + 4 * l);
      f_layer<OP, M, V, OP == OP_BWD ? KIND_MIS : 0>(t0, G, j, r, u, w);
      f_layer<OP, M, V, OP == OP_BWD ? 0 : KIND_MIS>(t1, G, j, r, u, w);
      if (OP == OP_BWD) due = c & STEP_RESCALE;
    } while (left > 0 && !due);
    if (OP == OP_FWD && due) rescale(l - 1);
  }
}

// ---- field I/O: lane j's modes [j*M, j*M+M) of V vectors; vectors from vend on and modes from N on read 0
template <int M, int V>
__device__ __forceinline__ void f_load(Fields<M, V>& u, const void* src, int vb0, int vend, int N, int ldu, int j) {
  auto at = [&](int v, int m) {   // modes m, m + 1
    const float4* p = reinterpret_cast<const float4*>(static_cast<const float2*>(src) + (size_t)(vb0 + v) * ldu + j * M);
    return vb0 + v < vend && j * M + m < N ? p[m / 2] : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  auto two = [](float4 x, float4 y, P2* p) {
    p[0] = P2{p_pack(x.x, y.x), p_pack(x.y, y.y)};
    p[1] = P2{p_pack(x.z, y.z), p_pack(x.w, y.w)};
  };
#pragma unroll
  for (int p = 0; p < V / 2; ++p)
#pragma unroll
    for (int k = 0; k < M; k += 2) two(at(2 * p, k), at(2 * p + 1, k), &u.v[p][k]);
  if constexpr (V & 1)
#pragma unroll
    for (int k = 0; k < M / 2; k += 2) two(at(V - 1, k), at(V - 1, M / 2 + k), &u.m[0][k]);
}
template <int M, int V>
__device__ __forceinline__ void f_store(const Fields<M, V>& u, void* dst, int vb0, int vend, int N, int ldu, int j) {
  auto put = [&](int v, int m, float4 x) {
    float4* p = reinterpret_cast<float4*>(static_cast<float2*>(dst) + (size_t)(vb0 + v) * ldu + j * M);
    if (vb0 + v < vend && j * M + m < N) p[m / 2] = x;
  };
  auto two = [&](const P2* p, int v0, int m0, int v1, int m1) {
    const float2 ar = p_split(p[0].r), ai = p_split(p[0].i), br = p_split(p[1].r), bi = p_split(p[1].i);
    put(v0, m0, make_float4(ar.x, ai.x, br.x, bi.x));
    put(v1, m1, make_float4(ar.y, ai.y, br.y, bi.y));
  };
#pragma unroll
  for (int p = 0; p < V / 2; ++p)
#pragma unroll
    for (int k = 0; k < M; k += 2) two(&u.v[p][k], 2 * p, k, 2 * p + 1, k);
  if constexpr (V & 1)
#pragma unroll
    for (int k = 0; k < M / 2; k += 2) two(&u.m[0][k], V - 1, k, V - 1, M / 2 + k);
}
// the frames d of the lane's modes as f_diag's factors
template <int M>
__device__ __forceinline__ ulonglong2 frame_pair(const float2* __restrict__ d, int j, int k) {
  const float2 d0 = __ldg(d + j * M + k), d1 = __ldg(d + j * M + M / 2 + k);
  return make_ulonglong2(p_pack(d0.x, d1.x), p_pack(d0.y, d1.y));
}
// CTA barrier by number: with MIX, warps of both kinds meet at it from their own copies of the body
__device__ __forceinline__ void cta_sync() { asm volatile("barrier.cta.sync.aligned 0;" ::: "memory"); }

// Sum of the W warps' staged gradients of a chunk (W a multiple of 4), in warp order, at the least of their scales, into this
// CTA's partials of the layers from lo on: n float4 of consecutive layers.  Equal scales, nearly always, have a loop of their
// own: with the factors in one loop for both, N = 400, B = 2432 took 393 us instead of 383.  turn: the chunk; the warps that the last round of a chunk leaves over
// change with it (the same two of eight at M = 20: back-propagation at N = 600, B = 2048 727 us, in turns 684)
__device__ __forceinline__ void f_reduce(uint32_t gst, uint32_t warp_bytes, int W, int n, int turn, const int* scales,
                                         const int* scale, ulonglong2* out) {
  const int least = scales[0];
  int first = threadIdx.x + (64 * turn) % (int)blockDim.x;
  if (first >= (int)blockDim.x) first -= blockDim.x;
  if (least >= scales[1]) {
#pragma unroll 1
    for (int idx = first; idx < n; idx += blockDim.x) {
      uint32_t p = gst + (uint32_t)idx * 16u;
      ulonglong2 t = make_ulonglong2(0, 0);
#pragma unroll 1
      for (int w = 0; w < W; w += 4, p += 4 * warp_bytes) {
        const ulonglong2 a = lds16(p), b = lds16(p + warp_bytes), c = lds16(p + 2 * warp_bytes), d = lds16(p + 3 * warp_bytes);
        t.x = padd(padd(padd(padd(t.x, a.x), b.x), c.x), d.x);
        t.y = padd(padd(padd(padd(t.y, a.y), b.y), c.y), d.y);
      }
      out[idx] = t;
    }
    return;
  }
#pragma unroll 1
  for (int idx = first; idx < n; idx += blockDim.x) {
    uint32_t p = gst + (uint32_t)idx * 16u;
    ulonglong2 t = make_ulonglong2(0, 0);
#pragma unroll 1
    for (int w = 0; w < W; w += 4, p += 4 * warp_bytes) {
      ulonglong2 x[4];
      float f[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        x[i] = lds16(p + i * warp_bytes);
        f[i] = pow2f(max(least - scale[kWarpScales * (w + i) + 8], -126));
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        t.x = padd(t.x, pmul(p_pack(f[i], f[i]), x[i].x));
        t.y = padd(t.y, pmul(p_pack(f[i], f[i]), x[i].y));
      }
    }
    out[idx] = t;
  }
}

// The warp's vectors [vb0, vb0 + V) (per lane group) through all layers.  The pipeline's barriers are initialised, the
// step codes and the layer of zeros are in shared memory.
//
// No CTA barrier between the first chunk and the last: a warp that has its chunk's stage goes through the chunk, sums
// its share of the chunk before (kGradSlots of them are staged) and arrives; the only wait is for the others to have
// finished that earlier chunk, so the warps of a scheduler may drift apart by up to a chunk and keep each other's
// latency covered.  The copies are issued by one thread, of another warp for every chunk (those of V - 1 vectors where
// there are some): what a warp does beyond its layers holds all the others up.  Measured on GB300 against two CTA barriers
// and the sum at every chunk's end, copies issued by warp 0: N = 600, L = 600, B = 2048 803 -> 684 us, N = 400, B = 2432
// 432 -> 368 us, N = 128, B = 4000 68 -> 60 us.
struct FramedSmem {
  unsigned char* base;
  uint32_t zero, gst;
  uint32_t bars;        // [kFrameStages] the stage has its copies, [kFrameStages] every warp is done with the stage
  uint32_t codes;       // of layer 0
  uint32_t resc;        // per chunk: the layers of its first framed_resc_rows RESCALE, -1 behind the last
  volatile int* state;  // [0] a wait ran out, [1] chunks whose copies were issued
  int* scales;          // least and largest of the warps' scales (gradients' products)
  int* scale;           // kWarpScales per warp: its vectors' exponents (4 of u, 4 of w), its scale
};
// Layers of the walk in chunks of CL; the first chunk is one shorter where that keeps pairs of layers whole
template <int OP>
struct Chunks {
  int L, CL, cut, n;
  __device__ __forceinline__ Chunks(const FramedArgs& a) : L(a.L), CL(a.fcl) {
    const int first = __ldg(a.fkinds + (OP == OP_BWD ? L - 1 : 0));
    cut = (OP == OP_BWD ? !(first & KIND_MIS) : (first & KIND_MIS) != 0) && CL > 1 ? 1 : 0;
    n = (L + cut + CL - 1) / CL;
  }
  __device__ __forceinline__ int walked(int c) const { return min(L, max(0, c * CL - cut)); }   // layers before chunk c
  __device__ __forceinline__ int lo(int c) const { return OP == OP_BWD ? L - walked(c + 1) : walked(c); }
  __device__ __forceinline__ int hi(int c) const { return OP == OP_BWD ? L - walked(c) : walked(c + 1); }
};
template <int OP, int M, int V, int GT>
__device__ __forceinline__ void framed_body(const FramedArgs& a, const FramedSmem& sm, const Chunks<OP>& ch, int vb0, int issuer) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const Lanes<GT> ln(a.G, a.logG);
  const int G = ln.G, j = ln.j, r = ln.r;
  const int np2 = (G * M) >> 1, CL = a.fcl;
  constexpr int S = kFrameStages;
  const uint32_t layer = framed_layer<OP>(a, np2), row = (uint32_t)np2 * 16u, warp_bytes = (uint32_t)CL * (row / 2), j16 = (uint32_t)j * 16u;
  const uint32_t stage = (uint32_t)framed_stage_bytes(layer, np2, CL), ring = smem_u32(sm.base);
  const uint32_t slot_bytes = (uint32_t)a.W * warp_bytes;
  Fields<M, V> u, w;
  f_load<M, V>(u, a.in0, vb0, a.vend, a.N, a.ldu, j);
  if constexpr (OP == OP_BWD) f_load<M, V>(w, a.target ? a.target : a.in1, vb0, a.vend, a.N, a.ldu, j);

  const int nch = ch.n;
  auto wait = [&](uint32_t bar, uint32_t phase) {
    return __all_sync(0xffffffffu, mbar_wait_bounded(bar, phase, a.wait_ns ? a.wait_ns : kWaitLimitNs));
  };
  // one thread: the copies of chunk c into stage s
  auto issue = [&](int c, int s) {
    sm.state[1] = c + 1;
    if (c + 1 == a.unarmed) return;
    const int lo = ch.lo(c), n = ch.hi(c) - lo, xr = framed_resc_rows(CL);
    int rows = 0;
    while (rows < xr && lds4(sm.resc + 4u * (c * xr + rows)) >= 0) ++rows;
    const uint32_t bar = sm.bars + 8u * s, at = ring + (uint32_t)s * stage;
    mbar_arrive_expect_tx(bar, n * layer + rows * row);
    tma_load_1d(at, reinterpret_cast<const unsigned char*>(a.main) + (size_t)lo * layer, n * layer, bar);
    for (int k = 0; k < rows; ++k)
      tma_load_1d(at + (uint32_t)CL * layer + (uint32_t)k * row, a.resc + (size_t)lds4(sm.resc + 4u * (c * xr + k)) * np2, row, bar);
  };
  if (tid == 0)
    for (int c = 0; c < min(S, nch); ++c) issue(c, c);
  int* const scale = sm.scale + kWarpScales * warp;
  if constexpr (OP == OP_FWD) {
    int ku[V];
    f_wanted<M, V>(u, ku);
#pragma unroll
    for (int v = 0; v < V; ++v) {
      if (ku[v] == kNoScale) ku[v] = 0;
      if (lane == 0) scale[v] = ku[v];
    }
    f_scale<M, V>([&](int v) { return ku[v] - kFrameTop; }, u);
  } else {
    if (a.target)   // fused L2 loss to a target: g = 2 (y - t)
      f_each<M, V>(u, w, [](P2& y, P2& t) {
        const p64 two = p_pack(2.f, 2.f);
        t = P2{pmul(two, psub(y.r, t.r)), pmul(two, psub(y.i, t.i))};
      });
    // one scale for all products of the warp, since its vectors' are added: that of the largest, in the range where a float
    // holds it, in steps of 16 (most launches then have one scale; unit vectors of 64 to 640 modes and gradients of their size
    // want 46 to 54, the middle of a step).  What a vector's own product is short of that, u and
    // w bear half each, up to 2^80, within which neither loses bits (a product below 2^-160 of the largest counts as up to that).
    int ku[V], kw[V], all = kNoScale;
#pragma unroll
    for (int v = 0; v < V; ++v) ku[v] = kw[v] = 0;
    if (a.scales) {
      f_wanted<M, V>(u, ku);
      f_wanted<M, V>(w, kw);
#pragma unroll
      for (int v = 0; v < V; ++v)
        if (ku[v] != kNoScale && kw[v] != kNoScale) all = min(all, ku[v] + kw[v]);
      if (all != kNoScale) all = ((max(all, -80) + 8) & ~15) - 8;
      if (lane == 0) {
        scale[8] = all;
        if (all != kNoScale) {
          atomicMin(sm.scales, all);
          atomicMax(sm.scales + 1, all);
        }
      }
    }
#pragma unroll
    for (int v = 0; v < V; ++v) {   // (a product with 0 or infinity has no scale)
      if (a.scales && ku[v] != kNoScale && kw[v] != kNoScale) {
        kw[v] -= min(max((ku[v] + kw[v] - all) >> 1, 0), 80);
        ku[v] = max(all - kw[v], ku[v] - 80);
      }
      if (ku[v] == kNoScale) ku[v] = 0;
      if (kw[v] == kNoScale) kw[v] = 0;
      if (lane == 0) {
        scale[v] = ku[v];
        scale[4 + v] = kw[v];
      }
    }
    f_scale<M, V>([&](int v) { return ku[v]; }, u);
    f_scale<M, V>([&](int v) { return kw[v]; }, w);
    f_diag<M, V, true>([&](int k) { return frame_pair<M>(a.dfin, j, k); }, u);
    f_diag<M, V, true>([&](int k) { return frame_pair<M>(a.dfin, j, k); }, w);
  }

  // chunk c: stage and gradient slot s = c % S, of whose barriers it is phase ph = (c / S) & 1
  auto reduce = [&](int c, int s) {
    const int lo = ch.lo(c);
    f_reduce(sm.gst + (uint32_t)s * slot_bytes, warp_bytes, a.W, (ch.hi(c) - lo) * (np2 / 2), c, sm.scales, sm.scale,
             reinterpret_cast<ulonglong2*>(a.partial + (size_t)lo * np2));
  };
  const FTile none{sm.zero + j16, sm.gst + (uint32_t)S * slot_bytes + j16};
  int c = 0, s = 0;
  uint32_t ph = 0;
  bool ok = true;
#pragma unroll 1
  for (; c < nch; ++c) {
    ok = wait(sm.bars + 8u * s, ph);
    if (!ok) break;
    const uint32_t at = ring + (uint32_t)s * stage + j16;
    f_chunk<OP, M, V>(a, sm.codes, FTile{at, sm.gst + (uint32_t)s * slot_bytes + (uint32_t)warp * warp_bytes + j16},
                      at + (uint32_t)CL * layer, none, np2, ch.lo(c), ch.hi(c), G, j, r, u, w);
    const bool mine = warp == issuer + (c & 3);
    if (c > 0 && (OP == OP_BWD || mine)) {
      // every warp is done with chunk c - 1 (and, having waited as this one does, with the sum of chunk c - 2, whose slot
      // is the next chunk's)
      const int prev = s ? s - 1 : S - 1;
      ok = wait(sm.bars + 8u * (S + prev), s ? ph : ph ^ 1);
      if (!ok) break;
      if (mine && lane == 0 && c + S - 1 < nch) issue(c + S - 1, prev);
      if constexpr (OP == OP_BWD) reduce(c - 1, prev);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(sm.bars + 8u * (S + s));
    if (++s == S) {
      s = 0;
      ph ^= 1;
    }
  }
  if (!ok && lane == 0) sm.state[0] = 1;
  cta_sync();
  if (sm.state[0]) {
    // a wait ran out: record, wait (bounded) for the copies still in flight, release the barriers, leave
    if (tid == 0) {
      set_status(a.status, ST_TIMEOUT);
      for (int cc = c; cc < sm.state[1]; ++cc)
        if (cc + 1 != a.unarmed)
          mbar_wait_bounded(sm.bars + 8u * (cc % S), (uint32_t)((cc / S) & 1), a.wait_ns ? a.wait_ns : kWaitLimitNs);
      for (int k = 0; k < 2 * S; ++k) mbar_inval(sm.bars + 8u * k);
    }
    return;
  }
  if (tid == 0)
    for (int k = 0; k < 2 * S; ++k) mbar_inval(sm.bars + 8u * k);
  if constexpr (OP == OP_BWD) {
    if (nch > 0) reduce(nch - 1, (nch - 1) % S);
    if (tid == 0 && a.scales) *a.scales = sm.scales[0];
  }
  if constexpr (OP == OP_FWD) {
    f_diag<M, V, false>([&](int k) { return frame_pair<M>(a.dfin, j, k); }, u);
    f_scale<M, V>([&](int v) { return -scale[v]; }, u);
    f_store<M, V>(u, a.out0, vb0, a.vend, a.N, a.ldu, j);
  } else {
    if (a.out0 != nullptr) {
      f_scale<M, V>([&](int v) { return -scale[v] - kFrameTop; }, u);
      f_store<M, V>(u, a.out0, vb0, a.vend, a.N, a.ldu, j);
    }
    f_scale<M, V>([&](int v) { return -scale[4 + v] - kFrameTop; }, w);
    f_store<M, V>(w, a.out1, vb0, a.vend, a.N, a.ldu, j);
  }
}

// The vectors [v0, vend) of a by one CTA: W warps of V vectors per lane group; MIX: warps 4-7 (12-15) take V - 1, so that
// every scheduler carries 2V - 1.  The two kinds have a body each, chosen once per warp.  A mesh that the frames do not
// suit (a.refuse) takes the unframed body of mg_prop.cuh on the same vectors.
template <int OP, int M, int V, int GT, bool MIX>
__device__ __forceinline__ void framed_run(const FramedArgs& a, unsigned char* smem) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = GT ? GT : a.G, R = 32 / G, np2 = (G * M) >> 1, r = lane / G, v0 = a.v0;
  if (__ldg(a.count) >= a.refuse) {
    prop_body<OP, M, V, false, GT, OP == OP_BWD ? 1 : 0, false, true>(a, smem);
    return;
  }
  const uint32_t layer = framed_layer<OP>(a, np2);
  const size_t bars = framed_bars_offset(OP, layer, np2, a.W, a.fcl);
  const Chunks<OP> ch(a);
  FramedSmem sm;
  sm.base = smem;
  sm.zero = smem_u32(smem + kFrameStages * framed_stage_bytes(layer, np2, a.fcl));
  sm.gst = sm.zero + layer;
  sm.bars = smem_u32(smem + bars);
  sm.state = reinterpret_cast<volatile int*>(smem + bars + 16 * kFrameStages);
  sm.scales = reinterpret_cast<int*>(smem + bars + 16 * kFrameStages + 8);
  sm.scale = reinterpret_cast<int*>(smem + bars + 16 * kFrameStages + 16);
  int* codes = sm.scale + kWarpScales * a.W + kCodePad;
  int* resc = codes + a.L + kCodePad;
  sm.codes = smem_u32(codes);
  sm.resc = smem_u32(resc);
  for (int c = tid; c < ch.n; c += blockDim.x) {
    const int lo = ch.lo(c), n = ch.hi(c) - lo, xr = framed_resc_rows(a.fcl);
    int rows = 0;
    for (int i = 0; i < n && rows < xr; ++i) {
      const int l = OP == OP_BWD ? lo + n - 1 - i : lo + i;
      if (__ldg(a.fkinds + l) & KIND_RESCALE) resc[c * xr + rows++] = l;
    }
    if (rows < xr) resc[c * xr + rows] = -1;
  }
  for (int l = tid - kCodePad; l < a.L + kCodePad; l += blockDim.x) codes[l] = step_code<OP>(a.fkinds, a.L, l);
  for (int i = tid; i < (int)layer / 16; i += blockDim.x) sts16(sm.zero + (uint32_t)i * 16u, 0, 0);
  if (tid == 0) {
    for (int s = 0; s < kFrameStages; ++s) {
      mbar_init(sm.bars + 8u * s, 1);
      mbar_init(sm.bars + 8u * (kFrameStages + s), a.W);
    }
    sm.state[0] = sm.state[1] = 0;
    sm.scales[0] = kNoScale;
    sm.scales[1] = -kNoScale;
    fence_mbar_init();
  }
  __syncthreads();
  if constexpr (MIX) {
    // warps of four alternate between V and V - 1 vectors
    const int base = v0 + (warp >> 3) * R * 4 * (2 * V - 1), in = (warp & 3) * R + r;
    if (warp & 4) framed_body<OP, M, V - 1, GT>(a, sm, ch, base + R * 4 * V + in * (V - 1), 4);
    else framed_body<OP, M, V, GT>(a, sm, ch, base + in * V, 4);
  } else {
    framed_body<OP, M, V, GT>(a, sm, ch, v0 + (warp * R + r) * V, 0);
  }
}

template <int OP, int M, int V, int GT, bool MIX>
__global__ void __launch_bounds__(framed_max_threads(M, V), 1) framed_kernel(const FramedArgs a0) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int G = GT ? GT : a0.G, cap = framed_cta_vectors(a0.W, 32 / G, V, MIX);
  FramedArgs a = a0;
  a.v0 = blockIdx.x * cap;
  a.vend = min(a.B, a.v0 + cap);
  if (OP == OP_BWD) {
    a.partial = a0.partial + (size_t)blockIdx.x * a.L * ((G * M) >> 1);
    a.scales = a0.scales + blockIdx.x;
  }
  framed_run<OP, M, V, GT, MIX>(a, smem);
}

// dp[l][q][k] (= or +=) the sum over the nC per-CTA partials, each 2^scales[c] of its own size, times the frames' weights, in the CTAs' order (as
// dp_reduce_kernel, whose layout of threads it shares); a float2 holds gradient k of the crossings e and e + M/4
constexpr int kFReduceCols = 32, kFReduceRows = 8;
struct FramedReduceArgs {
  const float2* partial;
  int nC, L, np2, M, G, N;
  float* dp;
  int ldp, accumulate;
  const int* geo;
  const float2* wts;
  const int* count;
  int refuse;
  const int* scales;   // null: 0
};
// columns [2 kFReduceCols blk, ..), two a thread (16-byte loads: with 8-byte ones a batch's 134 MB took 82 us, 20 at the
// measured copy rate); the caller's threads meet before acc is used again
__device__ __forceinline__ void framed_reduce_block(const FramedReduceArgs& a, int blk, float4 (&acc)[kFReduceRows][kFReduceCols]) {
  constexpr int kCols = kFReduceCols, kRows = kFReduceRows;
  const int nC = a.nC, L = a.L, np2 = a.np2, M = a.M, G = a.G, N = a.N;
  const int* geo = a.geo;
  const int col = threadIdx.x % kCols, row = threadIdx.x / kCols;
  const int idx0 = 2 * (blk * kCols + col);
  const bool valid = idx0 < L * np2;
  const size_t stride = (size_t)L * np2 / 2;
  auto add = [](float4 x, float4 y) { return make_float4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w); };
  float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
  // t is at the least scale of the row's partials
  const bool framed = __ldg(a.count) < a.refuse;
  int scale = framed && a.scales ? kNoScale : 0, most = scale == 0 ? 0 : -kNoScale;
  if (scale != 0) {
    for (int c = row + kRows * (threadIdx.x & 31); c < nC; c += 32 * kRows) {
      const int s = __ldg(a.scales + c);
      scale = min(scale, s);
      most = max(most, s);
    }
    scale = __reduce_min_sync(0xffffffffu, scale);
    most = __reduce_max_sync(0xffffffffu, most);
  }
  auto times = [](float4 x, int k) {
    const float f = pow2f(max(k, -126));
    return make_float4(x.x * f, x.y * f, x.z * f, x.w * f);
  };
  __shared__ int row_scale[kRows];
  if (valid) {
    const float4* p = reinterpret_cast<const float4*>(a.partial) + idx0 / 2;
    int c = row;
    if (scale < most)   // (seldom)
      for (; c < nC; c += kRows) t = add(t, times(__ldg(p + (size_t)c * stride), scale - __ldg(a.scales + c)));
    for (; c + 3 * kRows < nC; c += 4 * kRows) {
      const float4 a0 = __ldg(p + (size_t)c * stride), a1 = __ldg(p + (size_t)(c + kRows) * stride);
      const float4 a2 = __ldg(p + (size_t)(c + 2 * kRows) * stride), a3 = __ldg(p + (size_t)(c + 3 * kRows) * stride);
      t = add(add(add(add(t, a0), a1), a2), a3);
    }
    for (; c < nC; c += kRows) t = add(t, __ldg(p + (size_t)c * stride));
  }
  acc[row][col] = t;
  if (col == 0) row_scale[row] = scale;
  __syncthreads();
  if (row != 0 || !valid) return;
  for (int k = 1; k < kRows; ++k) {
    const int s = row_scale[k], to = min(s, scale);
    if (s == scale) {
      t = add(t, acc[k][col]);
    } else {
      t = add(times(t, to - scale), times(acc[k][col], to - s));
      scale = to;
    }
  }
  if (scale == kNoScale) scale = 0;
  const int l = idx0 / np2, sh = geo[2 * l] / 2, ln = geo[2 * l + 1];
  auto put = [&](int q, int k, float v) {
    if (q >= N / 2) return;
    float* o = a.dp + (size_t)l * a.ldp + 2 * (size_t)q + k;
    v = q >= sh && q < sh + ln ? v : 0.f;
    *o = a.accumulate ? *o + v : v;
  };
  const int rem = idx0 - l * np2;
  if (!framed) {   // partials of the unframed body: (dJ/dth, dJ/dph) of one slot each
    const int q0 = pos_slot(rem, M, G), q1 = pos_slot(rem + 1, M, G);
    put(q0, 0, t.x);
    put(q0, 1, t.y);
    put(q1, 0, t.z);
    put(q1, 1, t.w);
    return;
  }
  // (th, th'), (ph, ph') of one pair of crossings
  const int pos = rem >> 1, j = pos % G, q = j * (M / 2) + pos / G;
  const float4 w = __ldg(reinterpret_cast<const float4*>(a.wts) + idx0 / 2);
  const int k0 = min(scale, 120), k1 = min(scale - k0, 120);   // (beyond 2^-240 nothing is left)
  const float s0 = pow2f(-k0), s1 = pow2f(-k1);
  put(q, 0, t.x * w.x * s0 * s1);
  put(q + M / 4, 0, t.y * w.y * s0 * s1);
  put(q, 1, t.z * w.z * s0 * s1);
  put(q + M / 4, 1, t.w * w.w * s0 * s1);
}

static __global__ void __launch_bounds__(256) framed_reduce_kernel(const FramedReduceArgs a) {
  __shared__ float4 acc[kFReduceRows][kFReduceCols];
  framed_reduce_block(a, blockIdx.x, acc);
}

}  // namespace mg
