// The frame pass: transfer matrices of nearest-neighbour meshes -> the unit-diagonal tiles of mg_framed.cuh.
//
// A 2x2 complex crossing costs 16 real FMAs per vector, a crossing with a unit diagonal 8.  Any diagonal can be
// pushed through a mesh: with a complex factor D_m(l) per mode and layer boundary ("frame", u = D u~), the layer
//   K = D(l+1)^-1 T D(l),   D_m(l+1) = t_mm D_m(l)  (t_mm: the mode's own diagonal entry in its slot)
// has K_aa = K_bb = 1, and only alpha = (t01 D_b)/(t00 D_a) and beta = (t10 D_a)/(t11 D_b) are left.  The same
// alpha and beta serve back-propagation: in the frames E = D^-H the reversed layer is K^H = [[1, beta*], [alpha*, 1]].
//
// |D| shrinks by |t_mm| per layer.  Frames start at 2^kFrameTop; behind a layer that took one below 2^kFrameDue they
// start again, the fields being multiplied by D 2^-kFrameTop (RESCALE: 4 FMAs per mode), put off by one layer where
// that leaves a pair of layers whole, unless one is below 2^kFrameNow.  A |t_mm| below 2^-30 (a cross state) counts as
// 2^-30: an entry's float32 rounding is worth up to 2^-25.  A row's scale does not change how its sum rounds, and T
// reaches this pass unrounded (float-float), so a framed layer rounds less than an unframed one (forward, N = 256,
// against complex128: 6.2e-7 and 7.3e-7).
//
// What bounds the pass: the serial chain of frames along the layers.  The layers are cut into segments of about
// kFrameSeg with a RESCALE behind each (3% more arithmetic in the forward kernel, for 16 times the parallelism of the
// chain).  A CTA does 32 to 160 modes of one segment (as
// many as keep the pass to one wave); where the frames start again is found from |t_mm|^2 of all
// modes by every CTA of the segment alike.  Frames and quotients are float-float (about 48 bits): GB300's FP64 pipe
// would take ten times as long for them.
#pragma once
#include "mg_framed_args.cuh"

namespace mg {

// float nearest (to about an ulp) to n / d for d > 0
__device__ __forceinline__ float ff_quot(ff n, ff d) {
  const float inv = __frcp_rn(d.h);
  const float q = n.h * inv;
  const float r = __fmaf_rn(-q, d.h, n.h) + __fmaf_rn(-q, d.l, n.l);
  return __fmaf_rn(r, inv, q);
}
// num / den (float2)
__device__ __forceinline__ float2 ffz_quot(ffz num, ffz den) {
  const ff s = ff_add(ff_mul(den.x, den.x), ff_mul(den.y, den.y));
  const ffz n = ffz_mul(num, ffz{den.x, ff_neg(den.y)});
  return make_float2(ff_quot(n.x, s), ff_quot(n.y, s));
}
__device__ __forceinline__ ffz ffz_of(float4 v) { return ffz{ff{v.x, v.y}, ff{v.z, v.w}}; }
__device__ __forceinline__ ffz ffz_scale2(ffz a, float s) {   // s a power of two
  return ffz{ff{s * a.x.h, s * a.x.l}, ff{s * a.y.h, s * a.y.l}};
}

// last layer of the segments before s (-1: none); an odd-shift one, where that is the next
__device__ __forceinline__ int frame_segment_end(const FrameArgs& a, int s) {
  if (s == 0) return -1;
  if (s == (int)gridDim.x) return a.L - 1;
  const int l = min(s * kFrameSeg - 1, a.L - 1);
  const int k0 = __ldg(a.kinds + l), k1 = __ldg(a.kinds + min(l + 1, a.L - 1));
  return k0 == 0 && k1 == KIND_MIS ? l + 1 : l;
}

template <int kRows>
__global__ void __launch_bounds__(kFrameThreads) frame_kernel(const FrameArgs a) {
  extern __shared__ __align__(16) unsigned char fsm[];
  static_assert(kFrameThreads == 32 * kFrameBatch, "a thread takes one row of each 32 modes");
  constexpr int kFrameModes = 32 * kRows, NB = kFrameModes + 2;
  const int np2 = a.G * a.M / 2, modes = 2 * np2, tid = threadIdx.x, M2 = a.M / 2;
  float4* fr = reinterpret_cast<float4*>(fsm);                                    // [kFrameBatch + 1][NB]: frames of modes m0 - 1 ..
  float* cur2 = reinterpret_cast<float*>(fr + (size_t)(kFrameBatch + 1) * NB);    // [modes]: |D|^2 at the batch's start
  float* mag = cur2 + modes;                                                      // [kFrameBatch][modes]: |t_mm|^2
  __shared__ int s_first;
  const int lo = frame_segment_end(a, blockIdx.x) + 1, hi = frame_segment_end(a, blockIdx.x + 1) + 1;
  if (lo >= hi) return;
  constexpr float top = 1ull << kFrameTop, inv = 1.f / top, top2 = top * top;
  constexpr float due2 = 1.f / (1ull << (-2 * kFrameDue)), now2 = 1.f / (1ull << (-2 * kFrameNow));
  const int m0 = blockIdx.y * kFrameModes;
  for (int m = tid; m < modes; m += blockDim.x) cur2[m] = top2;
  const ffz start = {ff{top, 0.f}, ff{0.f, 0.f}};
  ffz d = start;                                  // threads 0 .. NB-1: the frame of mode m0 - 1 + tid
  const int mc = m0 - 1 + tid;
  const bool chain = tid < NB && mc >= 0 && mc < modes;

  for (int base = lo; base < hi; base += kFrameBatch) {
    const int n = min(kFrameBatch, hi - base);
    // everything the batch reads from global memory is asked for at once
    float4 td[kFrameBatch], to[kRows];
    if (chain) {
#pragma unroll
      for (int i = 0; i < kFrameBatch; ++i)
        if (i < n) td[i] = __ldg(a.tdiag + (size_t)(base + i) * modes + mc);
    }
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
      const int idx = tid + k * kFrameThreads, i = idx / kFrameModes, m = m0 + idx % kFrameModes;
      if (i < n && m < modes) to[k] = __ldg(a.toff + (size_t)(base + i) * modes + m);
    }
    // bit i: layer base + i odd-shift
    const int lane = tid & 31;
    const unsigned mis = __ballot_sync(0xffffffffu, __ldg(a.kinds + min(base + lane, a.L - 1)) == KIND_MIS);
    float2 cs[kRows];
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
      const int idx = tid + k * kFrameThreads, i = idx / kFrameModes, m = m0 + idx % kFrameModes, sh = mis >> i & 1u;
      cs[k] = make_float2(0.f, 0.f);
      if (a.bwd && i < n && m >= sh && m < modes && ((m - sh) & 1) == 0) cs[k] = __ldg(a.tcs + (size_t)(base + i) * np2 + ((m - sh) >> 1));
    }
    bool nan = false;
    for (int idx = tid; idx < n * modes / 4; idx += blockDim.x) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(a.tmag + (size_t)base * modes) + idx);
      reinterpret_cast<float4*>(mag)[idx] = v;
      nan |= !(v.x + v.y + v.z + v.w >= 0.f);
    }
    if (blockIdx.y == 0 && nan) atomicOr(a.count, 1 << 30);
    // bit i: there is a layer behind layer base + i; no pair is broken up behind it; RESCALE
    const unsigned inner = a.L - 1 - base >= 32 ? 0xffffffffu : (1u << (a.L - 1 - base)) - 1u;
    const unsigned whole = mis | ~(mis >> 1);
    unsigned resc = base + n == hi && hi < a.L ? 1u << (n - 1) : 0u;   // a segment's end, unless it is the mesh's
    __syncthreads();
    // where the frames start again, first to last (each changes the frames behind it, so the search goes on from there)
    for (unsigned todo = (n < 32 ? (1u << n) - 1u : 0xffffffffu) & inner;;) {
      if (tid == 0) s_first = n;
      __syncthreads();
      int first = n;
      for (int m = tid; m < modes; m += blockDim.x) {
        float g[kFrameBatch], cur = cur2[m];
#pragma unroll
        for (int i = 0; i < kFrameBatch; ++i) g[i] = i < n ? mag[i * modes + m] : 1.f;
#pragma unroll
        for (int i = 0; i < kFrameBatch; ++i) {
          cur *= g[i];
          if ((todo & ~resc) >> i & 1u)
            if (!(cur >= (whole >> i & 1u ? due2 : now2))) first = min(first, i);
          if (resc >> i & 1u) cur = top2;
        }
      }
      if (first < n) atomicMin(&s_first, first);
      __syncthreads();
      const int f = s_first;
      __syncthreads();
      if (f >= n) break;
      resc |= 1u << f;
      todo &= ~((2u << f) - 1u);
    }
    if (base + n < hi)
      for (int m = tid; m < modes; m += blockDim.x) {
        float cur = cur2[m];
        for (int i = 0; i < n; ++i) cur = resc >> i & 1u ? top2 : cur * mag[i * modes + m];
        cur2[m] = cur;
      }
    // the frames behind every layer of the batch (before a RESCALE)
    if (chain) {
      fr[tid] = make_float4(d.x.h, d.x.l, d.y.h, d.y.l);
#pragma unroll
      for (int i = 0; i < kFrameBatch; ++i)
        if (i < n) {
          d = ffz_mul(d, ffz_of(td[i]));
          fr[(i + 1) * NB + tid] = make_float4(d.x.h, d.x.l, d.y.h, d.y.l);
          if (resc >> i & 1u) d = start;
        }
    }
    __syncthreads();
    // each mode's row of its slot
#pragma unroll
    for (int kr = 0; kr < kRows; ++kr) {
      const int idx = tid + kr * kFrameThreads;
      const int i = idx / kFrameModes, k = idx % kFrameModes, m = m0 + k, l = base + i, sh = mis >> i & 1u;
      if (i >= n || m >= modes) continue;
      const int q = (m - sh) >> 1, h = (m - sh) & 1, k2 = k + 1 - 2 * h;     // k2: the partner's place
      const bool fresh = i > 0 && (resc >> (i - 1) & 1u);
      auto before = [&](int at) { return fresh ? start : ffz_of(fr[i * NB + at + 1]); };
      auto behind = [&](int at) { return ffz_of(fr[(i + 1) * NB + at + 1]); };
      auto put = [&](float4* p, int c, float2 v) {
        reinterpret_cast<float*>(p)[c] = v.x;
        reinterpret_cast<float*>(p)[2 + c] = v.y;
      };
      const ffz after = behind(k);
      if (resc >> i & 1u) {
        const int jl = m / a.M, ml = m - jl * a.M, c = ml >= M2 ? 1 : 0;
        put(a.resc + (size_t)l * np2 + (size_t)(ml - c * M2) * a.G + jl, c, ffz_round(ffz_scale2(after, inv)));
      }
      if (m < sh) continue;
      const int j = q / M2, e = q - j * M2, c = e >= a.M / 4 ? 1 : 0, ep = e - c * (a.M / 4);
      const bool pair = m + 1 - 2 * h < modes;                                // the last odd-shift slot has one mode
      const size_t o16 = (size_t)l * (a.bwd ? 3 * np2 / 2 : np2) + (size_t)(2 * ep) * a.G + j;   // h = 0; h = 1 lies G further
      float2 kk = make_float2(0.f, 0.f);
      if (pair) kk = ffz_quot(ffz_mul(before(k2), ffz_of(to[kr])), after);
      else put(a.main + o16 + a.G, c, kk);   // its second row: nothing from outside reaches it
      put(a.main + o16 + h * a.G, c, kk);
      if (a.bwd && h == 0) {
        // m = (S(beta)^H y)_a = c E_a (y~_a + gamma y~_b), gamma = -i (s/c) conj(D_a / D_b) behind the layer
        const float2 ratio = ffz_quot(after, pair ? behind(k2) : start);
        const float t = cs[kr].x != 0.f ? cs[kr].y / cs[kr].x : 0.f;
        const ffz own = before(k);
        const size_t o8 = (size_t)l * (np2 / 2) + (size_t)ep * a.G + j;
        put(a.main + (size_t)l * (3 * np2 / 2) + np2 + (size_t)ep * a.G + j, c, make_float2(-t * ratio.y, -t * ratio.x));
        reinterpret_cast<float*>(a.wts + o8)[c] = cs[kr].x * cs[kr].x / (after.x.h * after.x.h + after.y.h * after.y.h);
        reinterpret_cast<float*>(a.wts + o8)[2 + c] = 1.f / (own.x.h * own.x.h + own.y.h * own.y.h);
      }
    }
    if (blockIdx.y == 0 && tid < n) {
      const unsigned b = 1u << tid;
      a.fkinds[base + tid] = (mis & b ? KIND_MIS : 0) | (resc & b ? KIND_RESCALE : 0);
      // a pair of layers is (aligned, odd-shift) without a RESCALE between
      const bool next_mis = mis & (b << 1);
      if ((inner & b) && (mis & b ? next_mis : !next_mis || (resc & b))) atomicAdd(a.count, 1);
    }
    if (base + n == a.L && chain && tid >= 1 && tid <= kFrameModes) a.dfin[mc] = ffz_round(d);
    __syncthreads();
  }
}

}  // namespace mg
