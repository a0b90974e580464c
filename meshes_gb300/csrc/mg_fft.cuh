// Butterfly (FFT) meshes of 2^k modes over large batches: forward, and back-propagation with direct MZI gradients.
//
// A layer crosses the modes n and n + 2^e.  With M modes per lane and G <= M lanes to a vector (N = M G) every layer is
// within a lane in one of two orders: lane j holds the modes j M .. j M + M - 1 (rows: strides below M) or the modes j, j + G,
// j + 2 G .. (columns: strides of G and above).  So the walk turns the fields from one order to the other, through shared
// memory, where the next layer asks for it - once in the layers 0 .. k - 1 - instead of exchanging them between lanes by
// shuffles in every layer beyond the lane.  Fields come and leave in columns.
//
// The launch's tiles are the one-mesh kernel's (mg_prop.cuh); a CTA lays them out by slots of its own lanes in shared memory
// once, for all of its vectors, and its warps go through batches of 32 / G x V vectors on their own.  Every field is computed
// by the same operations as there.
//
// What bounds it: nothing alone - shared-memory wavefronts (coefficients, the turns: 52% forward), the packed FMAs (32%) and
// the latency between them at two (back-propagation) to four warps per scheduler.  Measured on GB300 at N = 256, B = 20000
// against the general kernel: forward 52 -> 34 us, back-propagation 124 -> 86 us, its reduction 9.5 -> 4 us (152 sets of
// partials instead of 625).
#pragma once
#include "mg_fft_args.cuh"
#include "mg_framed.cuh"

namespace mg {

// order of a layer's fields and log2 of its stride in places of that order
constexpr int FFT_COLUMNS = 16;
template <int M, int G>
__host__ __device__ __forceinline__ int fft_code(int e) {
  return (2 << e) <= M ? e : FFT_COLUMNS | (e - (G == 32 ? 5 : G == 16 ? 4 : G == 8 ? 3 : 2));
}

// u(place) from one order to the other: 16 bytes a place, a gap after every M
template <int M, int G, bool TO_COLUMNS>
__device__ __forceinline__ void fft_turn(P2 (&u)[M], uint32_t buf, int j) {
  auto rows = [&](int i) { return buf + (uint32_t)(j * (M + 1) + i) * 16u; };
  auto columns = [&](int i) {
    const int n = j + G * i;
    return buf + (uint32_t)(n + n / M) * 16u;
  };
  __syncwarp();
#pragma unroll
  for (int i = 0; i < M; ++i) sts16(TO_COLUMNS ? rows(i) : columns(i), u[i].r, u[i].i);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < M; ++i) {
    const ulonglong2 v = lds16(TO_COLUMNS ? columns(i) : rows(i));
    u[i] = P2{v.x, v.y};
  }
}

// y = c1 b + c0 a, and conj(c1) b + conj(c0) a
__device__ __forceinline__ P2 fft_lin(const PK& c0, const PK& c1, const P2& a, const P2& b) {
  return P2{pfma(c1.r, b.r, pfma(c1.n, b.i, pfma(c0.r, a.r, pmul(c0.n, a.i)))),
            pfma(c1.r, b.i, pfma(c1.i, b.r, pfma(c0.r, a.i, pmul(c0.i, a.r))))};
}
__device__ __forceinline__ P2 fft_clin(const PK& c0, const PK& c1, const P2& a, const P2& b) {
  return P2{pfma(c1.r, b.r, pfma(c1.i, b.i, pfma(c0.r, a.r, pmul(c0.i, a.i)))),
            pfma(c1.r, b.i, pfma(c1.n, b.r, pfma(c0.r, a.i, pmul(c0.n, a.r))))};
}

// One layer, its pairs 2^LOG places apart.  t: the lane's T rows, cs: its splitter pairs, acc: its gradient sums
template <int OP, int M, int G, int LOG>
__device__ __forceinline__ void fft_layer(uint32_t t, uint32_t cs, uint32_t acc, int r, P2 (&u)[M], P2 (&w)[OP == OP_BWD ? M : 1]) {
  constexpr int st = 1 << LOG;
#pragma unroll
  for (int s = 0; s < M / 2; ++s) {
    const int a = 2 * st * (s / st) + s % st, b = a + st;
    const ulonglong2 q0 = lds16(t + (uint32_t)(2 * s * G) * 16u), q1 = lds16(t + (uint32_t)((2 * s + 1) * G) * 16u);
    const float2 c00 = p_split(q0.x), c01 = p_split(q0.y), c10 = p_split(q1.x), c11 = p_split(q1.y);
    const PK t00 = pk_dup(c00.x, c00.y), t01 = pk_dup(c01.x, c01.y), t10 = pk_dup(c10.x, c10.y), t11 = pk_dup(c11.x, c11.y);
    const P2 ua = u[a], ub = u[b];
    if constexpr (OP == OP_FWD) {
      u[a] = fft_lin(t00, t01, ua, ub);
      u[b] = fft_lin(t10, t11, ua, ub);
    } else {
      const float2 k = p_split(lds8(cs + (uint32_t)(s * G) * 8u));
      const p64 c = p_pack(k.x, k.x), sn = p_pack(k.y, k.y), ns = pneg(sn), nc = pneg(c);
      const P2 ga = w[a], gb = w[b];
      const p64 m0x = pfma(c, ua.r, pmul(sn, ub.i)), m0y = pfma(c, ua.i, pmul(ns, ub.r));
      const p64 nh0x = pfma(nc, ga.r, pmul(ns, gb.i)), h0y = pfma(c, ga.i, pmul(ns, gb.r));
      const float2 th = p_split(pfma(h0y, m0x, pmul(nh0x, m0y)));
      u[a] = fft_clin(t00, t10, ua, ub);
      u[b] = fft_clin(t01, t11, ua, ub);
      w[a] = fft_clin(t00, t10, ga, gb);
      w[b] = fft_clin(t01, t11, ga, gb);
      const float2 ph = p_split(psub(pmul(w[a].i, u[a].r), pmul(w[a].r, u[a].i)));
      float ath = th.x + th.y, aph = ph.x + ph.y;
#pragma unroll
      for (int off = G; off < 32; off <<= 1) {
        ath += __shfl_xor_sync(0xffffffffu, ath, off, 32);
        aph += __shfl_xor_sync(0xffffffffu, aph, off, 32);
      }
      if (r == 0) {
        const uint32_t p = acc + (uint32_t)(s * G) * 8u;
        const float2 v = p_split(lds8(p));
        asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(p), "f"(v.x + ath), "f"(v.y + aph) : "memory");
      }
    }
  }
}
template <int OP, int M, int G>
__device__ __forceinline__ void fft_step(int log, uint32_t t, uint32_t cs, uint32_t acc, int r, P2 (&u)[M],
                                         P2 (&w)[OP == OP_BWD ? M : 1]) {
  switch (log) {
    case 0: fft_layer<OP, M, G, 0>(t, cs, acc, r, u, w); break;
    case 1: fft_layer<OP, M, G, 1>(t, cs, acc, r, u, w); break;
    case 2: fft_layer<OP, M, G, 2>(t, cs, acc, r, u, w); break;
    case 3: if constexpr (M > 8) { fft_layer<OP, M, G, 3>(t, cs, acc, r, u, w); } break;
    default: if constexpr (M > 16) { fft_layer<OP, M, G, 4>(t, cs, acc, r, u, w); } break;
  }
}

// two vectors from vb0 on, in columns (G lanes side by side; in rows every lane's access is a line of its own); those from
// vend on read 0
template <int M, int G>
__device__ __forceinline__ void fft_load(P2 (&u)[M], const void* src, int vb0, int vend, int ldu, int j) {
  const float2* p0 = static_cast<const float2*>(src) + (size_t)vb0 * ldu + j;
  const float2* p1 = p0 + ldu;
  const bool in0 = vb0 < vend, in1 = vb0 + 1 < vend;
  const float2 z = make_float2(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < M; ++i) {
    const float2 x = in0 ? p0[G * i] : z, y = in1 ? p1[G * i] : z;
    u[i] = P2{p_pack(x.x, y.x), p_pack(x.y, y.y)};
  }
}
template <int M, int G>
__device__ __forceinline__ void fft_store(const P2 (&u)[M], void* dst, int vb0, int vend, int ldu, int j) {
  float2* p0 = static_cast<float2*>(dst) + (size_t)vb0 * ldu + j;
  float2* p1 = p0 + ldu;
  const bool in0 = vb0 < vend, in1 = vb0 + 1 < vend;
#pragma unroll
  for (int i = 0; i < M; ++i) {
    const float2 re = p_split(u[i].r), im = p_split(u[i].i);
    if (in0) p0[G * i] = make_float2(re.x, im.x);
    if (in1) p1[G * i] = make_float2(re.y, im.y);
  }
}

template <int OP, int M, int G>
__global__ void __launch_bounds__(kFftThreads, fft_ctas_per_sm(OP, M)) fft_kernel(const FftArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int N = M * G, np2 = N / 2, R = 32 / G, V = kFftVectors, W = kFftThreads / 32;
  const FftLayout lay = fft_layout(OP, M, G, a.L);
  const uint32_t base = smem_u32(smem);
  int* codes = reinterpret_cast<int*>(smem + lay.codes);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, j = lane % G, r = lane / G;

  for (int l = tid; l < a.L; l += kFftThreads) codes[l] = __ldg(a.kinds + l);
  __syncthreads();
  // the tiles, by slots of this kernel's lanes
#pragma unroll 4
  for (int idx = tid; idx < a.L * np2; idx += kFftThreads) {
    const int l = idx / np2, q = idx - l * np2;
    const int kind = codes[l];
    const bool xl = kind >= KIND_XL;
    const int e = xl ? kind - KIND_XL : kind, code = fft_code<M, G>(e), st = 1 << e;
    const int n = 2 * st * (q / st) + (q & (st - 1));   // first mode of slot q
    const float4* tl = reinterpret_cast<const float4*>(a.tiles + (size_t)l * a.layer_bytes);
    const float2* ct = reinterpret_cast<const float2*>(tl + a.M * a.G);
    float4 row0, row1;
    float2 cs = make_float2(0.f, 0.f);
    if (!xl) {
      const int jt = q / (a.M / 2), s = q % (a.M / 2);
      row0 = __ldg(tl + (2 * s) * a.G + jt);
      row1 = __ldg(tl + (2 * s + 1) * a.G + jt);
      if (OP == OP_BWD) cs = __ldg(ct + s * a.G + jt);
    } else {
      const int m = n + st;
      const float4 ra = __ldg(tl + (n % a.M) * a.G + n / a.M), rb = __ldg(tl + (m % a.M) * a.G + m / a.M);
      if (OP == OP_BWD) {   // rows of T^H: (conj t00, conj t10), (conj t11, conj t01)
        row0 = make_float4(ra.x, -ra.y, rb.z, -rb.w);
        row1 = make_float4(ra.z, -ra.w, rb.x, -rb.y);
        cs = __ldg(ct + (n % a.M) * (a.G / 2) + a_lane_index(n / a.M, st / a.M));
      } else {              // rows of T: (t00, t01), (t11, t10)
        row0 = ra;
        row1 = make_float4(rb.z, rb.w, rb.x, rb.y);
      }
    }
    const bool columns = code & FFT_COLUMNS;
    const int jn = columns ? n % G : n / M, i = columns ? n / G : n % M, ls = code & 15;
    const int s = ((i >> (ls + 1)) << ls) | (i & ((1 << ls) - 1));
    float4* t = reinterpret_cast<float4*>(smem + lay.tiles) + (size_t)l * N;
    t[(2 * s) * G + jn] = row0;
    t[(2 * s + 1) * G + jn] = row1;
    if (OP == OP_BWD) reinterpret_cast<float2*>(smem + lay.cs)[(size_t)l * np2 + s * G + jn] = cs;
  }
  __syncthreads();
  for (int l = tid; l < a.L; l += kFftThreads) {
    const int kind = codes[l];
    codes[l] = fft_code<M, G>(kind >= KIND_XL ? kind - KIND_XL : kind);
  }
  if (OP == OP_BWD)
    for (int i = tid; i < W * a.L * np2; i += kFftThreads) reinterpret_cast<float2*>(smem + lay.acc)[i] = make_float2(0.f, 0.f);
  __syncthreads();

  const uint32_t turn = base + lay.turn + (uint32_t)(warp * R + r) * (N + G) * 16u;
  const uint32_t t0 = base + lay.tiles + (uint32_t)j * 16u, cs0 = base + lay.cs + (uint32_t)j * 8u;
  const uint32_t acc0 = base + lay.acc + (uint32_t)(warp * a.L * np2 + j) * 8u;
  const int batches = (a.B + R * V - 1) / (R * V);
#pragma unroll 1
  for (int b = blockIdx.x + gridDim.x * warp; b < batches; b += gridDim.x * W) {
    const int vb0 = (b * R + r) * V;
    P2 u[M], w[OP == OP_BWD ? M : 1];
    bool columns = true;
    fft_load<M, G>(u, a.in0, vb0, a.B, a.ldu, j);
    if constexpr (OP == OP_BWD) {
      fft_load<M, G>(w, a.target ? a.target : a.in1, vb0, a.B, a.ldu, j);
      if (a.target) {   // fused L2 loss to a target: g = 2 (y - t)
        const p64 two = p_pack(2.f, 2.f);
#pragma unroll
        for (int i = 0; i < M; ++i) w[i] = P2{pmul(two, psub(u[i].r, w[i].r)), pmul(two, psub(u[i].i, w[i].i))};
      }
    }
#pragma unroll 1
    for (int i = 0; i <= a.L; ++i) {
      const int l = OP == OP_BWD ? a.L - 1 - i : i;
      const int code = i < a.L ? codes[l] : FFT_COLUMNS;
      if (((code & FFT_COLUMNS) != 0) != columns) {
        if (columns) {
          fft_turn<M, G, false>(u, turn, j);
          if constexpr (OP == OP_BWD) fft_turn<M, G, false>(w, turn, j);
        } else {
          fft_turn<M, G, true>(u, turn, j);
          if constexpr (OP == OP_BWD) fft_turn<M, G, true>(w, turn, j);
        }
        columns = !columns;
      }
      if (i == a.L) break;
      fft_step<OP, M, G>(code & 15, t0 + (uint32_t)l * N * 16u, cs0 + (uint32_t)l * np2 * 8u, acc0 + (uint32_t)l * np2 * 8u, r, u,
                         w);
    }
    if (a.out0) fft_store<M, G>(u, a.out0, vb0, a.B, a.ldu, j);
    if constexpr (OP == OP_BWD) fft_store<M, G>(w, a.out1, vb0, a.B, a.ldu, j);
  }
  if constexpr (OP == OP_BWD) {
    __syncthreads();
    for (int idx = tid; idx < a.L * np2; idx += kFftThreads) {
      const int l = idx / np2, q = idx - l * np2, code = codes[l], ls = code & 15;
      const bool columns = code & FFT_COLUMNS;
      const int st = (1 << ls) * (columns ? G : 1);
      const int n = 2 * st * (q / st) + q % st, jn = columns ? n % G : n / M, i = columns ? n / G : n % M;
      const int s = ((i >> (ls + 1)) << ls) | (i & ((1 << ls) - 1));
      float2 sum = make_float2(0.f, 0.f);
      for (int k = 0; k < W; ++k)
        sum = cadd(sum, reinterpret_cast<const float2*>(smem + lay.acc)[((size_t)k * a.L + l) * np2 + s * G + jn]);
      a.partial[((size_t)blockIdx.x * a.L + l) * np2 + slot_pos(q, a.M, a.G)] = sum;
    }
  }
}

}  // namespace mg
