// Four-step z pass of the complex128 operator in float-float arithmetic
// (n3 = 16*NB): z-DFT, Green product and inverse z-DFT of W = TX*R contiguous
// elements of every (component, z) row, in shared memory.  Every complex value is
// held in packed FP32 pairs with (re, im) in the two lanes (ffpair.cuh).  The
// transform takes the three small steps of the x and y passes (xy4f.cuh) and the
// PWL product one thread per output group of a point, for the same reason:
// instruction latency and tasks that do not fill their last round are the cost.
// 96^3 PWL 4.21 -> 3.28 ms, the FMA pipe four fifths busy; 32^3 PWC 31 -> 26 us.
// Places: half h at h*C*W*S, sequence (c, e) at (c*W + e)*S in it, (klo, j) at
// klo*P4 + j in that; S and P4 put the lanes of a quarter-warp (e, then j or klo)
// on distinct 16-byte bank groups (kzf_stride).
#pragma once

#include "fastpath.cuh"
#include "ffpair.cuh"
#include "xy4f.cuh"

namespace marie {

// ---------------------------------------------------------------------------
// Float-float PWL multiply of one point for N / N^H: the four outputs of group P.
// Unrolled like zpoint, the 144 entries of a point are thousands of instructions
// in float-float and overflow the instruction cache, so the input group Q runs as
// a loop of three trips over a body holding the ten Tucker indices j unrolled:
// block (j, k) with k = PQ_N(P, Q) - 1, entries (l, lp) with |LLP(l, lp)| = j + 1
// (the same for every (P, Q) since PQ_N carries no sign).  The arithmetic runs in
// packed FP32 pairs with (re, im) in the two lanes; accumulators stay unnormalised
// (hi, lo) pairs until the end.
// ---------------------------------------------------------------------------
struct PwlPQ {
  int jl[4][4];          // Tucker index j of entry (l, lp)
  int sg[4][4];          // its sign
};

template <int OP>
constexpr PwlPQ make_pwl_pq() {
  using Tab = OpTab<true, OP>;
  PwlPQ t{};
  for (int i = 0; i < Tab::NE; ++i) {
    const OpEntry e = Tab::L.e[i];
    if (e.p < 4 && e.q < 4) {      // (P, Q) = (0, 0): block (j, 0)
      t.jl[e.p][e.q] = e.blk / 6;
      t.sg[e.p][e.q] = e.sgn;
    }
  }
  return t;
}

// acc += a*b per lane (NEG: acc -= a*b) on unnormalised float-float pairs:
// product error by FMA, sum error by two-sum, both collected in acc.lo.  na
// is -a; the error term is accumulated negated (p - a*b) so that every FMA
// adds, which gives the same values as the scalar form a*b - p.
template <bool NEG>
__device__ __forceinline__ void ff_acc2(ffc2& acc, const ffc2& a, const ffc2& na, const ffc2& b) {
  const ffc2& A = NEG ? na : a;
  const ffc2& NA = NEG ? a : na;
  const f2 p = A.hi * b.hi;
  f2 e = fma2(NA.hi, b.hi, p);
  e = fma2(NA.hi, b.lo, e);
  e = fma2(NA.lo, b.hi, e);
  const f2 s = acc.hi + p;
  const f2 bb = s - acc.hi;
  const f2 sl = (acc.hi - (s - bb)) + (p - bb);
  acc.hi = s;
  acc.lo = acc.lo + (sl - e);
}


// y += sgn * g * x for g = gr + i gi: lanes (re, im) += gr * (xr, xi) and
// (re, im) += (-gi, gi) * (xi, xr), in the order of the scalar form (the
// exchanged lanes (xi, xr) are formed at each use: keeping them costs 16
// registers and spills).
template <int OP>
__device__ __forceinline__ void zpoint_pwl_ff(ffc2* y, const ffc2* v, int qstride, const cplx<ff>* gp, int gstride,
                                              int P) {
  constexpr PwlPQ TB = make_pwl_pq<OP>();
  const f2 zero = f2_make(0.f, 0.f);
#pragma unroll
  for (int l = 0; l < 4; ++l) y[l] = ffc2{zero, zero};
#pragma unroll 1
  for (int Q = 0; Q < 3; ++Q) {
    ffc2 x[4];
#pragma unroll
    for (int lp = 0; lp < 4; ++lp) x[lp] = lds_ffc2(v + (4 * Q + lp) * qstride);
    const int k = P + Q + ((P > 0 && Q > 0) ? 1 : 0);    // PQ_N(P, Q) - 1
    const cplx<ff>* gk = gp + k * gstride;                // block (j, k) is 6j + k
#pragma unroll
    for (int j = 0; j < 10; ++j) {
      const float4 g = __ldg(reinterpret_cast<const float4*>(gk + 6 * j * gstride));   // (gr.hi, gr.lo, gi.hi, gi.lo)
      const ffc2 a1{f2_bc(g.x), f2_bc(g.y)};
      const ffc2 na1{zero - a1.hi, zero - a1.lo};
      ffc2 a2{f2_make(-g.z, g.z), f2_make(-g.w, g.w)};
      ffc2 na2{zero - a2.hi, zero - a2.lo};
      if constexpr ((OP & 1) != 0) {   // conj(g)
        const ffc2 t = a2;
        a2 = na2;
        na2 = t;
      }
#pragma unroll
      for (int l = 0; l < 4; ++l) {
#pragma unroll
        for (int lp = 0; lp < 4; ++lp) {
          if (TB.jl[l][lp] == j) {
            if (TB.sg[l][lp] > 0) {
              ff_acc2<false>(y[l], a1, na1, x[lp]);
              ff_acc2<false>(y[l], a2, na2, ffc2_swap(x[lp]));
            } else {
              ff_acc2<true>(y[l], a1, na1, x[lp]);
              ff_acc2<true>(y[l], a2, na2, ffc2_swap(x[lp]));
            }
          }
        }
      }
    }
  }
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    const f2 s = y[l].hi + y[l].lo;
    y[l] = ffc2{s, y[l].lo - (s - y[l].hi)};
  }
}

// PWC (C = 3): one entry of the 3 x 3 product, entries sorted by block.
template <int OP, int K>
struct ZPointFF {
  static __device__ __forceinline__ void run(ffc2* y, const ffc2* x, const ffc2* xs, ffc2& a1, ffc2& na1, ffc2& a2,
                                             ffc2& na2, const cplx<ff>* gp, int gstride) {
    using Tab = OpTab<false, OP>;
    constexpr int blk = Tab::L.e[K].blk;
    constexpr int p = Tab::L.e[K].p, q = Tab::L.e[K].q, sg = Tab::L.e[K].sgn;
    constexpr bool first = (K == 0) || (Tab::L.e[K == 0 ? 0 : K - 1].blk != blk);
    if constexpr (first) {
      const f2 zero = f2_make(0.f, 0.f);
      const float4 g = __ldg(reinterpret_cast<const float4*>(gp + blk * gstride));
      a1 = ffc2{f2_bc(g.x), f2_bc(g.y)};
      na1 = ffc2{zero - a1.hi, zero - a1.lo};
      a2 = ffc2{f2_make(-g.z, g.z), f2_make(-g.w, g.w)};
      na2 = ffc2{zero - a2.hi, zero - a2.lo};
      if constexpr ((OP & 1) != 0) {
        const ffc2 t = a2;
        a2 = na2;
        na2 = t;
      }
    }
    ff_acc2<(sg < 0)>(y[p], a1, na1, x[q]);
    ff_acc2<(sg < 0)>(y[p], a2, na2, xs[q]);
  }
};

template <int OP, int... Ks>
__device__ __forceinline__ void zpoint_pwc_ff(std::integer_sequence<int, Ks...>, ffc2* v, int qstride,
                                              const cplx<ff>* gp, int gstride) {
  const f2 zero = f2_make(0.f, 0.f);
  ffc2 x[3], xs[3], y[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    x[q] = lds_ffc2(v + q * qstride);
    xs[q] = ffc2_swap(x[q]);
    y[q] = ffc2{zero, zero};
  }
  ffc2 a1, na1, a2, na2;
  (ZPointFF<OP, Ks>::run(y, x, xs, a1, na1, a2, na2, gp, gstride), ...);
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    const f2 s = y[p].hi + y[p].lo;
    sts_ffc2(v + p * qstride, ffc2{s, y[p].lo - (s - y[p].hi)});
  }
}

// 384 threads: at n3 = 96 PWL the tasks of every phase are 1.5, 2 or 3 times as many.
constexpr int kZfThreads = 384;

template <int NB, bool PWL, int OP>
__global__ void __launch_bounds__(kZfThreads, 2) k4_zf(MvArgs<ff> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int N = 16 * NB, J = 4 * NB;
  constexpr int C = PWL ? 12 : 3;
  constexpr int NE = OpTab<PWL, OP>::NE;
  const int bu = blockIdx.x;
  if (!bundle_active(a, bu)) return;
  // blockIdx.z walks y in slot order: mirrored ky run back to back
  const int n1 = a.n1, n2 = a.n2, g3 = a.g3, m1 = 2 * n1, R = a.R;
  const int k0 = blockIdx.y * a.TX;
  bool my;
  const int kyo = slot_octant(blockIdx.z, n2, my);
  const int ky = my ? 2 * n2 - kyo : kyo;
  const int kyp = (ky & 1) * n2 + (ky >> 1);
  const int W = a.TX * R;                       // a power of two; TX divides 2*n1
  const int lgW = 31 - __clz(W);
  const int S = kzf_stride(N, W), P4 = J + kzf_pad(W);
  const int H = C * W * S;                      // start of the odd half
  ulonglong2* tw = reinterpret_cast<ulonglong2*>(smem_raw);
  ffc2* buf = reinterpret_cast<ffc2*>(tw + 2 * xyf_tw(N));
  load_twx<NB>(tw, a.az.tw2);
  __syncthreads();
  const int64_t row = (int64_t)m1 * R;
  const int64_t cstride = (int64_t)2 * n2 * g3 * row;
  cplx<ff>* base = a.S + (int64_t)bu * C * cstride + (int64_t)kyp * g3 * row + (int64_t)k0 * R;
  // x frequency of element e, and its components' sign changes where a
  // frequency is mirrored (mirror_mask)
  auto kx_of = [&](int e) {
    const int kxp = k0 + (e >> a.lgR), alpha = kxp >= n1 ? 1 : 0;
    return 2 * (kxp - alpha * n1) + alpha;
  };
  auto flip_of = [&](int e, int c) { return (mirror_flips<PWL>(kx_of(e) > n1, my) >> c) << 31; };
  // live bit of slice z = j + J*q, q < 4, at bit 4q
  auto live_of = [&](int j) {
    const int b = j % NB;
    return (a.zq ? (unsigned)a.zq[b] : inside_bits(g3, NB, b)) >> (j / NB);
  };

  for (int t = threadIdx.x; t < W * J * C; t += kZfThreads) {   // task (e, j, c), e fastest
    const int e = t & (W - 1), r = t >> lgW;
    const int j = r % J, c = r / J;
    const unsigned live = live_of(j), flip = flip_of(e, c);
    const cplx<ff>* src = base + c * cstride + (int64_t)j * row + e;
    ffc2 v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      v[q] = to_ffc2(flip_c((live >> (4 * q)) & 1u ? src[(int64_t)(J * q) * row] : cplx<ff>{ff(0), ff(0)}, flip));
    xyf_split<NB>(v, buf + (c * W + e) * S, H, P4, j, tw);
  }
  __syncthreads();
  xyf_mid<false, NB>(buf, lgW, 2 * C, S, P4, tw, [](int) { return true; });
  __syncthreads();
  // task (e, k1, s), e fastest; NB-point DFT in place: frequency k1 + 16*k3
  for (int t = threadIdx.x; t < 2 * C * W * 16; t += kZfThreads) {
    const int e = t & (W - 1), r = t >> lgW;
    const int k1 = r & 15, s = r >> 4;
    ffc2* p = buf + (s * W + e) * S + (k1 & 3) * P4 + (k1 >> 2) * NB;
    ffc2 w[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) w[b] = lds_ffc2(p + b);
    dftf<false, NB>(w);
#pragma unroll
    for (int k3 = 0; k3 < NB; ++k3) sts_ffc2(p + k3, w[k3]);
  }
  __syncthreads();

  // Green block multiply: point (e, kz = 2k + g); block blk of it is in the
  // spectrum at ((kyo*(n1+1) + kxo)*U + blk)*2N + g*N + k (octant columns; with
  // the blocks of a point side by side the lanes of a load meet 32 lines and the pass
  // takes 3.82 ms at 96^3 instead of 3.37).  PWL: one thread per output group P of a point, each reading the
  // twelve inputs where they are; the outputs go back when all have read.
  constexpr int U = OpTab<PWL, OP>::L.nblk;
  constexpr int kPoints = PWL ? kZfThreads / 3 : kZfThreads;   // per round
  for (int i0 = 0; i0 < 2 * N * W; i0 += kPoints) {
    const int P = threadIdx.x / kPoints;
    const int i = i0 + threadIdx.x - P * kPoints;
    const bool act = i < 2 * N * W;
    const int e = i & (W - 1), pp = i >> lgW;
    const int g = pp / N, k = pp - g * N;
    const int kx = kx_of(e), kxo = kx > n1 ? 2 * n1 - kx : kx;
    const cplx<ff>* gp = a.G + ((int64_t)kyo * (n1 + 1) + kxo) * (2 * N * U) + pp;
    ffc2* v = buf + g * H + e * S + (k & 3) * P4 + ((k >> 2) & 3) * NB + (k >> 4);
    if constexpr (PWL) {
      ffc2 y[4];
      if (act) zpoint_pwl_ff<OP>(y, v, W * S, gp, 2 * N, P);
      __syncthreads();
      if (act) {
#pragma unroll
        for (int l = 0; l < 4; ++l) sts_ffc2(v + (4 * P + l) * W * S, y[l]);
      }
    } else if (act) {
      zpoint_pwc_ff<OP>(std::make_integer_sequence<int, NE>{}, v, W * S, gp, 2 * N);
    }
  }
  __syncthreads();
  // the same steps back
  for (int t = threadIdx.x; t < 2 * C * W * 16; t += kZfThreads) {
    const int e = t & (W - 1), r = t >> lgW;
    const int k1 = r & 15, s = r >> 4;
    ffc2* p = buf + (s * W + e) * S + (k1 & 3) * P4 + (k1 >> 2) * NB;
    ffc2 w[NB];
#pragma unroll
    for (int k3 = 0; k3 < NB; ++k3) w[k3] = lds_ffc2(p + k3);
    dftf<true, NB>(w);
#pragma unroll
    for (int b = 0; b < NB; ++b) sts_ffc2(p + b, w[b]);
  }
  __syncthreads();
  xyf_mid<true, NB>(buf, lgW, 2 * C, S, P4, tw, [](int) { return true; });
  __syncthreads();
  for (int t = threadIdx.x; t < W * J * C; t += kZfThreads) {
    const int e = t & (W - 1), r = t >> lgW;
    const int j = r % J, c = r / J;
    const unsigned live = live_of(j), flip = flip_of(e, c);
    if (!(live & 0x1111u)) continue;
    ffc2 v[4];
    xyf_join<NB>(v, buf + (c * W + e) * S, H, P4, j, tw);
    cplx<ff>* dst = base + c * cstride + (int64_t)j * row + e;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if ((live >> (4 * q)) & 1u) dst[(int64_t)(J * q) * row] = flip_c(from_ffc2(v[q]), flip);
  }
}

}  // namespace marie
