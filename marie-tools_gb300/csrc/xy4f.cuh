// Float-float x and y passes of the four-step grids (edges n = 16*NB).
//
// A float-float addition is eleven dependent FP32 instructions, so these passes
// are bound by instruction latency, not by memory: what they need is many threads
// with little code each.  A line of n = 4*J points (J = 4*NB, point j + J*q) goes
// through three steps in place in shared memory, one task per small DFT:
//   1 (per j): the four values of a point set to the eight frequencies m = f mod 8
//     of the zero-padded length-2n transform, times w_2n^(j*m).  Even m are half
//     alpha = 0, odd m half alpha = 1; the padding costs no arithmetic.
//   2 (per half, klo = m/2, b): DFT4 over a of j = NB*a + b, times w_J^(b*khi)
//   3 (per half, klo, khi): DFT of NB points over b -> frequency klo + 4*khi + 16*k3
// (inverse: the same steps backwards, conjugated, keeping the first n points).
// Element e of W has its half alpha in sequence alpha*W + e, (klo, j) at place
// klo*P4 + j of it, P4 = J + 1; the sequences' stride 16*NB + 5 is odd, so lanes on
// neighbouring ones meet distinct bank groups.  Against one thread per 16-point DFT
// and both halves, X / Y / YI / XI: 96^3 PWL, one right-hand side, 0.427 / 0.602 /
// 0.572 / 0.608 -> 0.18 / 0.42 / 0.40 / 0.22 ms (the FP32 work alone 0.16 to 0.32);
// 32^3 PWC 32 / 18 / 13 / 32 -> 12 / 11 / 10 / 13 us.
#pragma once

#include "fastpath.cuh"
#include "ffpair.cuh"
#include "matvec.cuh"

namespace marie {

// Twiddles as the tasks read them, neighbouring lanes neighbouring entries:
// w_2n^(j*m) at (m - 1)*J + j, m in [1, 8), then w_J^(b*khi) at 7*J + (khi - 1)*NB + b;
// high parts, then the negated low parts.
template <int NB>
__device__ __forceinline__ void load_twx(ulonglong2* tw, const cplx<ff>* tw2) {
  constexpr int N = 16 * NB, J = 4 * NB, E = xyf_tw(N);
  const f2 zero = f2_make(0.f, 0.f);
  for (int i = threadIdx.x; i < E; i += blockDim.x) {
    const int r = i - 7 * J, k = r < 0 ? (i % J) * (i / J + 1) : 8 * (r % NB) * (r / NB + 1);
    cplx<ff> w = tw2[k < N ? k : k - N];
    if (k >= N) w = {-w.x, -w.y};
    const fftw t = fftw_make(w);
    tw[i] = make_ulonglong2(t.rh.v, t.ih.v);
    tw[E + i] = make_ulonglong2((zero - t.rl).v, (zero - t.il).v);
  }
}

// v times table entry i (INV: its conjugate)
template <bool INV, int NB>
__device__ __forceinline__ ffc2 tw_mulx(ffc2 v, const ulonglong2* tw, int i) {
  const ulonglong2 h = tw[i], l = tw[xyf_tw(16 * NB) + i];
  const f2 zero = f2_make(0.f, 0.f), rh{h.x}, ih{h.y}, nih = zero - ih, nrl{l.x}, nil{l.y};
  const f2 nrh = zero - rh, kh = INV ? nih : ih, nkh = INV ? ih : nih, nkl = INV ? zero - nil : nil;
  const ffc2 w = ffc2_swap(v);
  const f2 a = v.hi * rh, b = w.hi * kh;
  f2 e = fma2(v.hi, nrh, a), g = fma2(w.hi, nkh, b);
  e = fma2(v.lo, nrh, fma2(v.hi, nrl, e));
  g = fma2(w.lo, nkh, fma2(w.hi, nkl, g));
  return sum2(a, e, b, g);
}

// DFT of (v0 .. v3, 0, 0, 0, 0): frequencies 2k in e[k], 2k + 1 in o[k]
__device__ __forceinline__ void pad8(const ffc2* v, ffc2* e, ffc2* o) {
  const double h = 0.707106781186547524401;
  e[0] = v[0], e[1] = v[1], e[2] = v[2], e[3] = v[3];
  o[0] = v[0];
  o[1] = rotf<false>(v[1], h, h);
  o[2] = mul_w<false>(v[2]);
  o[3] = rotf<false>(v[3], -h, h);
  dftf4<false>(e);
  dftf4<false>(o);
}
// the first four values of the inverse
__device__ __forceinline__ void crop8(ffc2* e, ffc2* o) {
  const double h = 0.707106781186547524401;
  dftf4<true>(e);
  dftf4<true>(o);
  e[0] = e[0] + o[0];
  e[1] = e[1] + rotf<true>(o[1], h, h);
  e[2] = e[2] + mul_w<true>(o[2]);
  e[3] = e[3] + rotf<true>(o[3], -h, h);
}

// step 1 of one point set j of element p (its halves H apart), v[q] its values
template <int NB>
__device__ __forceinline__ void xyf_split(const ffc2* v, ffc2* p, int H, int P4, int j, const ulonglong2* tw) {
  constexpr int J = 4 * NB;
  ffc2 e[4], o[4];
  pad8(v, e, o);
  p += j;
  sts_ffc2(p, e[0]);
#pragma unroll
  for (int k = 1; k < 4; ++k) sts_ffc2(p + k * P4, tw_mulx<false, NB>(e[k], tw, (2 * k - 1) * J + j));
#pragma unroll
  for (int k = 0; k < 4; ++k) sts_ffc2(p + H + k * P4, tw_mulx<false, NB>(o[k], tw, 2 * k * J + j));
}
// its inverse: v[q] the values of point set j
template <int NB>
__device__ __forceinline__ void xyf_join(ffc2* v, const ffc2* p, int H, int P4, int j, const ulonglong2* tw) {
  constexpr int J = 4 * NB;
  ffc2 o[4];
  p += j;
  v[0] = lds_ffc2(p);
#pragma unroll
  for (int k = 1; k < 4; ++k) v[k] = tw_mulx<true, NB>(lds_ffc2(p + k * P4), tw, (2 * k - 1) * J + j);
#pragma unroll
  for (int k = 0; k < 4; ++k) o[k] = tw_mulx<true, NB>(lds_ffc2(p + H + k * P4), tw, 2 * k * J + j);
  crop8(v, o);
}

// step 2 of n groups of 2^lgE sequences, the group's elements fastest; live(e): wanted
template <bool INV, int NB, typename Live>
__device__ __forceinline__ void xyf_mid(ffc2* buf, int lgE, int n, int S, int P4, const ulonglong2* tw, Live live) {
  constexpr int J = 4 * NB;
  for (int t = threadIdx.x; t < (n * J) << lgE; t += blockDim.x) {
    const int e = t & ((1 << lgE) - 1), r = t >> lgE;
    if (!live(e)) continue;
    const int i = r % J, b = i % NB;
    ffc2* p = buf + (((r / J) << lgE) + e) * S + (i / NB) * P4 + b;
    ffc2 w[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) w[a] = lds_ffc2(p + NB * a);
    if (INV && NB > 1) {
#pragma unroll
      for (int k = 1; k < 4; ++k) w[k] = tw_mulx<true, NB>(w[k], tw, 7 * J + (k - 1) * NB + b);
    }
    dftf4<INV>(w);
#pragma unroll
    for (int k = 0; k < 4; ++k) sts_ffc2(p + NB * k, !INV && NB > 1 && k ? tw_mulx<false, NB>(w[k], tw, 7 * J + (k - 1) * NB + b) : w[k]);
  }
}

// ---------------------------------------------------------------------------
// Pass X (forward).  grid (ceil(g2/TY), g3, nbundle*C); element yy*R + r
// ---------------------------------------------------------------------------
template <int NB>
__global__ void __launch_bounds__(256, 3) k4f_fwd_x(MvArgs<ff> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int N = 16 * NB, J = 4 * NB, S = xyf_stride(N), P4 = J + 1;
  const int bc = blockIdx.z, bu = bc / a.C, c = bc - bu * a.C;
  if (!bundle_active(a, bu)) return;
  const int z = blockIdx.y, y0 = blockIdx.x * a.TY;
  const int g1 = a.g1, g2 = a.g2, g3 = a.g3, R = a.R, lgR = a.lgR;
  const int ty = min(a.TY, g2 - y0), W = a.TY * R;
  unsigned rows = 0;   // live rows of the tile
  for (int yy = 0; yy < ty; ++yy) rows |= row_is_live(a, y0 + yy, z) ? 1u << yy : 0u;
  if (!rows) return;   // rows without body voxels stay unwritten: the y pass reads them as zero
  ulonglong2* tw = reinterpret_cast<ulonglong2*>(smem_raw);
  ffc2* buf = reinterpret_cast<ffc2*>(tw + 2 * xyf_tw(N));
  load_twx<NB>(tw, a.ax.tw2);
  __syncthreads();
  const int64_t nD = (int64_t)g1 * g2 * g3;
  for (int t = threadIdx.x; t < W * J; t += blockDim.x) {   // j fastest
    const int j = t % J, e = t / J;
    const int r = e & (R - 1), yy = e >> lgR;
    if (!((rows >> yy) & 1u)) continue;
    const int rhs = bu * R + r;
    const bool act = lane_active(a, rhs);
    const auto* in = a.in + (int64_t)rhs * a.in_rs;
    const int64_t grow = (int64_t)g1 * (y0 + yy + (int64_t)g2 * z);
    ffc2 v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int x = j + J * q;
      cplx<ff> val = {ff(0), ff(0)};
      if (act && x < g1) {
        if (a.mode == MV_GRID) {
          val = io_load<ff>(in[(int64_t)c * nD + grow + x]);
        } else {
          const int s = a.vox2sol[grow + x];
          if (s >= 0) {
            val = io_load<ff>(in[(int64_t)c * a.Ns + s]);
            if (a.mode == MV_VIE_ADJ) val = scale(mulc(val, a.chi[s]), a.invg[c]);
            else if (a.mode == MV_HFIELD_ADJ) val = scale(val, a.invg[c]);
          }
        }
      }
      v[q] = to_ffc2(val);
    }
    xyf_split<NB>(v, buf + e * S, W * S, P4, j, tw);
  }
  __syncthreads();
  xyf_mid<false, NB>(buf, 31 - __clz(W), 2, S, P4, tw, [&](int e) { return (rows >> (e >> lgR)) & 1u; });
  __syncthreads();
  // step 3: task (yy, alpha, k1, r), r fastest; output row [kx' = alpha*N + k][r]
  const int rowlen = 2 * N * R;
  cplx<ff>* dst = a.T1 + (((int64_t)bu * a.C + c) * g3 + z) * (int64_t)g2 * rowlen;
  for (int t = threadIdx.x; t < W * 32; t += blockDim.x) {
    const int r = t & (R - 1), q = t >> lgR;
    const int k1 = q & 15, alpha = (q >> 4) & 1, yy = q >> 5;
    if (!((rows >> yy) & 1u)) continue;
    const ffc2* src = buf + (alpha * W + yy * R + r) * S + (k1 & 3) * P4 + (k1 >> 2) * NB;
    ffc2 w[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) w[b] = lds_ffc2(src + b);
    dftf<false, NB>(w);
    cplx<ff>* o = dst + (int64_t)(y0 + yy) * rowlen + (alpha * N + k1) * R + r;
#pragma unroll
    for (int k3 = 0; k3 < NB; ++k3) o[16 * k3 * R] = from_ffc2(w[k3]);
  }
}

// ---------------------------------------------------------------------------
// Pass XI (inverse x + crop + epilogue)
// ---------------------------------------------------------------------------
template <int NB>
__global__ void __launch_bounds__(256, 3) k4f_inv_x(MvArgs<ff> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int N = 16 * NB, J = 4 * NB, S = xyf_stride(N), P4 = J + 1;
  const int bc = blockIdx.z, bu = bc / a.C, c = bc - bu * a.C;
  if (!bundle_active(a, bu)) return;
  const int z = blockIdx.y, y0 = blockIdx.x * a.TY;
  const int g1 = a.g1, g2 = a.g2, g3 = a.g3, R = a.R, lgR = a.lgR;
  const int ty = min(a.TY, g2 - y0), W = a.TY * R;
  unsigned rows = 0;
  for (int yy = 0; yy < ty; ++yy) rows |= row_is_live(a, y0 + yy, z) ? 1u << yy : 0u;
  if (!rows) return;   // no body voxel in these rows: no output
  ulonglong2* tw = reinterpret_cast<ulonglong2*>(smem_raw);
  ffc2* buf = reinterpret_cast<ffc2*>(tw + 2 * xyf_tw(N));
  load_twx<NB>(tw, a.ax.tw2);
  const int rowlen = 2 * N * R;
  const cplx<ff>* src = a.T1 + (((int64_t)bu * a.C + c) * g3 + z) * (int64_t)g2 * rowlen;
  for (int t = threadIdx.x; t < W * 32; t += blockDim.x) {
    const int r = t & (R - 1), q = t >> lgR;
    const int k1 = q & 15, alpha = (q >> 4) & 1, yy = q >> 5;
    if (!((rows >> yy) & 1u)) continue;
    const cplx<ff>* in = src + (int64_t)(y0 + yy) * rowlen + (alpha * N + k1) * R + r;
    ffc2 w[NB];
#pragma unroll
    for (int k3 = 0; k3 < NB; ++k3) w[k3] = to_ffc2(in[16 * k3 * R]);
    dftf<true, NB>(w);
    ffc2* d = buf + (alpha * W + yy * R + r) * S + (k1 & 3) * P4 + (k1 >> 2) * NB;
#pragma unroll
    for (int b = 0; b < NB; ++b) sts_ffc2(d + b, w[b]);
  }
  __syncthreads();
  xyf_mid<true, NB>(buf, 31 - __clz(W), 2, S, P4, tw, [&](int e) { return (rows >> (e >> lgR)) & 1u; });
  __syncthreads();
  const int64_t nD = (int64_t)g1 * g2 * g3;
  for (int t = threadIdx.x; t < W * J; t += blockDim.x) {   // j fastest
    const int j = t % J, e = t / J;
    const int r = e & (R - 1), yy = e >> lgR, rhs = bu * R + r;
    if (!((rows >> yy) & 1u) || !lane_active(a, rhs)) continue;
    ffc2 v[4];
    xyf_join<NB>(v, buf + e * S, W * S, P4, j, tw);
    const int64_t grow = (int64_t)g1 * (y0 + yy + (int64_t)g2 * z);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int x = j + J * q;
      if (x >= g1) break;
      if (a.mode == MV_GRID) {
        a.out[(int64_t)rhs * a.out_rs + (int64_t)c * nD + grow + x] = io_store(from_ffc2(v[q]));
      } else {
        const int s = a.vox2sol[grow + x];
        if (s >= 0) body_store(a, c, s, rhs, from_ffc2(v[q]));
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Pass Y (forward).  grid (ceil(2n1/TXY), g3, nbundle*C); element (kx', r) of a row
// ---------------------------------------------------------------------------
// live bit of row y = j + J*q, q < 4, at bit 4q (rows: bit a + 4q is y = NB*(a + 4q) + b)
template <int NB>
__device__ __forceinline__ unsigned xyf_rows(const MvArgs<ff>& a, int z, int j) {
  const int b = j % NB;
  return (a.rowq ? (unsigned)a.rowq[z * 8 + b] : inside_bits(a.g2, NB, b)) >> (j / NB);
}

template <int NB>
__global__ void __launch_bounds__(256, 3) k4f_fwd_y(MvArgs<ff> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int N = 16 * NB, J = 4 * NB, S = xyf_stride(N), P4 = J + 1;
  const int bc = blockIdx.z, bu = bc / a.C, c = bc - bu * a.C;
  if (!bundle_active(a, bu)) return;
  const int z = blockIdx.y, k0 = blockIdx.x * a.TXY;
  if (!z_is_live(a, z)) return;   // slice without body voxels: the z pass reads it as zero
  const int g2 = a.g2, g3 = a.g3, m1 = 2 * a.n1, R = a.R;
  const int W = a.TXY * R, wl = min(a.TXY, m1 - k0) * R;
  const int lgW = 31 - __clz(W);   // TXY*R is a power of two
  ulonglong2* tw = reinterpret_cast<ulonglong2*>(smem_raw);
  ffc2* buf = reinterpret_cast<ffc2*>(tw + 2 * xyf_tw(N));
  load_twx<NB>(tw, a.ay.tw2);
  __syncthreads();
  const int64_t row = (int64_t)m1 * R;
  const cplx<ff>* src = a.T1 + (((int64_t)bu * a.C + c) * g3 + z) * (int64_t)g2 * row + (int64_t)k0 * R;
  for (int t = threadIdx.x; t < W * J; t += blockDim.x) {   // e fastest
    const int e = t & (W - 1), j = t >> lgW;
    if (e >= wl) continue;
    const unsigned live = xyf_rows<NB>(a, z, j);
    ffc2 v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      v[q] = to_ffc2((live >> (4 * q)) & 1u ? src[(int64_t)(j + J * q) * row + e] : cplx<ff>{ff(0), ff(0)});
    xyf_split<NB>(v, buf + e * S, W * S, P4, j, tw);
  }
  __syncthreads();
  xyf_mid<false, NB>(buf, lgW, 2, S, P4, tw, [&](int e) { return e < wl; });
  __syncthreads();
  // step 3: task (beta, k1, e), e fastest; S_glob[bu][c][beta*N + k][z][kx'][r]
  cplx<ff>* dst = a.S + ((int64_t)bu * a.C + c) * (int64_t)2 * N * g3 * row + (int64_t)k0 * R;
  for (int t = threadIdx.x; t < 32 * W; t += blockDim.x) {
    const int e = t & (W - 1), q = t >> lgW;
    const int k1 = q & 15, beta = q >> 4;
    if (e >= wl) continue;
    const ffc2* p = buf + (beta * W + e) * S + (k1 & 3) * P4 + (k1 >> 2) * NB;
    ffc2 w[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) w[b] = lds_ffc2(p + b);
    dftf<false, NB>(w);
#pragma unroll
    for (int k3 = 0; k3 < NB; ++k3)
      dst[((int64_t)(beta * N + k1 + 16 * k3) * g3 + z) * row + e] = from_ffc2(w[k3]);
  }
}

// ---------------------------------------------------------------------------
// Pass YI (inverse y + crop)
// ---------------------------------------------------------------------------
template <int NB>
__global__ void __launch_bounds__(256, 3) k4f_inv_y(MvArgs<ff> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int N = 16 * NB, J = 4 * NB, S = xyf_stride(N), P4 = J + 1;
  const int bc = blockIdx.z, bu = bc / a.C, c = bc - bu * a.C;
  if (!bundle_active(a, bu)) return;
  const int z = blockIdx.y, k0 = blockIdx.x * a.TXY;
  if (!z_is_live(a, z)) return;   // no body voxel in slice z: no output
  const int g2 = a.g2, g3 = a.g3, m1 = 2 * a.n1, R = a.R;
  const int W = a.TXY * R, wl = min(a.TXY, m1 - k0) * R;
  const int lgW = 31 - __clz(W);   // TXY*R is a power of two
  ulonglong2* tw = reinterpret_cast<ulonglong2*>(smem_raw);
  ffc2* buf = reinterpret_cast<ffc2*>(tw + 2 * xyf_tw(N));
  load_twx<NB>(tw, a.ay.tw2);
  const int64_t row = (int64_t)m1 * R;
  const cplx<ff>* src = a.S + ((int64_t)bu * a.C + c) * (int64_t)2 * N * g3 * row + (int64_t)k0 * R;
  for (int t = threadIdx.x; t < 32 * W; t += blockDim.x) {
    const int e = t & (W - 1), q = t >> lgW;
    const int k1 = q & 15, beta = q >> 4;
    if (e >= wl) continue;
    ffc2 w[NB];
#pragma unroll
    for (int k3 = 0; k3 < NB; ++k3)
      w[k3] = to_ffc2(src[((int64_t)(beta * N + k1 + 16 * k3) * g3 + z) * row + e]);
    dftf<true, NB>(w);
    ffc2* p = buf + (beta * W + e) * S + (k1 & 3) * P4 + (k1 >> 2) * NB;
#pragma unroll
    for (int b = 0; b < NB; ++b) sts_ffc2(p + b, w[b]);
  }
  __syncthreads();
  xyf_mid<true, NB>(buf, lgW, 2, S, P4, tw, [&](int e) { return e < wl; });
  __syncthreads();
  cplx<ff>* dst = a.T1 + (((int64_t)bu * a.C + c) * g3 + z) * (int64_t)g2 * row + (int64_t)k0 * R;
  for (int t = threadIdx.x; t < W * J; t += blockDim.x) {   // e fastest
    const int e = t & (W - 1), j = t >> lgW;
    const unsigned live = xyf_rows<NB>(a, z, j);
    if (e >= wl || !(live & 0x1111u)) continue;
    ffc2 v[4];
    xyf_join<NB>(v, buf + e * S, W * S, P4, j, tw);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if ((live >> (4 * q)) & 1u) dst[(int64_t)(j + J * q) * row + e] = from_ffc2(v[q]);
  }
}

}  // namespace marie
