// Four-step x and y passes of the complex64 operator (n = 16*NB): the split of
// matvec4.cuh on work arrays whose slices z are contiguous,
//   T1[bundle][c][y][2n1][z][R],  S[bundle][c][2n2][2n1][z][R],
// over the caller's rows y < g2 and slices z < g3.  Every tile is W neighbouring
// elements, (slice, right-hand side) of one row in the x passes, (kx, slice,
// right-hand side) in the y passes, so all three transforms read and write runs of W
// elements (256 bytes at W = 32), and a z-pass column is one contiguous run.  (With
// rows of kx in T1 and columns of z in S one of the two sides of the y passes had runs
// of 64 bytes: 128^3 PWL, sixteen right-hand sides, a body in 95% of the slices and half
// of the rows, 4.4 + 4.5 ms; now 3.5 + 3.5.)
//
// Both halves of a zero-padded transform (even and odd frequencies) run in the
// two lanes of packed FP32 pairs (pair.cuh), one instruction for both, and pass
// through shared memory as 16-byte pairs: sequence e at e*S, S = 16*NB + 1
// pairs, [k1][b] (consecutive e on distinct 16-byte bank groups).  128^3 PWL,
// sixteen right-hand sides, against one half after the other: X 1.86 -> 1.41,
// YI 4.10 -> 3.58 ms (the body above).  A tile is skipped where all of its rows or
// slices are empty: with 28% of the rows live, X takes 0.97 ms where tiles of one row,
// both halves in turn, took 0.87.
#pragma once

#include "matvec4.cuh"
#include "pair.cuh"

namespace marie {

// Forward 16-point step of group b: both halves of the inputs v (element NB*q +
// b), then the four-step twiddle; d: the sequence's pairs, at b.
template <int NB>
__device__ __forceinline__ void pair_fwd16(const cplx<float>* v, cp* d, int b, const cplx<float>* tw,
                                           const cplx<float>* tw2) {
  cp u[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    const cplx<float> w = tw2[NB * q + b];
    u[q] = cp{f2_make(v[q].x, v[q].x * w.x - v[q].y * w.y), f2_make(v[q].y, v[q].x * w.y + v[q].y * w.x)};
  }
  dftp<false, 16>(u);
  d[0] = u[0];
#pragma unroll
  for (int k1 = 1; k1 < 16; ++k1) {
    const cplx<float> w = tw[b * k1];
    d[k1 * NB] = tw_mul(u[k1], f2_bc(w.x), f2_bc(w.y), f2_bc(-w.y));
  }
}
// Inverse 16-point step: v[q] = even(q) + odd(q) * conj(w_2n^(NB*q + b)).
template <int NB>
__device__ __forceinline__ void pair_inv16(cplx<float>* v, const cp* d, int b, const cplx<float>* tw2) {
  cp u[16];
#pragma unroll
  for (int k1 = 0; k1 < 16; ++k1) u[k1] = d[k1 * NB];
  dftp<true, 16>(u);
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    float ar, br, ai, bi;
    f2_split(u[q].re, ar, br);
    f2_split(u[q].im, ai, bi);
    const cplx<float> w = tw2[NB * q + b];
    v[q] = cplx<float>{fmaf(br, w.x, fmaf(bi, w.y, ar)), fmaf(bi, w.x, fmaf(-br, w.y, ai))};
  }
}
// NB-point steps of frequencies k1 + 16*k2: to (forward) or from (inverse) the
// even half's values at o0 and the odd half's at o1, stride st between k2.
template <int NB>
__device__ __forceinline__ void pair_fwdn(const cp* d, cplx<float>* o0, cplx<float>* o1, int64_t st) {
  cp w[NB];
#pragma unroll
  for (int b = 0; b < NB; ++b) w[b] = d[b];
  dftp<false, NB>(w);
#pragma unroll
  for (int k2 = 0; k2 < NB; ++k2) {
    cplx<float> e, o;
    f2_split(w[k2].re, e.x, o.x);
    f2_split(w[k2].im, e.y, o.y);
    o0[k2 * st] = e;
    o1[k2 * st] = o;
  }
}
template <int NB>
__device__ __forceinline__ void pair_invn(cp* d, const cplx<float>* o0, const cplx<float>* o1, int64_t st, int k1,
                                          const cplx<float>* tw) {
  cp w[NB];
#pragma unroll
  for (int k2 = 0; k2 < NB; ++k2) {
    const cplx<float> e = o0[k2 * st], o = o1[k2 * st];
    w[k2] = cp{f2_make(e.x, o.x), f2_make(e.y, o.y)};
  }
  dftp<true, NB>(w);
  d[0] = w[0];
#pragma unroll
  for (int b = 1; b < NB; ++b) {
    const cplx<float> q = tw[b * k1];
    d[b] = tw_mulc(w[b], f2_bc(q.x), f2_bc(q.y), f2_bc(-q.y));
  }
}

// Twiddles and pairs in dynamic shared memory.
struct XySmem {
  cplx<float>* tw;
  cp* buf;
};
__device__ __forceinline__ XySmem xy_smem(const cplx<float>* src, int N) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  XySmem m{reinterpret_cast<cplx<float>*>(smem_raw), reinterpret_cast<cp*>(smem_raw + N * sizeof(cplx<float>))};
  load_tw(m.tw, src, N);
  return m;
}

// ---------------------------------------------------------------------------
// Pass X (forward).  grid (ceil(g3/TZ), g2, nbundle*C)
// element e = zz*R + r
// ---------------------------------------------------------------------------
template <int NB>
__global__ void __launch_bounds__(256, 2) k4c_fwd_x(MvArgs<float> a) {
  constexpr int N = 16 * NB, S = N + 1;
  const int bc = blockIdx.z, bu = bc / a.C, c = bc - bu * a.C;
  if (!bundle_active(a, bu)) return;
  const int y = blockIdx.y, z0 = blockIdx.x * a.TY;
  const int g1 = a.g1, g2 = a.g2, g3 = a.g3, R = a.R, lgR = a.lgR;
  const int tz = min(a.TY, g3 - z0), W = a.TY * R, lgW = 31 - __clz(W);
  bool any = false;
  for (int zz = 0; zz < tz; ++zz) any = any || row_is_live(a, y, z0 + zz);
  if (!any) return;   // rows without body voxels stay unwritten: the y pass reads them as zero
  const XySmem sm = xy_smem(a.ax.tw, N);
  __syncthreads();
  const int64_t nD = (int64_t)g1 * g2 * g3;
  // step 1: task (zz, r, b), b fastest
  for (int t = threadIdx.x; t < tz * R * NB; t += blockDim.x) {
    const int b = t % NB, e = t / NB;
    const int r = e & (R - 1), zz = e >> lgR;
    if (!row_is_live(a, y, z0 + zz)) continue;
    const int rhs = bu * R + r;
    const bool act = lane_active(a, rhs);
    const int64_t grow = (int64_t)g1 * (y + (int64_t)g2 * (z0 + zz));
    cplx<float> v[16];
    if (a.mode == MV_GRID) {
      const cplx<float>* in = a.in + (int64_t)rhs * a.in_rs + (int64_t)c * nD + grow;
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const int x = NB * q + b;
        v[q] = act && x < g1 ? in[x] : cplx<float>{0.f, 0.f};
      }
    } else {
      const cplx<float>* in = a.in + (int64_t)rhs * a.in_rs + (int64_t)c * a.Ns;
      int s[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const int x = NB * q + b;
        s[q] = act && x < g1 ? a.vox2sol[grow + x] : -1;
      }
#pragma unroll
      for (int q = 0; q < 16; ++q) v[q] = s[q] >= 0 ? in[s[q]] : cplx<float>{0.f, 0.f};
      if (a.mode == MV_VIE_ADJ) {
#pragma unroll
        for (int q = 0; q < 16; ++q)
          if (s[q] >= 0) v[q] = scale(mulc(v[q], a.chi[s[q]]), a.invg[c]);
      } else if (a.mode == MV_HFIELD_ADJ) {
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = scale(v[q], a.invg[c]);
      }
    }
    pair_fwd16<NB>(v, sm.buf + e * S + b, b, sm.tw, a.ax.tw2);
  }
  __syncthreads();
  // step 2: task (k1, e), e fastest; kx' = alpha*N + k
  const int64_t col = (int64_t)g3 * R;
  cplx<float>* dst = a.T1 + (((int64_t)bu * a.C + c) * g2 + y) * 2 * N * col + (int64_t)z0 * R;
  for (int t = threadIdx.x; t < 16 * W; t += blockDim.x) {
    const int e = t & (W - 1), k1 = t >> lgW, zz = e >> lgR;
    if (zz >= tz || !row_is_live(a, y, z0 + zz)) continue;
    cplx<float>* o = dst + k1 * col + e;
    pair_fwdn<NB>(sm.buf + e * S + k1 * NB, o, o + N * col, 16 * col);
  }
}

// body_store (matvec.cuh) of eight values, s < 0: none; loads first.
__device__ __forceinline__ void body_store8(const MvArgs<float>& a, int c, const int* s, int rhs,
                                            const cplx<float>* v) {
  const cplx<float>* in = a.in + (int64_t)rhs * a.in_rs + (int64_t)c * a.Ns;
  const cplx<float>* add = a.addend ? a.addend + (int64_t)rhs * a.out_rs + (int64_t)c * a.Ns : nullptr;
  cplx<float>* out = a.out + (int64_t)rhs * a.out_rs + (int64_t)c * a.Ns;
  const cplx<float> zero{0.f, 0.f};
  cplx<float> r[8], x[8];
  if (a.mode == MV_HFIELD) {
#pragma unroll
    for (int q = 0; q < 8; ++q) r[q] = scale(v[q], a.invg[c]);
  } else if (a.mode == MV_HFIELD_ADJ) {
#pragma unroll
    for (int q = 0; q < 8; ++q) r[q] = v[q];
  } else {
#pragma unroll
    for (int q = 0; q < 8; ++q) x[q] = s[q] >= 0 ? in[s[q]] : zero;
    if (a.mode == MV_VIE) {
      cplx<float> h[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) h[q] = s[q] >= 0 ? a.chi[s[q]] : zero;
#pragma unroll
      for (int q = 0; q < 8; ++q) r[q] = x[q] - scale(h[q] * v[q], a.invg[c]);
    } else if (a.mode == MV_VIE_ADJ) {
#pragma unroll
      for (int q = 0; q < 8; ++q) r[q] = x[q] - v[q];
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q) r[q] = a.efac * (scale(v[q], a.invg[c]) - x[q]);
    }
  }
  if (add) {
#pragma unroll
    for (int q = 0; q < 8; ++q) x[q] = s[q] >= 0 ? add[s[q]] : zero;
#pragma unroll
    for (int q = 0; q < 8; ++q) r[q] = r[q] + x[q];
  }
#pragma unroll
  for (int q = 0; q < 8; ++q)
    if (s[q] >= 0) out[s[q]] = r[q];
}

// ---------------------------------------------------------------------------
// Pass XI (inverse x + crop + epilogue).
// ---------------------------------------------------------------------------
template <int NB>
__global__ void __launch_bounds__(256, 2) k4c_inv_x(MvArgs<float> a) {
  constexpr int N = 16 * NB, S = N + 1;
  const int bc = blockIdx.z, bu = bc / a.C, c = bc - bu * a.C;
  if (!bundle_active(a, bu)) return;
  const int y = blockIdx.y, z0 = blockIdx.x * a.TY;
  const int g1 = a.g1, g2 = a.g2, g3 = a.g3, R = a.R, lgR = a.lgR;
  const int tz = min(a.TY, g3 - z0), W = a.TY * R, lgW = 31 - __clz(W);
  bool any = false;
  for (int zz = 0; zz < tz; ++zz) any = any || row_is_live(a, y, z0 + zz);
  if (!any) return;   // no body voxel in these rows: no output
  const XySmem sm = xy_smem(a.ax.tw, N);
  __syncthreads();
  const int64_t col = (int64_t)g3 * R;
  const cplx<float>* src = a.T1 + (((int64_t)bu * a.C + c) * g2 + y) * 2 * N * col + (int64_t)z0 * R;
  // step A: task (k1, e), e fastest: inverse NB-point DFT over k2, twiddle
  for (int t = threadIdx.x; t < 16 * W; t += blockDim.x) {
    const int e = t & (W - 1), k1 = t >> lgW, zz = e >> lgR;
    if (zz >= tz || !row_is_live(a, y, z0 + zz)) continue;
    const cplx<float>* in = src + k1 * col + e;
    pair_invn<NB>(sm.buf + e * S + k1 * NB, in, in + N * col, 16 * col, k1, sm.tw);
  }
  __syncthreads();
  // step B: task (zz, r, b): inverse 16-point DFTs of both halves, combine, epilogue
  const int64_t nD = (int64_t)g1 * g2 * g3;
  for (int t = threadIdx.x; t < tz * R * NB; t += blockDim.x) {
    const int b = t % NB, e = t / NB;
    const int r = e & (R - 1), zz = e >> lgR;
    const int rhs = bu * R + r;
    if (!lane_active(a, rhs) || !row_is_live(a, y, z0 + zz)) continue;
    const int64_t grow = (int64_t)g1 * (y + (int64_t)g2 * (z0 + zz));
    cplx<float> v[16];
    if (a.mode == MV_GRID) {
      pair_inv16<NB>(v, sm.buf + e * S + b, b, a.ax.tw2);
      cplx<float>* out = a.out + (int64_t)rhs * a.out_rs + (int64_t)c * nD + grow;
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const int x = NB * q + b;
        if (x < g1) out[x] = v[q];
      }
    } else {
      // the body index loads during the transform, the epilogue's operands
      // eight at a time
      int s[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const int x = NB * q + b;
        s[q] = x < g1 ? a.vox2sol[grow + x] : -1;
      }
      pair_inv16<NB>(v, sm.buf + e * S + b, b, a.ax.tw2);
#pragma unroll
      for (int q = 0; q < 16; q += 8) body_store8(a, c, s + q, rhs, v + q);
    }
  }
}

// ---------------------------------------------------------------------------
// Pass Y (forward).  The elements (kx, z, r) of a row lie back to back and a tile takes
// WY of them: grid (g3*R / WY, 2n1, nbundle*C) where WY divides a column, else
// (ceil(2n1*g3*R / WY), 1, nbundle*C), wherever columns begin, so that a short or ragged
// z edge leaves no tile half empty (in tiles of one column's slices 64 x 16 x 16 PWL,
// one right-hand side, Y 16.8, YI 18.4 us; now 12.4 and 12.4).  The first form saves the
// division by g3 (96^3: 2% of the pass).
// ---------------------------------------------------------------------------
// The tile's first element of the row and whether any of its slices holds body voxels;
// the thread's slice z (-1: none, or without body voxels).
__device__ __forceinline__ bool y_tile(const MvArgs<float>& a, int& f0, int& z) {
  const int q = blockIdx.x * a.WY, e = threadIdx.x & (a.WY - 1);   // WY divides the block size
  int first = q >> a.lgR;
  if (gridDim.y > 1) {     // whole tiles in a column, blockIdx.y: the column
    f0 = blockIdx.y * a.g3 * a.R + q;
    z = first + (e >> a.lgR);
  } else {
    f0 = q;
    first %= a.g3;
    z = (first + (e >> a.lgR)) % a.g3;
    if (q + e >= 2 * a.n1 * a.g3 * a.R) z = -1;
  }
  bool any = false;
  for (int i = 0, s = first; i < a.WY && !any; i += a.R) {
    any = z_is_live(a, s);
    if (++s == a.g3) s = 0;
  }
  if (z >= 0 && !z_is_live(a, z)) z = -1;
  return any;
}

// One half at a time in scalar arithmetic at 80 registers (64 bytes a thread spilled):
// the pass waits for HBM, and three CTAs an SM hold more loads in flight than two of the packed
// form (48^3 PWL, eight right-hand sides: 139 against 158 us; 128^3: the same).
template <int NB>
__global__ void __launch_bounds__(256, 3) k4c_fwd_y(MvArgs<float> a) {
  constexpr int N = 16 * NB, S = N + 1;
  const int bc = blockIdx.z, bu = bc / a.C, c = bc - bu * a.C;
  if (!bundle_active(a, bu)) return;
  int f0, z;
  if (!y_tile(a, f0, z)) return;   // slices without body voxels: the z pass reads them as zero
  const int g2 = a.g2, W = a.WY, lgW = 31 - __clz(W);
  const XySmem sm = xy_smem(a.ay.tw, N);
  const cplx<float>* tw = sm.tw;
  cplx<float>* buf = reinterpret_cast<cplx<float>*>(sm.buf);   // half beta of sequence e at (beta*W + e)*S
  const int e = threadIdx.x & (W - 1);
  __syncthreads();
  const int64_t plane = (int64_t)2 * a.n1 * a.g3 * a.R;
  // step 1: task (b, e), e fastest
  for (int t = threadIdx.x; t < W * NB; t += blockDim.x) {
    const int b = t >> lgW;
    const unsigned live = z < 0 ? 0u : (a.rowq ? a.rowq[z * 8 + b] : inside_bits(g2, NB, b));   // rows y = NB*q + b
    const cplx<float>* src = a.T1 + ((int64_t)bc * g2 + b) * plane + f0 + e;
    cplx<float> v[16], u[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const cplx<float> val = ((live >> q) & 1u) ? src[NB * q * plane] : cplx<float>{0, 0};
      v[q] = val;
      u[q] = val;
    }
    dftn<float, false, 16>(u);
#pragma unroll
    for (int k1 = 0; k1 < 16; ++k1) buf[e * S + k1 * NB + b] = u[k1] * tw[b * k1];
#pragma unroll
    for (int q = 0; q < 16; ++q) u[q] = v[q] * a.ay.tw2[NB * q + b];
    dftn<float, false, 16>(u);
#pragma unroll
    for (int k1 = 0; k1 < 16; ++k1) buf[(W + e) * S + k1 * NB + b] = u[k1] * tw[b * k1];
  }
  __syncthreads();
  // step 2: task (beta, k1, e), e fastest; ky' = beta*N + k
  cplx<float>* dst = a.S + (int64_t)bc * 2 * N * plane + f0 + e;
  for (int t = threadIdx.x; t < 2 * 16 * W; t += blockDim.x) {
    const int q = t >> lgW;
    const int k1 = q & 15, beta = q >> 4;
    cplx<float> w[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) w[b] = buf[(beta * W + e) * S + k1 * NB + b];
    dftn<float, false, NB>(w);
    if (z >= 0) {
      cplx<float>* o = dst + (beta * N + k1) * plane;
#pragma unroll
      for (int k2 = 0; k2 < NB; ++k2) o[16 * k2 * plane] = w[k2];
    }
  }
}

// ---------------------------------------------------------------------------
// Pass YI (inverse y + crop).
// ---------------------------------------------------------------------------
template <int NB>
__global__ void __launch_bounds__(256, 2) k4c_inv_y(MvArgs<float> a) {
  constexpr int N = 16 * NB, S = N + 1;
  const int bc = blockIdx.z, bu = bc / a.C, c = bc - bu * a.C;
  if (!bundle_active(a, bu)) return;
  int f0, z;
  if (!y_tile(a, f0, z)) return;   // no body voxel in these slices: no output
  const int g2 = a.g2, W = a.WY, lgW = 31 - __clz(W);
  const XySmem sm = xy_smem(a.ay.tw, N);
  const int e = threadIdx.x & (W - 1);
  __syncthreads();
  const int64_t plane = (int64_t)2 * a.n1 * a.g3 * a.R;
  const cplx<float>* src = a.S + ((int64_t)bu * a.C + c) * 2 * N * plane + f0 + e;
  // step A: task (k1, e): inverse NB-point DFT over k2, twiddle
  for (int t = threadIdx.x; t < 16 * W && z >= 0; t += blockDim.x) {
    const int k1 = t >> lgW;
    const cplx<float>* in = src + k1 * plane;
    pair_invn<NB>(sm.buf + e * S + k1 * NB, in, in + N * plane, 16 * plane, k1, sm.tw);
  }
  __syncthreads();
  // step B: task (b, e): inverse 16-point DFTs of both halves, combine, store
  cplx<float>* dst = a.T1 + ((int64_t)bu * a.C + c) * g2 * plane + f0 + e;
  for (int t = threadIdx.x; t < W * NB; t += blockDim.x) {
    const int b = t >> lgW;
    const unsigned live = z < 0 ? 0u : (a.rowq ? a.rowq[z * 8 + b] : inside_bits(g2, NB, b));   // rows y = NB*q + b
    if (!live) continue;
    cplx<float> v[16];
    pair_inv16<NB>(v, sm.buf + e * S + b, b, a.ay.tw2);
#pragma unroll
    for (int q = 0; q < 16; ++q)
      if ((live >> q) & 1u) dst[(NB * q + b) * plane] = v[q];
  }
}

}  // namespace marie
