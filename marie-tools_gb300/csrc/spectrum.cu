// Green's-tensor spectra: one-time construction of the octant spectrum of each
// circulant block, either from the reference's Tucker factors (the expansion
// that mvp_N_pwl_tucker.m:31 repeats in every product) or from a dense I_V
// block (assembly_fft_circ_tucker_pwl.m:53 without the HOSVD truncation).
//
// Octant spectrum: for each block, G_hat(kx,ky,kz) for kx in [0,n1], ky in
// [0,n2], kz in [0,n3]; the remaining frequencies follow from the circulant
// symmetry G_hat(2n-k) = s * G_hat(k) per axis (s = +-1 per block and axis,
// see the mirror signs in BlockTab).  Layout [blk][ky][kx][kz], scaled by
// 1/(8 n1 n2 n3) so that the inverse transforms need no normalisation.
#include <cmath>
#include <vector>

#include "fastpath.cuh"
#include "internal.h"

namespace marie {

typedef cplx<double> zd;

// out[o][k][i] = sum_j in[o][j][i] * e(j,k),  e(0,k) = 1,
// e(j,k) = w_2m^{jk} + s * w_2m^{-jk}  (1 <= j < n), k in [0, m], m >= n: the
// circulant extension of length 2m, zero at the offsets n..m-1
__global__ void k_circ_axis(const zd* __restrict__ in, zd* __restrict__ out, int n, int m, int s, int64_t inner,
                            int64_t outer, const zd* __restrict__ w2m) {
  const int64_t total = outer * (m + 1) * inner;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t ii = idx % inner;
    const int64_t r = idx / inner;
    const int k = (int)(r % (m + 1));
    const int64_t o = r / (m + 1);
    const zd* src = in + o * n * inner + ii;
    zd acc = src[0];
    for (int j = 1; j < n; ++j) {
      const int e = (int)(((int64_t)j * k) % (2 * m));
      const zd w = w2m[e];
      const zd v = src[(int64_t)j * inner];
      // v * (w + s*conj(w))
      const zd ws = {w.x + s * w.x, w.y - s * w.y};
      acc = acc + v * ws;
    }
    out[idx] = acc;
  }
}

// The inverse of k_circ_axis with m = n: out[o][j][i], j < n, from the values
// in[o][k][i] at the octant frequencies k in [0, n].
__global__ void k_circ_inv(const zd* __restrict__ in, zd* __restrict__ out, int n, int s, int64_t inner,
                           int64_t outer, const zd* __restrict__ w2n) {
  const int64_t total = outer * n * inner;
  const double h = 0.5 / n;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t ii = idx % inner;
    const int64_t r = idx / inner;
    const int j = (int)(r % n);
    const int64_t o = r / n;
    const zd* src = in + o * (n + 1) * inner + ii;
    zd acc = (j & 1) ? src[0] - src[(int64_t)n * inner] : src[0] + src[(int64_t)n * inner];
    for (int k = 1; k < n; ++k) {
      const zd w = w2n[(int)(((int64_t)j * k) % (2 * n))];
      acc = acc + src[(int64_t)k * inner] * zd{w.x + s * w.x, -(w.y - s * w.y)};   // conj(w) + s w
    }
    out[idx] = scale(acc, h);
  }
}

// P1[a + r1(b + r2 kz)] = sum_c G[a + r1(b + r2 c)] U3[c + r3 kz]
__global__ void k_tk1(const zd* G, const zd* U3, zd* P1, int r1, int r2, int r3, int nk) {
  const int64_t total = (int64_t)r1 * r2 * nk;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t ab = idx % ((int64_t)r1 * r2);
    const int kz = (int)(idx / ((int64_t)r1 * r2));
    zd acc = {0, 0};
    for (int c = 0; c < r3; ++c) acc = acc + G[ab + (int64_t)r1 * r2 * c] * U3[c + (int64_t)r3 * kz];
    P1[idx] = acc;
  }
}

// P2[a + r1(ky + nky kz)] = sum_b P1[a + r1(b + r2 kz)] U2[b + r2 ky]
__global__ void k_tk2(const zd* P1, const zd* U2, zd* P2, int r1, int r2, int nky, int nkz) {
  const int64_t total = (int64_t)r1 * nky * nkz;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int a = (int)(idx % r1);
    const int64_t r = idx / r1;
    const int ky = (int)(r % nky);
    const int kz = (int)(r / nky);
    zd acc = {0, 0};
    for (int b = 0; b < r2; ++b) acc = acc + P1[a + (int64_t)r1 * (b + (int64_t)r2 * kz)] * U2[b + (int64_t)r2 * ky];
    P2[idx] = acc;
  }
}

// tmp[kx + nkx(ky + nky kz)] = sum_a P2[a + r1(ky + nky kz)] U1[a + r1 kx]
__global__ void k_tk3(const zd* P2, const zd* U1, zd* tmp, int r1, int nkx, int nky, int nkz) {
  const int64_t total = (int64_t)nkx * nky * nkz;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int kx = (int)(idx % nkx);
    const int64_t yz = idx / nkx;
    zd acc = {0, 0};
    for (int a = 0; a < r1; ++a) acc = acc + P2[a + (int64_t)r1 * yz] * U1[a + (int64_t)r1 * kx];
    tmp[idx] = acc;
  }
}

// dst[(ky*nkx + kx)*nkz + kz] = scale * tmp[kx + nkx(ky + nky kz)]
template <typename T>
__global__ void k_oct_store(const zd* tmp, cplx<T>* dst, int nkx, int nky, int nkz, double scl) {
  const int64_t total = (int64_t)nkx * nky * nkz;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int kz = (int)(idx % nkz);
    const int64_t r = idx / nkz;
    const int kx = (int)(r % nkx);
    const int ky = (int)(r / nkx);
    const zd v = tmp[kx + (int64_t)nkx * (ky + (int64_t)nky * kz)];
    dst[idx] = cplx<T>{(T)(v.x * scl), (T)(v.y * scl)};
  }
}

// Spectrum of one block for the four-step z pass, octant columns: for the
// columns kx in [0, n1], ky in [0, n2] all 2n3 frequencies kz, the z mirror
// sign applied; the mirrored columns follow by signs of the components
// (mirror_mask).  dst[((ky*(n1+1) + kx)*2n3 + kz)*U + blk]; float-float
// ((ky*(n1+1) + kx)*U + blk)*2n3 + (kz & 1)*n3 + kz/2: threads of neighbouring
// frequencies read neighbouring values.
template <typename T>
__global__ void k_full_store(const zd* tmp, cplx<T>* dst, int n1, int n2, int n3, int U, int blk, int s3, double scl) {
  const int m3 = 2 * n3;
  const int nkx = n1 + 1, nky = n2 + 1;
  const int64_t total = (int64_t)nkx * nky * m3;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int kz = (int)(idx % m3);
    const int64_t r = idx / m3;
    const int kx = (int)(r % nkx);
    const int ky = (int)(r / nkx);
    const bool mz = kz > n3;
    const double sg = (double)(mz ? s3 : 1) * scl;
    const zd v = tmp[kx + (int64_t)nkx * (ky + (int64_t)nky * (mz ? m3 - kz : kz))];
    const int64_t o = std::is_same<T, ff>::value ? (r * U + blk) * m3 + (kz & 1) * n3 + (kz >> 1) : idx * U + blk;
    dst[o] = cplx<T>{(T)(v.x * sg), (T)(v.y * sg)};
  }
}

// The twiddles and DFT constants of the complex64 passes are rounded to FP32, and
// their moduli with them: a transform multiplies frequency f by the product of its
// factors' moduli, and the inverse transform by the same product again, where phase
// errors take themselves back.  On most lengths the mean of that gain over an axis is
// 4e-8 to 6e-8 below one (sqrt(1/2) and cos(pi/8) round down), three axes of it more
// than half of the passes' whole error.  It is known, so the spectrum is divided by
// it.  Error of a product against complex128: 60 x 77 x 90 PWL 1.8e-7 -> 1.2e-7 (the
// mixed-radix passes on its own lengths 1.5e-7), 96^3 PWL 2.6e-7 -> 1.3e-7, 32^3 PWC
// 2.6e-7 -> 1.5e-7, at the same time.
// Returned: 1 / gain of the octant frequencies f = 0..n, the mean over the positions
// z < live (F: the transform's matrix; a frequency and its mirror image share a value
// of the spectrum and so the mean of theirs).
static std::vector<double> inverse_gain(int n, int live, bool zpass) {
  const int NB = n / 16;
  auto sq = [](long double ang) {   // squared modulus of exp(i ang) rounded to FP32
    const double c = (float)std::cos(ang), s = (float)std::sin(ang);
    return c * c + s * s;
  };
  const long double pi = 3.141592653589793238462643383279502884L;
  std::vector<double> w(2 * n);     // of w_2n^k
  for (int k = 0; k < 2 * n; ++k) w[k] = sq(pi * k / n);
  // factors of the small DFTs (dft16, and dft_small / dft6 of NB points): frequency k, input j
  const int R = NB == 6 ? 3 : NB;
  double m16[10], mr[8], m8 = sq(pi / 4), m6 = sq(pi / 3);
  for (int m = 0; m < 10; ++m) m16[m] = m & 3 ? sq(2 * pi * m / 16) : 1.0;
  for (int m = 0; m < 8; ++m) mr[m] = m % R ? sq(2 * pi * m / R) : 1.0;
  auto small16 = [&](int k, int j) { return m16[(k & 3) * (j & 3)]; };
  auto smalln = [&](int k, int j) {
    if (NB == 8) return (j & k & 1) ? m8 : 1.0;
    if (NB == 6) return ((k & 1) && j % 3 ? m6 : 1.0) * mr[(k >> 1) * (j % 3) % 3];
    return NB == 3 || NB == 5 || NB == 7 ? mr[j * k % NB] : 1.0;
  };
  const bool split_nb = zpass && zp_outer(NB) == NB;   // k4_zp: NB points first, 16 after the twiddles
  std::vector<double> g(2 * n, 0.0);
  for (int h = 0; h < 2; ++h)
    for (int k = 0; k < n; ++k)
      for (int z = 0; z < live; ++z) {
        const int b = split_nb ? z % 16 : z % NB, q = split_nb ? z / 16 : z / NB;
        const int k1 = split_nb ? k % NB : k % 16, k2 = split_nb ? k / NB : k / 16;
        g[2 * k + h] += (h ? w[z] : 1.0) * w[2 * b * k1] *
                        (split_nb ? smalln(k1, q) * small16(k2, b) : small16(k1, q) * smalln(k2, b));
      }
  std::vector<double> out(n + 1);
  for (int f = 0; f <= n; ++f) out[f] = 2.0 * live / (g[f] + g[(2 * n - f) % (2 * n)]);
  return out;
}

std::vector<double> four_step_inverse_gain(const marie_vie* h, int axis) {
  const PrecState<float>& ps = h->p32;
  return axis == 0 ? inverse_gain(ps.m1, h->n1, false)
                   : axis == 1 ? inverse_gain(ps.m2, h->n2, false) : inverse_gain(ps.m3, h->n3, true);
}

// The same for the complex64 z pass (k4_zp), pair layout: frequencies 2k and
// 2k+1 of a column share one 16-byte entry (re, re, im, im) at
// ((ky*(n1+1) + kx)*U + blk)*n3 + p, k = zp_freq(n3/16, p).  gx, gy, gz: inverse
// gains of the axes.
__global__ void k_full_store_pair(const zd* tmp, float4* dst, int n1, int n2, int n3, int U, int blk, int s3,
                                  double scl, const double* gx, const double* gy, const double* gz) {
  const int m3 = 2 * n3;
  const int nkx = n1 + 1, nky = n2 + 1;
  const int64_t total = (int64_t)nkx * nky * n3;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int p = (int)(idx % n3);
    const int k = zp_freq(n3 >> 4, p);
    const int64_t r = idx / n3;
    const int kx = (int)(r % nkx);
    const int ky = (int)(r / nkx);
    const double sxy = scl * gx[kx] * gy[ky];
    zd v[2];
#pragma unroll
    for (int o = 0; o < 2; ++o) {
      const int kz = 2 * k + o;
      const bool mz = kz > n3;
      const int kzo = mz ? m3 - kz : kz;
      v[o] = scale(tmp[kx + (int64_t)nkx * (ky + (int64_t)nky * kzo)], (double)(mz ? s3 : 1) * sxy * gz[kzo]);
    }
    dst[(r * U + blk) * n3 + p] = make_float4((float)v[0].x, (float)v[1].x, (float)v[0].y, (float)v[1].y);
  }
}

static unsigned grid_for(int64_t n) {
  int64_t b = (n + 255) / 256;
  if (b > 65535LL * 16) b = 65535LL * 16;
  return (unsigned)std::max<int64_t>(1, b);
}

// The octant storage needs the circulant parity of every block: a block that
// is odd along an axis (mirror sign -1) must vanish on that axis' zero-offset
// plane, otherwise G_hat(2n-k) != -G_hat(k).  Operators assembled by
// assembly_N/K satisfy it to rounding (symmetric Gauss rules); reject others.
static const double kParityTol = 1e-9;

static marie_status check_parity_dense(const double* A, int n1, int n2, int n3, const int8_t s[3], int id) {
  const int64_t nD = (int64_t)n1 * n2 * n3;
  double mx = 0, bad = 0;
  for (int64_t g = 0; g < nD; ++g) {
    const double v = std::hypot(A[2 * g], A[2 * g + 1]);
    mx = std::max(mx, v);
    const int x = (int)(g % n1), y = (int)((g / n1) % n2), z = (int)(g / ((int64_t)n1 * n2));
    if ((s[0] < 0 && x == 0) || (s[1] < 0 && y == 0) || (s[2] < 0 && z == 0)) bad = std::max(bad, v);
  }
  if (bad > kParityTol * mx) {
    set_error("operator block %d violates the circulant parity (odd block nonzero on its zero-offset plane, "
              "relative %.3e)", id, mx > 0 ? bad / mx : bad);
    return MARIE_ERR_BAD_ARG;
  }
  return MARIE_OK;
}

// Tucker block: the zero-offset sample of factor column a along axis d is
// u0[a] = (1/2n) sum_k U_d[a + r k] (inverse FFT at index 0).  Weighted by the
// norm of the core slice it multiplies (the HOSVD singular value), it bounds
// the block's value on the zero-offset plane relative to the block.
static marie_status check_parity_tucker(const marie_tucker_block& t, int n1, int n2, int n3, const int8_t s[3],
                                        int id) {
  const int r[3] = {t.r1, t.r2, t.r3};
  const int n[3] = {n1, n2, n3};
  const double* U[3] = {t.U1, t.U2, t.U3};
  for (int d = 0; d < 3; ++d) {
    if (s[d] > 0) continue;
    std::vector<double> sl(r[d], 0.0);
    for (int c = 0; c < t.r3; ++c)
      for (int b = 0; b < t.r2; ++b)
        for (int a = 0; a < t.r1; ++a) {
          const int64_t g = a + (int64_t)t.r1 * (b + (int64_t)t.r2 * c);
          const double v2 = t.G[2 * g] * t.G[2 * g] + t.G[2 * g + 1] * t.G[2 * g + 1];
          sl[d == 0 ? a : (d == 1 ? b : c)] += v2;
        }
    double smax = 0, worst = 0;
    for (int a = 0; a < r[d]; ++a) smax = std::max(smax, std::sqrt(sl[a]));
    for (int a = 0; a < r[d]; ++a) {
      double sx = 0, sy = 0;
      for (int k = 0; k < 2 * n[d]; ++k) {
        sx += U[d][2 * (a + (int64_t)r[d] * k)];
        sy += U[d][2 * (a + (int64_t)r[d] * k) + 1];
      }
      worst = std::max(worst, std::hypot(sx, sy) / (2.0 * n[d]) * std::sqrt(sl[a]));
    }
    if (worst > kParityTol * std::max(smax, 1e-300)) {
      set_error("Tucker block %d violates the circulant parity along axis %d (odd block nonzero on its "
                "zero-offset plane, relative %.3e)", id, d + 1, worst / smax);
      return MARIE_ERR_BAD_ARG;
    }
  }
  return MARIE_OK;
}

// Build all blocks of one operator (N or K) into the handle's spectra.
// Spectrum destinations of one operator: octant per precision (generic
// path, K) and octant columns (four-step path, N); null = not built.
struct SpecDst {
  cplx<double>* o64 = nullptr;
  cplx<float>* o32 = nullptr;
  cplx<double>* f64 = nullptr;
  cplx<float>* f32 = nullptr;
  cplx<ff>* fff = nullptr;
  cplx<float>* pad = nullptr;    // complex64 octant columns of the padded lengths m (PrecState::padded)
};

static marie_status build_op(marie_vie* h, const marie_tucker_block* tk, const double* dense, int ncomp,
                             const SpecDst& dst) {
  const int n1 = h->n1, n2 = h->n2, n3 = h->n3;
  const int pwx = h->pwl ? 10 : 1;
  const int nblk = pwx * ncomp;
  const int nkx = n1 + 1, nky = n2 + 1, nkz = n3 + 1;
  const int64_t oct = (int64_t)nkx * nky * nkz;
  const int64_t nD = (int64_t)n1 * n2 * n3;
  const double scl = 1.0 / (8.0 * (double)n1 * (double)n2 * (double)n3);
  // scratch
  zd *tmp = nullptr, *a = nullptr, *b = nullptr, *w1 = nullptr, *w2 = nullptr, *w3 = nullptr;
  zd *dG = nullptr, *dU1 = nullptr, *dU2 = nullptr, *dU3 = nullptr;
  std::vector<void*> scratch;
  auto salloc = [&](zd** p, size_t count) -> marie_status {
    if (count == 0) count = 1;
    cudaError_t e = cudaMalloc((void**)p, count * sizeof(zd));
    if (e != cudaSuccess) {
      cudaGetLastError();
      set_error("scratch allocation of %zu bytes failed", count * sizeof(zd));
      return MARIE_ERR_OOM;
    }
    scratch.push_back(*p);
    return MARIE_OK;
  };
  auto cleanup = [&]() {
    cudaDeviceSynchronize();
    for (void* p : scratch) cudaFree(p);
  };
  marie_status st = MARIE_OK;
  const int tabk = ncomp == 6 ? 0 : 2;   // N or K table (mirror signs)
  const BlockTab& bt = h->tab[tabk];
  const int64_t full = (int64_t)nkx * nky * 2 * n3;
  // padded complex64 spectrum: transform lengths m, tables, scratch (pa: the
  // block at offsets; pb, pc: after one and two axes; pt: its octant)
  const int m[3] = {h->p32.m1, h->p32.m2, h->p32.m3}, nn[3] = {n1, n2, n3};
  const int64_t poct = (int64_t)(m[0] + 1) * (m[1] + 1) * (m[2] + 1);
  const double pscl = 1.0 / (8.0 * (double)m[0] * (double)m[1] * (double)m[2]);
  zd *pa = nullptr, *pb = nullptr, *pc = nullptr, *pt = nullptr, *wn[3] = {}, *wm[3] = {};
  auto root_table = [&](zd** p, int n) -> marie_status {
    MARIE_TRY(salloc(p, 2 * n));
    std::vector<zd> w(2 * n);
    for (int k = 0; k < 2 * n; ++k) {
      const long double ang = -3.141592653589793238462643383279502884L * (long double)k / (long double)n;
      w[k] = zd{(double)std::cos(ang), (double)std::sin(ang)};
    }
    cudaMemcpy(*p, w.data(), 2 * n * sizeof(zd), cudaMemcpyHostToDevice);
    return MARIE_OK;
  };
  const double* gain[3] = {};
  auto gain_alloc = [&]() -> marie_status {
    if (!dst.f32 && !dst.pad) return MARIE_OK;
    for (int d = 0; d < 3; ++d) {
      const std::vector<double> g = four_step_inverse_gain(h, d);
      zd* p = nullptr;
      MARIE_TRY(salloc(&p, (g.size() + 1) / 2));
      cudaMemcpy(p, g.data(), g.size() * sizeof(double), cudaMemcpyHostToDevice);
      gain[d] = reinterpret_cast<const double*>(p);
    }
    return MARIE_OK;
  };
  auto pad_alloc = [&]() -> marie_status {
    if (!dst.pad) return MARIE_OK;
    for (int d = 0; d < 3; ++d) {
      MARIE_TRY(root_table(&wn[d], nn[d]));
      MARIE_TRY(root_table(&wm[d], m[d]));
    }
    MARIE_TRY(salloc(&pa, nD));
    MARIE_TRY(salloc(&pb, (int64_t)(m[0] + 1) * (n2 + 1) * (n3 + 1)));
    MARIE_TRY(salloc(&pc, (int64_t)(m[0] + 1) * (m[1] + 1) * (n3 + 1)));
    MARIE_TRY(salloc(&pt, poct));
    return MARIE_OK;
  };
  // block: its values at the offsets (dense), or null: recovered from tmp
  auto store_pad = [&](int id, const zd* block) {
    if (!dst.pad) return;
    const int s1 = bt.s1[id], s2 = bt.s2[id], s3 = bt.s3[id];
    if (!block) {
      k_circ_inv<<<grid_for((int64_t)nkx * nky * n3), 256>>>(tmp, pc, n3, s3, (int64_t)nkx * nky, 1, wn[2]);
      k_circ_inv<<<grid_for((int64_t)nkx * n2 * n3), 256>>>(pc, pb, n2, s2, nkx, n3, wn[1]);
      k_circ_inv<<<grid_for(nD), 256>>>(pb, pa, n1, s1, 1, (int64_t)n2 * n3, wn[0]);
      g_launches += 3;
      block = pa;
    }
    const int64_t kx = m[0] + 1, ky = m[1] + 1;
    k_circ_axis<<<grid_for(kx * n2 * n3), 256>>>(block, pb, n1, m[0], s1, 1, (int64_t)n2 * n3, wm[0]);
    k_circ_axis<<<grid_for(kx * ky * n3), 256>>>(pb, pc, n2, m[1], s2, kx, n3, wm[1]);
    k_circ_axis<<<grid_for(poct), 256>>>(pc, pt, n3, m[2], s3, kx * ky, 1, wm[2]);
    k_full_store_pair<<<grid_for(kx * ky * m[2]), 256>>>(pt, reinterpret_cast<float4*>(dst.pad), m[0], m[1], m[2], nblk,
                                                         id, s3, pscl, gain[0], gain[1], gain[2]);
    g_launches += 4;
  };
  auto store_block = [&](int id) {
    if (dst.o64) { k_oct_store<double><<<grid_for(oct), 256>>>(tmp, dst.o64 + id * oct, nkx, nky, nkz, scl); g_launches++; }
    if (dst.o32) { k_oct_store<float><<<grid_for(oct), 256>>>(tmp, dst.o32 + id * oct, nkx, nky, nkz, scl); g_launches++; }
    const int s3 = bt.s3[id];
    if (dst.f64) {
      k_full_store<double><<<grid_for(full), 256>>>(tmp, dst.f64, n1, n2, n3, nblk, id, s3, scl);
      g_launches++;
    }
    if (dst.f32) {
      k_full_store_pair<<<grid_for(full / 2), 256>>>(tmp, reinterpret_cast<float4*>(dst.f32), n1, n2, n3, nblk, id, s3,
                                                     scl, gain[0], gain[1], gain[2]);
      g_launches++;
    }
    if (dst.fff) {
      k_full_store<ff><<<grid_for(full), 256>>>(tmp, dst.fff, n1, n2, n3, nblk, id, s3, scl);
      g_launches++;
    }
  };
  do {
    if ((st = salloc(&tmp, oct)) != MARIE_OK) break;
    if ((st = gain_alloc()) != MARIE_OK || (st = pad_alloc()) != MARIE_OK) break;
    // a padded handle without complex128 needs nothing on the grid's own lengths
    const bool own = dst.o64 || dst.o32 || dst.f64 || dst.f32 || dst.fff;
    if (dense) {
      if ((st = salloc(&a, nD)) != MARIE_OK) break;
      if ((st = salloc(&b, (int64_t)nkx * nky * n3)) != MARIE_OK) break;
      if ((st = root_table(&w1, n1)) != MARIE_OK || (st = root_table(&w2, n2)) != MARIE_OK ||
          (st = root_table(&w3, n3)) != MARIE_OK)
        break;
      zd* c = nullptr;
      if ((st = salloc(&c, (int64_t)nkx * nky * n3)) != MARIE_OK) break;
      for (int id = 0; id < nblk; ++id) {
        // dense I_V is (n1,n2,n3,pwx,ncomp) column-major: block (j,k) at (j + pwx*k)*nD
        const int j = id / ncomp, k = id % ncomp;
        const double* src = dense + 2 * ((int64_t)(j + pwx * k) * nD);
        const int8_t sg[3] = {bt.s1[id], bt.s2[id], bt.s3[id]};
        if ((st = check_parity_dense(src, n1, n2, n3, sg, id)) != MARIE_OK) break;
        if (cudaMemcpy(a, src, nD * sizeof(zd), cudaMemcpyHostToDevice) != cudaSuccess) {
          set_error("upload of dense I_V failed");
          st = MARIE_ERR_CUDA;
          break;
        }
        if (own) {
          k_circ_axis<<<grid_for((int64_t)nkx * n2 * n3), 256>>>(a, b, n1, n1, bt.s1[id], 1, (int64_t)n2 * n3, w1);
          k_circ_axis<<<grid_for((int64_t)nkx * nky * n3), 256>>>(b, c, n2, n2, bt.s2[id], nkx, n3, w2);
          k_circ_axis<<<grid_for(oct), 256>>>(c, tmp, n3, n3, bt.s3[id], (int64_t)nkx * nky, 1, w3);
          g_launches += 3;
          store_block(id);
        }
        store_pad(id, a);
        if (cudaGetLastError() != cudaSuccess) { set_error("spectrum kernel launch failed"); st = MARIE_ERR_CUDA; break; }
        cudaDeviceSynchronize();
      }
    } else {
      int mr1 = 1, mr2 = 1, mr3 = 1;
      int64_t mg = 1, mp1 = 1, mp2 = 1;
      for (int id = 0; id < nblk; ++id) {
        const marie_tucker_block& t = tk[id];
        if (t.r1 < 1 || t.r2 < 1 || t.r3 < 1 || !t.G || !t.U1 || !t.U2 || !t.U3) {
          set_error("Tucker block %d is incomplete", id);
          st = MARIE_ERR_BAD_ARG;
          break;
        }
        const int8_t sg[3] = {bt.s1[id], bt.s2[id], bt.s3[id]};
        if ((st = check_parity_tucker(t, n1, n2, n3, sg, id)) != MARIE_OK) break;
        mr1 = std::max(mr1, t.r1); mr2 = std::max(mr2, t.r2); mr3 = std::max(mr3, t.r3);
        mg = std::max<int64_t>(mg, (int64_t)t.r1 * t.r2 * t.r3);
        mp1 = std::max<int64_t>(mp1, (int64_t)t.r1 * t.r2 * nkz);
        mp2 = std::max<int64_t>(mp2, (int64_t)t.r1 * nky * nkz);
      }
      if (st != MARIE_OK) break;
      if ((st = salloc(&dG, mg)) != MARIE_OK) break;
      if ((st = salloc(&dU1, (int64_t)mr1 * 2 * n1)) != MARIE_OK) break;
      if ((st = salloc(&dU2, (int64_t)mr2 * 2 * n2)) != MARIE_OK) break;
      if ((st = salloc(&dU3, (int64_t)mr3 * 2 * n3)) != MARIE_OK) break;
      if ((st = salloc(&a, mp1)) != MARIE_OK) break;
      if ((st = salloc(&b, mp2)) != MARIE_OK) break;
      for (int id = 0; id < nblk; ++id) {
        const marie_tucker_block& t = tk[id];
        cudaMemcpy(dG, t.G, (size_t)t.r1 * t.r2 * t.r3 * sizeof(zd), cudaMemcpyHostToDevice);
        cudaMemcpy(dU1, t.U1, (size_t)t.r1 * 2 * n1 * sizeof(zd), cudaMemcpyHostToDevice);
        cudaMemcpy(dU2, t.U2, (size_t)t.r2 * 2 * n2 * sizeof(zd), cudaMemcpyHostToDevice);
        cudaMemcpy(dU3, t.U3, (size_t)t.r3 * 2 * n3 * sizeof(zd), cudaMemcpyHostToDevice);
        k_tk1<<<grid_for((int64_t)t.r1 * t.r2 * nkz), 256>>>(dG, dU3, a, t.r1, t.r2, t.r3, nkz);
        g_launches++;
        k_tk2<<<grid_for((int64_t)t.r1 * nky * nkz), 256>>>(a, dU2, b, t.r1, t.r2, nky, nkz);
        g_launches++;
        k_tk3<<<grid_for(oct), 256>>>(b, dU1, tmp, t.r1, nkx, nky, nkz);
        g_launches++;
        store_block(id);
        store_pad(id, nullptr);
        if (cudaGetLastError() != cudaSuccess) { set_error("spectrum kernel launch failed"); st = MARIE_ERR_CUDA; break; }
        cudaDeviceSynchronize();
      }
    }
  } while (0);
  cleanup();
  return st;
}

marie_status build_spectra(marie_vie* h, const marie_vie_desc* d) {
  const int64_t oct = (int64_t)(h->n1 + 1) * (h->n2 + 1) * (h->n3 + 1);
  const int64_t full = (int64_t)(h->n1 + 1) * (h->n2 + 1) * 2 * h->n3;   // octant columns
  const bool fast = four_step_grid(h);
  if (h->precisions & 1) {
    MARIE_TRY(dev_alloc(h, (void**)&h->p64.GN, (size_t)h->nblkN * oct * sizeof(cplx<double>)));
    if (h->has_K) MARIE_TRY(dev_alloc(h, (void**)&h->p64.GK, (size_t)h->nblkK * oct * sizeof(cplx<double>)));
    if (fast) MARIE_TRY(dev_alloc(h, (void**)&h->p64.GNf, (size_t)h->nblkN * full * sizeof(cplx<double>)));
  }
  if (h->precisions & 2) {
    const PrecState<float>& ps = h->p32;
    const int64_t cols = (int64_t)(ps.m1 + 1) * (ps.m2 + 1) * 2 * ps.m3;
    if (!ps.padded) {
      MARIE_TRY(dev_alloc(h, (void**)&h->p32.GN, (size_t)h->nblkN * oct * sizeof(cplx<float>)));
      if (h->has_K) MARIE_TRY(dev_alloc(h, (void**)&h->p32.GK, (size_t)h->nblkK * oct * sizeof(cplx<float>)));
    }
    if (fast || ps.padded) {
      MARIE_TRY(dev_alloc(h, (void**)&h->p32.GNf, (size_t)h->nblkN * cols * sizeof(cplx<float>)));
      if (h->has_K) MARIE_TRY(dev_alloc(h, (void**)&h->p32.GKf, (size_t)h->nblkK * cols * sizeof(cplx<float>)));
    }
  }
  if (h->precisions & 4)   // float-float: four-step path only (N and N^H)
    MARIE_TRY(dev_alloc(h, (void**)&h->pff.GNf, (size_t)h->nblkN * full * sizeof(cplx<ff>)));
  SpecDst dN;
  dN.o64 = h->p64.GN;
  dN.o32 = h->p32.GN;
  dN.f64 = h->p64.GNf;
  (h->p32.padded ? dN.pad : dN.f32) = h->p32.GNf;
  dN.fff = h->pff.GNf;
  MARIE_TRY(build_op(h, d->tucker_N, d->tucker_N ? nullptr : d->dense_N, 6, dN));
  if (h->has_K) {
    SpecDst dK;
    dK.o64 = h->p64.GK;
    dK.o32 = h->p32.GK;
    (h->p32.padded ? dK.pad : dK.f32) = h->p32.GKf;
    MARIE_TRY(build_op(h, d->tucker_K, d->tucker_K ? nullptr : d->dense_K, 3, dK));
  }
  return MARIE_OK;
}

}  // namespace marie
