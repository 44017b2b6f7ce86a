// Producers of the hot path's operands, computed on the GPU in FP64:
//  - I_V of assembly_N.m:16-81 / assembly_K.m:16-81 (volume-volume Green's
//    tensor integrals per voxel offset, VV_Nop.m:1-48, VV_Kop.m:1-50,
//    G_N.m:3-19, G_K.m:3-13);
//  - incident fields of unit-current closed loops and of a plane wave, tested
//    onto the PWC/PWL basis (the loop right-hand sides).
#include "green_host.h"
#include <algorithm>
#include <cmath>
#include <vector>

#include "fp64math.cuh"
#include "internal.h"

namespace marie {

typedef cplx<double> zd;

// The kernels without their factor 1/(4 pi), which the callers' weights carry.
// G_N.m entries [-Gyy-Gzz, Gxy, Gxz, -Gxx-Gzz, Gyz, -Gxx-Gyy]
__device__ __forceinline__ void gn_kernel(double dx, double dy, double dz, double k0, zd* f) {
  const double R2 = dx * dx + dy * dy + dz * dz;
  double R;
  const double iR = inv_sqrt(R2, R);
  const double iR2 = iR * iR, iR3 = iR2 * iR, iR4 = iR2 * iR2, iR5 = iR4 * iR;
  double sn, cs;
  sin_cos(k0 * R, &sn, &cs);
  const zd Ge = {cs, -sn};                         // exp(-i k0 R)
  const double k2 = k0 * k0;
  // diag: 3d^2/R^5 + 3i k0 d^2/R^4 - (1 + k0^2 d^2)/R^3 - i k0/R^2
  auto diag = [&](double d) -> zd {
    return zd{3 * d * d * iR5 - (1 + k2 * d * d) * iR3, 3 * k0 * d * d * iR4 - k0 * iR2};
  };
  auto off = [&](double a, double b) -> zd {
    return zd{3 * a * b * iR5 - k2 * a * b * iR3, 3 * k0 * a * b * iR4};
  };
  const zd xx = Ge * diag(dx), yy = Ge * diag(dy), zz = Ge * diag(dz);
  f[0] = zd{-(yy.x + zz.x), -(yy.y + zz.y)};
  f[1] = Ge * off(dx, dy);
  f[2] = Ge * off(dx, dz);
  f[3] = zd{-(xx.x + zz.x), -(xx.y + zz.y)};
  f[4] = Ge * off(dy, dz);
  f[5] = zd{-(xx.x + yy.x), -(xx.y + yy.y)};
}

// G_K.m entries [Gx, Gy, Gz] = exp(-ik0R) * (-d) * (1/R^3 + i k0/R^2)
__device__ __forceinline__ void gk_kernel(double dx, double dy, double dz, double k0, zd* f) {
  double R;
  const double iR = inv_sqrt(dx * dx + dy * dy + dz * dz, R);
  double sn, cs;
  sin_cos(k0 * R, &sn, &cs);
  const zd Ge = {cs, -sn};
  const zd fac = Ge * zd{iR * iR * iR, k0 * iR * iR};
  f[0] = scale(fac, -dx);
  f[1] = scale(fac, -dy);
  f[2] = scale(fac, -dz);
}

// ---------------------------------------------------------------------------
// I_V of one voxel offset m is a six-dimensional Gauss sum over the point
// pairs (r, r') of two voxels, but the kernel sees only r - r', and along one
// axis the n x n' pairs have few distinct differences: a symmetric n-point
// rule used on both sides gives the same difference for (i, j) and
// (n-1-j, n-1-i), so 9 of 16 for the far rule (n = 4) and 33 of 64 for the
// medium one (n = 8).  The pair weights and the moments (T_l, B_l' linear or
// constant along the axis) are summed per difference on the host, and the
// kernel is evaluated at D^3 points instead of (n n')^3: 729 for 4096, 35937
// for 262144.  The moments are then applied axis by axis: one thread per
// (x, y) line sums its D kernel values over z with the three z weights, and
// the CTA's outputs sum the lines with the x weights, row by row, and the rows with
// the y weights.  Rows are summed in two parts and the sum over the rows carries
// its rounding (two-sum), and the common factor is applied in two parts, so that
// fewer points do not mean a larger error: 1.7e-16 and 1.9e-16 of a far offset's
// values at 2 and 5 mm (with one running sum over the lines 3.8e-16 at 5 mm; the sum
// over all point pairs 2.4e-16 and 2.2e-16).
//
// The sum is also symmetric under axis permutations (a permuted offset holds
// the same values with components and moments permuted), so only offsets
// a >= b >= c are computed and written to their (up to six) places.
//
// Bound: FP64 arithmetic (two FMAs per clock and SM), almost all of it the
// D^3 kernel values.  48^3 PWL, N, the whole call with its copy to the host:
// 405 -> 9.8 ms (with k_near, which took 95 ms of it on the host).
// ---------------------------------------------------------------------------
struct AxisRule {
  const double* d;      // D differences X - X' on [-1, 1] nodes
  const double* w;      // [4][D]: weights for (T, B) = (1, 1), (x, 1), (1, x), (x, x)
  int D;
};
constexpr int kVvThreads = 128;
constexpr int kVvLines = 243;     // most lines per pass: three offsets of the far rule (3 * 9^2), odd: conflict-free rows

enum WType { W_CC = 0, W_LC = 1, W_CL = 2, W_LL = 3 };
// weight type of moment product j (VV_Nop.m:27-28) along axis d (0 x, 1 y, 2 z)
__host__ __device__ constexpr int pair_l(int j) { return j < 4 ? j : (j < 7 ? 0 : (j < 9 ? 1 : 2)); }
__host__ __device__ constexpr int pair_lp(int j) { return j < 4 ? j : (j < 7 ? j - 3 : (j == 7 ? 2 : 3)); }
__host__ __device__ constexpr int pair_of(int l, int lp) {
  return l == lp ? l : (l == 0 || lp == 0 ? l + lp + 3 : l + lp + 4);
}
__host__ __device__ constexpr int pair_type(int j, int d) {
  return (pair_l(j) == d + 1 ? 1 : 0) + (pair_lp(j) == d + 1 ? 2 : 0);
}
// components of the symmetric N tensor: xx, xy, xz, yy, yz, zz
__host__ __device__ constexpr int comp_of(int p, int q) { return p + q + (p > 0 && q > 0 ? 1 : 0); }
__host__ __device__ constexpr int comp_p(int c) { return c < 3 ? 0 : (c < 5 ? 1 : 2); }
__host__ __device__ constexpr int comp_q(int c) { return c < 3 ? c : (c < 5 ? c - 2 : 2); }

// Axis permutation s (of 0..5): destination axis d takes canonical axis perm(s, d).
__host__ __device__ constexpr int perm_axis(int s, int d) {
  const int first = s >> 1, r0 = first == 0 ? 1 : 0, r1 = first == 2 ? 1 : 2;
  return d == 0 ? first : ((d == 1) == ((s & 1) == 0) ? r0 : r1);
}

// offs: (a, b, c, rule | 8 * permute).  The first nspec blocks take one offset
// each (medium rule and the near stand-in), the others three offsets of the
// far rule.  J: (dx/2)^6 / (4 pi) in two parts (its rounding would be in every value).
// out[(mx + n1(my + n2 mz)) + nD*(llp + pwx*comp)]
template <int PWX, int NC, bool ISN>
__global__ void __launch_bounds__(kVvThreads) k_vv(const int4* offs, int nspec, int noff, AxisRule r0, AxisRule r1,
                                                   AxisRule r2, double dx, double2 J, double k0, int n1, int n2,
                                                   int n3, double* out) {
  extern __shared__ __align__(16) double vsm[];
  constexpr int NZ = PWX == 1 ? 1 : 3;          // z weight types in use: cc, cl, ll
  constexpr int NA = NZ * NC * 2;
  constexpr int NOUT = PWX * NC * 2;
  constexpr int PER = (3 * NOUT + kVvThreads - 1) / kVvThreads;
  double* A = vsm;                              // [NA][kVvLines]
  double* wt = A + NA * kVvLines;               // [4][D], then the differences
  const int b = blockIdx.x;
  const bool one = b < nspec;
  const int o0 = one ? b : nspec + 3 * (b - nspec);
  const int cnt = one ? 1 : min(3, noff - o0);
  const int rid = offs[o0].w & 7;
  const AxisRule r = rid == 0 ? r0 : (rid == 1 ? r1 : r2);
  const int D = r.D, D2 = D * D;
  double* dd = wt + 4 * D;
  const double h = dx / 2;
  for (int i = threadIdx.x; i < 4 * D; i += kVvThreads) wt[i] = r.w[i];
  for (int i = threadIdx.x; i < D; i += kVvThreads) dd[i] = h * r.d[i];
  double acc[PER], err[PER];
#pragma unroll
  for (int v = 0; v < PER; ++v) acc[v] = err[v] = 0;
  const int total = cnt * D2;
  const int pass = kVvLines / D * D;            // whole rows
  for (int base = 0; base < total; base += pass) {
    const int nl = min(pass, total - base);
    __syncthreads();
    for (int t = threadIdx.x; t < nl; t += kVvThreads) {
      const int o = (base + t) / D2, line = base + t - o * D2;
      const int iy = line / D, ix = line - iy * D;
      const int4 m = offs[o0 + o];
      const double x = m.x * dx + dd[ix], y = m.y * dx + dd[iy], z0 = m.z * dx;
      zd a[NZ][NC];
#pragma unroll
      for (int q = 0; q < NZ; ++q)
#pragma unroll
        for (int c = 0; c < NC; ++c) a[q][c] = zd{0, 0};
      for (int iz = 0; iz < D; ++iz) {
        zd f[NC];
        if (ISN) gn_kernel(x, y, z0 + dd[iz], k0, f);
        else gk_kernel(x, y, z0 + dd[iz], k0, f);
#pragma unroll
        for (int q = 0; q < NZ; ++q) {
          const double w = wt[(q == 0 ? W_CC : (q == 1 ? W_CL : W_LL)) * D + iz];
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            a[q][c].x = fma(w, f[c].x, a[q][c].x);
            a[q][c].y = fma(w, f[c].y, a[q][c].y);
          }
        }
      }
#pragma unroll
      for (int q = 0; q < NZ; ++q)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          A[((q * NC + c) * 2 + 0) * kVvLines + t] = a[q][c].x;
          A[((q * NC + c) * 2 + 1) * kVvLines + t] = a[q][c].y;
        }
    }
    __syncthreads();
#pragma unroll
    for (int v = 0; v < PER; ++v) {
      const int u = threadIdx.x + v * kVvThreads;
      if (u >= cnt * NOUT) break;
      const int o = u / NOUT, e = u - o * NOUT, ri = e & 1, jc = e >> 1, j = jc / NC, c = jc - j * NC;
      const int zt = pair_type(j, 2);
      const double* wx = wt + pair_type(j, 0) * D;
      const double* wy = wt + pair_type(j, 1) * D;
      const double* row = A + (((zt == W_CC ? 0 : (zt == W_CL ? 1 : 2)) * NC + c) * 2 + ri) * kVvLines;
      const int lo = max(o * D2 - base, 0), hi = min((o + 1) * D2 - base, nl);
      const int iy0 = (base + lo - o * D2) / D;
      for (int t = lo, iy = iy0; t < hi; t += D, ++iy) {
        double s0 = 0, s1 = 0;
        int ix = 0;
#pragma unroll 4
        for (; ix + 1 < D; ix += 2) {
          s0 = fma(wx[ix], row[t + ix], s0);
          s1 = fma(wx[ix + 1], row[t + ix + 1], s1);
        }
        if (ix < D) s0 = fma(wx[ix], row[t + ix], s0);
        const double r = s0 + s1, p = __dmul_rn(wy[iy], r);
        const double sum = acc[v] + p, back = sum - acc[v];
        err[v] += ((acc[v] - (sum - back)) + (p - back)) + fma(wy[iy], r, -p);
        acc[v] = sum;
      }
    }
  }
  const int64_t nD = (int64_t)n1 * n2 * n3;
#pragma unroll
  for (int v = 0; v < PER; ++v) {
    const int u = threadIdx.x + v * kVvThreads;
    if (u >= cnt * NOUT) break;
    const int o = u / NOUT, e = u - o * NOUT, ri = e & 1, jc = e >> 1, j = jc / NC, c = jc - j * NC;
    const int4 m = offs[o0 + o];
    const int t[3] = {m.x, m.y, m.z};
    const int np = (m.w & 8) ? 6 : 1;
    for (int s = 0; s < np; ++s) {
      const int p0 = perm_axis(s, 0), p1 = perm_axis(s, 1), p2 = perm_axis(s, 2);
      const int mx = t[p0], my = t[p1], mz = t[p2];
      if (mx >= n1 || my >= n2 || mz >= n3) continue;
      bool again = false;          // equal offsets: the first permutation writes the place
      for (int q = 0; q < s; ++q)
        again = again || (t[perm_axis(q, 0)] == mx && t[perm_axis(q, 1)] == my && t[perm_axis(q, 2)] == mz);
      if (again) continue;
      auto back = [&](int ax) { return p0 == ax ? 0 : (p1 == ax ? 1 : 2); };
      const int l = pair_l(j), lp = pair_lp(j);
      const int jj = PWX == 1 ? 0 : pair_of(l ? back(l - 1) + 1 : 0, lp ? back(lp - 1) + 1 : 0);
      int cc;
      if (ISN) cc = comp_of(back(comp_p(c)), back(comp_q(c)));
      else cc = back(c);
      out[2 * (mx + (int64_t)n1 * (my + (int64_t)n2 * mz) + nD * (jj + PWX * cc)) + ri] = fma(acc[v], J.x, fma(acc[v], J.y, err[v] * J.x));
    }
  }
}

// The accurate near zone (green_host.h, near_zone_offset) of the offsets
// {0,1}^3 on the GPU: the same cubature, its points spread over the CTAs
// (Gauss node i of the first variable, piece and pyramid, offset).  Each CTA
// leaves the partial sums of its order^2 points; k_near_sum adds the CTAs of
// an offset in a fixed order.  On the host this took 95 ms of every assembly
// (one core, 480 thousand points, three kernel values each).
constexpr int kNearOrder = 16;
constexpr int kNearThreads = 128;

template <int PWX, int NC, bool ISN>
__global__ void __launch_bounds__(kNearThreads) k_near(const double* gx, const double* gw, double res, double k0,
                                                       int n1, int n2, int n3, double* part) {
  __shared__ double F[kNearThreads][2][2 * NC];   // the two terms' kernel values with the quadrature weight
  __shared__ double Wm[kNearThreads][2][PWX];     // W_l and W_l - W_l(0)
  const int m[3] = {(int)(blockIdx.z & 1), (int)(blockIdx.z >> 1 & 1), (int)(blockIdx.z >> 2)};
  if (m[0] >= n1 || m[1] >= n2 || m[2] >= n3) return;
  const int i = blockIdx.x, piece = blockIdx.y / 3, e = blockIdx.y - 3 * piece;
  double L[3], a[3], sg[3];
  bool corner = true;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int upper = piece >> (2 - d) & 1;
    const double lo = m[d] == 0 ? (upper ? 0.0 : -res) : (upper ? res : 0.0);
    const double hi = m[d] == 0 ? (upper ? res : 0.0) : (upper ? 2 * res : res);
    a[d] = lo;
    L[d] = hi - lo;
    if (!(lo == 0.0 || hi == 0.0)) corner = false;
    sg[d] = hi > 0.0 ? 1.0 : -1.0;
  }
  const double vol = L[0] * L[1] * L[2];
  auto weights = [&](const double* u, double* W) {
    double ov[3][4];
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
      for (int q = 0; q < 4; ++q)
        ov[d][q] = PWX == 1 && q ? 0.0 : green_host::moment_overlap(u[d], m[d], res, (q & 1) != 0, (q & 2) != 0);
#pragma unroll
    for (int j = 0; j < PWX; ++j) W[j] = ov[0][pair_type(j, 0)] * ov[1][pair_type(j, 1)] * ov[2][pair_type(j, 2)];
  };
  const double zero[3] = {0.0, 0.0, 0.0};
  double W0[PWX], W[PWX];
  weights(zero, W0);
  const int f = (e + 1) % 3;
  double acc = 0;
  const bool run = corner || e == 0;              // pieces away from 0 take one tensor rule
  for (int base = 0; run && base < kNearOrder * kNearOrder; base += kNearThreads) {
    const int j = (base + threadIdx.x) / kNearOrder, k = (base + threadIdx.x) - j * kNearOrder;
    const double wq = gw[i] * gw[j] * gw[k] * (vol * (0.25 / 3.14159265358979323846));
    zd Kf[NC], Ks[NC], Kt[NC];
    double u[3], ut[3];
    double c1 = wq, c2 = 0;
    if (!corner) {
      u[0] = a[0] + L[0] * gx[i];
      u[1] = a[1] + L[1] * gx[j];
      u[2] = a[2] + L[2] * gx[k];
#pragma unroll
      for (int d = 0; d < 3; ++d) ut[d] = u[d];
    } else {
      const double t = gx[i];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        ut[d] = sg[d] * L[d] * (d == e ? 1.0 : (d == f ? gx[j] : gx[k]));
        u[d] = t * ut[d];
      }
      c1 = wq * t * t;
      c2 = ISN ? wq / t : 0.0;
    }
    if (ISN) gn_kernel(u[0], u[1], u[2], k0, Kf);
    else gk_kernel(u[0], u[1], u[2], k0, Kf);
    if (ISN && corner) {
      gn_kernel(u[0], u[1], u[2], 0.0, Ks);
      gn_kernel(ut[0], ut[1], ut[2], 0.0, Kt);
    } else {
#pragma unroll
      for (int c = 0; c < NC; ++c) Ks[c] = Kt[c] = zd{0, 0};
    }
    weights(u, W);
    __syncthreads();
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      F[threadIdx.x][0][2 * c] = c1 * (Kf[c].x - Ks[c].x);
      F[threadIdx.x][0][2 * c + 1] = c1 * (Kf[c].y - Ks[c].y);
      F[threadIdx.x][1][2 * c] = c2 * Kt[c].x;
      F[threadIdx.x][1][2 * c + 1] = c2 * Kt[c].y;
    }
#pragma unroll
    for (int l = 0; l < PWX; ++l) {
      Wm[threadIdx.x][0][l] = W[l];
      Wm[threadIdx.x][1][l] = W[l] - W0[l];
    }
    __syncthreads();
    if (threadIdx.x < PWX * NC * 2) {
      const int l = threadIdx.x / (2 * NC), q = threadIdx.x - l * 2 * NC;
      for (int t = 0; t < kNearThreads; ++t)
        acc += F[t][0][q] * Wm[t][0][l] + F[t][1][q] * Wm[t][1][l];
    }
  }
  if (threadIdx.x < PWX * NC * 2)
    part[(((int64_t)blockIdx.z * 24 + blockIdx.y) * kNearOrder + i) * (PWX * NC * 2) + threadIdx.x] = acc;
}

// out at offset blockIdx.x of {0,1}^3: its CTAs' partial sums, in order
template <int PWX, int NC>
__global__ void k_near_sum(const double* part, int n1, int n2, int n3, double* out) {
  const int mx = blockIdx.x & 1, my = blockIdx.x >> 1 & 1, mz = blockIdx.x >> 2;
  if (mx >= n1 || my >= n2 || mz >= n3 || threadIdx.x >= PWX * NC * 2) return;
  const int l = threadIdx.x / (2 * NC), q = threadIdx.x - l * 2 * NC, c = q >> 1, ri = q & 1;
  double s = 0;
  for (int b = 0; b < 24 * kNearOrder; ++b)
    s += part[((int64_t)blockIdx.x * 24 * kNearOrder + b) * (PWX * NC * 2) + threadIdx.x];
  const int64_t nD = (int64_t)n1 * n2 * n3;
  out[2 * (mx + (int64_t)n1 * (my + (int64_t)n2 * mz) + nD * (l + PWX * c)) + ri] = s;
}

void gauss_legendre(int n, std::vector<double>& x, std::vector<double>& w) {
  // Newton iteration on P_n; nodes ascending.
  x.assign(n, 0.0);
  w.assign(n, 0.0);
  for (int i = 0; i < n; ++i) {
    long double z = std::cos(3.141592653589793238462643383279502884L * (i + 0.75L) / (n + 0.5L));
    long double pp = 0;
    for (int it = 0; it < 100; ++it) {
      long double p1 = 1, p2 = 0;
      for (int j = 1; j <= n; ++j) {
        const long double p3 = p2;
        p2 = p1;
        p1 = ((2.0L * j - 1.0L) * z * p2 - (j - 1.0L) * p3) / j;
      }
      pp = n * (z * p1 - p2) / (z * z - 1.0L);
      const long double z1 = z;
      z = z1 - p1 / pp;
      if (std::fabs((double)(z - z1)) < 1e-19) {
        // recompute derivative at the converged node
        p1 = 1; p2 = 0;
        for (int j = 1; j <= n; ++j) {
          const long double p3 = p2;
          p2 = p1;
          p1 = ((2.0L * j - 1.0L) * z * p2 - (j - 1.0L) * p3) / j;
        }
        pp = n * (z * p1 - p2) / (z * z - 1.0L);
        break;
      }
    }
    x[n - 1 - i] = (double)z;
    w[n - 1 - i] = (double)(2.0L / ((1.0L - z * z) * pp * pp));
  }
}

struct DevRule {
  double* mem = nullptr;
  AxisRule r{};
};

// Differences and weights of an no x ns point rule along one axis (see k_vv).
static marie_status make_rule(int no, int ns, DevRule& dr, std::vector<void*>& scratch) {
  std::vector<double> xo, wo, xs, ws;
  gauss_legendre(no, xo, wo);
  gauss_legendre(ns, xs, ws);
  std::vector<double> d, w[4];
  std::vector<int> at((size_t)no * ns, -1);
  for (int i = 0; i < no; ++i)
    for (int j = 0; j < ns; ++j) {
      int k = -1;
      if (no == ns) {            // the same difference: i = j, and (no-1-j, no-1-i)
        if (i == j && i > 0) k = at[0];
        else if (i != j) k = at[(size_t)(no - 1 - j) * ns + (no - 1 - i)];
      }
      if (k < 0) {
        k = (int)d.size();
        d.push_back(i == j && no == ns ? 0.0
                    : no == ns         ? 0.5 * ((xo[i] - xs[j]) + (xo[no - 1 - j] - xs[no - 1 - i]))
                                       : xo[i] - xs[j]);
        for (auto& v : w) v.push_back(0.0);
      }
      at[(size_t)i * ns + j] = k;
      const double ww = wo[i] * ws[j];
      w[W_CC][k] += ww;
      w[W_LC][k] += ww * (0.5 * xo[i]);
      w[W_CL][k] += ww * (0.5 * xs[j]);
      w[W_LL][k] += ww * (0.5 * xo[i]) * (0.5 * xs[j]);
    }
  const int D = (int)d.size();
  for (auto& v : w) d.insert(d.end(), v.begin(), v.end());
  if (cudaMalloc(&dr.mem, d.size() * sizeof(double)) != cudaSuccess) return MARIE_ERR_OOM;
  scratch.push_back(dr.mem);
  cudaMemcpy(dr.mem, d.data(), d.size() * sizeof(double), cudaMemcpyHostToDevice);
  dr.r = AxisRule{dr.mem, dr.mem + D, D};
  return MARIE_OK;
}

template <int PWX, int NC, bool ISN>
static cudaError_t run_vv(const int4* offs, int nspec, int noff, const DevRule* rules, bool near_exact,
                          const double* gauss, double* part, double dx, double k0, int n1, int n2, int n3,
                          double* out) {
  constexpr int NZ = PWX == 1 ? 1 : 3;
  int D = 0;
  for (int i = 0; i < 3; ++i) D = std::max(D, rules[i].r.D);
  const size_t smem = ((size_t)NZ * NC * 2 * kVvLines + 5 * (size_t)D) * sizeof(double);
  static std::atomic<uint64_t> done{0};
  smem_opt_in_device((const void*)k_vv<PWX, NC, ISN>, done);
  if (near_exact) {
    k_near<PWX, NC, ISN><<<dim3(kNearOrder, 24, 8), kNearThreads>>>(gauss, gauss + kNearOrder, dx, k0, n1, n2, n3, part);
    k_near_sum<PWX, NC><<<8, kNearThreads>>>(part, n1, n2, n3, out);
    g_launches += 2;
  }
  const int blocks = nspec + (noff - nspec + 2) / 3;
  if (blocks > 0) {
    const long double h = 0.5L * dx, J = h * h * h * h * h * h / (4.0L * 3.141592653589793238462643383279502884L);
    const double2 J2{(double)J, (double)(J - (double)J)};
    k_vv<PWX, NC, ISN><<<blocks, kVvThreads, smem>>>(offs, nspec, noff, rules[0].r, rules[1].r, rules[2].r, dx,
                                                     J2, k0, n1, n2, n3, out);
    g_launches++;
  }
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Incident fields
// ---------------------------------------------------------------------------

// Ue[l][comp*Ns + s] = coef of loop l on voxel s; one thread per (voxel, loop).
// Segments: seg[(l*nseg + i)*6 + {mid xyz, dl xyz}]; whole[7l + {sum of the loop's dl
// xyz, its centre xyz, mean squared distance of its mid-points from the centre}].
//
// Bound by FP64: 27 points (three Gauss points per axis) times nseg segments per
// voxel, each 1/R and exp(-iR).  So the squares of the coordinate differences are
// formed per axis, in units of 1/k0; the moments are summed axis by axis for each
// segment (its dl factors out of the points); and with SMALL (k0 times the distance
// to the voxel's centre point at most 0.05) the phase is the centre's times that of
// R - R_centre, a short series.  About thirty FP64 operations a value instead of
// seventy: 64^3 PWL, four loops of 64 segments, 55.6 -> 31.8 ms.
//
// Rounding: the dl of a closed loop add up to zero, so the field is a small
// difference of the segments' values.  The value at the root mean square distance of
// the voxel's centre from the loop is subtracted from all of them where they are formed
// (an FMA in place of a product) and its part of the sum added at the end, with the dl
// summed on the host: what the sums then round is the difference (error 4.0e-16 of the
// field at 24^3 PWL, 7.8 mm, where the values themselves give 1.4e-15 and plain FP64
// point by point 1.7e-15).  That distance is a typical one at every voxel and never
// small, also where a segment passes through the voxel.
constexpr int kLoopThreads = 128;
constexpr int kLoopTile = 64;      // segments staged in shared memory

template <bool PWL, bool SMALL>
__global__ void __launch_bounds__(kLoopThreads) k_loops(const int64_t* idxS, int64_t Ns, int n1, int n2, double ox,
                                                        double oy, double oz, double res, const double* seg, int nseg,
                                                        const double* whole, const double* qx, const double* qw,
                                                        double k0, double f, zd* out) {
  __shared__ double tile[kLoopTile * 6];
  constexpr int L = PWL ? 4 : 1;
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int l = blockIdx.y;
  const bool on = s < Ns;
  const int64_t g = on ? idxS[s] : 0;
  const int ix = (int)(g % n1), iy = (int)((g / n1) % n2), iz = (int)(g / ((int64_t)n1 * n2));
  const double cx = ox + res * ix, cy = oy + res * iy, cz = oz + res * iz;
  double o[3], w[3], v[3];       // point offsets, weights, weights times the linear moment
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    o[a] = 0.5 * res * k0 * qx[a];
    w[a] = 0.5 * qw[a];
    v[a] = w[a] * (0.5 * qx[a]);
  }
  zd acc[3][L];
#pragma unroll
  for (int p = 0; p < 3; ++p)
#pragma unroll
    for (int q = 0; q < L; ++q) acc[p][q] = zd{0, 0};
  const double* sg = seg + (int64_t)l * nseg * 6;
  double g0x = 0, g0y = 0;       // cos(R)/R and sin(R)/R subtracted from every value
  if (on) {
    const double* m = whole + 7 * l + 3;
    const double dx = cx - m[0], dy = cy - m[1], dz = cz - m[2];
    double R, sn, cs;
    const double iR = inv_sqrt(k0 * k0 * (dx * dx + dy * dy + dz * dz + m[3]), R);
    sin_cos(R, &sn, &cs);
    g0x = cs * iR;
    g0y = sn * iR;
  }
  for (int t0 = 0; t0 < nseg; t0 += kLoopTile) {
    const int nt = min(kLoopTile, nseg - t0);
    __syncthreads();
    for (int i = threadIdx.x; i < nt * 6; i += blockDim.x) tile[i] = sg[6 * t0 + i];
    __syncthreads();
    if (!on) continue;
    for (int i = 0; i < nt; ++i) {
      const double* q = tile + 6 * i;
      double x2[3], y2[3], z2[3];
      // a point's offset is added to the centre's difference: where a segment is near, the
      // coordinates' own rounding does not enter
      const double ex = cx - q[0], ey = cy - q[1], ez = cz - q[2];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const double dx = fma(k0, ex, o[a]), dy = fma(k0, ey, o[a]), dz = fma(k0, ez, o[a]);
        x2[a] = dx * dx;
        y2[a] = dy * dy;
        z2[a] = dz * dz;
      }
      // the middle Gauss point is the centre
      double Rc = 0, sc = 0, cc = 1;
      if (SMALL) {
        inv_sqrt(x2[1] + y2[1] + z2[1], Rc);
        sin_cos(Rc, &sc, &cc);
      }
      double gx[L], gy[L];         // moments of cos(R)/R and sin(R)/R
#pragma unroll
      for (int m = 0; m < L; ++m) gx[m] = gy[m] = 0;
#pragma unroll 1
      for (int a = 0; a < 3; ++a) {
        const double xa = a == 0 ? x2[0] : (a == 1 ? x2[1] : x2[2]);
        double ax = 0, ay = 0, bx = 0, by = 0, dx = 0, dy = 0;
#pragma unroll
        for (int b = 0; b < 3; ++b) {
          const double xy = xa + y2[b];
          double px = 0, py = 0, ux = 0, uy = 0;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            double R, sn, cs;
            const double iR = inv_sqrt(xy + z2[c], R);
            if (SMALL) {
              double st, ct;
              sin_cos_small(R - Rc, &st, &ct);
              cs = fma(cc, ct, -(sc * st));
              sn = fma(sc, ct, cc * st);
            } else {
              sin_cos(R, &sn, &cs);
            }
            cs = fma(cs, iR, -g0x);
            sn = fma(sn, iR, -g0y);
            px = fma(w[c], cs, px);
            py = fma(w[c], sn, py);
            if (PWL && c != 1) {
              ux = fma(v[c], cs, ux);
              uy = fma(v[c], sn, uy);
            }
          }
          ax = fma(w[b], px, ax);
          ay = fma(w[b], py, ay);
          if (PWL) {
            if (b != 1) {
              bx = fma(v[b], px, bx);
              by = fma(v[b], py, by);
            }
            dx = fma(w[b], ux, dx);
            dy = fma(w[b], uy, dy);
          }
        }
        const double wa = a == 1 ? w[1] : w[0], va = a == 0 ? v[0] : (a == 1 ? 0.0 : v[2]);
        gx[0] = fma(wa, ax, gx[0]);
        gy[0] = fma(wa, ay, gy[0]);
        if constexpr (PWL) {
          gx[1] = fma(va, ax, gx[1]);
          gy[1] = fma(va, ay, gy[1]);
          gx[2] = fma(wa, bx, gx[2]);
          gy[2] = fma(wa, by, gy[2]);
          gx[3] = fma(wa, dx, gx[3]);
          gy[3] = fma(wa, dy, gy[3]);
        }
      }
#pragma unroll
      for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int m = 0; m < L; ++m) {
          acc[p][m].x = fma(q[3 + p], gx[m], acc[p][m].x);
          acc[p][m].y = fma(q[3 + p], gy[m], acc[p][m].y);
        }
    }
  }
  if (!on) return;
#pragma unroll
  for (int p = 0; p < 3; ++p) {   // the weights of the constant moment add up to one, of the linear ones to zero
    acc[p][0].x = fma(whole[7 * l + p], g0x, acc[p][0].x);
    acc[p][0].y = fma(whole[7 * l + p], g0y, acc[p][0].y);
  }
  // E = -i omega mu0 sum exp(-ikR)/(4 pi R) dl, f = omega mu0 k0 / (4 pi)
#pragma unroll
  for (int p = 0; p < 3; ++p)
#pragma unroll
    for (int q = 0; q < L; ++q) {
      const double nrm = f * (q == 0 ? 1.0 : 12.0);
      out[(int64_t)l * 3 * L * Ns + (int64_t)(p * L + q) * Ns + s] = zd{-nrm * acc[p][q].y, -nrm * acc[p][q].x};
    }
}

template <bool PWL>
__global__ void k_plane(const int64_t* idxS, int64_t Ns, int n1, int n2, double ox, double oy, double oz, double res,
                        const double* qx, const double* qw, int nq, double k0, zd* out) {
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= Ns) return;
  const int64_t g = idxS[s];
  const int ix = (int)(g % n1), iy = (int)((g / n1) % n2), iz = (int)(g / ((int64_t)n1 * n2));
  const double cx = ox + res * ix, cy = oy + res * iy, cz = oz + res * iz;
  (void)cx; (void)cy;
  constexpr int L = PWL ? 4 : 1;
  zd acc[L];
#pragma unroll
  for (int q = 0; q < L; ++q) acc[q] = zd{0, 0};
  for (int a = 0; a < nq; ++a)
    for (int b = 0; b < nq; ++b)
      for (int c = 0; c < nq; ++c) {
        const double pz = cz + qx[c] * res * 0.5;
        const double wt = qw[a] * qw[b] * qw[c] * 0.125;
        double sn, cs;
        sincos(k0 * pz, &sn, &cs);
        const zd e = {cs, -sn};
        const double fl[4] = {1.0, qx[a] * 0.5, qx[b] * 0.5, qx[c] * 0.5};
#pragma unroll
        for (int q = 0; q < L; ++q) acc[q] = acc[q] + scale(e, wt * fl[q]);
      }
  for (int p = 0; p < 3; ++p)
    for (int q = 0; q < L; ++q) {
      const double nrm = q == 0 ? 1.0 : 12.0;
      out[(int64_t)(p * L + q) * Ns + s] = p == 0 ? scale(acc[q], nrm) : zd{0, 0};
    }
}

}  // namespace marie

using namespace marie;

static marie_status assemble(int32_t n1, int32_t n2, int32_t n3, double res, double freq, int32_t basis,
                             int32_t kernel, bool near_exact, double* out_host) {
  if (n1 < 1 || n2 < 1 || n3 < 1 || !(res > 0) || !(freq > 0) || !out_host || (basis != 0 && basis != 1) ||
      (kernel != 0 && kernel != 1)) {
    set_error("marie_assemble_green: invalid argument");
    return MARIE_ERR_BAD_ARG;
  }
  const bool pwl = basis == MARIE_PWL, isN = kernel == 0;
  const int pwx = pwl ? 10 : 1, nc = isN ? 6 : 3;
  const double c0 = 299792458.0;
  const double k0 = 2 * M_PI / (c0 / freq);
  const int64_t nD = (int64_t)n1 * n2 * n3;
  // rules: 0 far (4^3 x 4^3), 1 medium (8^3 x 8^3 or min(n)), 2 near stand-in (8^3 x 7^3)
  const int thr = isN ? 5 : 2;
  const int Npm = (n1 <= thr || n2 <= thr || n3 <= thr) ? std::min(n1, std::min(n2, n3)) : 8;
  // canonical offsets a >= b >= c of which some permutation lies in the box;
  // the long ones (near stand-in, medium) first, one CTA each
  int ed[3] = {n1, n2, n3};
  std::sort(ed, ed + 3, [](int p, int q) { return p > q; });
  std::vector<int4> offs, far_offs;
  if (!near_exact)
    for (int z = 0; z < std::min(2, n3); ++z)
      for (int y = 0; y < std::min(2, n2); ++y)
        for (int x = 0; x < std::min(2, n1); ++x) offs.push_back(int4{x, y, z, 2});   // unequal rules: no permutations
  for (int a = 0; a < ed[0]; ++a)
    for (int b = 0; b < std::min(a + 1, ed[1]); ++b)
      for (int c = 0; c < std::min(b + 1, ed[2]); ++c) {
        if (a < 2) continue;                     // {0,1}^3: the near zone
        if (a < Npm) offs.push_back(int4{a, b, c, 1 | 8});
        else far_offs.push_back(int4{a, b, c, 0 | 8});
      }
  const int nspec = (int)offs.size();
  offs.insert(offs.end(), far_offs.begin(), far_offs.end());
  if (offs.empty()) offs.push_back(int4{0, 0, 0, 0});
  const int noff = (int)(nspec + far_offs.size());
  std::vector<void*> scratch;
  auto done = [&](marie_status s) {
    cudaDeviceSynchronize();
    for (void* p : scratch) cudaFree(p);
    return s;
  };
  DevRule rules[3];
  marie_status st;
  if ((st = make_rule(4, 4, rules[0], scratch)) != MARIE_OK) return done(st);
  if ((st = make_rule(Npm, Npm, rules[1], scratch)) != MARIE_OK) return done(st);
  if ((st = make_rule(8, 7, rules[2], scratch)) != MARIE_OK) return done(st);
  int4* d_offs = nullptr;
  double *d_out = nullptr, *d_gauss = nullptr, *d_part = nullptr;
  auto alloc = [&](void** p, size_t bytes) {
    if (cudaMalloc(p, bytes) != cudaSuccess) return false;
    scratch.push_back(*p);
    return true;
  };
  if (!alloc((void**)&d_offs, offs.size() * sizeof(int4)) || !alloc((void**)&d_out, (size_t)nD * pwx * nc * sizeof(zd)) ||
      !alloc((void**)&d_gauss, 2 * kNearOrder * sizeof(double)) ||
      !alloc((void**)&d_part, (size_t)8 * 24 * kNearOrder * pwx * nc * sizeof(zd)))
    return done(MARIE_ERR_OOM);
  std::vector<double> gx, gw;
  green_host::gauss01(kNearOrder, gx, gw);
  cudaMemcpy(d_gauss, gx.data(), kNearOrder * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemcpy(d_gauss + kNearOrder, gw.data(), kNearOrder * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemcpy(d_offs, offs.data(), offs.size() * sizeof(int4), cudaMemcpyHostToDevice);
  cudaError_t e;
  if (pwl && isN) e = run_vv<10, 6, true>(d_offs, nspec, noff, rules, near_exact, d_gauss, d_part, res, k0, n1, n2, n3, d_out);
  else if (pwl) e = run_vv<10, 3, false>(d_offs, nspec, noff, rules, near_exact, d_gauss, d_part, res, k0, n1, n2, n3, d_out);
  else if (isN) e = run_vv<1, 6, true>(d_offs, nspec, noff, rules, near_exact, d_gauss, d_part, res, k0, n1, n2, n3, d_out);
  else e = run_vv<1, 3, false>(d_offs, nspec, noff, rules, near_exact, d_gauss, d_part, res, k0, n1, n2, n3, d_out);
  if (e != cudaSuccess) {
    set_error("assembly kernel launch failed");
    return done(MARIE_ERR_CUDA);
  }
  if (cudaMemcpy(out_host, d_out, (size_t)nD * pwx * nc * sizeof(zd), cudaMemcpyDeviceToHost) != cudaSuccess) {
    set_error("assembly: device error %s", cudaGetErrorString(cudaGetLastError()));
    return done(MARIE_ERR_CUDA);
  }
  return done(MARIE_OK);
}

extern "C" marie_status marie_assemble_green(int32_t n1, int32_t n2, int32_t n3, double res, double freq,
                                             int32_t basis, int32_t kernel, double* out_host) {
  return assemble(n1, n2, n3, res, freq, basis, kernel, false, out_host);
}

extern "C" marie_status marie_assemble_green_ex(int32_t n1, int32_t n2, int32_t n3, double res, double freq,
                                                int32_t basis, int32_t kernel, int32_t flags, double* out_host) {
  if (flags & ~(MARIE_GREEN_SELF_POINT_TERM | MARIE_GREEN_NEAR_EXACT)) {
    set_error("marie_assemble_green_ex: unknown flags 0x%x", (unsigned)flags);
    return MARIE_ERR_BAD_ARG;
  }
  MARIE_TRY(assemble(n1, n2, n3, res, freq, basis, kernel, (flags & MARIE_GREEN_NEAR_EXACT) != 0, out_host));
  // the point term of N at the self offset (near_zone_exact holds it too)
  if (kernel == 0 && flags)
    green_host::add_self_point_term(out_host, (int64_t)n1 * n2 * n3, basis == MARIE_PWL ? 10 : 1, res);
  return MARIE_OK;
}

static marie_status quad_rule(int nq, double** qx, double** qw, std::vector<void*>& scratch) {
  std::vector<double> x, w;
  gauss_legendre(nq, x, w);
  if (cudaMalloc(qx, nq * sizeof(double)) != cudaSuccess) return MARIE_ERR_OOM;
  scratch.push_back(*qx);
  if (cudaMalloc(qw, nq * sizeof(double)) != cudaSuccess) return MARIE_ERR_OOM;
  scratch.push_back(*qw);
  cudaMemcpy(*qx, x.data(), nq * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemcpy(*qw, w.data(), nq * sizeof(double), cudaMemcpyHostToDevice);
  return MARIE_OK;
}

extern "C" marie_status marie_incident_loops(marie_vie* h, const double* origin, const double* loops, int32_t nloop,
                                             double radius, int32_t nseg, void* out_dev, void* stream) {
  if (!h || !origin || !loops || nloop < 1 || !(radius > 0) || nseg < 3 || !out_dev) {
    set_error("marie_incident_loops: invalid argument");
    return MARIE_ERR_BAD_ARG;
  }
  // regular nseg-gon inscribed in each circle: mid-points and chord vectors
  std::vector<double> seg((size_t)nloop * nseg * 6 + 7 * (size_t)nloop);
  double* const whole = seg.data() + (size_t)nloop * nseg * 6;
  for (int l = 0; l < nloop; ++l) {
    const double* L = loops + 6 * l;
    double nx = L[3], ny = L[4], nz = L[5];
    const double nn = std::sqrt(nx * nx + ny * ny + nz * nz);
    if (!(nn > 0)) { set_error("loop %d has a zero normal", l); return MARIE_ERR_BAD_ARG; }
    nx /= nn; ny /= nn; nz /= nn;
    double ax = 1, ay = 0, az = 0;
    if (std::fabs(nx) >= 0.9) { ax = 0; ay = 1; }
    // e1 = n x a / |.|, e2 = n x e1
    double e1x = ny * az - nz * ay, e1y = nz * ax - nx * az, e1z = nx * ay - ny * ax;
    const double n1 = std::sqrt(e1x * e1x + e1y * e1y + e1z * e1z);
    e1x /= n1; e1y /= n1; e1z /= n1;
    const double e2x = ny * e1z - nz * e1y, e2y = nz * e1x - nx * e1z, e2z = nx * e1y - ny * e1x;
    for (int i = 0; i < nseg; ++i) {
      const double t0 = 2 * M_PI * i / nseg, t1 = 2 * M_PI * (i + 1) / nseg;
      const double p0x = L[0] + radius * (std::cos(t0) * e1x + std::sin(t0) * e2x);
      const double p0y = L[1] + radius * (std::cos(t0) * e1y + std::sin(t0) * e2y);
      const double p0z = L[2] + radius * (std::cos(t0) * e1z + std::sin(t0) * e2z);
      const double p1x = L[0] + radius * (std::cos(t1) * e1x + std::sin(t1) * e2x);
      const double p1y = L[1] + radius * (std::cos(t1) * e1y + std::sin(t1) * e2y);
      const double p1z = L[2] + radius * (std::cos(t1) * e1z + std::sin(t1) * e2z);
      double* sgp = &seg[((size_t)l * nseg + i) * 6];
      sgp[0] = 0.5 * (p0x + p1x); sgp[1] = 0.5 * (p0y + p1y); sgp[2] = 0.5 * (p0z + p1z);
      sgp[3] = p1x - p0x; sgp[4] = p1y - p0y; sgp[5] = p1z - p0z;
    }
    for (int p = 0; p < 3; ++p) {
      long double sum = 0;
      for (int i = 0; i < nseg; ++i) sum += seg[((size_t)l * nseg + i) * 6 + 3 + p];
      whole[7 * l + p] = (double)sum;
      whole[7 * l + 3 + p] = L[p];
    }
    const double rm = radius * std::cos(M_PI / nseg);
    whole[7 * l + 6] = rm * rm;
  }
  std::vector<void*> scratch;
  auto done = [&](marie_status s) {
    cudaStreamSynchronize((cudaStream_t)stream);
    for (void* p : scratch) cudaFree(p);
    return s;
  };
  double* d_seg = nullptr;
  if (cudaMalloc(&d_seg, seg.size() * sizeof(double)) != cudaSuccess) return done(MARIE_ERR_OOM);
  scratch.push_back(d_seg);
  cudaMemcpy(d_seg, seg.data(), seg.size() * sizeof(double), cudaMemcpyHostToDevice);
  double *qx = nullptr, *qw = nullptr;
  marie_status st;
  if ((st = quad_rule(3, &qx, &qw, scratch)) != MARIE_OK) return done(st);
  const double mu0 = 4e-7 * M_PI;
  const double f = (double)((long double)h->omega * mu0 * h->k0 / (4.0L * 3.141592653589793238462643383279502884L));
  dim3 grid((unsigned)((h->Ns + kLoopThreads - 1) / kLoopThreads), (unsigned)nloop);
  cudaStream_t s = (cudaStream_t)stream;
  // the outermost Gauss point is sqrt(3) * sqrt(0.6) * res / 2 from the centre
  const bool small = 0.671 * h->k0 * h->res <= 0.05;
  auto run = [&](auto kernel) {
    kernel<<<grid, kLoopThreads, 0, s>>>(h->idxS, h->Ns, h->n1, h->n2, origin[0], origin[1], origin[2], h->res, d_seg,
                                         nseg, d_seg + (size_t)nloop * nseg * 6, qx, qw, h->k0, f, (zd*)out_dev);
  };
  if (h->pwl) small ? run(k_loops<true, true>) : run(k_loops<true, false>);
  else small ? run(k_loops<false, true>) : run(k_loops<false, false>);
  g_launches++;
  if (cudaGetLastError() != cudaSuccess) { set_error("incident-field kernel launch failed"); return done(MARIE_ERR_CUDA); }
  return done(MARIE_OK);
}

extern "C" marie_status marie_incident_plane_wave(marie_vie* h, const double* origin, void* out_dev, void* stream) {
  if (!h || !origin || !out_dev) { set_error("marie_incident_plane_wave: invalid argument"); return MARIE_ERR_BAD_ARG; }
  std::vector<void*> scratch;
  auto done = [&](marie_status s) {
    cudaStreamSynchronize((cudaStream_t)stream);
    for (void* p : scratch) cudaFree(p);
    return s;
  };
  double *qx = nullptr, *qw = nullptr;
  marie_status st;
  if ((st = quad_rule(3, &qx, &qw, scratch)) != MARIE_OK) return done(st);
  cudaStream_t s = (cudaStream_t)stream;
  const unsigned gb = (unsigned)((h->Ns + 127) / 128);
  if (h->pwl) k_plane<true><<<gb, 128, 0, s>>>(h->idxS, h->Ns, h->n1, h->n2, origin[0], origin[1], origin[2], h->res, qx, qw, 3, h->k0, (zd*)out_dev);
  else k_plane<false><<<gb, 128, 0, s>>>(h->idxS, h->Ns, h->n1, h->n2, origin[0], origin[1], origin[2], h->res, qx, qw, 3, h->k0, (zd*)out_dev);
  g_launches++;
  if (cudaGetLastError() != cudaSuccess) { set_error("plane-wave kernel launch failed"); return done(MARIE_ERR_CUDA); }
  return done(MARIE_OK);
}
