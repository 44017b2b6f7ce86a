// Block GMRES with few right-hand sides (p <= 16): the tall products of the
// block solver in complex64 with FP32 accumulation.  Included by bgmres.cuh.
//
//   k_tall_cn:   H (M x p) = A^H B    (A: N_b x M, B: N_b x p)
//   k_tall_comb: C (N_b x p) = alpha A X + beta C    (X: M x p)
//
// With p this small both are bound by reading A once (M vectors of N_b), which
// a GEMM's 128-wide tiles of a p-wide result are far from: 48^3 PWL, eight
// right-hand sides, the emulated GEMMs took 0.8 ms for a step's projection and
// update and 1.3 ms for its block QR, two and a half times the operator's 0.95
// ms (the whole solve 947 -> 463 ms, on the operator of that time).  At 240 vectors of 396960 the two take 219 and
// 228 us (HBM alone 116, the FP32 work alone 82): many loads in flight beside the
// arithmetic are what counts, so few registers a thread, and sums over a warp that
// exchange each value once (k_tall_cn with four columns a pass and a butterfly per
// value 266 us; k_tall_comb with half the loads in flight and CTAs of 256 414 us).
#pragma once

namespace marie {

constexpr int kTallMax = 16;          // largest p of these kernels
constexpr int kTallThreads = 256;
constexpr int kTallCtas = 3 * 152;    // most row ranges (partial sums per entry)
constexpr int kCombThreads = 128;

// Rows of B staged in shared memory per piece and columns of A per warp pass.
template <int P>
struct Tall {
  static constexpr int rows = 4096 / P;
  static constexpr int cols = P <= 4 ? 4 : 2;
  static constexpr int ctas = P <= 8 ? 3 : 2;   // per SM, of k_tall_cn
};

// The V (a multiple of 32) values of every lane summed over the warp: value
// lane*V/32 + i ends in a[i] of its lane.  Each step halves the values a lane
// keeps: V - V/32 exchanges, where a butterfly per value takes 5*V.
template <int V>
__device__ __forceinline__ void warp_transpose_sum(float* a, int lane) {
#pragma unroll
  for (int o = 16, h = V / 2; o > 0; o >>= 1, h >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < V / 2; ++i) {
      if (i < h) {
        const float keep = up ? a[i + h] : a[i], send = up ? a[i] : a[i + h];
        a[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
  }
}

// Partial products of the CTA's rows: part[(c*M + m)*gridDim.x + blockIdx.x].
// The CTA stages `rows` rows of B, its warps take groups of `cols` columns of A
// (when there are fewer groups than warps, several warps share a group and split
// the rows), each lane its rows; the warp's sums are added into the CTA's FP32
// accumulators in shared memory.  flag (may be null): set to 2 if a value of B
// is not finite.
template <int P>
__global__ void __launch_bounds__(kTallThreads, Tall<P>::ctas) k_tall_cn(const cplx<float>* __restrict__ A,
                                                          const cplx<float>* __restrict__ B, int64_t Nb, int M, int p,
                                                          cplx<float>* __restrict__ part, int* flag) {
  extern __shared__ __align__(16) unsigned char tall_smem[];
  constexpr int RC = Tall<P>::rows, CW = Tall<P>::cols, V = 2 * CW * P, kWarps = kTallThreads / 32;
  float2* bt = reinterpret_cast<float2*>(tall_smem);        // [P][RC]
  const int ngroups = (M + CW - 1) / CW;
  int split = 1;
  while (split * 2 * ngroups <= kWarps) split *= 2;
  float2* acc = bt + P * RC;                                // [split][M*p]
  for (int i = threadIdx.x; i < split * M * p; i += kTallThreads) acc[i] = make_float2(0.f, 0.f);
  const int64_t per = ((Nb + gridDim.x - 1) / gridDim.x + 31) / 32 * 32;
  const int64_t r0 = blockIdx.x * per, r1 = r0 + per < Nb ? r0 + per : Nb;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float2* A2 = reinterpret_cast<const float2*>(A);
  const float2* B2 = reinterpret_cast<const float2*>(B);
  bool bad = false;
  for (int64_t base = r0; base < r1; base += RC) {
    const int n = (int)(r1 - base < RC ? r1 - base : RC);
    __syncthreads();
    for (int i = threadIdx.x; i < P * RC; i += kTallThreads) {
      const int c = i / RC, r = i - c * RC;
      const float2 v = c < p && r < n ? B2[(int64_t)c * Nb + base + r] : make_float2(0.f, 0.f);
      bad |= !(isfinite(v.x) && isfinite(v.y));
      bt[i] = v;
    }
    __syncthreads();
    // (group, part of the rows) items
    for (int it = warp; it < ngroups * split; it += kWarps) {
      const int g = it % ngroups, sp = it / ngroups;
      const int steps = (n + 31) / 32, per_s = (steps + split - 1) / split;
      const int s0 = sp * per_s, s1 = min(steps, s0 + per_s);
      const float2* a[CW];
#pragma unroll
      for (int k = 0; k < CW; ++k) a[k] = A2 + (int64_t)min(g * CW + k, M - 1) * Nb + base;
      float s[V];
#pragma unroll
      for (int i = 0; i < V; ++i) s[i] = 0.f;
#pragma unroll 4
      for (int st = s0; st < s1; ++st) {
        const int r = st * 32 + lane;
        float2 v[CW];
#pragma unroll
        for (int k = 0; k < CW; ++k) v[k] = r < n ? a[k][r] : make_float2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < P; ++c) {
          const float2 w = bt[c * RC + (r < RC ? r : RC - 1)];
#pragma unroll
          for (int k = 0; k < CW; ++k) {
            float* q = s + 2 * (k * P + c);
            q[0] = fmaf(v[k].x, w.x, fmaf(v[k].y, w.y, q[0]));
            q[1] = fmaf(v[k].x, w.y, fmaf(-v[k].y, w.x, q[1]));
          }
        }
      }
      warp_transpose_sum<V>(s, lane);
#pragma unroll
      for (int i = 0; i < V / 32; ++i) {
        const int id = lane * (V / 32) + i, k = id / (2 * P), c = (id >> 1) % P;
        if (g * CW + k < M && c < p)
          reinterpret_cast<float*>(acc)[2 * ((int64_t)sp * M * p + c * M + g * CW + k) + (id & 1)] += s[i];
      }
    }
  }
  if (__syncthreads_or(bad) && flag && threadIdx.x == 0) *(volatile int*)flag = 2;
  for (int i = threadIdx.x; i < M * p; i += kTallThreads) {
    float2 t = acc[i];
    for (int q = 1; q < split; ++q) {
      t.x += acc[q * M * p + i].x;
      t.y += acc[q * M * p + i].y;
    }
    part[(int64_t)i * gridDim.x + blockIdx.x] = cplx<float>{t.x, t.y};
  }
}

// H[e] = the nparts partial products of entry e, summed in FP64 in a fixed order
// (one warp per entry).
__global__ void k_tall_sum(const cplx<float>* __restrict__ part, int nparts, int n, cplx<float>* __restrict__ H) {
  const int e = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (e >= n) return;
  double x = 0, y = 0;
  for (int q = lane; q < nparts; q += 32) {
    const cplx<float> v = part[(int64_t)e * nparts + q];
    x += v.x;
    y += v.y;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    x += __shfl_xor_sync(0xffffffffu, x, o);
    y += __shfl_xor_sync(0xffffffffu, y, o);
  }
  if (lane == 0) H[e] = cplx<float>{(float)x, (float)y};
}

// C_c[i] = alpha * sum_m A_m[i] X[m + M*c] + beta * C_c[i], two rows per thread
// (each coefficient read from shared memory serves both); beta 0 or 1.
template <int P>
__global__ void __launch_bounds__(kCombThreads) k_tall_comb(const cplx<float>* __restrict__ A,
                                                            const cplx<float>* __restrict__ X, int64_t Nb, int M,
                                                            int p, float alpha, float beta, cplx<float>* C) {
  extern __shared__ __align__(16) unsigned char tall_smem[];
  float2* x = reinterpret_cast<float2*>(tall_smem);         // [M][P]
  for (int i = threadIdx.x; i < M * P; i += kCombThreads) {
    const int m = i / P, c = i - m * P;
    const cplx<float> v = c < p ? X[m + (int64_t)M * c] : cplx<float>{0.f, 0.f};
    x[i] = make_float2(alpha * v.x, alpha * v.y);
  }
  __syncthreads();
  const int64_t stride = (int64_t)gridDim.x * kCombThreads * 2;
  for (int64_t i0 = (int64_t)blockIdx.x * kCombThreads * 2 + threadIdx.x; i0 < Nb; i0 += stride) {
    const int64_t i1 = i0 + kCombThreads;
    const bool two = i1 < Nb;
    float2 s[2][P];
#pragma unroll
    for (int c = 0; c < P; ++c) {
      s[0][c] = s[1][c] = make_float2(0.f, 0.f);
      if (beta != 0.f && c < p) {
        const cplx<float> u = C[(int64_t)c * Nb + i0];
        s[0][c] = make_float2(u.x, u.y);
        if (two) {
          const cplx<float> t = C[(int64_t)c * Nb + i1];
          s[1][c] = make_float2(t.x, t.y);
        }
      }
    }
#pragma unroll 8
    for (int m = 0; m < M; ++m) {
      const cplx<float> u = A[(int64_t)m * Nb + i0];
      const cplx<float> t = two ? A[(int64_t)m * Nb + i1] : cplx<float>{0.f, 0.f};
#pragma unroll
      for (int c = 0; c < P; ++c) {
        const float2 w = x[m * P + c];
        s[0][c].x = fmaf(u.x, w.x, fmaf(-u.y, w.y, s[0][c].x));
        s[0][c].y = fmaf(u.x, w.y, fmaf(u.y, w.x, s[0][c].y));
        s[1][c].x = fmaf(t.x, w.x, fmaf(-t.y, w.y, s[1][c].x));
        s[1][c].y = fmaf(t.x, w.y, fmaf(t.y, w.x, s[1][c].y));
      }
    }
#pragma unroll
    for (int c = 0; c < P; ++c) {
      if (c >= p) break;
      C[(int64_t)c * Nb + i0] = cplx<float>{s[0][c].x, s[0][c].y};
      if (two) C[(int64_t)c * Nb + i1] = cplx<float>{s[1][c].x, s[1][c].y};
    }
  }
}

// Shared memory of the two kernels; M beyond it goes to cuBLAS.
template <int P>
inline size_t tall_cn_smem(int M, int p) { return (size_t)(P * Tall<P>::rows + std::max(M * p, 8 * 2 * Tall<P>::cols * p)) * 8; }
template <int P>
inline size_t tall_comb_smem(int M) { return (size_t)M * P * 8; }

template <int P>
static marie_status tall_cn(int64_t Nb, int M, int p, const cplx<float>* A, const cplx<float>* B, cplx<float>* H,
                            cplx<float>* part, int64_t part_cap, int* flag, cudaStream_t s) {
  static std::atomic<uint64_t> done{0};
  smem_opt_in_device((const void*)k_tall_cn<P>, done);
  const int64_t rows = std::min<int64_t>(Tall<P>::ctas * 152, (Nb + 255) / 256);
  const int ctas = (int)std::min<int64_t>(rows, part_cap / ((int64_t)M * p));
  k_tall_cn<P><<<ctas, kTallThreads, tall_cn_smem<P>(M, p), s>>>(A, B, Nb, M, p, part, flag);
  MARIE_LAUNCH_CHECK();
  k_tall_sum<<<(M * p + 7) / 8, 256, 0, s>>>(part, ctas, M * p, H);
  MARIE_LAUNCH_CHECK();
  return MARIE_OK;
}
template <int P>
static marie_status tall_comb(int64_t Nb, int M, int p, float alpha, const cplx<float>* A, const cplx<float>* X,
                              float beta, cplx<float>* C, cudaStream_t s) {
  static std::atomic<uint64_t> done{0};
  smem_opt_in_device((const void*)k_tall_comb<P>, done);
  const int64_t need = (Nb + 2 * kCombThreads - 1) / (2 * kCombThreads);
  k_tall_comb<P><<<(unsigned)std::min<int64_t>(need, 16 * 152), kCombThreads, tall_comb_smem<P>(M), s>>>(
      A, X, Nb, M, p, alpha, beta, C);
  MARIE_LAUNCH_CHECK();
  return MARIE_OK;
}

static bool tall_fits(int64_t M, int p) {
  return p <= kTallMax && tall_cn_smem<16>((int)std::min<int64_t>(M, 1 << 20), p) <= kSmemOptin &&
         tall_comb_smem<16>((int)std::min<int64_t>(M, 1 << 20)) <= kSmemOptin;
}
static marie_status tall_cn(int64_t Nb, int M, int p, const cplx<float>* A, const cplx<float>* B, cplx<float>* H,
                            cplx<float>* part, int64_t part_cap, int* flag, cudaStream_t s) {
  if (p <= 4) return tall_cn<4>(Nb, M, p, A, B, H, part, part_cap, flag, s);
  if (p <= 8) return tall_cn<8>(Nb, M, p, A, B, H, part, part_cap, flag, s);
  return tall_cn<16>(Nb, M, p, A, B, H, part, part_cap, flag, s);
}
static marie_status tall_comb(int64_t Nb, int M, int p, float alpha, const cplx<float>* A, const cplx<float>* X,
                              float beta, cplx<float>* C, cudaStream_t s) {
  if (p <= 4) return tall_comb<4>(Nb, M, p, alpha, A, X, beta, C, s);
  if (p <= 8) return tall_comb<8>(Nb, M, p, alpha, A, X, beta, C, s);
  return tall_comb<16>(Nb, M, p, alpha, A, X, beta, C, s);
}

}  // namespace marie
