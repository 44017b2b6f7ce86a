// Four-step z pass of the complex64 operator (n3 = 16*NB) in packed FP32
// pairs: one task carries the even- and odd-frequency halves of the
// zero-padded 2N-point transform in the two lanes of every value (pair.cuh),
// so each complex operation of the z-DFTs and of the Green block product is
// issued once for both halves.
// A length-N transform is split N = P x Q, {P, Q} = {NB, 16} (ZpSplit): input
// slice z = Q*a + b, frequency k = j + P*k2; step 1 is the P-point DFT over a of
// slice group b, then the twiddle w_N^(b*j), step 2 the Q-point DFT over b.
// Shared memory: sequence (c, e) of the tile (component c, tile element e)
// starts at (c*W + e)*S; its N positions hold 16-byte pairs (re_even, re_odd,
// im_even, im_odd).  Pair (j, i), i = b before step 2 and k2 after it, sits at
// row*16 + (col ^ row) with row the NB-side index and col the 16-side one; with
// S = N + 2 (N + 8/W for W < 4) the eight lanes of every quarter-warp of a
// 128-bit access (four elements and two neighbouring b or j, or eight columns)
// fall on distinct 16-byte bank groups in all five phases.
//
// Green spectrum: octant columns (kyo <= n2, kxo <= n1) in pair layout: for a
// column, block blk and place p = row*16 + col (zp_freq), one 16-byte entry (re
// G(2k), re G(2k+1), im G(2k), im G(2k+1)) at ((kyo*(n1+1) + kxo)*U + blk)*N + p.
// The mirrored columns are the same values
// between sign changes of the components (mirror_mask), applied where the
// inputs enter and the outputs leave.
//
// Measured against the kernel before it (full spectrum, one tile per CTA, rows
// of kx in S), ellipsoids that leave 5% of the slices empty: 96^3 PWL one right-hand
// side 0.814 -> 0.532 ms, 128^3 PWL sixteen 21.3 -> 18.1 ms, 112^3 PWC seven 1.38 ->
// 1.08 ms.  What bounds it: at few
// right-hand sides the Green columns were (a quarter of them is read now), then
// the data path of shared memory and L1 (60-70% busy: 13 thousand clocks a
// 128^3 PWL tile, 6 of them the product's inputs and Green values) and the FMA
// pipe (45%), in phases separated by barriers:
//  * a column's slices are contiguous in S (z, then right-hand side), so a
//    warp's access in steps 1 and B is one run of 256 bytes;
//  * each CTA walks tiles and loads the next tile's first inputs into
//    registers during the last inverse step (a task of step B and the same task
//    of the next tile's step 1 own the same place in shared memory, so no
//    barrier stands between them);
//  * tasks are small enough for 128 registers, sixteen warps an SM (a few of them
//    spill: 8 to 28 bytes a thread at n3 = 64 and more, 20 to 150 at 16 to 48, whose
//    tasks hold sixteen inputs at once);
//  * the product gives a thread the outputs of one moment l (of the three
//    vector components) for two elements that share their Green column, and
//    loads the Green values of its next input moment while it multiplies by the
//    current ones.
#pragma once

#include "fastpath.cuh"
#include "matvec4.cuh"
#include "pair.cuh"

namespace marie {

// Bulk prefetch of [p, p + bytes) into L2 (no data returned to the SM);
// p and bytes multiples of 16.
__device__ __forceinline__ void prefetch_l2_bulk(const void* p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

__device__ __forceinline__ cp lds_cp(const cp* p) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  return cp{f2{v.x}, f2{v.y}};
}
__device__ __forceinline__ void sts_cp(cp* p, cp v) {
  *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(v.re.v, v.im.v);
}

__device__ __forceinline__ float flip_sign(float v, unsigned m) { return __uint_as_float(__float_as_uint(v) ^ m); }

// One Green value in the lanes (G(2k), G(2k+1)), conj(g) in the adjoint, times
// a sign known at compile time.
template <bool CONJ, bool NEG>
struct ZGreen {
  f2 gr, gi, ngi;
  __device__ __forceinline__ explicit ZGreen(const float4& v) {
    constexpr unsigned sr = NEG ? 0x80000000u : 0u, si = sr ^ (CONJ ? 0x80000000u : 0u), sn = si ^ 0x80000000u;
    gr = f2_make(flip_sign(v.x, sr), flip_sign(v.y, sr));
    gi = f2_make(flip_sign(v.z, si), flip_sign(v.w, si));
    ngi = f2_make(flip_sign(v.z, sn), flip_sign(v.w, sn));
  }
  // y += g x:  re += gr*xr - gi*xi,  im += gr*xi + gi*xr
  __device__ __forceinline__ void add(cp& y, const cp& x) const {
    y.re = fma2(gr, x.re, fma2(ngi, x.im, y.re));
    y.im = fma2(gr, x.im, fma2(gi, x.re, y.im));
  }
};

// PWC: the 3 x 3 product of one frequency pair of one element.
template <int OP, int K>
__device__ __forceinline__ void zentry_pwc(cp* y, const cp* x, const float4* g) {
  constexpr OpEntry e = OpTab<false, OP>::L.e[K];
  ZGreen<(OP & 1) != 0, (e.sgn < 0)>(g[e.blk]).add(y[e.p], x[e.q]);
}
template <int OP, int... Ks>
__device__ __forceinline__ void zpoint_pwc(std::integer_sequence<int, Ks...>, cp* v, int qstride, const float4* g) {
  const f2 zero = f2_make(0.f, 0.f);
  cp x[3], y[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    x[q] = lds_cp(v + q * qstride);
    y[q] = cp{zero, zero};
  }
  (zentry_pwc<OP, Ks>(y, x, g), ...);
#pragma unroll
  for (int p = 0; p < 3; ++p) sts_cp(v + p * qstride, y[p]);
}

// PWL: Tucker index of the moment pair (l, l') (LLP without its signs) and
// whether the entry is negative: N, K: l' = 0 < l; adjoint: l = 0 < l'.
__device__ __forceinline__ int ll_index(int l, int lp) {
  return l == lp ? l : (l == 0 || lp == 0 ? l + lp + 3 : l + lp + 4);
}
template <int OP>
__device__ __forceinline__ bool ll_negative(int l, int lp) {
  return (OP & 1) ? (l == 0 && lp > 0) : (lp == 0 && l > 0);
}
// component of the vector pair (P, Q) and its sign: N symmetric, K the third
// axis, - for Q = P + 1 (cyclic) and, in the adjoint, the other way round
template <int OP>
__device__ __forceinline__ constexpr int pq_comp(int P, int Q) {
  return OP >= 2 ? 3 - P - Q : P + Q + ((P > 0 && Q > 0) ? 1 : 0);
}
template <int OP>
__device__ __forceinline__ constexpr bool pq_negative(int P, int Q) {
  return OP >= 2 && ((Q == (P + 1) % 3) != ((OP & 1) != 0));
}

// y[2P + e] += sum over Q of G_(P,Q) x_Q for one input moment and two elements
// (stride S); xq: element 0 of component l'; QS: stride of the vector index Q.
template <int OP>
__device__ __forceinline__ void zstage_pwl(cp* y, const float4* g, const cp* xq, int S, int QS) {
#pragma unroll
  for (int Q = 0; Q < 3; ++Q) {
    const cp x0 = lds_cp(xq + Q * QS), x1 = lds_cp(xq + Q * QS + S);
#pragma unroll
    for (int P = 0; P < 3; ++P) {
      if (OP >= 2 && P == Q) continue;
      if (pq_negative<OP>(P, Q)) {
        const ZGreen<(OP & 1) != 0, true> G(g[pq_comp<OP>(P, Q)]);
        G.add(y[2 * P], x0);
        G.add(y[2 * P + 1], x1);
      } else {
        const ZGreen<(OP & 1) != 0, false> G(g[pq_comp<OP>(P, Q)]);
        G.add(y[2 * P], x0);
        G.add(y[2 * P + 1], x1);
      }
    }
  }
}

__device__ __forceinline__ void bar_named(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// 512 threads an SM (zp_threads): 128 registers.  Steps 1 and B have C*W*Q tasks,
// steps 2 and A C*W*P (768 and 384 at 128^3).

// An element of a tile: its first value in S (-1: no such column) and its
// components' sign changes (bit 31: one more of all outputs).
struct __align__(16) ZpElem {
  long long off;
  unsigned flips;
  int kxo;
};
struct ZpTile {
  int kyo, kx0, first, more;   // first: starts a column; more: there is such a tile
};

template <int NB, bool PWL, int OP>
__global__ void __launch_bounds__(zp_threads(NB, PWL), 512 / zp_threads(NB, PWL)) k4_zp(MvArgs<float> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int N = 16 * NB, kZpThreads = zp_threads(NB, PWL);
  constexpr int C = PWL ? 12 : 3;
  constexpr int NE = OpTab<PWL, OP>::NE;
  constexpr int U = OpTab<PWL, OP>::L.nblk;
  constexpr int P = zp_outer(NB), Q = N / P;
  constexpr bool wide = P == 16;                // the 16-side index is j, not b
  constexpr int A = P >= 5 ? 1 : 2;             // step 1 tasks of a thread whose inputs are in flight
  const int n1 = a.n1, n2 = a.n2, g3 = a.g3, R = a.R;
  const int W = a.TX * R;                       // a power of two
  const ZpTiles zt = kzp_tiles(n1, n2, W, R, (a.nrhs + R - 1) / R);
  const int lgW = zt.lgW, lgR = zt.lgR;
  const int S = kzp_stride(N, W);
  const int T1 = C * W * Q;                     // tasks of forward step 1 / inverse step B
  const int T2 = C * W * P;                     // tasks of forward step 2 / inverse step A
  // pair (j, i) of a sequence, and twiddle w_N^(i*j) (neighbouring i and
  // neighbouring j on different banks)
  auto place = [](int j, int i) { return wide ? zpos(i, j) : zpos(j, i); };
  auto twid = [](int j, int i) { return wide ? i * 18 + j : j * 18 + i; };
  // four-step twiddles; w_2N^z; live slices Q*a + b of group b as bits a; the
  // elements of this and the next tile
  float2* tws = reinterpret_cast<float2*>(smem_raw);
  float2* tw2s = tws + 18 * NB;
  unsigned* zqs = reinterpret_cast<unsigned*>(tw2s + N);     // [16]
  ZpElem* elem = reinterpret_cast<ZpElem*>(zqs + 16);        // [2][16]
  ZpTile* info = reinterpret_cast<ZpTile*>(elem + 32);       // [2]
  cp* buf = reinterpret_cast<cp*>(info + 2);
  for (int i = threadIdx.x; i < 18 * NB; i += blockDim.x) {
    const int m = i / 18, k = i - 18 * m;
    const cplx<float> w = k < 16 ? a.az.tw[m * k] : cplx<float>{0.f, 0.f};
    tws[i] = make_float2(w.x, w.y);
  }
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    const cplx<float> t2 = a.az.tw2[i];
    tw2s[i] = make_float2(t2.x, t2.y);
  }
  if (threadIdx.x < Q) {
    unsigned m = 0;
    for (int q = 0; q < P; ++q) {
      const int z = Q * q + (int)threadIdx.x;
      if (z < g3 && z_is_live(a, z)) m |= 1u << q;
    }
    zqs[threadIdx.x] = m;
  }
  const int64_t colR = (int64_t)g3 * R;                      // one column of one component
  const int64_t cstride = (int64_t)2 * n2 * 2 * n1 * colR;

  // The last warp walks the CTA's tiles blockIdx.x, + gridDim.x, ...: octant columns
  // kx0.. of row kyo, mirrors outside the tile's own (m), bundle bu, advanced
  // digit by digit (divisions by run-time values cost a thousand clocks here).
  // Tiles without work are passed over: a bundle whose right-hand sides are all
  // inactive, the mirror of a self-mirror frequency.
  struct Digits {
    int bu, m, kx, ky;
  };
  const int nm = zt.nsub / zt.nb;
  auto digits = [&](int t) {
    const int q = t / zt.nsub, sub = t - q * zt.nsub, m = sub / zt.nb, ky = q / zt.ncx;
    return Digits{sub - m * zt.nb, m, q - ky * zt.ncx, ky};
  };
  Digits at = digits(blockIdx.x);
  const Digits step = digits(gridDim.x);
  auto find = [&](bool advance, int u) {
    const int lane = threadIdx.x & 31;
    bool tmx = false, tmy = false;
    for (;; advance = true) {
      if (advance) {
        at.bu += step.bu;
        int carry = at.bu >= zt.nb;
        at.bu -= carry ? zt.nb : 0;
        at.m += step.m + carry;
        carry = at.m >= nm;
        at.m -= carry ? nm : 0;
        at.kx += step.kx + carry;
        carry = at.kx >= zt.ncx;
        at.kx -= carry ? zt.ncx : 0;
        at.ky += step.ky + carry;
      }
      if (at.ky > n2) break;
      tmx = !zt.mx && (at.m & 1);
      tmy = zt.mx ? (!zt.my && (at.m & 1)) : (at.m >> 1) != 0;
      if (tmx && (at.kx == 0 || at.kx == n1)) continue;
      if (tmy && (at.ky == 0 || at.ky == n2)) continue;
      if (a.active == nullptr || bundle_active(a, at.bu)) break;
    }
    const bool more = at.ky <= n2;
    const int kyo = at.ky, kx0 = at.kx * zt.cols, bu = at.bu;
    if (lane == 0) info[u] = ZpTile{kyo, kx0, bu == 0 && at.m == 0, more};
    if (lane < W) {
      const int em = lane >> lgR;
      const bool mx = zt.mx ? (em & 1) != 0 : tmx;
      const bool my = zt.my ? (em & 2) != 0 : tmy;
      const int kxo = kx0 + (zt.my ? em >> 2 : 0);
      const bool ok = more && kxo <= n1 && !(mx && (kxo == 0 || kxo == n1)) &&
                      !(my && (kyo == 0 || kyo == n2));
      const int kx = mx ? 2 * n1 - kxo : kxo, kxp = (kx & 1) * n1 + (kx >> 1);
      const int ky = my ? 2 * n2 - kyo : kyo, kyp = (ky & 1) * n2 + (ky >> 1);
      ZpElem el;
      el.off = ok ? (int64_t)bu * C * cstride + ((int64_t)kyp * 2 * n1 + kxp) * colR + (lane & (R - 1)) : -1;
      el.flips = mirror_flips<PWL>(mx, my);
      if (OP >= 2 && mx != my) el.flips |= 0x80000000u;    // K: one more sign
      el.kxo = min(kxo, n1);
      elem[u * 16 + lane] = el;
    }
  };
  // Tasks: lanes are four elements (e_lo), then the group i of the sequence (of
  // n: slice groups b in steps 1 and B, j in steps 2 and A), then the elements'
  // high bits and the component, so that a warp's access to S is runs of 64
  // bytes or more and its accesses to shared memory spread over all banks.
  const int lgE = lgW < 2 ? lgW : 2;
  auto task = [&](int t, int n, int& i, int& e, int& c) {
    const int r = t >> lgE, q = r / n;
    i = r - q * n;
    e = (t & ((1 << lgE) - 1)) | ((q & ((W >> lgE) - 1)) << lgE);
    c = q >> (lgW - lgE);
  };
  // inputs of step 1 task t of tile u: slices z = Q*q + b
  auto fetch = [&](int t, int u, float2* x) {
    int b, e, c;
    task(t, Q, b, e, c);
    const long long off = elem[u * 16 + e].off;
    const unsigned live = off >= 0 ? zqs[b] : 0u;
    const float2* src = reinterpret_cast<const float2*>(a.S) + (off >= 0 ? off + c * cstride : 0) + b * R;
#pragma unroll
    for (int q = 0; q < P; ++q) x[q] = ((live >> q) & 1u) ? src[Q * q * R] : make_float2(0.f, 0.f);
  };

  int u = 0;
  __syncthreads();
  if (threadIdx.x >= kZpThreads - 32) find(false, 0);
  __syncthreads();
  if (!info[0].more) return;
  float2 pre[A][P];
#pragma unroll
  for (int i = 0; i < A; ++i)
    if ((int)threadIdx.x + i * kZpThreads < T1) fetch(threadIdx.x + i * kZpThreads, 0, pre[i]);

  for (;; u ^= 1) {
    const ZpTile cur = info[u];
    // the column's Green rows (U blocks x N pairs x 16 bytes, contiguous)
    // start towards L2 with the first tile that uses them
    if (cur.first) {
      const int64_t colb = (int64_t)U * N * 16;
      const unsigned piece = (unsigned)(colb / 8);      // U * N * 2 bytes: a multiple of 16
      const int ncol = min(zt.cols, n1 + 1 - cur.kx0);
      const char* col = reinterpret_cast<const char*>(a.G) + ((int64_t)cur.kyo * (n1 + 1) + cur.kx0) * colb;
      for (int c = threadIdx.x; c < ncol * 8; c += blockDim.x) prefetch_l2_bulk(col + (int64_t)c * piece, piece);
    }
    // forward step 1: lanes (even half, odd half = inputs times w_2N^z) of the
    // P-point DFT, then the four-step twiddle (the same for both halves)
    float2 w2[P], w4[P];
    auto twiddles = [&](int b) {
#pragma unroll
      for (int q = 0; q < P; ++q) {
        w2[q] = tw2s[Q * q + b];
        w4[q] = tws[twid(q, b)];
      }
    };
    if constexpr (!wide) twiddles((threadIdx.x >> lgE) & 15);   // Q = 16: b is the same in all of a thread's tasks
    for (int t0 = threadIdx.x; t0 < T1; t0 += A * kZpThreads) {
#pragma unroll
      for (int i = 0; i < A; ++i) {
        const int t = t0 + i * kZpThreads;
        if (t >= T1) break;
        int b, e, c;
        task(t, Q, b, e, c);
        const unsigned neg = (elem[u * 16 + e].flips >> c) << 31;
        float2 in[P];
#pragma unroll
        for (int q = 0; q < P; ++q) in[q] = pre[i][q];
        if (t + A * kZpThreads < T1) fetch(t + A * kZpThreads, u, pre[i]);
        cp v[P];
#pragma unroll
        for (int q = 0; q < P; ++q) {
          const float2 x = make_float2(flip_sign(in[q].x, neg), flip_sign(in[q].y, neg));
          const float2 w = wide ? tw2s[Q * q + b] : w2[q];
          v[q] = cp{f2_make(x.x, x.x * w.x - x.y * w.y), f2_make(x.y, x.x * w.y + x.y * w.x)};
        }
        dftp<false, P>(v);
        cp* d = buf + (c * W + e) * S;
        sts_cp(d + place(0, b), v[0]);
#pragma unroll
        for (int j = 1; j < P; ++j) {
          const float2 w = wide ? tws[twid(j, b)] : w4[j];
          sts_cp(d + place(j, b), tw_mul(v[j], f2_bc(w.x), f2_bc(w.y), f2_bc(-w.y)));
        }
      }
    }
    __syncthreads();
    // forward step 2 (in place): task (j, e, c); Q-point DFT over b.  The last
    // warp, which has one task less than the first where T2 is no multiple of
    // the block size, finds the next tile.  (N = 16: Q = 1, nothing to do here or in
    // inverse step A; with both passing over the tile all the same 16 x 32 x 16,
    // sixteen right-hand sides, PWL 87.4 us, now 82.5, PWC 39.0, now 36.2.)
    if constexpr (Q > 1) {
      for (int t = threadIdx.x; t < T2; t += blockDim.x) {
        int j, e, c;
        task(t, P, j, e, c);
        cp* p = buf + (c * W + e) * S;
        cp v[Q];
#pragma unroll
        for (int b = 0; b < Q; ++b) v[b] = lds_cp(p + place(j, b));
        dftp<false, Q>(v);
#pragma unroll
        for (int k2 = 0; k2 < Q; ++k2) sts_cp(p + place(j, k2), v[k2]);
      }
    }
    if (threadIdx.x >= kZpThreads - 32) find(true, u ^ 1);
    if constexpr (Q > 1) __syncthreads();

    // Green block product: place p = row*16 + col of every component at
    // zpos(row, col).
    const float4* gcol = reinterpret_cast<const float4*>(a.G) + (int64_t)cur.kyo * (n1 + 1) * U * N;
    if constexpr (PWL) {
      // Item (p, pair of elements): sixteen p per half-warp, the W/2 pairs of a
      // block of sixteen next to each other.  Four warps l = 0..3 take a block
      // of 32 items: they read all twelve inputs, meet, and write their three
      // outputs in place.  The two sets of four warps take blocks in turn.
      constexpr int NC = OP >= 2 ? 3 : 6;
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l = warp & 3, set = warp >> 2;
      const int nblk = NB * (W >> 2);
      // element pair and place of block blk; a block past the end repeats the last
      auto item = [&](int blk, int& e, int& j) {
        const int u16 = 2 * min(blk, nblk - 1) + (lane >> 4);
        j = u16 >> (lgW - 1);
        e = 2 * (u16 - (j << (lgW - 1)));
        return gcol + (int64_t)elem[u * 16 + e].kxo * U * N + j * 16 + (lane & 15);
      };
      float4 g[NC];
      int e, j;
      const float4* gp = item(set, e, j);
#pragma unroll
      for (int c = 0; c < NC; ++c) g[c] = __ldg(gp + (ll_index(l, 0) * NC + c) * N);
      for (int blk = set; blk < nblk; blk += 2) {
        cp* v = buf + e * S + zpos(j, lane & 15);
        cp y[6];
        const f2 zero = f2_make(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 6; ++i) y[i] = cp{zero, zero};
#pragma unroll
        for (int lp = 0; lp < 4; ++lp) {
          if (lp == 3) gp = item(blk + 2, e, j);
          float4 gn[NC];
#pragma unroll
          for (int c = 0; c < NC; ++c) gn[c] = __ldg(gp + (ll_index(l, (lp + 1) & 3) * NC + c) * N);
          if (ll_negative<OP>(l, lp)) {
#pragma unroll
            for (int c = 0; c < NC; ++c) g[c] = make_float4(-g[c].x, -g[c].y, -g[c].z, -g[c].w);
          }
          zstage_pwl<OP>(y, g, v + lp * W * S, S, 4 * W * S);
#pragma unroll
          for (int c = 0; c < NC; ++c) g[c] = gn[c];
        }
        bar_named(1 + set, 128);
#pragma unroll
        for (int P = 0; P < 3; ++P) {
          sts_cp(v + (4 * P + l) * W * S, y[2 * P]);
          sts_cp(v + (4 * P + l) * W * S + S, y[2 * P + 1]);
        }
      }
    } else {
      // Item (p, group of up to four elements that share their column), p
      // fastest; the next item's Green values load meanwhile.
      const int eg = 1 << lgE, items = N * (W >> lgE);
      auto item = [&](int i, int& e, int& p) {
        i = min(i, items - 1);
        const int g = i / N;
        p = i - g * N;
        e = g << lgE;
        return gcol + (int64_t)elem[u * 16 + e].kxo * U * N + p;
      };
      int e, p;
      const float4* gp = item(threadIdx.x, e, p);
      float4 g[U];
#pragma unroll
      for (int j = 0; j < U; ++j) g[j] = __ldg(gp + j * N);
      for (int i = threadIdx.x; i < items; i += blockDim.x) {
        cp* v = buf + e * S + zpos(p >> 4, p & 15);
        gp = item(i + blockDim.x, e, p);
        float4 gn[U];
#pragma unroll
        for (int j = 0; j < U; ++j) gn[j] = __ldg(gp + j * N);
        for (int q = 0; q < eg; ++q) zpoint_pwc<OP>(std::make_integer_sequence<int, NE>{}, v + q * S, W * S, g);
#pragma unroll
        for (int j = 0; j < U; ++j) g[j] = gn[j];
      }
    }
    __syncthreads();
    // inverse step A (in place): task (j, e, c); inverse Q-point DFT over k2
    // and the conjugate four-step twiddle
    if constexpr (Q > 1) {
      for (int t = threadIdx.x; t < T2; t += blockDim.x) {
        int j, e, c;
        task(t, P, j, e, c);
        cp* p = buf + (c * W + e) * S;
        cp v[Q];
#pragma unroll
        for (int k2 = 0; k2 < Q; ++k2) v[k2] = lds_cp(p + place(j, k2));
        dftp<true, Q>(v);
        sts_cp(p + place(j, 0), v[0]);
#pragma unroll
        for (int b = 1; b < Q; ++b) {
          const float2 q = tws[twid(j, b)];
          sts_cp(p + place(j, b), tw_mulc(v[b], f2_bc(q.x), f2_bc(q.y), f2_bc(-q.y)));
        }
      }
      __syncthreads();
    }
    // inverse step B: task as in step 1, inverse P-point DFT of both halves;
    // output z = Q*q + b is even(q) + odd(q) * conj(w_2N^z).  The last tasks of a
    // thread start the loads of its first tasks of the next tile.
    const bool more = info[u ^ 1].more;
    if constexpr (!wide) twiddles((threadIdx.x >> lgE) & 15);
    for (int t0 = threadIdx.x; t0 < T1; t0 += A * kZpThreads) {
#pragma unroll
      for (int i = 0; i < A; ++i) {
        const int t = t0 + i * kZpThreads;
        if (t >= T1) break;
        int b, e, c;
        task(t, Q, b, e, c);
        const cp* sp = buf + (c * W + e) * S;
        cp v[P];
#pragma unroll
        for (int j = 0; j < P; ++j) v[j] = lds_cp(sp + place(j, b));
        if (more && t + A * kZpThreads >= T1) fetch(threadIdx.x + i * kZpThreads, u ^ 1, pre[i]);
        dftp<true, P>(v);
        const ZpElem el = elem[u * 16 + e];
        const unsigned live = el.off >= 0 ? zqs[b] : 0u;
        const unsigned neg = ((el.flips >> c) << 31) ^ (el.flips & 0x80000000u);
        cplx<float>* dst = a.S + (el.off + c * cstride + b * R);
#pragma unroll
        for (int q = 0; q < P; ++q) {
          float ar, br, ai, bi;
          f2_split(v[q].re, ar, br);
          f2_split(v[q].im, ai, bi);
          const float2 w = wide ? tw2s[Q * q + b] : w2[q];
          const float ox = fmaf(br, w.x, fmaf(bi, w.y, ar)), oy = fmaf(bi, w.x, fmaf(-br, w.y, ai));
          if ((live >> q) & 1u) dst[Q * q * R] = cplx<float>{flip_sign(ox, neg), flip_sign(oy, neg)};
        }
      }
    }
    if (!more) break;
  }
}

}  // namespace marie
