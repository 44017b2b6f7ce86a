// Launch code of the four-step matvec passes (xy4c, xy4f, matvec4, kz4p, kz4f, kz4).
//
// The per-pass launchers (switch over NB = n/16) are declared here and
// defined in fastpath_impl.cuh, so that one precision's kernels can be spread
// over several translation units that compile in parallel (the float-float
// kernels: x and y passes in two units, the z pass in one object per NB).
#pragma once

#include <algorithm>

#include "internal.h"

namespace marie {

__host__ __device__ constexpr int kz4_stride(int N, int W) { return N + (W >= 16 ? 1 : 16 / W); }
__host__ __device__ constexpr int kz4_halfpad(int W) { return W >= 16 ? 0 : 8 / W; }

// Float-float x and y passes (xy4f.cuh): twiddles (32 bytes each), sequence stride
// in 16-byte elements, and shared memory of a tile of w lines.
__host__ __device__ constexpr int xyf_tw(int n) { return 31 * (n / 16); }
__host__ __device__ constexpr int xyf_stride(int n) { return n + 5; }
__host__ __device__ constexpr size_t xyf_smem(int n, int w) {
  return (size_t)32 * xyf_tw(n) + (size_t)2 * w * xyf_stride(n) * 16;
}

// Sequence stride of k4_zp (complex64, packed pairs) in 16-byte pairs.
__host__ __device__ constexpr int kzp_stride(int N, int W) { return N + (W >= 4 ? 2 : 8 / W); }
// k4_zf (float-float, 16-byte elements): sequence stride, and pad of a quarter of
// a sequence, per tile width (with eight elements or more those alone spread).
__host__ __device__ constexpr int kzf_stride(int N, int W) { return N + (W >= 8 ? 1 : W == 4 ? 6 : W == 2 ? 4 : 3); }
__host__ __device__ constexpr int kzf_pad(int W) { return W >= 8 ? 0 : 1; }

// Shared-memory bytes of the z pass: k4_z (native complex128: twiddles +
// both halves), k4_zf (float-float: twiddles of 32 bytes + both halves)
// or k4_zp (complex64: twiddle tables, slice masks, tile elements, pairs).
template <typename T>
__host__ inline size_t kz4_smem(int N, int C, int W) {
  const size_t NB = N / 16;
  if (sizeof(T) == 4) return 272 * NB + 64 + 544 + (size_t)C * W * kzp_stride(N, W) * 16;
  if (std::is_same<T, ff>::value) return (size_t)32 * xyf_tw(N) + 2 * (size_t)C * W * kzf_stride(N, W) * 16;
  const size_t half = (size_t)C * W * kz4_stride(N, W);
  return (N + 2 * half + kz4_halfpad(W)) * sizeof(cplx<T>);
}

// Outer length of the complex64 z pass' split N = P x Q: the step that touches
// HBM.  The short one where it has enough values in flight (NB >= 4: 1.08 against
// 1.15 ms in the z pass at 112^3 PWC and seven right-hand sides), 16 below.
__host__ __device__ constexpr int zp_outer(int NB) { return NB >= 4 ? NB : 16; }
// frequency k of place p (row*16 + col) of a column of the pair layout
__host__ __device__ constexpr int zp_freq(int NB, int p) { return zp_outer(NB) == NB ? (p >> 4) + NB * (p & 15) : p; }

// Tiles of the complex64 z pass (k4_zp): W = TX*R elements are, from the
// lowest bit up, R right-hand sides, then the x mirror, then the y mirror,
// then neighbouring columns, as far as W reaches; mirrors that do not fit
// are tiles of their own.  As many CTAs as run at once, each walking the tiles.
struct ZpTiles {
  int lgW, lgR, cols;       // cols: octant columns kx per tile
  bool mx, my;              // mirrors inside the tile
  int ncx, nsub, nb;
  int total;
};
__host__ __device__ inline ZpTiles kzp_tiles(int n1, int n2, int W, int R, int nb) {
  ZpTiles t;
  t.lgW = t.lgR = 0;
  while ((1 << t.lgW) < W) ++t.lgW;
  while ((1 << t.lgR) < R) ++t.lgR;
  const int extra = t.lgW - t.lgR;
  t.mx = extra >= 1;
  t.my = extra >= 2;
  t.cols = extra > 2 ? 1 << (extra - 2) : 1;
  t.ncx = (n1 + t.cols) / t.cols;               // ceil((n1 + 1) / cols)
  t.nb = nb;
  t.nsub = nb * (t.mx ? 1 : 2) * (t.my ? 1 : 2);
  t.total = (n2 + 1) * t.ncx * t.nsub;
  return t;
}
constexpr int kSms = 152;
// Threads of k4_zp: 512 an SM at 128 registers, in CTAs of 256; PWC of n3 = 16 has 48
// tasks a tile and takes CTAs of 64 (16 x 32 x 16, sixteen right-hand sides: z pass
// 36.2 -> 20.3 us).  Tiles that run at once.
__host__ __device__ constexpr int zp_threads(int NB, bool pwl) { return NB == 1 && !pwl ? 64 : 256; }
__host__ __device__ constexpr int zp_slots(int NB, bool pwl) { return kSms * (512 / zp_threads(NB, pwl)); }
template <typename T>
inline unsigned kzp_grid(const MvArgs<T>& a, int nb) {
  const int tiles = kzp_tiles(a.n1, a.n2, a.TX * a.R, a.R, nb).total;
  return (unsigned)std::min(tiles, zp_slots(a.n3 / 16, a.C == 12));
}

template <typename T>
void launch_x_nb(int nb, bool inv, const MvArgs<T>& a, dim3 g, size_t smem, cudaStream_t s);
template <typename T>
void launch_y_nb(int nb, bool inv, const MvArgs<T>& a, dim3 g, size_t smem, cudaStream_t s);
template <typename T, bool PWL, int NB>
void launch_z_one(int op, const MvArgs<T>& a, dim3 g, size_t smem, cudaStream_t s);

#define MARIE_NB_SWITCH(nb, CALL) \
  switch (nb) {                   \
    case 1: CALL(1); break;       \
    case 2: CALL(2); break;       \
    case 3: CALL(3); break;       \
    case 4: CALL(4); break;       \
    case 5: CALL(5); break;       \
    case 6: CALL(6); break;       \
    case 7: CALL(7); break;       \
    default: CALL(8); break;      \
  }

template <typename T, bool PWL>
void launch_z_nb(int nb, int op, const MvArgs<T>& a, dim3 g, size_t smem, cudaStream_t s) {
#define Z_CALL(NB) launch_z_one<T, PWL, NB>(op, a, g, smem, s)
  MARIE_NB_SWITCH(nb, Z_CALL);
#undef Z_CALL
}

// The five passes of one chunk on the four-step path; ev (optional) as in
// launch_matvec_ev.  Tiles in `a` are set by the caller.
template <typename T>
marie_status launch_fast_chunk(marie_vie* h, int op, MvArgs<T>& a, int nb, cudaStream_t stream, cudaEvent_t* ev) {
  const int n1 = a.n1, n2 = a.n2, n3 = a.n3, C = h->C;
  const size_t sz = sizeof(cplx<T>);
  constexpr bool c64 = std::is_same<T, float>::value;
  auto smxy = [&](int n, int w) {
    return std::is_same<T, ff>::value ? xyf_smem(n, w) : (n + (size_t)2 * w * (n + 1)) * sz;
  };
  const size_t smx = smxy(n1, a.TY * a.R);
  const size_t smy = smxy(n2, c64 ? a.WY : a.TXY * a.R);
  const size_t smz = kz4_smem<T>(n3, C, a.TX * a.R);
  // x: TY rows (complex64: slices) per tile; y: TXY kx of a row (complex64: WY elements)
  dim3 gx(c64 ? (a.g3 + a.TY - 1) / a.TY : (a.g2 + a.TY - 1) / a.TY, c64 ? a.g2 : a.g3, nb * C);
  dim3 gy((2 * n1 + a.TXY - 1) / a.TXY, a.g3, nb * C);
  if constexpr (c64) {
    const int col = a.g3 * a.R;
    gy = col % a.WY == 0 ? dim3(col / a.WY, 2 * n1, nb * C) : dim3((2 * n1 * col + a.WY - 1) / a.WY, 1, nb * C);
  }
  dim3 gz(nb, (2 * n1 + a.TX - 1) / a.TX, 2 * n2);
  if constexpr (c64) gz = dim3(kzp_grid(a, nb));
  if (ev) cudaEventRecord(ev[0], stream);
  launch_x_nb<T>(n1 / 16, false, a, gx, smx, stream);
  MARIE_LAUNCH_CHECK();
  if (ev) cudaEventRecord(ev[1], stream);
  launch_y_nb<T>(n2 / 16, false, a, gy, smy, stream);
  MARIE_LAUNCH_CHECK();
  if (ev) cudaEventRecord(ev[2], stream);
  if (h->pwl) launch_z_nb<T, true>(n3 / 16, op, a, gz, smz, stream);
  else launch_z_nb<T, false>(n3 / 16, op, a, gz, smz, stream);
  MARIE_LAUNCH_CHECK();
  if (ev) cudaEventRecord(ev[3], stream);
  launch_y_nb<T>(n2 / 16, true, a, gy, smy, stream);
  MARIE_LAUNCH_CHECK();
  if (ev) cudaEventRecord(ev[4], stream);
  launch_x_nb<T>(n1 / 16, true, a, gx, smx, stream);
  MARIE_LAUNCH_CHECK();
  if (ev) cudaEventRecord(ev[5], stream);
  return MARIE_OK;
}

}  // namespace marie
