// fc_fused.cu -- correlations as five fused, hand-written FFT passes over HBM
// (no cuFFT), with the Y_lm weighting, the conjugate product, the k-subgrid
// extraction and the r-subgrid extraction folded into them, and the inverse
// transform pruned to the rows the r-subgrid needs: a survey correlation's,
// (ell, m) by (ell, m), and a periodic one's, once without the weights (those of
// all its multipoles are in the histograms).
//
// Per (ell, m), for the half-complex work array W[x][y][kz] (kz < N2/2+1):
//   zfwd   W[x][y][:] = R2C_z( Y_lm(cell) * rho[x][y][:] )   (make_ylm + r2c
//          along z; spherical_harmonics.h:32-179, fft_grid.cc:125-150)
//   yfwd   W = DFT_y(W)
//   xcorr  per (ky, kz) column: F = DFT_x(W); P = F * conj(G)
//          (array_ops.cc:139-163); ksub += Y_lm(k) W(k)^-2 4 pi Re P on the
//          k-subgrid (fft_grid.cc:215-258); Wr[ri][ky][kz] = IDFT_x(P) only
//          at the rs rows x = (N0 - rs/2 + ri) mod N0 of the r-subgrid (in W's
//          place, where it has no more rows than the grid)
//   yinv   Wry[ri][rj][kz] = IDFT_y(Wr) at the rs rows of the r-subgrid
//   zinv   rsub[ri][rj][rk] += Y_lm(r) 4 pi/N * C2R_z(Wry)[rk] (fft_grid.cc:
//          182-210)
// Both histograms are over |k| and |r|, and Y_lm is even for even ell, so only
// the part of P that is even in k contributes: Re P, whose inverse transform
// is even in r.  The k-subgrid is stored for kz >= 0 alone.  Where every
// r-subgrid cell and its mirror image fall into the same bin (the bins of r
// and -r are computed from rounded coordinates, so this is checked when a
// correlator is made), the inverse takes Re P -- two real columns ride
// through one complex transform -- and stops at the rows x >= 0, half the
// work of the inverse passes; otherwise it transforms P itself.  Per launch
// at 512^3 FP32: x pass 324 -> 279 us, inverse y 37 -> 22 us, inverse z 23 ->
// 14 us (a correlation 11.8 -> 10.8 ms); at 256^3 FP64: 105 -> 85 us, 15 -> 9
// us, 9 -> 8 us; the x pass at 64^3, whose extraction walked the k-subgrid's
// rows one after another, 27 -> 11 us.
// Two columns that share a transform share its rounding too: the larger one's
// reaches the smaller, of order 1e-7 (FP32) of the larger per value, and a
// column of zeros beside one that is not comes out at that level instead of
// zero.  The same holds of the rows that share one in fc_fused_gen.cuh.  The sum
// of the squared errors is that of separate transforms, but the two halves of r
// no longer average separate ones.  Errors of xi against 64 bits (2-norm, mean of
// 6 fields; in brackets cuFFT's or the passes' before): survey 64^3 1.58e-7
// (1.83e-7), 125 x 180 x 126 7.2e-8 (8.0e-8), 128^3 2.17e-7 (2.41e-7); periodic
// 125 x 126 x 120 8.6e-8 (1.15e-7), 128^3 2.55e-7 (3.04e-7), 125 x 81 x 105
// 1.27e-7 (1.05e-7) and in FP64 4.4e-16 (2.8e-16); survey 128^3 FP64 3.1e-16
// (3.3e-16).
// grid2's transform G (correlator.h:53-77) is zfwd (no weighting) + yfwd +
// DFT_x.  Bytes per (ell, m) at 512^3 FP32: ~4 GB instead of ~11 GB for
// separate make_ylm / cuFFT r2c / multiply / extract / cuFFT c2r passes.
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "fc_common.cuh"
#include "fc_fft.cuh"
#include "fc_fused.h"
#include "fc_internal.h"

namespace fc {
namespace {

template <typename T>
using C2 = typename Vec2<T>::type;

// Columns (or rows) per CTA: 64-byte segments of complex values.
template <typename T>
struct Tile {
  static constexpr int B = 64 / (2 * sizeof(T));  // 8 for FP32, 4 for FP64
};

// FP32-mixed weighting of one grid row: with (x, y) fixed, Y_lm * r^ell is
// a polynomial in z, so the row's coefficients (normalisation folded in)
// are formed once in FP64 and each cell costs a Horner evaluation and one
// reciprocal:  Y = D * (c0 + c1 z + c2 z^2 + c3 z^3 + c4 z^4) / r^ell.
struct RowPoly {
  float c[5];
  float rxy2;  // x^2 + y^2
  int ell;
  float value0;
};

__device__ __forceinline__ RowPoly row_poly(const YlmParams &p, double x,
                                            double y) {
  RowPoly r;
  r.ell = p.ell;
  r.value0 = (float)p.value0;
  double c[5];
  row_poly_coefs(p, x, y, c);
  for (int i = 0; i < 5; ++i) r.c[i] = (float)c[i];
  r.rxy2 = (float)(x * x + y * y);
  return r;
}

// The row polynomial of an (ell, m) term has only the powers of z of one
// parity up to ell - |m| (spherical_harmonics.h:100-176): its form is one
// of five (POLY, below), chosen once per thread instead of a full Horner
// evaluation per cell.
//   0: c0    1: c1 z    2: c0 + c2 z^2    3: (c1 + c3 z^2) z
//   4: c0 + (c2 + c4 z^2) z^2
__host__ __device__ __forceinline__ int row_poly_form(int ell, int m) {
  const int a = m < 0 ? -m : m;
  if (ell == 2) return a == 2 ? 0 : a == 1 ? 1 : 2;
  return a == 4 ? 0 : a == 3 ? 1 : a == 2 ? 2 : a == 1 ? 3 : 4;
}

// z of the cell `i` after the one at z0 (FP32: zt), rounded once in rows of 32
// pairs, which stood with the mixed-radix rows before, as these round it.
template <int L>
__device__ __forceinline__ float row_z(double z0, float zt, int i) {
  if constexpr (L == 32) return (float)(z0 + i);
  else return zt + (float)i;
}

template <int POLY, int ELL>
__device__ __forceinline__ float row_weight_form(const RowPoly &r, float D,
                                                 float z) {
  const float z2 = z * z;
  float poly;
  if constexpr (POLY == 0) poly = r.c[0];
  else if constexpr (POLY == 1) poly = r.c[1] * z;
  else if constexpr (POLY == 2) poly = r.c[2] * z2 + r.c[0];
  else if constexpr (POLY == 3) poly = (r.c[3] * z2 + r.c[1]) * z;
  else poly = (r.c[4] * z2 + r.c[2]) * z2 + r.c[0];
  const float ir2 = __fdividef(1.0f, r.rxy2 + z2 + 1e-20f);
  // (1 / r^2 twice: its square is infinite in FP32 at the observer, r = 0,
  // where poly is 0 and the weight must be.)
  if constexpr (ELL == 2) return D * poly * ir2;
  else return D * poly * ir2 * ir2;
}

// (Plain loads: k_rowpoly writes the table just before, see grid_chain.)
__device__ __forceinline__ RowPoly load_row_poly(const float4 *tab, int64_t row,
                                                 const YlmParams &p) {
  const float4 a = tab[2 * row];
  const float4 b = tab[2 * row + 1];
  RowPoly r;
  r.c[0] = a.x;
  r.c[1] = a.y;
  r.c[2] = a.z;
  r.c[3] = a.w;
  r.c[4] = b.x;
  r.rxy2 = b.y;
  r.ell = p.ell;
  r.value0 = (float)p.value0;
  return r;
}

// --------------------------------------------------------------------------
// Power-of-two lengths, with the register-resident engine (reg_fft in
// fc_fft.cuh); other lengths are fc_fused_gen.cuh's.  B2 columns per CTA keep the CTA at <= 1024
// threads (TPC = L/8 threads per column).
template <typename T, int L>
struct P2 {
  // (Rows of 32 elements, which only the z passes take, need more of them.)
  static constexpr int B = L == 32 ? 4 * Tile<T>::B
                           : (Tile<T>::B < 8192 / L) ? Tile<T>::B : 8192 / L;
  static constexpr int TPC = L / 8;
  static constexpr int THREADS = TPC * B;
  // Exchange rows of B elements: a 128-byte shared-memory line holds R of
  // them.  Row i is stored at row i ^ ((i >> 3) & (R - 1)), which spreads
  // the rows a warp touches in every Stockham write and read evenly over
  // the line's R parts (bank-conflict free), with no padding.
  static constexpr int RB = B * (int)sizeof(C2<T>);
  static constexpr int R = RB >= 128 ? 1 : 128 / RB;
  __device__ static __forceinline__ int row(int i) {
    return i ^ ((i >> 3) & (R - 1));
  }
  // Element index of row t + TPC u, column b: when TPC / 8 is a multiple
  // of R the swizzle only depends on t, so it is a per-thread base plus u
  // times a constant.
  static constexpr bool kFastRead = (TPC / 8) % R == 0;
  __device__ static __forceinline__ int rd_base(int t, int b) {
    return kFastRead ? row(t) * B + b : 0;
  }
  __device__ static __forceinline__ int rd(int base, int t, int b, int u) {
    return kFastRead ? base + u * TPC * B : row(t + TPC * u) * B + b;
  }
};

// The same layout with BB columns.
template <typename T, int L, int BB>
struct P2B {
  static constexpr int TPC = L / 8;
  static constexpr int THREADS = TPC * BB;
  static constexpr int RB = BB * (int)sizeof(C2<T>);
  static constexpr int R = RB >= 128 ? 1 : 128 / RB;
  __device__ static __forceinline__ int row(int i) {
    return i ^ ((i >> 3) & (R - 1));
  }
  static constexpr bool kFastRead = (TPC / 8) % R == 0;
  __device__ static __forceinline__ int rd_base(int t, int b) {
    return kFastRead ? row(t) * BB + b : 0;
  }
  __device__ static __forceinline__ int rd(int base, int t, int b, int u) {
    return kFastRead ? base + u * TPC * BB : row(t + TPC * u) * BB + b;
  }
};

template <typename T, int L>
__global__ void __launch_bounds__(P2<T, L>::THREADS)
    k_yfwd_p2(C2<T> *W, FusedGeom g, const C2<T> *__restrict__ taby) {
  grid_chain();
  using C = C2<T>;
  using Q = P2<T, L>;
  extern __shared__ unsigned char smem_raw[];
  C *ex = reinterpret_cast<C *>(smem_raw);
  const int t = threadIdx.x / Q::B;
  const int b = threadIdx.x - t * Q::B;
  const int kz0 = blockIdx.x * Q::B;
  const bool valid = kz0 + b < g.h;
  const int64_t base = (int64_t)blockIdx.y * L * g.hp + kz0 + b;
  C v[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    v[u].x = 0;
    v[u].y = 0;
    if (valid) v[u] = W[base + (int64_t)(t + Q::TPC * u) * g.hp];
  }
  const int rb = Q::rd_base(t, b);
  reg_fft<L>(v, t, [&](int i) { return &ex[Q::row(i) * Q::B + b]; },
             [&](int u) { return &ex[Q::rd(rb, t, b, u)]; }, taby, -1);
  if (valid) {
#pragma unroll
    for (int u = 0; u < 8; ++u) W[base + (int64_t)(t + Q::TPC * u) * g.hp] = v[u];
  }
}

template <typename T, int L>
__global__ void __launch_bounds__(P2<T, L>::THREADS)
    k_yinv_p2(const C2<T> *Wr, C2<T> *Wry, FusedGeom g,
              const C2<T> *__restrict__ taby) {
  grid_chain();
  using C = C2<T>;
  using Q = P2<T, L>;
  extern __shared__ unsigned char smem_raw[];
  C *ex = reinterpret_cast<C *>(smem_raw);
  const int t = threadIdx.x / Q::B;
  const int b = threadIdx.x - t * Q::B;
  const int kz0 = blockIdx.x * Q::B;
  const int ri = blockIdx.y;
  const bool valid = kz0 + b < g.h;
  const int64_t base = (int64_t)ri * L * g.hp + kz0 + b;
  C v[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    v[u].x = 0;
    v[u].y = 0;
    if (valid) v[u] = Wr[base + (int64_t)(t + Q::TPC * u) * g.hp];
  }
  const int rb = Q::rd_base(t, b);
  reg_fft<L>(v, t, [&](int i) { return &ex[Q::row(i) * Q::B + b]; },
             [&](int u) { return &ex[Q::rd(rb, t, b, u)]; }, taby, +1);
  if (!valid) return;
  const int64_t obase = (int64_t)ri * g.rs * g.hp + kz0 + b;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int y = t + Q::TPC * u;
    for (int rj = (y + g.ro) & (L - 1); rj < g.rs; rj += L)
      Wry[obase + (int64_t)rj * g.hp] = v[u];
  }
}

// Adds a thread's real parts re[u] of P at rows t + TPC u, columns kz ..
// kz + W - 1, to the stored half of the k-subgrid (half_k_cell; the last cell
// may be the row's padding), or overwrites it when `first`.  A cell has one
// source element, so nothing collides.
template <int L, int W, typename KT, typename Re>
__device__ __forceinline__ void to_half_k(double *ksub, const KT *__restrict__ ktab,
                                          const FusedGeom &g, int t, int jr, int kz,
                                          bool first, Re re) {
  constexpr int TPC = L / 8;
  constexpr int N = 4 / W;  // rows whose loads go out together
  const int ox = g.ks0 / 2;
  for (int j = jr; j < g.ks1; j += g.n1)
#pragma unroll
    for (int u0 = 0; u0 < 8; u0 += N) {
      size_t cell[N];
      double w[N][W], acc[N][W];
      bool on[N];
#pragma unroll
      for (int s = 0; s < N; ++s) {
        const int i = (t + TPC * (u0 + s) + ox) & (L - 1);
        on[s] = i < g.ks0;
        cell[s] = ((size_t)i * g.ks1 + j) * g.kp + kz;
#pragma unroll
        for (int l = 0; l < W; ++l) {
          w[s][l] = acc[s][l] = 0.0;
          if (on[s]) {
            w[s][l] = ktab ? (double)ktab[cell[s] + l] : 1.0;
            if (!first) acc[s][l] = ksub[cell[s] + l];
          }
        }
      }
#pragma unroll
      for (int s = 0; s < N; ++s)
#pragma unroll
        for (int l = 0; l < W; ++l)
          if (on[s]) ksub[cell[s] + l] = acc[s][l] + w[s][l] * re(u0 + s, l);
    }
  // A k-subgrid of L + 1 rows holds row L / 2 of P at both of its ends.
  if (g.ks0 > L && t == (L / 2) % TPC)
    for (int j = jr; j < g.ks1; j += g.n1) {
      const size_t c = ((size_t)L * g.ks1 + j) * g.kp + kz;
      for (int l = 0; l < W; ++l)
        ksub[c + l] = (first ? 0.0 : ksub[c + l]) +
                      (ktab ? (double)ktab[c + l] : 1.0) * re(L / 2 / TPC, l);
    }
}

// The columns A and B of Z = DFT(a + i b), a and b real, from Z at x and at
// -x: A = (Z(x) + conj Z(-x)) / 2, B = (Z(x) - conj Z(-x)) / 2i.
template <typename C>
__device__ __forceinline__ void split_pair(const C &z, const C &m, C *a, C *b) {
  using T = decltype(z.x);
  a->x = (T)0.5 * (z.x + m.x);
  a->y = (T)0.5 * (z.y - m.y);
  b->x = (T)0.5 * (z.y + m.y);
  b->y = (T)0.5 * (m.x - z.x);
}

// FP64.  MODE 0: out = G = DFT_x(W).  MODE 1: the product, extraction and
// inverse described at the top; MODE 2 (ell = 0 of an autocorrelation): the
// weighted field is w00 * rho, whose transform is w00 * G, so P = w00 |G|^2
// and neither W nor a forward transform is needed; MODE 3 (periodic
// autocorrelation): P = |DFT_x(W)|^2.  Without ktab the k-subgrid's weights
// are 1.  EVEN: the inverse of Re P, two real columns to a complex one:
// half of the CTA's threads transform half as many columns, the others
// leave.
template <int L, int MODE, bool EVEN>
__global__ void __launch_bounds__(P2<double, L>::THREADS)
    k_xcorr_p2(const double2 *W, const double2 *G, double2 *out, double *ksub, FusedGeom g,
               const double2 *__restrict__ tabx, const double *__restrict__ ktab,
               double w00, int first) {
  grid_chain();
  using C = double2;
  using Q = P2<double, L>;
  extern __shared__ unsigned char smem_raw[];
  C *ex = reinterpret_cast<C *>(smem_raw);
  const int t = threadIdx.x / Q::B;
  const int b = threadIdx.x - t * Q::B;
  const int kz0 = blockIdx.x * Q::B;
  const int yy = blockIdx.y;
  const int kzi = kz0 + b;
  const bool valid = kzi < g.h;
  const int64_t stride = (int64_t)g.n1 * g.hp;
  const int64_t base = (int64_t)yy * g.hp + kzi;
  auto exf = [&](int i) { return &ex[Q::row(i) * Q::B + b]; };
  C v[8];
  // In product mode the G column is loaded together with the W column, so
  // both streams are in flight during the forward transform.
  C gv[MODE == 1 ? 8 : 1];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    v[u] = make_double2(0, 0);
    const int64_t at = base + (t + Q::TPC * u) * stride;
    if constexpr (MODE == 2) {
      if (valid) {
        const C q = G[at];
        v[u].x = w00 * (q.x * q.x + q.y * q.y);
      }
    } else {
      if (valid) v[u] = W[at];
    }
    if constexpr (MODE == 1) gv[u] = valid ? G[at] : make_double2(0, 0);
  }
  const int rb = Q::rd_base(t, b);
  auto exr = [&](int u) { return &ex[Q::rd(rb, t, b, u)]; };
  if constexpr (MODE != 2) reg_fft<L>(v, t, exf, exr, tabx, -1);
  if constexpr (MODE == 0) {
    if (valid) {
#pragma unroll
      for (int u = 0; u < 8; ++u) out[base + (t + Q::TPC * u) * stride] = v[u];
    }
  } else {
    if constexpr (MODE == 1) {
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = cmulc(v[u], gv[u]);
    } else if constexpr (MODE == 3) {
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u].x = v[u].x * v[u].x + v[u].y * v[u].y;
    }
    const int jr = (yy + g.ks1 / 2) % g.n1;
    if (ksub != nullptr && jr < g.ks1 && kzi <= g.ks2 / 2)
      to_half_k<L, 1>(ksub, ktab, g, t, jr, kzi, first != 0,
                      [&](int u, int) { return v[u].x; });
    if constexpr (EVEN) {
      constexpr int H = Q::B / 2;
      using QH = P2B<double, L, H>;
      double *st = reinterpret_cast<double *>(smem_raw);
#pragma unroll
      for (int u = 0; u < 8; ++u) st[(t + Q::TPC * u) * Q::B + b] = v[u].x;
      __syncthreads();
      if (threadIdx.x >= QH::THREADS) return;
      const int t2 = threadIdx.x / H, b2 = threadIdx.x % H;
      C z[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) z[u] = ex[(t2 + Q::TPC * u) * H + b2];
      __syncthreads();
      const int rb2 = QH::rd_base(t2, b2);
      auto zf = [&](int i) { return &ex[QH::row(i) * H + b2]; };
      reg_fft<L>(z, t2, zf, [&](int u) { return &ex[QH::rd(rb2, t2, b2, u)]; }, tabx, +1);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int x = t2 + Q::TPC * u;
        if (x <= g.ro || x >= L - g.ro) *zf(x) = z[u];
      }
      __syncthreads();
      const int c = kz0 + 2 * b2;
      for (int x = t2; x <= g.ro; x += Q::TPC) {
        C A, B;
        split_pair(*zf(x & (L - 1)), *zf((L - x) & (L - 1)), &A, &B);
        C *o = out + x * stride + (int64_t)yy * g.hp + c;
        if (c < g.h) o[0] = A;
        if (c + 1 < g.h) o[1] = B;
      }
    } else {
      reg_fft<L>(v, t, exf, exr, tabx, +1);
      if (valid) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int x = t + Q::TPC * u;
          for (int ri = (x + g.ro) & (L - 1); ri < g.rs; ri += L)
            out[base + ri * stride] = v[u];
        }
      }
    }
  }
}

// FP64 rows of the z transform: thread t of row b holds z[t + TPC u].  The
// weight of a cell is its row's polynomial in z over r^ell (row_poly_coefs),
// formed per thread: with the evaluation of Y_lm from (x, y, z) at every cell
// the pass took 108 us at 256^3 against 66, bound by FP64 instructions.
template <int L, bool WEIGHT>
__global__ void __launch_bounds__(P2<double, L>::THREADS)
    k_zfwd_p2(const double *rho, double2 *W, FusedGeom g,
              YlmParams p, double x0, double y0, double z0,
              const double2 *__restrict__ tabz) {
  grid_chain();
  using C = double2;
  using Q = P2<double, L>;
  // Row pitch in shared memory, with one pad slot every 8 elements so the
  // strided Stockham writes spread over the banks.
  constexpr int RP = L + L / 8 + 1;
  extern __shared__ unsigned char smem_raw[];
  C *ex = reinterpret_cast<C *>(smem_raw);
  const int b = threadIdx.x / Q::TPC;
  const int t = threadIdx.x - b * Q::TPC;
  const int64_t nrows = (int64_t)g.n0 * g.n1;
  const int64_t row = (int64_t)blockIdx.x * Q::B + b;
  const bool valid = row < nrows;
  const C *src = reinterpret_cast<const C *>(rho + (valid ? row : 0) * g.n2);
  C v[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) v[u] = valid ? src[t + Q::TPC * u] : make_double2(0, 0);
  if constexpr (WEIGHT) {
    if (p.ell == 0) {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        v[u].x *= p.value0;
        v[u].y *= p.value0;
      }
    } else {
      const int x = (int)((unsigned)row / (unsigned)g.n1);
      const int y = (int)row - x * g.n1;
      const double cx = x0 + x * 1.0, cy = y0 + y * 1.0;
      const double rxy2 = cx * cx + cy * cy;
      double c[5];
      row_poly_coefs(p, cx, cy, c);
      auto weigh = [&](auto ell, double d, double z) {
        const double z2 = z * z;
        const double ir2 = 1.0 / (rxy2 + z2 + 1e-20);
        if constexpr (decltype(ell)::value == 2)
          return d * ((c[2] * z + c[1]) * z + c[0]) * ir2;
        else
          return d * ((((c[4] * z + c[3]) * z + c[2]) * z + c[1]) * z + c[0]) * ir2 * ir2;
      };
      auto row_of = [&](auto ell) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const double z = z0 + (2 * (t + Q::TPC * u)) * 1.0;
          v[u].x = weigh(ell, v[u].x, z);
          v[u].y = weigh(ell, v[u].y, z + 1.0);
        }
      };
      if (p.ell == 2) row_of(std::integral_constant<int, 2>());
      else row_of(std::integral_constant<int, 4>());
    }
  }
  auto exf = [&](int i) { return &ex[b * RP + i + (i >> 3)]; };
  reg_fft<L>(v, t, exf, tabz, -1, 2);
  // Real-to-complex split needs Z_k and Z_{M-k}.
#pragma unroll
  for (int u = 0; u < 8; ++u) *exf(t + Q::TPC * u) = v[u];
  __syncthreads();
  if (!valid) return;
  C *dst = W + row * g.hp;
  for (int k = t; k <= L; k += Q::TPC) {
    const C a = *exf(k == L ? 0 : k);
    const C c = cconj(*exf(k == 0 ? 0 : L - k));
    C e, o;
    e.x = 0.5 * (a.x + c.x);
    e.y = 0.5 * (a.y + c.y);
    const C d = csub(a, c);
    o.x = 0.5 * d.y;
    o.y = -0.5 * d.x;
    dst[k] = cadd(e, cmul(__ldg(&tabz[k]), o));
  }
}

template <typename T, int L>
__global__ void __launch_bounds__(P2<T, L>::THREADS)
    k_zinv_p2(const C2<T> *Wry, double *rsub, FusedGeom g,
              const C2<T> *__restrict__ tabz,
              const T *__restrict__ rtab, int first) {
  grid_chain();
  using C = C2<T>;
  using Q = P2<T, L>;
  constexpr int RP = L + L / 8 + 1;
  extern __shared__ unsigned char smem_raw[];
  C *ex = reinterpret_cast<C *>(smem_raw);
  const int b = threadIdx.x / Q::TPC;
  const int t = threadIdx.x - b * Q::TPC;
  const int nrows = g.nri * g.rs;
  const int row = blockIdx.x * Q::B + b;
  const bool valid = row < nrows;
  C v[8];
  const C *X = Wry + (int64_t)(valid ? row : 0) * g.hp;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int k = t + Q::TPC * u;
    v[u].x = 0;
    v[u].y = 0;
    if (valid) {
      C a = X[k];
      C c = cconj(X[L - k]);
      if (k == 0) {
        a.y = 0;
        c.y = 0;
      }
      const C e = cadd(a, c);
      const C o = cmul(csub(a, c), cconj(__ldg(&tabz[k])));
      v[u].x = e.x - o.y;
      v[u].y = e.y + o.x;
    }
  }
  auto exf = [&](int i) { return &ex[b * RP + i + (i >> 3)]; };
  reg_fft<L>(v, t, exf, tabz, +1, 2);
  if (!valid) return;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int jj = t + Q::TPC * u;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int z = 2 * jj + h;
      const double val = (double)(h ? v[u].y : v[u].x);
      for (int rk = (z + g.ro) % g.n2; rk < g.rs; rk += g.n2) {
        const size_t cell = (size_t)row * g.rs + rk;
        rsub[cell] = rtab == nullptr ? val
                                     : (first ? 0.0 : rsub[cell]) + (double)rtab[cell] * val;
      }
    }
  }
}

// ------------------------------------------------- FP32 two-per-thread
// FP32 y and z passes with two independent transforms per thread: the same
// B columns (or rows) per CTA as the kernels above with half the threads.
// The two transforms share every twiddle load and index computation and the
// shared-memory exchanges move 16 bytes per access.  The y passes carry the
// pair as CPair (packed two-lane instructions), the z pass as CPairS
// (one-lane instructions), whichever measured faster for the pass.
// Thread (t, p) holds columns p and p + PB of the CTA's B, so each global
// access of a warp stays contiguous per row.  (The FP32 x passes pair
// adjacent columns like the y passes, below.)
template <int L>
struct PP {
  static constexpr int B = P2<float, L>::B;
  static constexpr int PB = B / 2;
  static constexpr int TPC = L / 8;
  static constexpr int THREADS = TPC * PB;
  static constexpr int RB = PB * (int)sizeof(CPair);
  static constexpr int R = RB >= 128 ? 1 : 128 / RB;
  __device__ static __forceinline__ int row(int i) {
    return i ^ ((i >> 3) & (R - 1));
  }
  static constexpr bool kFastRead = (TPC / 8) % R == 0;
  __device__ static __forceinline__ int rd_base(int t, int p) {
    return kFastRead ? row(t) * PB + p : 0;
  }
  __device__ static __forceinline__ int rd(int base, int t, int p, int u) {
    return kFastRead ? base + u * TPC * PB : row(t + TPC * u) * PB + p;
  }
};

// The FP32 y passes pair ADJACENT columns: thread (t, p) holds columns 2p
// and 2p + 1 of the CTA's B and moves both with one 16-byte access, and B
// is 16 where the CTA allows it, so a warp's access covers whole 128-byte
// row segments.  (Row pitches are multiples of 16 columns, so the pair of
// the last valid column lies in the padding and is read but never stored.)
template <int L, int BW = 16>
struct PY {
  static constexpr int B = BW < 8192 / L ? BW : 8192 / L;
  static constexpr int PB = B / 2;
  static constexpr int TPC = L / 8;
  static constexpr int THREADS = TPC * PB;
  static constexpr int RB = PB * (int)sizeof(CPair);
  static constexpr int R = RB >= 128 ? 1 : 128 / RB;
  __device__ static __forceinline__ int row(int i) {
    return i ^ ((i >> 3) & (R - 1));
  }
  static constexpr bool kFastRead = (TPC / 8) % R == 0;
  __device__ static __forceinline__ int rd_base(int t, int p) {
    return kFastRead ? row(t) * PB + p : 0;
  }
  __device__ static __forceinline__ int rd(int base, int t, int p, int u) {
    return kFastRead ? base + u * TPC * PB : row(t + TPC * u) * PB + p;
  }
  static constexpr size_t smem = (size_t)L * PB * sizeof(CPair);
};

__device__ __forceinline__ CPair load_pair(const float2 *p) {
  const float4 q = *reinterpret_cast<const float4 *>(p);
  return cpack(make_float2(q.x, q.y), make_float2(q.z, q.w));
}
__device__ __forceinline__ void store_pair(float2 *p, const CPair &v, bool v0,
                                           bool v1) {
  if (v1) {
    const float2 a = clane0(v), b = clane1(v);
    *reinterpret_cast<float4 *>(p) = make_float4(a.x, a.y, b.x, b.y);
  } else if (v0) {
    *p = clane0(v);
  }
}

// The column pair of thread p in a column pass.  Ordinary CTAs hold
// adjacent columns c0, c0 + 1 of one plane (one 16-byte access).  When the
// pass runs with `nyq`, the CTAs of the last column group (SPLIT) instead
// hold the last column (kz = N2/2, alone in its 16-column group) of planes
// 2p and 2p + 1 of their group of B planes, so that column does not take a
// whole group of mostly padding columns per plane.  The kernels branch once
// per CTA between the two forms, each compiled separately.
template <bool SPLIT>
struct ColPair {
  int64_t b0, b1;  // element offsets of the two columns' first rows
  bool v0, v1;     // whether each column exists
  __device__ CPair load(const float2 *a, int64_t row) const {
    if constexpr (!SPLIT) return load_pair(a + b0 + row);
    else return cpack(a[b0 + row], a[b1 + row]);
  }
  __device__ void store(float2 *a, int64_t row, const CPair &v) const {
    if constexpr (!SPLIT) {
      store_pair(a + b0 + row, v, v0, v1);
    } else {
      if (v0) a[b0 + row] = clane0(v);
      if (v1) a[b1 + row] = clane1(v);
    }
  }
  // Asynchronous copy of the pair at `row` into a 16-byte shared slot, laid
  // out as in memory (re, im of each column).
  __device__ void copy_async(CPair *slot, const float2 *a, int64_t row) const {
    if constexpr (!SPLIT) {
      cp_async16(slot, a + b0 + row);
    } else {
      float2 *d = reinterpret_cast<float2 *>(slot);
      cp_async8(d, a + b0 + row);
      cp_async8(d + 1, a + b1 + row);
    }
  }
};

// Column pair of thread p in the CTA of group blockIdx.x and plane (or, for
// SPLIT, plane group) `plane`, in a pass whose `nplanes` planes are `pitch`
// elements apart.  Returns false when a SPLIT CTA has no planes left.
template <int B, bool SPLIT>
__device__ __forceinline__ bool col_pair(ColPair<SPLIT> &c, int p, int plane,
                                         int64_t pitch, int nplanes,
                                         const FusedGeom &g) {
  if constexpr (SPLIT) {
    const int pl0 = plane * B;
    if (pl0 >= nplanes) return false;
    const int pa = pl0 + 2 * p;
    c.v0 = pa < nplanes;
    c.v1 = pa + 1 < nplanes;
    c.b0 = (int64_t)(c.v0 ? pa : 0) * pitch + g.h - 1;
    c.b1 = (int64_t)(c.v1 ? pa + 1 : 0) * pitch + g.h - 1;
  } else {
    const int c0 = blockIdx.x * B + 2 * p;
    c.v0 = c0 < g.h;
    c.v1 = c0 + 1 < g.h;
    c.b0 = (int64_t)plane * pitch + c0;
    c.b1 = c.b0 + 1;
  }
  return true;
}

// Whether this CTA takes the last column of a group of planes.
__device__ __forceinline__ bool split_cta(int nyq) {
  return nyq != 0 && blockIdx.x == gridDim.x - 1;
}

template <int L, bool SPLIT>
__device__ __forceinline__ void yfwd_pp_body(float2 *W, const FusedGeom &g,
                                             const float2 *__restrict__ taby) {
  using Q = PY<L>;
  extern __shared__ unsigned char smem_raw[];
  CPair *ex = reinterpret_cast<CPair *>(smem_raw);
  const int t = threadIdx.x / Q::PB;
  const int p = threadIdx.x - t * Q::PB;
  // Planes are x, L * g.hp elements apart.
  ColPair<SPLIT> cp;
  if (!col_pair<Q::B>(cp, p, blockIdx.y, (int64_t)L * g.hp, g.n0, g)) return;
  CPair v[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) v[u] = cp.load(W, (int64_t)(t + Q::TPC * u) * g.hp);
  const int rb = Q::rd_base(t, p);
  reg_fft<L>(v, t, [&](int i) { return &ex[Q::row(i) * Q::PB + p]; },
             [&](int u) { return &ex[Q::rd(rb, t, p, u)]; }, taby, -1);
#pragma unroll
  for (int u = 0; u < 8; ++u) cp.store(W, (int64_t)(t + Q::TPC * u) * g.hp, v[u]);
}

template <int L>
__global__ void __launch_bounds__(PY<L>::THREADS, 1024 / PY<L>::THREADS)
    k_yfwd_pp(float2 *W, FusedGeom g, const float2 *__restrict__ taby) {
  grid_chain();
  // (Splitting off the last column measured slower here: 194 vs 183 us.)
  yfwd_pp_body<L, false>(W, g, taby);
}

// grid2's x transform in the FP32 form: G = DFT_x(W), the same column
// pairing as the y passes, with rows N1 * hp elements apart.
template <int L, bool SPLIT>
__device__ __forceinline__ void xfwd_pp_body(const float2 *W, float2 *G,
                                             const FusedGeom &g,
                                             const float2 *__restrict__ tabx) {
  using Q = PY<L>;
  extern __shared__ unsigned char smem_raw[];
  CPair *ex = reinterpret_cast<CPair *>(smem_raw);
  const int t = threadIdx.x / Q::PB;
  const int p = threadIdx.x - t * Q::PB;
  const int64_t stride = (int64_t)g.n1 * g.hp;
  // Planes are y, g.hp elements apart.
  ColPair<SPLIT> cp;
  if (!col_pair<Q::B>(cp, p, blockIdx.y, g.hp, g.n1, g)) return;
  CPair v[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) v[u] = cp.load(W, (t + Q::TPC * u) * stride);
  const int rb = Q::rd_base(t, p);
  reg_fft<L>(v, t, [&](int i) { return &ex[Q::row(i) * Q::PB + p]; },
             [&](int u) { return &ex[Q::rd(rb, t, p, u)]; }, tabx, -1);
#pragma unroll
  for (int u = 0; u < 8; ++u) cp.store(G, (t + Q::TPC * u) * stride, v[u]);
}

template <int L>
__global__ void __launch_bounds__(PY<L>::THREADS, 1024 / PY<L>::THREADS)
    k_xfwd_pp(const float2 *W, float2 *G, FusedGeom g,
              const float2 *__restrict__ tabx) {
  grid_chain();
  xfwd_pp_body<L, false>(W, G, g, tabx);
}

// The FP32 x pass of one (ell, m) term with the same column pairing.
// MODE 1: P = DFT_x(W) conj(G); MODE 2 (ell = 0 of an autocorrelation):
// P = w00 |G|^2 with no forward transform; MODE 3 (periodic
// autocorrelation): P = |DFT_x(W)|^2 (see k_xcorr_p2).  Then the
// k-subgrid extraction and the inverse transform, stored only at the
// r-subgrid's rows.  G is read after the forward transform, so a thread
// holds one pair of columns at a time and two CTAs fit an SM; the other
// CTA's warps cover those loads.  EVEN: the inverse of Re P: a pair of real
// columns is one complex column, so half of the CTA's threads carry the
// columns of two pairs through one transform each and the others leave.
constexpr int kXB = 16;  // columns per CTA of the FP32 x passes

template <int L, int MODE, bool SPLIT, bool EVEN>
__device__ __forceinline__ void xcorr_pp_body(
    const float2 *W, const float2 *G, float2 *out, double *ksub, const FusedGeom &g,
    const float2 *__restrict__ tabx, const float *__restrict__ ktab, float w00,
    int first) {
  using Q = PY<L, kXB>;
  extern __shared__ unsigned char smem_raw[];
  CPair *ex = reinterpret_cast<CPair *>(smem_raw);
  const int t = threadIdx.x / Q::PB;
  const int p = threadIdx.x - t * Q::PB;
  const int yy = blockIdx.y;
  const int64_t stride = (int64_t)g.n1 * g.hp;
  // Planes are y, g.hp elements apart; with nyq the host has made sure the
  // last column lies outside the k-subgrid.
  ColPair<SPLIT> cp;
  if (!col_pair<Q::B>(cp, p, yy, g.hp, g.n1, g)) return;
  const int cb = SPLIT ? g.h - 1 : blockIdx.x * Q::B;
  const int c0 = SPLIT ? g.h - 1 : cb + 2 * p;
  auto exf = [&](int i) { return &ex[Q::row(i) * Q::PB + p]; };
  const int rb = Q::rd_base(t, p);
  auto exr = [&](int u) { return &ex[Q::rd(rb, t, p, u)]; };
  CPair v[8];
  if constexpr (MODE == 2) {
    const float2 w = f2splat(w00);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const CPair q = cp.load(G, (t + Q::TPC * u) * stride);
      v[u].x = w * __ffma2_rn(q.x, q.x, q.y * q.y);
      v[u].y = f2splat(0.f);
    }
  } else if constexpr (MODE == 3) {
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = cp.load(W, (t + Q::TPC * u) * stride);
    reg_fft<L>(v, t, exf, exr, tabx, -1);
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u].x = __ffma2_rn(v[u].x, v[u].x, v[u].y * v[u].y);
  } else {
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = cp.load(W, (t + Q::TPC * u) * stride);
    // G's pairs are copied into this thread's own exchange slots while the
    // last pass of the forward transform computes.  A slot then holds the
    // two columns as stored in memory, (re, im) of each, so it is read back
    // with load_pair like a global pair.
    reg_fft<L>(v, t, exf, exr, tabx, -1, 1, [&] {
#pragma unroll
      for (int u = 0; u < 8; ++u)
        cp.copy_async(exr(u), G, (t + Q::TPC * u) * stride);
    });
    cp_async_wait_all();
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const CPair gp = load_pair(reinterpret_cast<const float2 *>(exr(u)));
      if constexpr (EVEN) v[u].x = __ffma2_rn(v[u].y, gp.y, __fmul2_rn(v[u].x, gp.x));
      else v[u] = cmulc(v[u], gp);
    }
  }
  const int jr = (yy + g.ks1 / 2) % g.n1;
  if (!SPLIT && ksub != nullptr && jr < g.ks1 && c0 <= g.ks2 / 2)
    to_half_k<L, 2>(ksub, ktab, g, t, jr, c0, first != 0, [&](int u, int l) {
      return (double)(l ? v[u].x.y : v[u].x.x);
    });
  // Every thread has read G from its slots before anything is written over
  // them.
  if constexpr (MODE == 1) __syncthreads();
  if constexpr (EVEN) {
    constexpr int H = Q::PB / 2;
    using QH = PY<L, Q::B / 2>;
    static_assert(QH::PB == H && 2 * QH::THREADS == Q::THREADS);
    // A column that does not exist must not reach its neighbour's transform.
    float2 *st = reinterpret_cast<float2 *>(smem_raw);
#pragma unroll
    for (int u = 0; u < 8; ++u)
      st[(t + Q::TPC * u) * Q::PB + p] =
          make_float2(cp.v0 ? v[u].x.x : 0.f, cp.v1 ? v[u].x.y : 0.f);
    __syncthreads();
    if (threadIdx.x >= QH::THREADS) return;
    const int t2 = threadIdx.x / H, p2 = threadIdx.x % H;
    CPair z[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      z[u] = load_pair(st + (t2 + Q::TPC * u) * Q::PB + 2 * p2);
    __syncthreads();
    const int rb2 = QH::rd_base(t2, p2);
    auto zf = [&](int i) { return &ex[QH::row(i) * H + p2]; };
    // Only rows |x| <= ro are stored: when they all lie in the first and last
    // TPC rows, only outputs u = 0 and 7 are computed.
    const bool edges = g.ro < Q::TPC;
    reg_fft<L>(z, t2, zf, [&](int u) { return &ex[QH::rd(rb2, t2, p2, u)]; }, tabx, +1,
               1, NoHook{}, edges);
    if (edges) {
      *zf(t2) = z[0];
      *zf(t2 + 7 * Q::TPC) = z[7];
    } else {
#pragma unroll
      for (int u = 0; u < 8; ++u) *zf(t2 + Q::TPC * u) = z[u];
    }
    __syncthreads();
    for (int x = t2; x <= g.ro; x += Q::TPC) {
      const CPair zp = *zf(x & (L - 1)), zm = *zf((L - x) & (L - 1));
      float2 c[4];
      split_pair(clane0(zp), clane0(zm), &c[0], &c[1]);
      split_pair(clane1(zp), clane1(zm), &c[2], &c[3]);
      float2 *o = out + x * stride;
      if constexpr (SPLIT) {
        const int pl = yy * Q::B + 4 * p2;
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (pl + i < g.n1) o[(int64_t)(pl + i) * g.hp + g.h - 1] = c[i];
      } else {
        const int k = cb + 4 * p2;
        o += (int64_t)yy * g.hp + k;
        if (k + 3 < g.h) {
          reinterpret_cast<float4 *>(o)[0] = make_float4(c[0].x, c[0].y, c[1].x, c[1].y);
          reinterpret_cast<float4 *>(o)[1] = make_float4(c[2].x, c[2].y, c[3].x, c[3].y);
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (k + i < g.h) o[i] = c[i];
        }
      }
    }
  } else {
    // Rows x whose r-subgrid row (x + ro) mod L is below rs; when they all
    // lie in the first and last TPC rows, only outputs u = 0 and 7 are
    // computed.
    const bool edges = g.ro <= Q::TPC && g.rs - g.ro <= Q::TPC;
    reg_fft<L>(v, t, exf, exr, tabx, +1, 1, NoHook{}, edges);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (edges && u != 0 && u != 7) continue;
      const int x = t + Q::TPC * u;
      for (int ri = (x + g.ro) & (L - 1); ri < g.rs; ri += L)
        cp.store(out, ri * stride, v[u]);
    }
  }
}

template <int L, int MODE, bool EVEN>
__global__ void __launch_bounds__(PY<L, kXB>::THREADS, 1024 / PY<L, kXB>::THREADS)
    k_xcorr_pp(const float2 *W, const float2 *G, float2 *out, double *ksub, FusedGeom g,
               const float2 *__restrict__ tabx, const float *__restrict__ ktab,
               float w00, int nyq, int first) {
  grid_chain();
  // The last column split off (nyq) pays in the product mode only; the
  // ell = 0 mode compiles without it (with it: 215 vs 188 us).
  if constexpr (MODE == 1) {
    if (split_cta(nyq)) {
      xcorr_pp_body<L, MODE, true, EVEN>(W, G, out, ksub, g, tabx, ktab, w00, first);
      return;
    }
  }
  xcorr_pp_body<L, MODE, false, EVEN>(W, G, out, ksub, g, tabx, ktab, w00, first);
}

template <int L, bool SPLIT>
__device__ __forceinline__ void yinv_pp_body(const float2 *Wr, float2 *Wry,
                                             const FusedGeom &g,
                                             const float2 *__restrict__ taby) {
  using Q = PY<L>;
  extern __shared__ unsigned char smem_raw[];
  CPair *ex = reinterpret_cast<CPair *>(smem_raw);
  const int t = threadIdx.x / Q::PB;
  const int p = threadIdx.x - t * Q::PB;
  // Planes are the r-subgrid's x rows: L * g.hp elements apart in Wr,
  // rs * g.hp in Wry.
  ColPair<SPLIT> cp;
  if (!col_pair<Q::B>(cp, p, blockIdx.y, (int64_t)L * g.hp, g.nri, g)) return;
  CPair v[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) v[u] = cp.load(Wr, (int64_t)(t + Q::TPC * u) * g.hp);
  const int rb = Q::rd_base(t, p);
  const bool edges = g.ro <= Q::TPC && g.rs - g.ro <= Q::TPC;  // see k_xcorr_pp
  reg_fft<L>(v, t, [&](int i) { return &ex[Q::row(i) * Q::PB + p]; },
             [&](int u) { return &ex[Q::rd(rb, t, p, u)]; }, taby, +1, 1,
             NoHook{}, edges);
  ColPair<SPLIT> co;  // the same columns of the same planes in Wry
  col_pair<Q::B>(co, p, blockIdx.y, (int64_t)g.rs * g.hp, g.nri, g);
  if (edges) {
#pragma unroll
    for (int u = 0; u < 8; u += 7) {
      const int rj = (t + Q::TPC * u + g.ro) & (L - 1);
      if (rj < g.rs) co.store(Wry, (int64_t)rj * g.hp, v[u]);
    }
    return;
  }
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int y = t + Q::TPC * u;
    for (int rj = (y + g.ro) & (L - 1); rj < g.rs; rj += L)
      co.store(Wry, (int64_t)rj * g.hp, v[u]);
  }
}

template <int L>
__global__ void __launch_bounds__(PY<L>::THREADS, 1024 / PY<L>::THREADS)
    k_yinv_pp(const float2 *Wr, float2 *Wry, FusedGeom g,
              const float2 *__restrict__ taby, int nyq) {
  grid_chain();
  if (split_cta(nyq))
    yinv_pp_body<L, true>(Wr, Wry, g, taby);
  else
    yinv_pp_body<L, false>(Wr, Wry, g, taby);
}

// Rows of the z transform, two rows per thread: rows b and b + PB of the
// CTA's B, thread t of a row pair holding z[t + TPC u] of both.
template <int L, bool WEIGHT>
__global__ void __launch_bounds__(PP<L>::THREADS)
    k_zfwd_pp(const float *rho, float2 *W, FusedGeom g,
              YlmParams p, double x0, double y0, double z0,
              const float2 *__restrict__ tabz, const float4 *rowtab) {
  grid_chain();
  using Q = PP<L>;
  constexpr int RP = L + L / 8 + 1;
  extern __shared__ unsigned char smem_raw[];
  CPairS *ex = reinterpret_cast<CPairS *>(smem_raw);
  const int pb = threadIdx.x / Q::TPC;
  const int t = threadIdx.x - pb * Q::TPC;
  const int64_t nrows = (int64_t)g.n0 * g.n1;
  const int64_t row0 = (int64_t)blockIdx.x * Q::B + pb;
  const int64_t row1 = row0 + Q::PB;
  const bool v0 = row0 < nrows, v1 = row1 < nrows;
  const float2 *src0 = reinterpret_cast<const float2 *>(rho + (v0 ? row0 : 0) * g.n2);
  const float2 *src1 = reinterpret_cast<const float2 *>(rho + (v1 ? row1 : 0) * g.n2);
  RowPoly rp0, rp1;
  float zt = 0.f;
  if constexpr (WEIGHT) {
    if (rowtab != nullptr) {
      // Per-row coefficients from k_rowpoly (the same FP64 evaluation).
      rp0 = load_row_poly(rowtab, v0 ? row0 : 0, p);
      rp1 = load_row_poly(rowtab, v1 ? row1 : 0, p);
    } else {
      const int xa = (int)(row0 / g.n1), ya = (int)(row0 - (int64_t)xa * g.n1);
      const int xb = (int)(row1 / g.n1), yb = (int)(row1 - (int64_t)xb * g.n1);
      rp0 = row_poly(p, x0 + xa * 1.0, y0 + ya * 1.0);
      rp1 = row_poly(p, x0 + xb * 1.0, y0 + yb * 1.0);
    }
    zt = (float)(z0 + (2 * t) * 1.0);
    z0 += 2 * t;
  }
  const float2 zero = make_float2(0.f, 0.f);
  float2 a[8], b[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int jj = t + Q::TPC * u;
    a[u] = v0 ? src0[jj] : zero;
    b[u] = v1 ? src1[jj] : zero;
  }
  if constexpr (WEIGHT) {
    // One uniform branch per thread picks the weight's form.
    auto weigh = [&](auto poly, auto ellc) {
      constexpr int POLY = decltype(poly)::value, ELL = decltype(ellc)::value;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float zu = row_z<L>(z0, zt, 2 * Q::TPC * u);
        const float zv = L == 32 ? row_z<L>(z0, zt, 2 * Q::TPC * u + 1) : zu + 1.0f;
        a[u].x = row_weight_form<POLY, ELL>(rp0, a[u].x, zu);
        a[u].y = row_weight_form<POLY, ELL>(rp0, a[u].y, zv);
        b[u].x = row_weight_form<POLY, ELL>(rp1, b[u].x, zu);
        b[u].y = row_weight_form<POLY, ELL>(rp1, b[u].y, zv);
      }
    };
    using std::integral_constant;
    using I2 = integral_constant<int, 2>;
    using I4 = integral_constant<int, 4>;
    if (p.ell == 0) {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        a[u] = make_float2(a[u].x * rp0.value0, a[u].y * rp0.value0);
        b[u] = make_float2(b[u].x * rp1.value0, b[u].y * rp1.value0);
      }
    } else if (p.ell == 2) {
      switch (row_poly_form(2, p.m)) {
        case 0: weigh(integral_constant<int, 0>(), I2()); break;
        case 1: weigh(integral_constant<int, 1>(), I2()); break;
        default: weigh(integral_constant<int, 2>(), I2()); break;
      }
    } else {
      switch (row_poly_form(4, p.m)) {
        case 0: weigh(integral_constant<int, 0>(), I4()); break;
        case 1: weigh(integral_constant<int, 1>(), I4()); break;
        case 2: weigh(integral_constant<int, 2>(), I4()); break;
        case 3: weigh(integral_constant<int, 3>(), I4()); break;
        default: weigh(integral_constant<int, 4>(), I4()); break;
      }
    }
  }
  CPairS v[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) v[u] = cpack_s(a[u], b[u]);
  auto exf = [&](int i) { return &ex[pb * RP + i + (i >> 3)]; };
  reg_fft<L>(v, t, exf, tabz, -1, 2);
#pragma unroll
  for (int u = 0; u < 8; ++u) *exf(t + Q::TPC * u) = v[u];
  __syncthreads();
  float2 *dst0 = W + row0 * g.hp;
  float2 *dst1 = W + row1 * g.hp;
  // Real-to-complex split, outputs k and L - k together: with
  // e = (Z_k + conj Z_{L-k}) / 2 and o = -i (Z_k - conj Z_{L-k}) / 2,
  // X_k = e + o w_k and X_{L-k} = conj(e - o w_k) (w_{L-k} = -conj w_k).
  // Unrolled so the twiddle loads of all outputs issue together.
#pragma unroll
  for (int i = 0; i <= L / 2 / Q::TPC; ++i) {
    const int k = t + Q::TPC * i;
    if (k > L / 2) break;
    const CPairS za = *exf(k);
    const CPairS c = cconj(*exf(k == 0 ? 0 : L - k));
    CPairS e, o;
    e.x = 0.5f * (za.x + c.x);
    e.y = 0.5f * (za.y + c.y);
    const CPairS d = csub(za, c);
    o.x = 0.5f * d.y;
    o.y = -0.5f * d.x;
    const CPairS ow = cmul(o, __ldg(&tabz[k]));
    const CPairS r = cadd(e, ow);
    if (v0) dst0[k] = clane0(r);
    if (v1) dst1[k] = clane1(r);
    if (k != L / 2) {
      const CPairS q = cconj(csub(e, ow));
      if (v0) dst0[L - k] = clane0(q);
      if (v1) dst1[L - k] = clane1(q);
    }
  }
}

// Calls f(POLY, ELL) with the compile-time form of an (ell > 0, m) term's
// row polynomial (row_poly_form).
template <typename F>
__device__ __forceinline__ void with_row_form(const YlmParams &p, F &&f) {
  using std::integral_constant;
  using I2 = integral_constant<int, 2>;
  using I4 = integral_constant<int, 4>;
  if (p.ell == 2) {
    switch (row_poly_form(2, p.m)) {
      case 0: f(integral_constant<int, 0>(), I2()); break;
      case 1: f(integral_constant<int, 1>(), I2()); break;
      default: f(integral_constant<int, 2>(), I2()); break;
    }
  } else {
    switch (row_poly_form(4, p.m)) {
      case 0: f(integral_constant<int, 0>(), I4()); break;
      case 1: f(integral_constant<int, 1>(), I4()); break;
      case 2: f(integral_constant<int, 2>(), I4()); break;
      case 3: f(integral_constant<int, 3>(), I4()); break;
      default: f(integral_constant<int, 4>(), I4()); break;
    }
  }
}

// The row polynomial of form POLY at z (z2 = z^2), as row_weight_form.
template <int POLY>
__device__ __forceinline__ float row_poly_at(const RowPoly &r, float z, float z2) {
  if constexpr (POLY == 0) return r.c[0];
  else if constexpr (POLY == 1) return r.c[1] * z;
  else if constexpr (POLY == 2) return r.c[2] * z2 + r.c[0];
  else if constexpr (POLY == 3) return (r.c[3] * z2 + r.c[1]) * z;
  else return (r.c[4] * z2 + r.c[2]) * z2 + r.c[0];
}

// One row weighted for two terms a and q: b = Y_q * a, then a = Y_a * a,
// with the same operations as row_weight_form; z^2 and 1/r^2 depend only
// on the row and z, so they are computed once for both terms.
template <int L>
__device__ __forceinline__ void weigh_row_pair(const RowPoly &ra,
                                               const YlmParams &pa,
                                               const RowPoly &rq,
                                               const YlmParams &pq, double z0, float zt,
                                               float2 *a, float2 *b) {
  constexpr int TPC = L / 8;
  with_row_form(pa, [&](auto polya, auto ella) {
    with_row_form(pq, [&](auto polyq, auto ellq) {
      constexpr int PA = decltype(polya)::value, EA = decltype(ella)::value;
      constexpr int PQ = decltype(polyq)::value, EQ = decltype(ellq)::value;
      auto one = [&](float d, float z, float &wa, float &wq) {
        const float z2 = z * z;
        const float ir2 = __fdividef(1.0f, ra.rxy2 + z2 + 1e-20f);
        wq = d * row_poly_at<PQ>(rq, z, z2) * ir2;
        wa = d * row_poly_at<PA>(ra, z, z2) * ir2;
        if constexpr (EQ == 4) wq *= ir2;
        if constexpr (EA == 4) wa *= ir2;
      };
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float zu = row_z<L>(z0, zt, 2 * TPC * u);
        const float zv = L == 32 ? row_z<L>(z0, zt, 2 * TPC * u + 1) : zu + 1.0f;
        one(a[u].x, zu, a[u].x, b[u].x);
        one(a[u].y, zv, a[u].y, b[u].y);
      }
    });
  });
}

// The weighted z pass of two (ell > 0, m) terms at once: thread t of row
// group pb holds z[t + TPC u] of one row, and its two transforms are that
// row weighted for term a and for term b.  The density row is read once
// for both terms and each term's W gets its row, so a pair of terms reads
// the density once instead of twice; the transform and the real-to-complex
// split are those of k_zfwd_pp.
template <int L>
__global__ void __launch_bounds__(PP<L>::THREADS, 1024 / PP<L>::THREADS)
    k_zfwd_pp2(const float *rho, float2 *Wa, float2 *Wb, FusedGeom g, YlmParams pa,
               YlmParams pq,
               double z0, const float2 *__restrict__ tabz,
               const float4 *rowtab_a, const float4 *rowtab_b) {
  grid_chain();
  using Q = PP<L>;
  constexpr int RP = L + L / 8 + 1;
  extern __shared__ unsigned char smem_raw[];
  CPairS *ex = reinterpret_cast<CPairS *>(smem_raw);
  const int pb = threadIdx.x / Q::TPC;
  const int t = threadIdx.x - pb * Q::TPC;
  const int64_t nrows = (int64_t)g.n0 * g.n1;
  const int64_t row = (int64_t)blockIdx.x * Q::PB + pb;
  const bool valid = row < nrows;
  const int64_t r = valid ? row : 0;
  const float2 *src = reinterpret_cast<const float2 *>(rho + r * g.n2);
  const RowPoly ra = load_row_poly(rowtab_a, r, pa);
  const RowPoly rq = load_row_poly(rowtab_b, r, pq);
  const float zt = (float)(z0 + (2 * t) * 1.0);
  const float2 zero = make_float2(0.f, 0.f);
  float2 a[8], b[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) a[u] = valid ? src[t + Q::TPC * u] : zero;
  weigh_row_pair<L>(ra, pa, rq, pq, z0 + 2 * t, zt, a, b);
  CPairS v[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) v[u] = cpack_s(a[u], b[u]);
  auto exf = [&](int i) { return &ex[pb * RP + i + (i >> 3)]; };
  reg_fft<L>(v, t, exf, tabz, -1, 2);
#pragma unroll
  for (int u = 0; u < 8; ++u) *exf(t + Q::TPC * u) = v[u];
  __syncthreads();
  if (!valid) return;
  float2 *dst0 = Wa + row * g.hp;
  float2 *dst1 = Wb + row * g.hp;
#pragma unroll
  for (int i = 0; i <= L / 2 / Q::TPC; ++i) {
    const int k = t + Q::TPC * i;
    if (k > L / 2) break;
    const CPairS za = *exf(k);
    const CPairS c = cconj(*exf(k == 0 ? 0 : L - k));
    CPairS e, o;
    e.x = 0.5f * (za.x + c.x);
    e.y = 0.5f * (za.y + c.y);
    const CPairS d = csub(za, c);
    o.x = 0.5f * d.y;
    o.y = -0.5f * d.x;
    const CPairS ow = cmul(o, __ldg(&tabz[k]));
    const CPairS rr = cadd(e, ow);
    dst0[k] = clane0(rr);
    dst1[k] = clane1(rr);
    if (k != L / 2) {
      const CPairS q = cconj(csub(e, ow));
      dst0[L - k] = clane0(q);
      dst1[L - k] = clane1(q);
    }
  }
}

// Per-row Horner coefficients of one (ell, m) (row_poly), two float4 per
// row, so the z pass does no FP64 work per row.
__global__ void k_rowpoly(float4 *tab, int64_t nrows, int n1,
                          YlmParams p, double x0, double y0) {
  grid_chain();
  for (int64_t row = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
       row < nrows; row += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(row / n1);
    const int y = (int)(row - (int64_t)x * n1);
    const RowPoly r = row_poly(p, x0 + x * 1.0, y0 + y * 1.0);
    tab[2 * row] = make_float4(r.c[0], r.c[1], r.c[2], r.c[3]);
    tab[2 * row + 1] = make_float4(r.c[4], r.rxy2, 0.f, 0.f);
  }
}

// Per-cell r-subgrid weight of one (ell, m): Y_lm(r) with the r-subgrid
// normalisation (make_ylm, correlator.h:477-480), computed once per
// correlator and multipole so the z inverse pass does a multiply-add.  In the
// even form a cell stands for its mirror image too, whose coordinates are not
// its own with the sign changed to the last bit (start + i step, rounded): its
// weight is the mean of the two, or the quadrupole near r = 0, where the cells
// of a bin cancel, is off by those bits.
template <typename RT>
__global__ void k_rtable(RT *__restrict__ tab, FusedGeom g,
                         const double *__restrict__ raxis, YlmParams pr) {
  const size_t n = (size_t)g.nri * g.rs * g.rs;
  const int x0 = g.rs - g.nri;  // the even form keeps the rows x >= 0
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const int rk = (int)(i % g.rs);
    const int rj = (int)((i / g.rs) % g.rs);
    const int ri = (int)(i / ((size_t)g.rs * g.rs));
    double y = ylm_eval(pr, 1.0, raxis[x0 + ri], raxis[rj], raxis[rk]);
    if (x0 > 0) {
      const int e = g.rs - 1;
      y = 0.5 * (y + ylm_eval(pr, 1.0, raxis[e - x0 - ri], raxis[e - rj], raxis[e - rk]));
    }
    tab[i] = (RT)y;
  }
}

// Per-cell k-subgrid weight of one (ell, m): Y_lm(k) * 4 pi / (W(kx) W(ky)
// W(kz)) with make_ylm's arithmetic (correlator.h:453-466), computed once
// per correlator and multipole so the extraction in the x pass is a
// multiply-add; the mean of a cell's and of its mirror image's (k_rtable).
template <typename KT>
__global__ void k_ktable(KT *__restrict__ tab, FusedGeom g, KAxes ax, YlmParams pk) {
  const int oz = g.ks2 / 2;
  const size_t n = (size_t)g.ks0 * g.ks1 * g.kp;
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n;
       c += (size_t)gridDim.x * blockDim.x) {
    const int k = (int)(c % g.kp) + oz;
    const int j = (int)((c / g.kp) % g.ks1);
    const int i = (int)(c / ((size_t)g.kp * g.ks1));
    if (k >= g.ks2) {  // padding of the row
      tab[c] = (KT)0;
      continue;
    }
    auto weight = [&](int a, int b, int d) {
      const double inv_w = 1.0 / (ax.wx[a] * ax.wy[b] * ax.wz[d]);
      return ylm_eval(pk, inv_w, ax.kx[a], ax.ky[b], ax.kz[d]);
    };
    tab[c] = (KT)(0.5 * (weight(i, j, k) +
                         weight(g.ks0 - 1 - i, g.ks1 - 1 - j, g.ks2 - 1 - k)));
  }
}

// One term's unweighted k- and r-subgrids times their weights and `scale`,
// added to the multipole's subgrids or (first) written over them.
__global__ void k_add_term(double *ksub, double *rsub, const double *kterm,
                           const double *rterm, const double *__restrict__ ktab,
                           const double *__restrict__ rtab, size_t nk, size_t nr,
                           double scale, int first) {
  grid_chain();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nk + nr;
       i += (size_t)gridDim.x * blockDim.x) {
    const bool k = i < nk;
    const size_t c = k ? i : i - nk;
    double *dst = k ? ksub : rsub;
    const double v = k ? ktab[c] * (scale * kterm[c]) : rtab[c] * (scale * rterm[c]);
    dst[c] = first ? v : dst[c] + v;
  }
}

__global__ void k_to_float(const double *__restrict__ in, float *__restrict__ out,
                           size_t n, double shift) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    out[i] = (float)(in[i] - shift);
}

template <typename C>
std::vector<C> root_table(int order) {
  std::vector<C> t(order);
  for (int m = 0; m < order; ++m) {
    // e^{-2 pi i m / order}, argument reduced exactly before the FP64 call.
    const double a = 2.0 * M_PI * (double)m / (double)order;
    t[m].x = (decltype(t[m].x))cos(a);
    t[m].y = (decltype(t[m].y))(-sin(a));
  }
  return t;
}

// ----------------------------------------------------- power-of-two dispatch

bool is_p2(int L) { return L >= 64 && L <= 1024 && (L & (L - 1)) == 0; }
// Longest row (z) of the passes (longer ones go through cuFFT, whose weights are
// FP64); columns end at 1280 (gen_supported).
constexpr int kMaxRow = 2560;

template <typename T, int L>
size_t p2_col_smem() {
  return (size_t)L * P2<T, L>::B * sizeof(C2<T>);
}
template <typename T, int L>
size_t p2_row_smem() {
  return (size_t)P2<T, L>::B * (L + L / 8 + 1) * sizeof(C2<T>);
}

// Calls f.template operator()<L>() for the power-of-two L of a column, and of a
// row's pairs.
template <typename F>
void with_p2(int L, F &&f) {
  switch (L) {
    case 64: f.template operator()<64>(); break;
    case 128: f.template operator()<128>(); break;
    case 256: f.template operator()<256>(); break;
    case 512: f.template operator()<512>(); break;
    default: f.template operator()<1024>(); break;
  }
}
template <typename F>
void with_p2_row(int L, F &&f) {
  if (L == 32) f.template operator()<32>();
  else with_p2(L, f);
}

template <typename K>
void big_smem(K kernel) {
  FC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               200 * 1024));
}

// Shared-memory limits of the kernels that a correlator launches, axis by axis.
template <typename T, int L>
void p2_z_limits(bool weighted, bool pairs) {
  big_smem(k_zinv_p2<T, L>);
  if constexpr (std::is_same_v<T, double>) {
    big_smem(k_zfwd_p2<L, false>);
    if (weighted) big_smem(k_zfwd_p2<L, true>);
  } else {
    big_smem(k_zfwd_pp<L, false>);
    if (weighted) big_smem(k_zfwd_pp<L, true>);
    if (weighted && pairs) big_smem(k_zfwd_pp2<L>);
  }
}
template <typename T, int L>
void p2_y_limits() {
  if constexpr (std::is_same_v<T, double>) {
    big_smem(k_yfwd_p2<T, L>);
    big_smem(k_yinv_p2<T, L>);
  } else {
    big_smem(k_yfwd_pp<L>);
    big_smem(k_yinv_pp<L>);
  }
}
template <typename T, int L>
void p2_x_limits(int mode, bool even) {
  if constexpr (std::is_same_v<T, double>) {
    if (mode == 0) big_smem(k_xcorr_p2<L, 0, false>);
    else if (mode == 3) big_smem(k_xcorr_p2<L, 3, true>);
    else if (mode == 2 && even) big_smem(k_xcorr_p2<L, 2, true>);
    else if (mode == 2) big_smem(k_xcorr_p2<L, 2, false>);
    else if (even) big_smem(k_xcorr_p2<L, 1, true>);
    else big_smem(k_xcorr_p2<L, 1, false>);
  } else {
    if (mode == 0) big_smem(k_xfwd_pp<L>);
    else if (mode == 3) big_smem(k_xcorr_pp<L, 3, true>);
    else if (mode == 2 && even) big_smem(k_xcorr_pp<L, 2, true>);
    else if (mode == 2) big_smem(k_xcorr_pp<L, 2, false>);
    else if (even) big_smem(k_xcorr_pp<L, 1, true>);
    else big_smem(k_xcorr_pp<L, 1, false>);
  }
}

}  // namespace

bool FusedSurvey::supported(const int shape[3], int rsize) {
  return shape[2] <= kMaxRow && gen_supported(shape[0], false) && gen_supported(shape[1], false) &&
         gen_supported(shape[2], true) && rsize > 0;
}

FusedSurvey::FusedSurvey(const int shape[3], int rsize, const int kshape[3],
                         bool fp64, bool even, bool survey)
    : fp64_(fp64) {
  // (A planned failure takes a periodic correlator's plan, cuFFT's or this; a
  // survey that makes no cuFFT plan passes it over.)
  if (!survey && fault_fires(kFaultFftPlan))
    FC_THROW(FC_ERR_CUFFT, "injected FFT plan creation failure");
  g.n0 = shape[0];
  g.n1 = shape[1];
  g.n2 = shape[2];
  g.m = shape[2] / 2;
  g.h = g.m + 1;
  g.hp = (g.h + 15) / 16 * 16;
  g.rs = rsize;
  g.ro = rsize / 2;
  g.ks0 = kshape[0];
  g.ks1 = kshape[1];
  g.ks2 = kshape[2];
  g.kp = (g.ks2 / 2 + 1 + 3) / 4 * 4;
  g.nri = even ? g.ro + 1 : g.rs;
  // Axes that the power-of-two passes do not take.
  if (!is_p2(g.n0)) gx.init(g.n0, fp64);
  if (!is_p2(g.n1)) gy.init(g.n1, fp64);
  if (!p2_rows()) gz.init(g.n2, fp64);
  const size_t eb = fp64 ? 16 : 8;
  auto roots = [&](DeviceBuffer &tab, int n) {
    if (fp64) upload(tab, root_table<double2>(n));
    else upload(tab, root_table<float2>(n));
  };
  if (is_p2(g.n0)) roots(tabx, g.n0);
  if (is_p2(g.n1)) roots(taby, g.n1);
  if (p2_rows()) roots(tabz, g.n2);
  const size_t nc = (size_t)g.n0 * g.n1 * g.hp;
  W.resize(nc * eb);
  if (survey) G.resize(nc * eb);
  if (g.nri > g.n0) Wr.resize((size_t)g.nri * g.n1 * g.hp * eb);
  Wry.resize((size_t)g.nri * g.rs * g.hp * eb);
  if (survey && wide()) {
    kterm.resize(k_cells() * sizeof(double));
    rterm.resize(r_cells() * sizeof(double));
  }
  if (survey && pairs()) {
    rowtab.resize((size_t)g.n0 * g.n1 * 2 * sizeof(float4));
    W2.resize(nc * eb);
    rowtab2.resize((size_t)g.n0 * g.n1 * 2 * sizeof(float4));
  }
  if (fp64) set_limits<double>(survey);
  else set_limits<float>(survey);
}

template <typename V>
void FusedSurvey::upload(DeviceBuffer &dst, const std::vector<V> &v) {
  dst.resize(v.size() * sizeof(V));
  FC_CUDA(cudaMemcpy(dst.get(), v.data(), v.size() * sizeof(V),
                     cudaMemcpyHostToDevice));
}

template <typename T>
void FusedSurvey::x_limits(int mode) {
  if (is_p2(g.n0)) with_p2(g.n0, [&]<int L>() { p2_x_limits<T, L>(mode, even()); });
  else gen_x_limits<T>(g.n0, mode, even());
}

template <typename T>
void FusedSurvey::set_limits(bool survey) {
  if (p2_rows())
    with_p2_row(g.m, [&]<int L>() { p2_z_limits<T, L>(survey, pairs()); });
  else
    gen_z_limits<T>(g.n2, survey);
  if (is_p2(g.n1)) with_p2(g.n1, [&]<int L>() { p2_y_limits<T, L>(); });
  else gen_y_limits<T>(g.n1);
  if (survey) {
    for (int mode : {0, 1, 2}) x_limits<T>(mode);
    product_ready = true;
  } else {
    x_limits<T>(3);
  }
}

void FusedSurvey::prepare_product() {
  G.resize(W.bytes());
  if (product_ready) return;
  for (int mode : {0, 1}) {
    if (fp64_) x_limits<double>(mode);
    else x_limits<float>(mode);
  }
  product_ready = true;
}

FusedSurvey::Cells FusedSurvey::prepare_input(const void *rho, bool f32,
                                              cudaStream_t s) {
  FC_REQUIRE(!(fp64_ && f32), FC_ERR_INVALID,
             "the FP64 passes take FP64 cells");
  if (reads_as_is(f32)) return {rho, f32};
  const size_t n = (size_t)g.n0 * g.n1 * g.n2;
  rho32.resize(n * sizeof(float));  // (for the first FP64 cells)
  k_to_float<<<grid_for(n, 256), 256, 0, s>>>(static_cast<const double *>(rho),
                                              rho32.as<float>(), n, 0.0);
  FC_LAUNCH_CHECK();
  return {rho32.get(), true};
}

template <typename T>
void FusedSurvey::zfwd(Cells in, bool weight, const YlmParams &p, const double xyz0[3],
                       cudaStream_t s) {
  if (p2_rows()) {
    const void *rho = in.p;
    with_p2_row(g.m, [&]<int L>() {
      using Q = P2<T, L>;
      const int64_t nrows = (int64_t)g.n0 * g.n1;
      const unsigned blocks = (unsigned)((nrows + Q::B - 1) / Q::B);
      if constexpr (std::is_same_v<T, float>) {
        using PQ = PP<L>;
        const float4 *rt = nullptr;
        if (weight && p.ell != 0) {
          launch_after(k_rowpoly, grid_for(nrows, 256), 256, 0, s, 
              rowtab.as<float4>(), nrows, g.n1, p, xyz0[0], xyz0[1]);
          FC_LAUNCH_CHECK();
          rt = rowtab.as<float4>();
        }
        if (weight)
          launch_after(k_zfwd_pp<L, true>, blocks, PQ::THREADS, p2_row_smem<T, L>(), s, 
              (const float *)rho, W.as<float2>(), g, p, xyz0[0], xyz0[1],
              xyz0[2], tabz.as<float2>(), rt);
        else
          launch_after(k_zfwd_pp<L, false>, blocks, PQ::THREADS, p2_row_smem<T, L>(), s, 
              (const float *)rho, W.as<float2>(), g, p, xyz0[0], xyz0[1],
              xyz0[2], tabz.as<float2>(), nullptr);
        return;
      }
      if constexpr (std::is_same_v<T, double>) {
        auto go = [&](auto kernel) {
          launch_small(kernel, blocks, Q::THREADS, p2_row_smem<T, L>(), s, 
              (const T *)rho, W.as<C2<T>>(), g, p, xyz0[0], xyz0[1], xyz0[2],
              tabz.as<C2<T>>());
        };
        if (weight) go(k_zfwd_p2<L, true>);
        else go(k_zfwd_p2<L, false>);
      }
    });
    FC_LAUNCH_CHECK();
    return;
  }
  gen_zfwd<T>(gz, g, in.p, in.f32, W.as<C2<T>>(), weight, p, xyz0, s);
}

template <typename T>
void FusedSurvey::yfwd(cudaStream_t s) {
  if (is_p2(g.n1)) {
    with_p2(g.n1, [&]<int L>() {
      using Q = P2<T, L>;
      if constexpr (std::is_same_v<T, float>) {
        using Y = PY<L>;
        dim3 grid((g.h + Y::B - 1) / Y::B, g.n0);
        launch_after(k_yfwd_pp<L>, grid, Y::THREADS, Y::smem, s, W.as<float2>(), g,
                                                        taby.as<float2>());
      } else {
        dim3 grid((g.h + Q::B - 1) / Q::B, g.n0);
        launch_small(k_yfwd_p2<T, L>, grid, Q::THREADS, p2_col_smem<T, L>(), s, 
            W.as<C2<T>>(), g, taby.as<C2<T>>());
      }
    });
    FC_LAUNCH_CHECK();
    return;
  }
  gen_yfwd<T>(gy, g, W.as<C2<T>>(), s);
}

template <typename T>
void FusedSurvey::grid2_x(cudaStream_t s) {
  if (!is_p2(g.n0)) {
    gen_x<T>(gx, g, 0, W.as<C2<T>>(), nullptr, G.as<C2<T>>(), nullptr, nullptr, T(0), true, s);
    return;
  }
  with_p2(g.n0, [&]<int L>() {
    if constexpr (std::is_same_v<T, float>) {
      using Y = PY<L>;
      launch_after(k_xfwd_pp<L>, dim3((g.h + Y::B - 1) / Y::B, g.n1), Y::THREADS, Y::smem, s, 
          W.as<float2>(), G.as<float2>(), g, tabx.as<float2>());
    } else {
      using Q = P2<T, L>;
      launch_small(k_xcorr_p2<L, 0, false>, dim3((g.h + Q::B - 1) / Q::B, g.n1), Q::THREADS, p2_col_smem<T, L>(), s, 
              W.as<C2<T>>(), nullptr, G.as<C2<T>>(), nullptr, g, tabx.as<C2<T>>(), nullptr,
              T(0), 1);
    }
  });
  FC_LAUNCH_CHECK();
}

template <typename T>
void FusedSurvey::xcorr(int mode, double *ksub, const void *ktab_v, double w00,
                        bool first, cudaStream_t s) {
  const T *ktab = static_cast<const T *>(ktab_v);
  if (!is_p2(g.n0)) {
    gen_x<T>(gx, g, mode, W.as<C2<T>>(), G.as<C2<T>>(), inverse_rows<T>(), ksub,
             ktab, (T)w00, first, s);
    return;
  }
  with_p2(g.n0, [&]<int L>() {
    if constexpr (std::is_same_v<T, float>) {
      using Y = PY<L, kXB>;
      auto go = [&](auto kernel, int nyq) {
        launch_after(kernel, dim3((g.h + Y::B - 1) / Y::B, g.n1), Y::THREADS, Y::smem, s, 
            W.as<float2>(), G.as<float2>(), inverse_rows<float>(), ksub, g, tabx.as<float2>(),
            ktab, (float)w00, nyq, first);
      };
      const int nyq = nyq_group<Y::B>(ksub != nullptr);
      if (mode == 3) go(k_xcorr_pp<L, 3, true>, 0);
      else if (mode == 2 && even()) go(k_xcorr_pp<L, 2, true>, 0);
      else if (mode == 2) go(k_xcorr_pp<L, 2, false>, 0);
      else if (even()) go(k_xcorr_pp<L, 1, true>, nyq);
      else go(k_xcorr_pp<L, 1, false>, nyq);
    } else {
      using Q = P2<T, L>;
      auto go = [&](auto kernel) {
        launch_small(kernel, dim3((g.h + Q::B - 1) / Q::B, g.n1), Q::THREADS, p2_col_smem<T, L>(), s, 
            W.as<C2<T>>(), G.as<C2<T>>(), inverse_rows<T>(), ksub, g, tabx.as<C2<T>>(), ktab,
            w00, first);
      };
      if (mode == 3) go(k_xcorr_p2<L, 3, true>);
      else if (mode == 2 && even()) go(k_xcorr_p2<L, 2, true>);
      else if (mode == 2) go(k_xcorr_p2<L, 2, false>);
      else if (even()) go(k_xcorr_p2<L, 1, true>);
      else go(k_xcorr_p2<L, 1, false>);
    }
  });
  FC_LAUNCH_CHECK();
}

template <typename T>
void FusedSurvey::yinv(cudaStream_t s) {
  if (is_p2(g.n1)) {
    with_p2(g.n1, [&]<int L>() {
      using Q = P2<T, L>;
      if constexpr (std::is_same_v<T, float>) {
        using Y = PY<L>;
        dim3 grid((g.h + Y::B - 1) / Y::B, g.nri);
        launch_after(k_yinv_pp<L>, grid, Y::THREADS, Y::smem, s, 
            inverse_rows<float>(), Wry.as<float2>(), g, taby.as<float2>(),
            nyq_group<Y::B>(false));
      } else {
        dim3 grid((g.h + Q::B - 1) / Q::B, g.nri);
        launch_small(k_yinv_p2<T, L>, grid, Q::THREADS, p2_col_smem<T, L>(), s, 
            inverse_rows<T>(), Wry.as<C2<T>>(), g, taby.as<C2<T>>());
      }
    });
    FC_LAUNCH_CHECK();
    return;
  }
  gen_yinv<T>(gy, g, inverse_rows<T>(), Wry.as<C2<T>>(), s);
}

template <typename T>
void FusedSurvey::zinv(double *rsub, const void *rtab_v, bool first, cudaStream_t s) {
  const T *rtab = static_cast<const T *>(rtab_v);
  if (p2_rows()) {
    with_p2_row(g.m, [&]<int L>() {
      using Q = P2<T, L>;
      const int nrows = g.nri * g.rs;
      const unsigned blocks = (unsigned)((nrows + Q::B - 1) / Q::B);
      launch_chain(!fp64_ || blocks <= 4u * sm_count(), k_zinv_p2<T, L>, blocks, Q::THREADS, p2_row_smem<T, L>(), s, 
          Wry.as<C2<T>>(), rsub, g, tabz.as<C2<T>>(), rtab, first);
    });
    FC_LAUNCH_CHECK();
    return;
  }
  gen_zinv<T>(gz, g, Wry.as<C2<T>>(), rsub, rtab, first, s);
}

const void *FusedSurvey::r_table(int ell, int m, const double *raxis,
                                 const YlmParams &pr, cudaStream_t s) {
  const int key = ell * 16 + (m + ell);
  auto it = rtabs.find(key);
  if (it != rtabs.end()) return it->second.get();
  const size_t n = (size_t)g.nri * g.rs * g.rs;
  DeviceBuffer &b = rtabs[key];
  // FP64 for the FP64 form and wide rows, else FP32 (the product with the
  // transform and the accumulation stay FP64).
  if (fp64_ || wide()) {
    b.resize(std::max<size_t>(n, 1) * sizeof(double));
    k_rtable<double><<<grid_for(n, 256), 256, 0, s>>>(b.as<double>(), g, raxis, pr);
  } else {
    b.resize(std::max<size_t>(n, 1) * sizeof(float));
    k_rtable<float><<<grid_for(n, 256), 256, 0, s>>>(b.as<float>(), g, raxis, pr);
  }
  FC_LAUNCH_CHECK();
  return b.get();
}

void FusedSurvey::prepare_tables(int maxell, double ncells, const double *raxis,
                                 const KAxes &ka, bool with_k, cudaStream_t s) {
  for (int ell = 0; ell <= maxell; ell += 2)
    for (int m = -ell; m <= ell; ++m) {
      r_table(ell, m, raxis, make_ylm_params(ell, m, 4.0 * M_PI / ncells), s);
      if (with_k) k_table(ell, m, ka, s);
    }
}

const void *FusedSurvey::k_table(int ell, int m, const KAxes &ka,
                                 cudaStream_t s) {
  const int key = ell * 16 + (m + ell);
  auto it = ktabs.find(key);
  if (it != ktabs.end()) return it->second.get();
  const size_t n = k_cells();
  DeviceBuffer &b = ktabs[key];
  const YlmParams pk = make_ylm_params(ell, m, 4.0 * M_PI);
  // FP64 weights for the FP64 form and wide rows; the others keep them in FP32
  // (a relative rounding of 6e-8, far inside their precision).
  if (fp64_ || wide()) {
    b.resize(std::max<size_t>(n, 1) * sizeof(double));
    k_ktable<double><<<grid_for(n, 256), 256, 0, s>>>(
        b.as<double>(), g, ka, pk);
  } else {
    b.resize(std::max<size_t>(n, 1) * sizeof(float));
    k_ktable<float><<<grid_for(n, 256), 256, 0, s>>>(
        b.as<float>(), g, ka, pk);
  }
  FC_LAUNCH_CHECK();
  return b.get();
}

void FusedSurvey::grid2(Cells in, cudaStream_t s, const KAxes &ka) {
  (void)ka;
  prepare_product();
  YlmParams none = make_ylm_params(0, 0, 1.0);
  const double zero[3] = {0, 0, 0};
  if (fp64_) {
    zfwd<double>(in, false, none, zero, s);
    yfwd<double>(s);
    grid2_x<double>(s);
  } else {
    zfwd<float>(in, false, none, zero, s);
    yfwd<float>(s);
    grid2_x<float>(s);
  }
}

bool FusedSurvey::p2_rows() const {
  return g.n2 % 2 == 0 && (g.m == 32 || is_p2(g.m));
}
bool FusedSurvey::pairs() const { return !fp64_ && p2_rows(); }

void FusedSurvey::zfwd_pair(Cells in, int ell_a, int m_a, int ell_b,
                            int m_b, const double xyz0[3], cudaStream_t s,
                            PhaseHook *hook) {
  FC_REQUIRE(pairs() && ell_a > 0 && ell_b > 0, FC_ERR_STATE,
             "paired z pass needs two weighted FP32 terms");
  const YlmParams pa = make_ylm_params(ell_a, m_a, 1.0);
  const YlmParams pb = make_ylm_params(ell_b, m_b, 1.0);
  const int64_t nrows = (int64_t)g.n0 * g.n1;
  launch_after(k_rowpoly, grid_for(nrows, 256), 256, 0, s, rowtab.as<float4>(), nrows,
                                                 g.n1, pa, xyz0[0], xyz0[1]);
  FC_LAUNCH_CHECK();
  launch_after(k_rowpoly, grid_for(nrows, 256), 256, 0, s, rowtab2.as<float4>(), nrows,
                                                 g.n1, pb, xyz0[0], xyz0[1]);
  FC_LAUNCH_CHECK();
  if (hook) hook->begin("zfwd2");
  with_p2_row(g.m, [&]<int L>() {
    using PQ = PP<L>;
    const unsigned blocks = (unsigned)((nrows + PQ::PB - 1) / PQ::PB);
    launch_after(k_zfwd_pp2<L>, blocks, PQ::THREADS, p2_row_smem<float, L>(), s, 
        static_cast<const float *>(in.p), W.as<float2>(), W2.as<float2>(), g,
        pa, pb, xyz0[2], tabz.as<float2>(), rowtab.as<float4>(),
        rowtab2.as<float4>());
  });
  FC_LAUNCH_CHECK();
  if (hook) hook->end();
}

int FusedSurvey::term(Cells in, int ell, int m, const double xyz0[3],
                       double ncells, double *ksub, double *rsub,
                       const double *raxis, const KAxes &ka, cudaStream_t s,
                       PhaseHook *hook, bool first, bool g_of_input, bool z_done) {
  const YlmParams pw = make_ylm_params(ell, m, 1.0);
  const YlmParams pr = make_ylm_params(ell, m, 4.0 * M_PI / ncells);
  const void *ktab = ksub ? k_table(ell, m, ka, s) : nullptr;
  const void *rtab = r_table(ell, m, raxis, pr, s);
  const bool from_g = ell == 0 && g_of_input;
  // Wide rows: the passes leave the term's subgrids unweighted, and
  // k_add_term weights them in FP64 (the constant of from_g among it).
  const bool w = wide();
  double *kdst = w && ksub ? kterm.as<double>() : ksub;
  double *rdst = w ? rterm.as<double>() : rsub;
  const void *kw = w ? nullptr : ktab, *rw = w ? nullptr : rtab;
  const bool over = w || first;
  auto run = [&](auto tag) {
    using T = decltype(tag);
    if (from_g) {
      // The weight is the constant pw.value0, so the term's transform is
      // value0 * G (see k_xcorr_p2, MODE 2).
      if (hook) hook->begin("xcorr00");
      xcorr<T>(2, kdst, kw, w ? 1.0 : pw.value0, over, s);
      if (hook) hook->end();
    } else {
      if (!z_done) {
        if (hook) hook->begin("zfwd");
        zfwd<T>(in, true, pw, xyz0, s);
        if (hook) hook->end();
      }
      if (hook) hook->begin("yfwd");
      yfwd<T>(s);
      if (hook) hook->end();
      if (hook) hook->begin("xcorr");
      xcorr<T>(1, kdst, kw, 0.0, over, s);
      if (hook) hook->end();
    }
    if (hook) hook->begin("yinv");
    yinv<T>(s);
    if (hook) hook->end();
    if (hook) hook->begin("zinv");
    zinv<T>(rdst, rw, over, s);
    if (w) {
      const size_t nk = ksub ? k_cells() : 0, nr = r_cells();
      launch_small(k_add_term, grid_for(nk + nr, 256), 256, 0, s, ksub, rsub,
                   kterm.as<double>(), rterm.as<double>(),
                   static_cast<const double *>(ktab), static_cast<const double *>(rtab),
                   nk, nr, from_g ? pw.value0 : 1.0, first);
      FC_LAUNCH_CHECK();
    }
    if (hook) hook->end();
  };
  if (fp64_)
    run(double());
  else
    run(float());
  return from_g ? 1 : 2;
}

void FusedSurvey::periodic(Cells in, bool cross, double *ksub, double *rsub,
                           cudaStream_t s, PhaseHook *hook) {
  const YlmParams none = make_ylm_params(0, 0, 1.0);
  const double zero[3] = {0, 0, 0};
  auto phase = [&](const char *name, auto f) {
    if (hook) hook->begin(name);
    f();
    if (hook) hook->end();
  };
  auto run = [&](auto tag) {
    using T = decltype(tag);
    phase("zfwd", [&] { zfwd<T>(in, false, none, zero, s); });
    phase("yfwd", [&] { yfwd<T>(s); });
    phase("xcorr", [&] { xcorr<T>(cross ? 1 : 3, ksub, nullptr, 0.0, true, s); });
    phase("yinv", [&] { yinv<T>(s); });
    phase("zinv", [&] { zinv<T>(rsub, nullptr, true, s); });
  };
  if (fp64_)
    run(double());
  else
    run(float());
}

}  // namespace fc
