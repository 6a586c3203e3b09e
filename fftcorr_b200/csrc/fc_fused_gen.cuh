// fc_fused_gen.cuh -- the passes of the fused correlator (fc_fused.cu) along
// an axis whose length is not a power of two, any product of 2, 3, 5 and 7,
// even or odd, with the transform of fc_gfft.cuh.
//
// The column passes (x, y) take adjacent columns of one plane per CTA, 128
// bytes of a row; the row passes (z) take pairs of rows, both of which ride
// through one complex transform of the full row length as its real and
// imaginary parts (so an odd row length needs nothing of its own) and are
// separated by X_a(k) = (Z(k) + conj Z(N-k)) / 2 and X_b(k) = (Z(k) -
// conj Z(N-k)) / 2i.  First passes read device memory into registers, last
// passes write it from registers.
//
// Measured per launch on a 250 x 360 x 378 FP32 grid (34M cells, one B200),
// against the engine before it (mixed radices chosen largest power of two
// first, loads and stores as passes of their own through shared memory, one
// column per thread, per-element modulos): z 339 -> 104 us, y 164 -> 67 us,
// x with product and inverse 611 -> 110 us (134 before the even form), inverse y
// 41 -> 15 us (19); a cross correlation at ell <= 4 18.4 -> 5.05 ms.  The y pass
// moves 274 MB at 4.1 TB/s; all are bound by instruction issue and by barriers
// between the passes (two CTAs of an SM at 64 registers in y and at 80 in x, five
// at up to 96 in z).  Before the even form, one column per thread instead of two
// took y 91 us and x 184 us; 64-byte rows (half the tile, more CTAs) y 76 and x
// 162 us, from bank conflicts and scattered twiddle loads.
//
// (fc_fused_gen_f32.cu and fc_fused_gen_f64.cu compile them, side by side.)
#pragma once

#include <algorithm>

#include "fc_fused_gen.h"

namespace fc {
namespace {

template <typename T>
using C2 = typename Vec2<T>::type;

constexpr int kRowThreads = 128;
constexpr size_t kGenSmem = 200 * 1024;

// What a thread carries through a transform: two complex columns (or row
// pairs) in FP32, which share twiddles, indices and 16-byte accesses and use
// the packed two-lane instructions, one in FP64.
template <typename T>
struct GElem;
template <>
struct GElem<float> {
  using E = CPair;
  static constexpr int W = 2;  // complex values per element
  // The element at p, of which n values exist; the others are zero.
  __device__ static CPair load(const float2 *p, int n) {
    const float4 q = n > 0 ? *reinterpret_cast<const float4 *>(p) : make_float4(0, 0, 0, 0);
    return cpack(make_float2(q.x, q.y), n > 1 ? make_float2(q.z, q.w) : make_float2(0, 0));
  }
  __device__ static void store(float2 *p, const CPair &v, int n) {
    const float2 a = clane0(v), b = clane1(v);
    if (n > 1) *reinterpret_cast<float4 *>(p) = make_float4(a.x, a.y, b.x, b.y);
    else if (n > 0) *p = a;
  }
};
template <>
struct GElem<double> {
  using E = double2;
  static constexpr int W = 1;
  __device__ static double2 load(const double2 *p, int n) {
    return n > 0 ? *p : make_double2(0, 0);
  }
  __device__ static void store(double2 *p, const double2 &v, int n) {
    if (n > 0) *p = v;
  }
};

// A column pass takes B elements of a row per CTA.  With B = 8 a row is 128
// bytes of device memory and of shared memory, which each 8-lane phase of a
// 16-byte access covers without bank conflicts; longer transforms take 4,
// padded, so that two CTAs still fit an SM.
constexpr int pitch_of(int B) { return B == 8 ? 8 : B + 1; }
template <typename T, int B>
constexpr int kCols = B * GElem<T>::W;
inline int col_width(int L) { return L <= 430 ? 8 : 4; }
// Most threads of a y and of an x pass.
constexpr int kYThreads = 512, kXThreads = 384;

// A middle (or, with first, the first) pass over B columns of elements
// between two shared buffers.
template <int SIGN, int B, typename E, typename Tw>
__device__ __forceinline__ void col_pass(const GPass &ps, const Tw *__restrict__ tw,
                                         const E *src, E *dst, bool first) {
  constexpr int BP = pitch_of(B);
  with_radix(ps.R, [&]<int R>() {
    for (int bf = threadIdx.x; bf < ps.LR * B; bf += blockDim.x) {
      const int j = bf / B, b = bf % B;
      E v[R];
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = src[(j + q * ps.LR) * BP + b];
      int k = 0;
      if (!first) {
        k = j - gdiv(j, ps.Ns, ps.mNs) * ps.Ns;
        g_twiddle<R, SIGN>(v, tw + ps.tw, ps.Ns, k);
      }
      GDft<R, SIGN, E>::run(v);
      E *o = dst + ((j - k) * R + k) * BP + b;
#pragma unroll
      for (int q = 0; q < R; ++q) o[q * ps.Ns * BP] = v[q];
    }
  });
  __syncthreads();
}

// The first pass, read from device memory (columns at and above nb are
// zero), into dst.
template <int SIGN, int B, typename T>
__device__ __forceinline__ void col_first(const GPass &ps, const C2<T> *src,
                                          int64_t stride, int nb,
                                          typename GElem<T>::E *dst) {
  using GE = GElem<T>;
  using E = typename GE::E;
  constexpr int BP = pitch_of(B);
  with_radix(ps.R, [&]<int R>() {
    for (int bf = threadIdx.x; bf < ps.LR * B; bf += blockDim.x) {
      const int j = bf / B, b = bf % B;
      const C2<T> *p = src + j * stride + GE::W * b;
      E v[R];
#pragma unroll
      for (int q = 0; q < R; ++q)
        v[q] = GE::load(p + (int64_t)(q * ps.LR) * stride, nb - GE::W * b);
      GDft<R, SIGN, E>::run(v);
      E *o = dst + j * R * BP + b;
#pragma unroll
      for (int q = 0; q < R; ++q) o[q * BP] = v[q];
    }
  });
  __syncthreads();
}

// The last pass: store(i, b, value) for every output row i.
template <int SIGN, int B, typename E, typename Tw, typename Store>
__device__ __forceinline__ void col_last(const GPass &ps, const Tw *__restrict__ tw,
                                         const E *src, Store store) {
  constexpr int BP = pitch_of(B);
  with_radix(ps.R, [&]<int R>() {
    for (int bf = threadIdx.x; bf < ps.LR * B; bf += blockDim.x) {
      const int j = bf / B, b = bf % B;
      E v[R];
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = src[(j + q * ps.LR) * BP + b];
      g_twiddle<R, SIGN>(v, tw + ps.tw, ps.Ns, j);
      GDft<R, SIGN, E>::run(v);
#pragma unroll
      for (int q = 0; q < R; ++q) store(j + q * ps.LR, b, v[q]);
    }
  });
}

// The passes between the first and the last; returns the buffer they end in.
template <int SIGN, int B, typename E, typename Tw>
__device__ __forceinline__ E *col_middle(const GPlan &p, const Tw *__restrict__ tw,
                                         E *src, E *dst) {
  for (int s = 1; s + 1 < p.npass; ++s) {
    col_pass<SIGN, B>(p.p[s], tw, src, dst, false);
    E *t = src;
    src = dst;
    dst = t;
  }
  return src;
}

// ------------------------------------------------------------------ y
template <typename T, int B>
__global__ void __launch_bounds__(kYThreads, sizeof(T) == 4 ? 2 : 1)
    k_gyfwd(C2<T> *W, FusedGeom g, const __grid_constant__ GPlan plan,
            const C2<T> *__restrict__ tw) {
  grid_chain();
  using GE = GElem<T>;
  using E = typename GE::E;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  E *buf = reinterpret_cast<E *>(smem_raw);
  const int kz0 = blockIdx.x * kCols<T, B>;
  const int nb = g.h - kz0;
  C2<T> *col = W + (int64_t)blockIdx.y * g.n1 * g.hp + kz0;
  col_first<-1, B, T>(plan.p[0], col, g.hp, nb, buf);
  const E *res = col_middle<-1, B>(plan, tw, buf, buf + g.n1 * pitch_of(B));
  col_last<-1, B>(plan.p[plan.npass - 1], tw, res, [&](int i, int b, const E &v) {
    GE::store(col + (int64_t)i * g.hp + GE::W * b, v, nb - GE::W * b);
  });
}

template <typename T, int B>
__global__ void __launch_bounds__(kYThreads, sizeof(T) == 4 ? 2 : 1)
    k_gyinv(const C2<T> *Wr, C2<T> *Wry, FusedGeom g,
            const __grid_constant__ GPlan plan, const C2<T> *__restrict__ tw) {
  grid_chain();
  using GE = GElem<T>;
  using E = typename GE::E;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  E *buf = reinterpret_cast<E *>(smem_raw);
  const int kz0 = blockIdx.x * kCols<T, B>;
  const int nb = g.h - kz0;
  const C2<T> *col = Wr + (int64_t)blockIdx.y * g.n1 * g.hp + kz0;
  C2<T> *out = Wry + (int64_t)blockIdx.y * g.rs * g.hp + kz0;
  col_first<1, B, T>(plan.p[0], col, g.hp, nb, buf);
  const E *res = col_middle<1, B>(plan, tw, buf, buf + g.n1 * pitch_of(B));
  col_last<1, B>(plan.p[plan.npass - 1], tw, res, [&](int y, int b, const E &v) {
    int rj = y + g.ro;
    if (rj >= g.n1) rj -= g.n1;
    for (; rj < g.rs; rj += g.n1)
      GE::store(out + (int64_t)rj * g.hp + GE::W * b, v, nb - GE::W * b);
  });
}

// ------------------------------------------------------------------ x
// The W real parts of an element (n of them valid, the others zero) as they
// are staged for the even form's inverse.
__device__ __forceinline__ float2 real_parts(const CPair &v, int n) {
  return make_float2(n > 0 ? v.x.x : 0.f, n > 1 ? v.x.y : 0.f);
}
__device__ __forceinline__ double real_parts(const double2 &v, int n) {
  return n > 0 ? v.x : 0.0;
}
__device__ __forceinline__ double part(float2 r, int l) { return (double)(l ? r.y : r.x); }
__device__ __forceinline__ double part(double r, int) { return r; }

// w |q|^2 as an element.
__device__ __forceinline__ CPair abs2_elem(const CPair &q, float w) {
  CPair r;
  r.x = f2splat(w) * __ffma2_rn(q.x, q.x, q.y * q.y);
  r.y = f2splat(0.f);
  return r;
}
__device__ __forceinline__ double2 abs2_elem(const double2 &q, double w) {
  return make_double2(w * (q.x * q.x + q.y * q.y), 0.0);
}

// Staged real parts of adjacent columns as elements: column pairs become the
// real and imaginary parts of one complex column.
__device__ __forceinline__ CPair from_staged(const CPair &raw) {
  // in memory: (a0, b0, a1, b1), the pairs (a, b) of two complex columns
  return cpack(raw.x, raw.y);
}
__device__ __forceinline__ double2 from_staged(const double2 &raw) { return raw; }

// The columns A and B of Z = DFT(a + i b), a and b real, at x from Z at x
// and -x: A = (Z(x) + conj Z(-x)) / 2, B = (Z(x) - conj Z(-x)) / 2i.  Of the
// 2 W columns at p, n exist.
template <typename C>
__device__ __forceinline__ void split_store(C *p, C z, C m, int n) {
  C a, b;
  a.x = 0.5f * (z.x + m.x);
  a.y = 0.5f * (z.y - m.y);
  b.x = 0.5f * (z.y + m.y);
  b.y = 0.5f * (m.x - z.x);
  if (n > 0) p[0] = a;
  if (n > 1) p[1] = b;
}
__device__ __forceinline__ void split_elem(float2 *p, const CPair &z, const CPair &m, int n) {
  split_store(p, clane0(z), clane0(m), n);
  split_store(p + 2, clane1(z), clane1(m), n - 2);
}
__device__ __forceinline__ void split_elem(double2 *p, const double2 &z, const double2 &m,
                                           int n) {
  split_store(p, z, m, n);
}

// MODE 0: G = DFT_x(W).  MODE 1: P = DFT_x(W) conj(G); MODE 2 (ell = 0 of an
// autocorrelation): P = w00 |G|^2; MODE 3 (periodic autocorrelation): P =
// |DFT_x(W)|^2.  Then the k-subgrid extraction (weights 1 without ktab), straight
// from the registers that hold P (every k-subgrid cell has one source
// element, so the read-modify-writes never collide; `first` overwrites), and
// the inverse, stored at the r-subgrid's rows.  EVEN: the inverse of Re P
// (fc_fused.h), two real columns to a complex one.
template <typename T, int B, int MODE, bool EVEN>
__global__ void __launch_bounds__(kXThreads, sizeof(T) == 4 ? 2 : 1)
    k_gx(const C2<T> *W, const C2<T> *G, C2<T> *out, double *ksub, FusedGeom g,
         const __grid_constant__ GPlan plan, const C2<T> *__restrict__ tw,
         const T *__restrict__ ktab, T w00, int first) {
  grid_chain();
  using GE = GElem<T>;
  using E = typename GE::E;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  E *buf = reinterpret_cast<E *>(smem_raw);
  constexpr int BP = pitch_of(B);
  E *other = buf + g.n0 * BP;
  const int kz0 = blockIdx.x * kCols<T, B>;
  const int nb = g.h - kz0;
  const int yy = blockIdx.y;
  const int64_t stride = (int64_t)g.n1 * g.hp;
  const int64_t base = (int64_t)yy * g.hp + kz0;
  const GPass &last = plan.p[plan.npass - 1];
  E *cur = buf;
  if constexpr (MODE != 2) {
    col_first<-1, B, T>(plan.p[0], W + base, stride, nb, buf);
    cur = col_middle<-1, B>(plan, tw, buf, other);
    other = cur == buf ? other : buf;
  }
  if constexpr (MODE == 0) {
    col_last<-1, B>(last, tw, cur, [&](int i, int b, const E &v) {
      GE::store(out + base + (int64_t)i * stride + GE::W * b, v, nb - GE::W * b);
    });
  } else {
    using RP = decltype(real_parts(E(), 0));
    const int ox = g.ks0 / 2, oz = g.ks2 / 2;
    int jr = yy + g.ks1 / 2;
    if (jr >= g.n1) jr -= g.n1;
    const bool extract = ksub != nullptr && kz0 <= oz && jr < g.ks1;
    // Row x of P: to the k-subgrid, and to shared memory for the inverse.
    auto take = [&](int x, int b, const E &v, E *dst) {
      const int n = nb - GE::W * b;
      const RP re = real_parts(v, n);
      if constexpr (EVEN) reinterpret_cast<RP *>(dst)[x * B + b] = re;
      else dst[x * BP + b] = v;
      const int kz = kz0 + GE::W * b;
      if (!extract || kz > oz) return;
      int i = x + ox;
      if (i >= g.n0) i -= g.n0;
      for (; i < g.ks0; i += g.n0)
        for (int j = jr; j < g.ks1; j += g.n1) {
          // (The second cell of a pair may be the row's padding.)
          const size_t cell = ((size_t)i * g.ks1 + j) * g.kp + kz;
#pragma unroll
          for (int l = 0; l < GE::W; ++l)
            ksub[cell + l] = (first ? 0.0 : ksub[cell + l]) +
                             (ktab ? (double)ktab[cell + l] : 1.0) * part(re, l);
        }
    };
    if constexpr (MODE == 1 || MODE == 3) {
      with_radix(last.R, [&]<int R>() {
        for (int bf = threadIdx.x; bf < last.LR * B; bf += blockDim.x) {
          const int j = bf / B, b = bf % B;
          const C2<T> *gp = G + base + j * stride + GE::W * b;
          E gv[R], v[R];
#pragma unroll
          for (int q = 0; q < (MODE == 1 ? R : 0); ++q)
            gv[q] = GE::load(gp + (int64_t)(q * last.LR) * stride, nb - GE::W * b);
#pragma unroll
          for (int q = 0; q < R; ++q) v[q] = cur[(j + q * last.LR) * BP + b];
          g_twiddle<R, -1>(v, tw + last.tw, last.Ns, j);
          GDft<R, -1, E>::run(v);
#pragma unroll
          for (int q = 0; q < R; ++q)
            v[q] = MODE == 1 ? cmulc(v[q], gv[q]) : abs2_elem(v[q], (T)1);
#pragma unroll
          for (int q = 0; q < R; ++q) take(j + q * last.LR, b, v[q], other);
        }
      });
      E *t = cur;
      cur = other;
      other = t;
    } else {
      for (int idx = threadIdx.x; idx < g.n0 * B; idx += blockDim.x) {
        const int x = idx / B, b = idx % B;
        take(x, b,
             abs2_elem(GE::load(G + base + x * stride + GE::W * b, nb - GE::W * b), w00),
             cur);
      }
    }
    __syncthreads();
    if constexpr (EVEN) {
      constexpr int H = B / 2, HP = pitch_of(H);
      const GPass &f = plan.p[0];
      with_radix(f.R, [&]<int R>() {
        for (int bf = threadIdx.x; bf < f.LR * H; bf += blockDim.x) {
          const int j = bf / H, b = bf % H;
          E v[R];
#pragma unroll
          for (int q = 0; q < R; ++q) v[q] = from_staged(cur[(j + q * f.LR) * H + b]);
          GDft<R, 1, E>::run(v);
          E *o = other + j * R * HP + b;
#pragma unroll
          for (int q = 0; q < R; ++q) o[q * HP] = v[q];
        }
      });
      __syncthreads();
      const E *res = col_middle<1, H>(plan, tw, other, cur);
      E *zb = res == cur ? other : cur;
      col_last<1, H>(last, tw, res, [&](int x, int b, const E &v) {
        if (x <= g.ro || x >= g.n0 - g.ro) zb[x * HP + b] = v;
      });
      __syncthreads();
      for (int idx = threadIdx.x; idx < (g.ro + 1) * H; idx += blockDim.x) {
        const int x = idx / H, b = idx % H;
        const int xp = x == g.n0 ? 0 : x, xm = xp == 0 ? 0 : g.n0 - xp;
        split_elem(out + base + x * stride + 2 * GE::W * b, zb[xp * HP + b],
                   zb[xm * HP + b], nb - 2 * GE::W * b);
      }
    } else {
      col_pass<1, B>(plan.p[0], tw, cur, other, true);
      const E *res = col_middle<1, B>(plan, tw, other, cur);
      col_last<1, B>(last, tw, res, [&](int x, int b, const E &v) {
        int ri = x + g.ro;
        if (ri >= g.n0) ri -= g.n0;
        for (; ri < g.rs; ri += g.n0)
          GE::store(out + base + ri * stride + GE::W * b, v, nb - GE::W * b);
      });
    }
  }
}

// ------------------------------------------------------------------ z
// The z polynomial of Y_lm r^ell with the row's (x, y) fixed (row_poly in
// fc_fused.cu), in the weights' precision WT, formed in FP64.
template <typename WT>
struct RowCoef {
  WT c[5], rxy2;
};

// Y_lm D of a cell at z: D (c0 + c1 z + .. + c4 z^4) / r^ell.  In FP32 1 / r^2
// is __fdividef's, off by 2 units in the last place at most, and z is rounded
// once (RowZ).  Error against 64 bits (2-norm, mean of 6 fields) of 125 x 180 x
// 126 surveys at ell <= 4: cross xi 8.6e-8 and P 8.1e-8 (rounded divide: 7.3e-8
// and 7.7e-8; z rounded twice: 9.3e-8 and 8.7e-8; the passes with a rounded divide
// before these: 1.16e-7 and 9.3e-8), auto xi 7.2e-8 (6.7e-8; 7.3e-8; 8.0e-8).
// The rounded divide costs 250 x 360 x 378 cross correlations 5.06 -> 5.27 ms.
template <typename WT, int ELL>
__device__ __forceinline__ WT row_value(const RowCoef<WT> &r, WT D, WT z) {
  const WT z2 = z * z;
  const WT r2 = r.rxy2 + z2 + (WT)1e-20;
  WT ir2;
  if constexpr (sizeof(WT) == 4) ir2 = __fdividef(1.0f, r2);
  else ir2 = 1.0 / r2;
  // (1 / r^2 twice: its square is infinite in FP32 at the observer, r = 0.)
  if constexpr (ELL == 2) return D * ((r.c[2] * z + r.c[1]) * z + r.c[0]) * ir2;
  return D * ((((r.c[4] * z + r.c[3]) * z + r.c[2]) * z + r.c[1]) * z + r.c[0]) * ir2 * ir2;
}

// z of the cell i of a row, z0 + i rounded to its type once.
template <typename T>
struct RowZ;
template <>
struct RowZ<double> {
  double z0;
  __device__ explicit RowZ(double z) : z0(z) {}
  __device__ double at(int i) const { return z0 + i; }
};
// FP32: Knuth's two-sum of the upper half and i, so that no cell converts from
// FP64.
template <>
struct RowZ<float> {
  float hi, lo;
  __device__ explicit RowZ(double z) : hi((float)z), lo((float)(z - (double)(float)z)) {}
  __device__ float at(int i) const {
    const float x = (float)i, s = hi + x, b = s - hi;
    return s + (((hi - (s - b)) + (x - b)) + lo);
  }
};

// Shared index of element i of a row: one pad element in 8 spreads the
// strided accesses over the banks.
__device__ __forceinline__ int rpos(int i) { return i + (i >> 3); }

// A pass over np rows of elements between shared buffers.
template <int SIGN, typename E, typename Tw>
__device__ __forceinline__ void row_pass(const GPass &ps, const Tw *__restrict__ tw,
                                         const E *src, E *dst, int np, int pitch) {
  with_radix(ps.R, [&]<int R>() {
    for (int bf = threadIdx.x; bf < ps.LR * np; bf += blockDim.x) {
      const int b = gdiv(bf, ps.LR, ps.mLR);
      const int j = bf - b * ps.LR;
      E v[R];
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = src[b * pitch + rpos(j + q * ps.LR)];
      const int k = j - gdiv(j, ps.Ns, ps.mNs) * ps.Ns;
      g_twiddle<R, SIGN>(v, tw + ps.tw, ps.Ns, k);
      GDft<R, SIGN, E>::run(v);
      const int o = (j - k) * R + k;
#pragma unroll
      for (int q = 0; q < R; ++q) dst[b * pitch + rpos(o + q * ps.Ns)] = v[q];
    }
  });
  __syncthreads();
}

// Real component c (grid row c of the element's 2 W) of an element.
__device__ __forceinline__ float &comp(CPair &v, int c) {
  return c == 0 ? v.x.x : c == 1 ? v.y.x : c == 2 ? v.x.y : v.y.y;
}
__device__ __forceinline__ double &comp(double2 &v, int c) { return c ? v.y : v.x; }

// ELL: the weight's multipole (unweighted: 0, with value0 = 1).  np elements per CTA, each
// of 2 W rows.  IN: the cells' type, WT: the precision in which they are
// weighted; the result is rounded to T once.
template <typename T, int ELL, typename IN, typename WT>
__global__ void __launch_bounds__(kRowThreads, sizeof(WT) == 4 ? 5 : 4)
    k_gzfwd(const IN *rho, C2<T> *W, FusedGeom g,
            const __grid_constant__ GPlan plan, const C2<T> *__restrict__ tw, int np,
            YlmParams p, double x0, double y0, double z0) {
  grid_chain();
  using E = typename GElem<T>::E;
  constexpr int NR = 2 * GElem<T>::W;  // grid rows per element
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ RowCoef<WT> rc[NR * kGenMaxPairs];
  const int N = g.n2;
  const int pitch = rpos(N - 1) + 1;
  E *buf = reinterpret_cast<E *>(smem_raw);
  E *other = buf + np * pitch;
  const int64_t nrows = (int64_t)g.n0 * g.n1;
  const int64_t row0 = (int64_t)blockIdx.x * NR * np;
  if constexpr (ELL > 0) {
    // (Short rows leave the CTA with fewer threads than table entries.)
    for (int e = threadIdx.x; e < NR * np; e += blockDim.x) {
      const int64_t row = min(row0 + e, nrows - 1);
      const int x = (int)(row / g.n1);
      const int y = (int)(row - (int64_t)x * g.n1);
      double c[5];
      row_poly_coefs(p, x0 + x * 1.0, y0 + y * 1.0, c);
      RowCoef<WT> r;
      for (int i = 0; i < 5; ++i) r.c[i] = (WT)c[i];
      r.rxy2 = (WT)((x0 + x) * (x0 + x) + (y0 + y) * (y0 + y));
      rc[e] = r;
    }
    __syncthreads();
  }
  const GPass &f = plan.p[0];
  const RowZ<WT> zs(z0);
  with_radix(f.R, [&]<int R>() {
    for (int bf = threadIdx.x; bf < f.LR * np; bf += blockDim.x) {
      const int b = gdiv(bf, f.LR, f.mLR);
      const int j = bf - b * f.LR;
      const int64_t ra = row0 + NR * b;
      const IN *src = rho + (ra < nrows ? ra : 0) * N + j;
      IN d[R][NR];
#pragma unroll
      for (int c = 0; c < NR; ++c) {
        const bool on = ra + c < nrows;
#pragma unroll
        for (int q = 0; q < R; ++q) d[q][c] = on ? src[c * N + q * f.LR] : (IN)0;
      }
      E v[R];
      if constexpr (ELL == 0) {
#pragma unroll
        for (int q = 0; q < R; ++q)
#pragma unroll
          for (int c = 0; c < NR; ++c) comp(v[q], c) = (T)((WT)d[q][c] * (WT)p.value0);
      } else {
        WT z[R];
#pragma unroll
        for (int q = 0; q < R; ++q) z[q] = zs.at(j + q * f.LR);
#pragma unroll
        for (int c = 0; c < NR; ++c) {
          const RowCoef<WT> a = rc[NR * b + c];
#pragma unroll
          for (int q = 0; q < R; ++q)
            comp(v[q], c) = (T)row_value<WT, ELL>(a, (WT)d[q][c], z[q]);
        }
      }
      GDft<R, -1, E>::run(v);
#pragma unroll
      for (int q = 0; q < R; ++q) buf[b * pitch + rpos(j * R + q)] = v[q];
    }
  });
  __syncthreads();
  for (int s = 1; s < plan.npass; ++s) {
    row_pass<-1>(plan.p[s], tw, buf, other, np, pitch);
    E *t = buf;
    buf = other;
    other = t;
  }
  for (int b = 0; b < np; ++b) {
    const int64_t ra = row0 + NR * b;
    if (ra >= nrows) break;
    C2<T> *dst = W + ra * g.hp;
    for (int k = threadIdx.x; k < g.h; k += blockDim.x) {
      E z = buf[b * pitch + rpos(k)];
      E c = buf[b * pitch + rpos(k == 0 ? 0 : N - k)];
#pragma unroll
      for (int l = 0; l < NR; l += 2) {
        const T zx = comp(z, l), zy = comp(z, l + 1);
        const T cx = comp(c, l), cy = -comp(c, l + 1);
        C2<T> xa, xb;
        xa.x = (T)0.5 * (zx + cx);
        xa.y = (T)0.5 * (zy + cy);
        xb.x = (T)0.5 * (zy - cy);
        xb.y = (T)0.5 * (cx - zx);
        if (ra + l < nrows) dst[l * g.hp + k] = xa;
        if (ra + l + 1 < nrows) dst[(l + 1) * g.hp + k] = xb;
      }
    }
  }
}

// Pairs of rows of Wry to real rows, accumulated into the r-subgrid.
template <typename T>
__global__ void __launch_bounds__(kRowThreads, sizeof(T) == 4 ? 5 : 4)
    k_gzinv(const C2<T> *Wry, double *rsub, FusedGeom g,
            const __grid_constant__ GPlan plan, const C2<T> *__restrict__ tw, int np,
            const T *__restrict__ rtab, int first) {
  grid_chain();
  using E = typename GElem<T>::E;
  constexpr int NR = 2 * GElem<T>::W;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = g.n2;
  const int pitch = rpos(N - 1) + 1;
  E *buf = reinterpret_cast<E *>(smem_raw);
  E *other = buf + np * pitch;
  const int nrows = g.nri * g.rs;
  const int row0 = blockIdx.x * NR * np;
  const GPass &f = plan.p[0];
  with_radix(f.R, [&]<int R>() {
    for (int bf = threadIdx.x; bf < f.LR * np; bf += blockDim.x) {
      const int b = gdiv(bf, f.LR, f.mLR);
      const int j = bf - b * f.LR;
      const int ra = row0 + NR * b;
      const C2<T> *src = Wry + (int64_t)(ra < nrows ? ra : 0) * g.hp;
      E v[R];
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const int k = j + q * f.LR;
        const int kk = k < g.h ? k : N - k;
        const bool real = kk == 0 || 2 * kk == N;  // DC and Nyquist
#pragma unroll
        for (int l = 0; l < NR; l += 2) {
          C2<T> xa, xb;
          xa.x = xa.y = xb.x = xb.y = 0;
          if (ra + l < nrows) xa = src[l * g.hp + kk];
          if (ra + l + 1 < nrows) xb = src[(l + 1) * g.hp + kk];
          const T sg = real ? (T)0 : k >= g.h ? (T)-1 : (T)1;
          comp(v[q], l) = xa.x - sg * xb.y;
          comp(v[q], l + 1) = sg * xa.y + xb.x;
        }
      }
      GDft<R, 1, E>::run(v);
#pragma unroll
      for (int q = 0; q < R; ++q) buf[b * pitch + rpos(j * R + q)] = v[q];
    }
  });
  __syncthreads();
  for (int s = 1; s + 1 < plan.npass; ++s) {
    row_pass<1>(plan.p[s], tw, buf, other, np, pitch);
    E *t = buf;
    buf = other;
    other = t;
  }
  const GPass &l = plan.p[plan.npass - 1];
  with_radix(l.R, [&]<int R>() {
    for (int bf = threadIdx.x; bf < l.LR * np; bf += blockDim.x) {
      const int b = gdiv(bf, l.LR, l.mLR);
      const int j = bf - b * l.LR;
      const int ra = row0 + NR * b;
      if (ra >= nrows) break;
      E v[R];
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = buf[b * pitch + rpos(j + q * l.LR)];
      g_twiddle<R, 1>(v, tw + l.tw, l.Ns, j);
      GDft<R, 1, E>::run(v);
#pragma unroll
      for (int q = 0; q < R; ++q) {
        int rk = j + q * l.LR + g.ro;
        if (rk >= N) rk -= N;
        for (; rk < g.rs; rk += N) {
#pragma unroll
          for (int c = 0; c < NR; ++c) {
            if (ra + c >= nrows) continue;
            const size_t cell = (size_t)(ra + c) * g.rs + rk;
            const double val = (double)comp(v[q], c);
            rsub[cell] = rtab == nullptr ? val
                                         : (first ? 0.0 : rsub[cell]) +
                                               (double)rtab[cell] * val;
          }
        }
      }
    }
  });
}

size_t col_smem(int L) { return 2 * (size_t)L * pitch_of(col_width(L)) * 16; }

// Threads of a column pass: one butterfly each of the pass with the most, or
// an equal share of several.
int col_threads(const GPlan &p, int most) {
  int n = 0;
  for (int s = 0; s < p.npass; ++s)
    if (p.p[s].R > 1) n = std::max(n, p.p[s].LR * col_width(p.L));
  const int rounds = (n + most - 1) / most;
  const int t = rounds > 0 ? (n + rounds - 1) / rounds : 32;
  return std::max(64, (t + 31) / 32 * 32);
}

// Elements (of 2 W rows) per CTA of a z pass: about one butterfly of the
// first pass per thread, within the shared memory and the coefficient table,
// and few enough that `total` elements still make two CTAs per SM.
size_t row_smem(int L, int np) { return 2 * (size_t)np * (L + L / 8 + 1) * 16; }
int row_elems(const GPlan &p, int64_t total) {
  int np = (kRowThreads + p.p[0].LR / 2) / p.p[0].LR;
  np = std::min(np, (int)(44 * 1024 / row_smem(p.L, 1)));
  np = (int)std::min<int64_t>(np, total / (2 * sm_count()));
  return std::max(1, std::min(np, kGenMaxPairs));
}
int row_threads(const GPlan &p, int np) {
  int n = 0;
  for (int s = 0; s < p.npass; ++s)
    if (p.p[s].R > 1) n = std::max(n, p.p[s].LR * np);
  return std::max(32, std::min(kRowThreads, (n + 31) / 32 * 32));
}

template <typename K>
void big_smem(K kernel) {
  FC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kGenSmem));
}

// Calls f.template operator()<B>() for a length's column width.
template <typename F>
void with_width(int L, F &&f) {
  if (col_width(L) == 8) f.template operator()<8>();
  else f.template operator()<4>();
}

// Calls f(kernel) for the x kernel of a mode.
template <typename T, int B, typename F>
void x_kernel(int mode, bool even, F &&f) {
  if (mode == 0) f(k_gx<T, B, 0, false>);
  else if (mode == 3) f(k_gx<T, B, 3, true>);
  else if (mode == 1 && even) f(k_gx<T, B, 1, true>);
  else if (mode == 1) f(k_gx<T, B, 1, false>);
  else if (even) f(k_gx<T, B, 2, true>);
  else f(k_gx<T, B, 2, false>);
}

}  // namespace

// Calls f(kernel) for every z kernel of a cell type and weights' precision.
template <typename T, typename IN, typename WT, typename F>
void z_kernels(bool weighted, F &&f) {
  f(k_gzfwd<T, 0, IN, WT>);
  if (!weighted) return;
  f(k_gzfwd<T, 2, IN, WT>);
  f(k_gzfwd<T, 4, IN, WT>);
}
template <typename T>
void gen_z_limits(int n2, bool weighted) {
  auto set = [](auto kernel) { big_smem(kernel); };
  if constexpr (sizeof(T) == 4) {
    if (wide_rows(n2)) {
      z_kernels<T, T, T>(false, set);
      if (weighted) z_kernels<T, T, double>(true, set);
      z_kernels<T, double, double>(weighted, set);
    } else {
      z_kernels<T, T, T>(weighted, set);
    }
  } else {
    z_kernels<T, T, T>(weighted, set);
  }
  big_smem(k_gzinv<T>);
}
template <typename T>
void gen_y_limits(int n1) {
  with_width(n1, [&]<int B>() {
    big_smem(k_gyfwd<T, B>);
    big_smem(k_gyinv<T, B>);
  });
}
template <typename T>
void gen_x_limits(int n0, int mode, bool even) {
  with_width(n0, [&]<int B>() {
    x_kernel<T, B>(mode, even, [](auto kernel) { big_smem(kernel); });
  });
}

template <typename T>
void gen_zfwd(const GenAxis &a, const FusedGeom &g, const void *rho, bool f32, C2<T> *W,
              bool weight, const YlmParams &p, const double xyz0[3], cudaStream_t s) {
  constexpr int NR = 2 * GElem<T>::W;
  const int64_t nrows = (int64_t)g.n0 * g.n1;
  const int np = row_elems(a.plan, (nrows + NR - 1) / NR);
  const unsigned blocks = (unsigned)((nrows + NR * np - 1) / (NR * np));
  const size_t sm = row_smem(g.n2, np);
  YlmParams one{};
  one.value0 = 1.0;
  auto run = [&](auto in, auto wt) {
    using IN = decltype(in);
    using WT = decltype(wt);
    auto go = [&](auto kernel) {
      launch_small(kernel, blocks, row_threads(a.plan, np), sm, s,
                   static_cast<const IN *>(rho), W, g, a.plan, a.tw.as<C2<T>>(), np,
                   weight ? p : one, xyz0[0], xyz0[1], xyz0[2]);
    };
    if (!weight || p.ell == 0) go(k_gzfwd<T, 0, IN, WT>);
    else if (p.ell == 2) go(k_gzfwd<T, 2, IN, WT>);
    else go(k_gzfwd<T, 4, IN, WT>);
  };
  if constexpr (sizeof(T) == 4) {
    if (wide_rows(g.n2) && !f32) run(double(), double());
    else if (wide_rows(g.n2) && weight) run(T(), double());
    else run(T(), T());  // (the cells as they are)
  } else {
    run(T(), T());
  }
  FC_LAUNCH_CHECK();
}

template <typename T>
void gen_yfwd(const GenAxis &a, const FusedGeom &g, C2<T> *W, cudaStream_t s) {
  with_width(a.plan.L, [&]<int B>() {
    constexpr int NC = kCols<T, B>;
    launch_small(k_gyfwd<T, B>, dim3((g.h + NC - 1) / NC, g.n0), col_threads(a.plan, kYThreads), col_smem(g.n1), s, W, g, a.plan, a.tw.as<C2<T>>());
  });
  FC_LAUNCH_CHECK();
}

template <typename T>
void gen_x(const GenAxis &a, const FusedGeom &g, int mode, const C2<T> *W, const C2<T> *G,
           C2<T> *out, double *ksub, const T *ktab, T w00, bool first, cudaStream_t s) {
  with_width(a.plan.L, [&]<int B>() {
    constexpr int NC = kCols<T, B>;
    auto go = [&](auto kernel) {
      launch_small(kernel, dim3((g.h + NC - 1) / NC, g.n1), col_threads(a.plan, kXThreads), col_smem(g.n0), s, 
          W, G, out, ksub, g, a.plan, a.tw.as<C2<T>>(), ktab, w00, first);
    };
    x_kernel<T, B>(mode, g.nri != g.rs, go);
  });
  FC_LAUNCH_CHECK();
}

template <typename T>
void gen_yinv(const GenAxis &a, const FusedGeom &g, const C2<T> *Wr, C2<T> *Wry,
              cudaStream_t s) {
  with_width(a.plan.L, [&]<int B>() {
    constexpr int NC = kCols<T, B>;
    launch_small(k_gyinv<T, B>, dim3((g.h + NC - 1) / NC, g.nri), col_threads(a.plan, kYThreads), col_smem(g.n1), s, Wr, Wry, g, a.plan, a.tw.as<C2<T>>());
  });
  FC_LAUNCH_CHECK();
}

template <typename T>
void gen_zinv(const GenAxis &a, const FusedGeom &g, const C2<T> *Wry, double *rsub,
              const T *rtab, bool first, cudaStream_t s) {
  constexpr int NR = 2 * GElem<T>::W;
  const int nrows = g.nri * g.rs;
  const int np = row_elems(a.plan, (nrows + NR - 1) / NR);
  launch_small(k_gzinv<T>, (nrows + NR * np - 1) / (NR * np), row_threads(a.plan, np), row_smem(g.n2, np), s, 
      Wry, rsub, g, a.plan, a.tw.as<C2<T>>(), np, rtab, first);
  FC_LAUNCH_CHECK();
}

#define FC_GEN(T)                                                                      \
  template void gen_z_limits<T>(int, bool);                                            \
  template void gen_y_limits<T>(int);                                                  \
  template void gen_x_limits<T>(int, int, bool);                                       \
  template void gen_zfwd<T>(const GenAxis &, const FusedGeom &, const void *, bool,    \
                            C2<T> *, bool, const YlmParams &, const double[3],         \
                            cudaStream_t);                                             \
  template void gen_yfwd<T>(const GenAxis &, const FusedGeom &, C2<T> *, cudaStream_t); \
  template void gen_x<T>(const GenAxis &, const FusedGeom &, int, const C2<T> *,       \
                         const C2<T> *, C2<T> *, double *, const T *, T, bool,        \
                         cudaStream_t); \
  template void gen_yinv<T>(const GenAxis &, const FusedGeom &, const C2<T> *,         \
                            C2<T> *, cudaStream_t);                                    \
  template void gen_zinv<T>(const GenAxis &, const FusedGeom &, const C2<T> *,         \
                            double *, const T *, bool, cudaStream_t);

}  // namespace fc
