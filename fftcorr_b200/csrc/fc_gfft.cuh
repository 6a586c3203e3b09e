// fc_gfft.cuh -- shared-memory FFT of any length with prime factors 2, 3, 5
// and 7 (the lengths that the power-of-two engine of fc_fft.cuh does not
// take), for the generic passes of fc_fused_gen.cuh.
//
// A length is split into as few radices of at most 10 as it has (378 = 9 x 7
// x 6, 1000 = 10 x 10 x 10), one Stockham pass each.  The first pass reads
// its inputs where they are (device memory) and the last hands its outputs to
// the caller in registers, so a transform of three passes crosses shared
// memory twice; passes alternate between two buffers and need one barrier
// each.  A pass reads its twiddles from a table laid out as it uses them,
// rounded from FP64.
#pragma once

#include <cmath>
#include <vector>

#include "fc_fft.cuh"

namespace fc {

// One pass: radix R over butterflies j < LR, inputs x[j + q LR], Ns the
// product of the radices before it, mNs = 2^32 / Ns rounded up (division of
// j by Ns), mLR the same of LR, tw the pass's first entry in the twiddle
// table.
struct GPass {
  int R, Ns, LR;
  unsigned mNs, mLR;
  int tw;
};

// n / d from m = 2^32 / d rounded up, exact for n d < 2^32.
__device__ __forceinline__ int gdiv(int n, int d, unsigned m) {
  return d == 1 ? n : (int)__umulhi((unsigned)n, m);
}
inline unsigned gdiv_magic(int d) {
  return d > 1 ? (unsigned)(0x100000000ull / (unsigned)d + 1) : 0;
}

struct GPlan {
  int L, npass;
  GPass p[6];
};

// Radices (at most 10, descending) of a length with the fewest passes, then
// the smallest sum; at least two passes (a last radix 1 where one would do),
// so that every transform has a first and a last one.  False if L has a
// prime factor above 7.
inline bool gplan_split(int L, int top, int left, std::vector<int> &cur, int sum,
                        int &best_sum, std::vector<int> &best) {
  if (left == 0) {
    if (L == 1 && (best.empty() || sum < best_sum)) {
      best = cur;
      best_sum = sum;
    }
    return !best.empty();
  }
  for (int r = top; r >= 1; --r) {
    if (L % r != 0 || (r == 1 && L != 1)) continue;
    cur.push_back(r);
    gplan_split(L / r, r, left - 1, cur, sum + r, best_sum, best);
    cur.pop_back();
  }
  return !best.empty();
}

inline bool gplan_length(int L, GPlan *p) {
  if (L < 1) return false;
  int n = L;
  for (int f : {2, 3, 5, 7})
    while (n % f == 0) n /= f;
  if (n != 1) return false;
  std::vector<int> cur, best;
  int best_sum = 0;
  for (int np = 2; np <= 6; ++np)
    if (gplan_split(L, 10, np, cur, 0, best_sum, best)) break;
  if (best.empty()) return false;
  p->L = L;
  p->npass = (int)best.size();
  int ns = 1, tw = 0;
  for (int s = 0; s < p->npass; ++s) {
    GPass &g = p->p[s];
    g.R = best[s];
    g.Ns = ns;
    g.LR = L / g.R;
    g.mNs = gdiv_magic(ns);
    g.mLR = gdiv_magic(g.LR);
    g.tw = tw;
    tw += ns * (g.R - 1);
    ns *= g.R;
  }
  return true;
}

// e^{-2 pi i q k / (R Ns)} for every pass, k < Ns and 0 < q < R.
template <typename C>
std::vector<C> gplan_twiddles(const GPlan &p) {
  std::vector<C> t;
  for (int s = 0; s < p.npass; ++s) {
    const GPass &g = p.p[s];
    for (int q = 1; q < g.R; ++q)
      for (int k = 0; k < g.Ns; ++k) {
        const int order = g.R * g.Ns;
        const double a = 2.0 * M_PI * (double)((q * k) % order) / (double)order;
        C w;
        w.x = (decltype(w.x))cos(a);
        w.y = (decltype(w.y))(-sin(a));
        t.push_back(w);
      }
  }
  if (t.empty()) t.push_back(C{1, 0});
  return t;
}

// ------------------------------------------------------ small transforms
// s a + b, by lane for a pair.
__device__ __forceinline__ float mad(float s, float a, float b) { return fmaf(s, a, b); }
__device__ __forceinline__ double mad(double s, double a, double b) { return fma(s, a, b); }
__device__ __forceinline__ float2 mad(float s, float2 a, float2 b) {
  return __ffma2_rn(f2splat(s), a, b);
}

// GDft<R, SIGN>: out[k] = sum_n v[n] e^{SIGN 2 pi i n k / R} in registers.
template <int R, int SIGN, typename C>
struct GDft {
  // Radices 2, 3, 4 and 8 as in fc_fft.cuh.
  __device__ __forceinline__ static void run(C *v) { Dft<R, C>::run(v, SIGN); }
};
template <int SIGN, typename C>
struct GDft<1, SIGN, C> {
  __device__ __forceinline__ static void run(C *) {}
};

// Odd prime R: with t_u = v_u + v_{R-u} and d_u = v_u - v_{R-u}, output k is
// v_0 + sum_u cos(2 pi u k / R) t_u + SIGN i sum_u sin(2 pi u k / R) d_u, and
// output R - k the same with the second sum subtracted: R - 1 real
// multiplications per output pair and component instead of R complex ones.
// cos and sin of 2 pi u / R, 1 <= u <= (R - 1) / 2.
template <int R>
__device__ constexpr double root_cos(int u) {
  if (R == 5) return u == 1 ? 0.30901699437494742410 : -0.80901699437494742410;
  return u == 1   ? 0.62348980185873353053
         : u == 2 ? -0.22252093395631440429
                  : -0.90096886790241912624;
}
template <int R>
__device__ constexpr double root_sin(int u) {
  if (R == 5) return u == 1 ? 0.95105651629515357212 : 0.58778525229247312917;
  return u == 1   ? 0.78183148246802980871
         : u == 2 ? 0.97492791218182360702
                  : 0.43388373911755812048;
}
template <int R, int SIGN, typename C>
struct GDftPrime {
  __device__ __forceinline__ static void run(C *v) {
    using T = typename Real<C>::type;
    constexpr int H = (R - 1) / 2;
    C t[H], d[H];
#pragma unroll
    for (int u = 0; u < H; ++u) {
      t[u] = cadd(v[u + 1], v[R - 1 - u]);
      d[u] = csub(v[u + 1], v[R - 1 - u]);
    }
    const C z = v[0];
#pragma unroll
    for (int u = 0; u < H; ++u) v[0] = cadd(v[0], t[u]);
#pragma unroll
    for (int k = 1; k <= H; ++k) {
      C m = z, e;
#pragma unroll
      for (int u = 1; u <= H; ++u) {
        const int uk = (u * k) % R;
        const int w = uk <= H ? uk : R - uk;  // cos is even, sin is odd
        const T cc = (T)root_cos<R>(w);
        const T ss = (T)(uk <= H ? root_sin<R>(w) : -root_sin<R>(w));
        m.x = mad(cc, t[u - 1].x, m.x);
        m.y = mad(cc, t[u - 1].y, m.y);
        e.x = u == 1 ? ss * d[0].x : mad(ss, d[u - 1].x, e.x);
        e.y = u == 1 ? ss * d[0].y : mad(ss, d[u - 1].y, e.y);
      }
      const C ie = cmuli(e, SIGN);
      v[k] = cadd(m, ie);
      v[R - k] = csub(m, ie);
    }
  }
};
template <int SIGN, typename C>
struct GDft<5, SIGN, C> : GDftPrime<5, SIGN, C> {};
template <int SIGN, typename C>
struct GDft<7, SIGN, C> : GDftPrime<7, SIGN, C> {};

// R = A B with A and B coprime (Good's prime-factor map): input A n2 + B n1
// is element (n1, n2), output k is element (k mod A, k mod B), no twiddles.
template <int A, int B, int SIGN, typename C>
struct GDftPfa {
  __device__ __forceinline__ static void run(C *v) {
    C t[A][B];
#pragma unroll
    for (int a = 0; a < A; ++a) {
#pragma unroll
      for (int b = 0; b < B; ++b) t[a][b] = v[(B * a + A * b) % (A * B)];
      GDft<B, SIGN, C>::run(t[a]);
    }
#pragma unroll
    for (int b = 0; b < B; ++b) {
      C u[A];
#pragma unroll
      for (int a = 0; a < A; ++a) u[a] = t[a][b];
      GDft<A, SIGN, C>::run(u);
#pragma unroll
      for (int a = 0; a < A; ++a) t[a][b] = u[a];
    }
#pragma unroll
    for (int k = 0; k < A * B; ++k) v[k] = t[k % A][k % B];
  }
};
template <int SIGN, typename C>
struct GDft<6, SIGN, C> : GDftPfa<2, 3, SIGN, C> {};
template <int SIGN, typename C>
struct GDft<10, SIGN, C> : GDftPfa<2, 5, SIGN, C> {};

template <int SIGN, typename C>
struct GDft<9, SIGN, C> {
  __device__ __forceinline__ static void run(C *v) {
    using T = typename Real<C>::type;
    // cos and sin of 2 pi m / 9
    constexpr double c1 = 0.76604444311897803520, s1 = 0.64278760968653932632;
    constexpr double c2 = 0.17364817766693034885, s2 = 0.98480775301220805937;
    constexpr double c4 = -0.93969262078590838405, s4 = 0.34202014332566873304;
    C t[3][3];
#pragma unroll
    for (int b = 0; b < 3; ++b) {
#pragma unroll
      for (int a = 0; a < 3; ++a) t[b][a] = v[3 * a + b];
      Dft<3, C>::run(t[b], SIGN);
    }
    auto rot = [](C z, double c, double s) {
      typename Vec2<T>::type w;
      w.x = (T)c;
      w.y = (T)(SIGN * s);
      return cmul(z, w);
    };
    t[1][1] = rot(t[1][1], c1, s1);
    t[1][2] = rot(t[1][2], c2, s2);
    t[2][1] = rot(t[2][1], c2, s2);
    t[2][2] = rot(t[2][2], c4, s4);
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1) {
      C u[3] = {t[0][k1], t[1][k1], t[2][k1]};
      Dft<3, C>::run(u, SIGN);
#pragma unroll
      for (int k2 = 0; k2 < 3; ++k2) v[k1 + 3 * k2] = u[k2];
    }
  }
};

// Calls f.template operator()<R>() for the pass's radix.
template <typename F>
__device__ __forceinline__ void with_radix(int R, F &&f) {
  switch (R) {
    case 10: f.template operator()<10>(); break;
    case 9: f.template operator()<9>(); break;
    case 8: f.template operator()<8>(); break;
    case 7: f.template operator()<7>(); break;
    case 6: f.template operator()<6>(); break;
    case 5: f.template operator()<5>(); break;
    case 4: f.template operator()<4>(); break;
    case 3: f.template operator()<3>(); break;
    case 2: f.template operator()<2>(); break;
    default: f.template operator()<1>(); break;
  }
}

// The twiddles of butterfly k of a pass applied to its inputs.  Neighbouring
// butterflies read neighbouring entries, so a warp's load is one line.
template <int R, int SIGN, typename C, typename Tw>
__device__ __forceinline__ void g_twiddle(C *v, const Tw *__restrict__ tw, int Ns,
                                          int k) {
#pragma unroll
  for (int q = 1; q < R; ++q) {
    Tw t = __ldg(&tw[(q - 1) * Ns + k]);
    if (SIGN > 0) t.y = -t.y;
    v[q] = cmul(v[q], t);
  }
}

}  // namespace fc
