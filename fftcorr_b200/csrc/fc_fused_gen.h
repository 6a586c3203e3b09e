// fc_fused_gen.h -- launchers of the fused passes along axes whose length is
// not a power of two (fc_fused_gen.cuh).
#pragma once

#include "fc_common.cuh"
#include "fc_fused_geom.h"
#include "fc_gfft.cuh"

namespace fc {

// Elements (two or four rows) a z pass takes per CTA, at most.
constexpr int kGenMaxPairs = 16;

// The plan and twiddles of one axis.
struct GenAxis {
  GPlan plan;
  DeviceBuffer tw;
  void init(int L, bool fp64);
};
// Shared-memory limits of an axis's kernels.
template <typename T>
void gen_z_limits(int n2, bool weighted);
template <typename T>
void gen_y_limits(int n1);
template <typename T>
void gen_x_limits(int n0, int mode, bool even);

// Whether an axis (of rows, or of columns) of this length fits, in either
// precision.
bool gen_supported(int L, bool row);

// FP32 transforms of rows of odd length weight their cells, and the cells of
// their subgrids, in FP64, of either cell type, and round the product once: as
// cuFFT's path does, which took these rows before.  (216 x 180 x 225, ell <= 4:
// by cuFFT 4.13 ms, weighted in FP32 1.95 ms, in FP64 2.18 ms.)
inline bool wide_rows(int n2) { return n2 % 2 != 0; }

// f32: the cells are FP32 (FP64 ones only in wide rows, or where T is double).
template <typename T>
void gen_zfwd(const GenAxis &a, const FusedGeom &g, const void *rho, bool f32,
              typename Vec2<T>::type *W, bool weight, const YlmParams &p,
              const double xyz0[3], cudaStream_t s);
template <typename T>
void gen_yfwd(const GenAxis &a, const FusedGeom &g, typename Vec2<T>::type *W,
              cudaStream_t s);
// mode 0: out = G = DFT_x(W); 1: the product with G; 2: w00 |G|^2;
// 3: |DFT_x(W)|^2.  first:
// the subgrid is overwritten, not added to.
template <typename T>
void gen_x(const GenAxis &a, const FusedGeom &g, int mode,
           const typename Vec2<T>::type *W, const typename Vec2<T>::type *G,
           typename Vec2<T>::type *out, double *ksub, const T *ktab, T w00, bool first,
           cudaStream_t s);
template <typename T>
void gen_yinv(const GenAxis &a, const FusedGeom &g, const typename Vec2<T>::type *Wr,
              typename Vec2<T>::type *Wry, cudaStream_t s);
template <typename T>
void gen_zinv(const GenAxis &a, const FusedGeom &g, const typename Vec2<T>::type *Wry,
              double *rsub, const T *rtab, bool first, cudaStream_t s);

// Coefficients of Y_lm r^ell (ell 2 or 4) as a polynomial in z with (x, y)
// fixed, in FP64 with the normalisation folded in (spherical_harmonics.h:
// 100-176).
__host__ __device__ __forceinline__ void row_poly_coefs(const YlmParams &p, double x,
                                                        double y, double c[5]) {
  const double x2 = x * x, y2 = y * y, s = x2 + y2;
  for (int i = 0; i < 5; ++i) c[i] = 0;
  if (p.ell == 2) {
    switch (p.m) {
      case 2: c[0] = x2 - y2; break;
      case 1: c[1] = x; break;
      case 0: c[0] = -s; c[2] = 2.0; break;
      case -1: c[1] = y; break;
      default: c[0] = x * y; break;
    }
  } else if (p.ell == 4) {
    switch (p.m) {
      case 4: c[0] = x2 * x2 - 6.0 * x2 * y2 + y2 * y2; break;
      case 3: c[1] = x * (x2 - 3.0 * y2); break;
      case 2: c[0] = y2 * y2 - x2 * x2; c[2] = 6.0 * (x2 - y2); break;
      case 1: c[1] = -x * s; c[3] = 4.0 / 3.0 * x; break;
      case 0: c[0] = 0.375 * s * s; c[2] = -3.0 * s; c[4] = 1.0; break;
      case -1: c[1] = -y * s; c[3] = 4.0 / 3.0 * y; break;
      case -2: c[0] = -2.0 * x * y * s; c[2] = 12.0 * x * y; break;
      case -3: c[1] = 3.0 * x2 * y - y2 * y; break;
      default: c[0] = 4.0 * x * (x2 * y - y2 * y); break;
    }
  }
  for (int i = 0; i < 5; ++i) c[i] *= p.norm;
}

}  // namespace fc
