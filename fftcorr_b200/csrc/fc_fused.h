// fc_fused.h -- fused hand-written FFT passes of the survey correlator
// (see fc_fused.cu for the algorithm).
#pragma once

#include <map>
#include <utility>
#include <vector>

#include "fc_common.cuh"
#include "fc_fused_gen.h"

namespace fc {

// Device pointers of the k axes and the per-axis |W|^2 window tables.
struct KAxes {
  const double *kx, *ky, *kz, *wx, *wy, *wz;
};

// Optional per-pass timing callbacks (the correlator's profiler).
struct PhaseHook {
  virtual void begin(const char *name) = 0;
  virtual void end() = 0;
  virtual ~PhaseHook() {}
};

class FusedSurvey {
 public:
  // True when every side factors into 2, 3, 5, 7 and the shared-memory tiles
  // fit: columns (x, y) of at most 1280 cells and rows (z) of at most 2560.
  static bool supported(const int shape[3], int rsize);

  // even: the r-subgrid's bins are those of its mirror image, so the inverse
  // transforms may take Re P (fc_fused.cu).
  // survey: the buffers of weighted terms and of G are allocated now.
  FusedSurvey(const int shape[3], int rsize, const int kshape[3], bool fp64,
              bool even, bool survey);
  bool even() const { return g.nri != g.rs; }
  // Cells of the stored subgrids (half_k_cell, half_r_cell).
  size_t k_cells() const { return (size_t)g.ks0 * g.ks1 * g.kp; }
  size_t r_cells() const { return (size_t)g.nri * g.rs * g.rs; }

  // Cells as the z passes read them.
  struct Cells {
    const void *p;
    bool f32;
  };
  // The grid's cells as they are where the passes read that type (f32: FP32
  // cells, in mixed precision only), else an FP32 copy of FP64 cells.
  Cells prepare_input(const void *rho, bool f32, cudaStream_t s);
  // What prepare_input(rho, f32) last returned -- valid only while that
  // density is unchanged.
  Cells input(const void *rho, bool f32) const {
    return reads_as_is(f32) ? Cells{rho, f32} : Cells{rho32.get(), true};
  }
  // G = 3-D DFT of the prepared grid (BaseCorrelator::set_grid2).
  void grid2(Cells in, cudaStream_t s, const KAxes &ka);
  // Builds the r- (and, with with_k, k-) subgrid weight tables of every
  // (ell, m) up to maxell, so that later correlations allocate nothing.
  void prepare_tables(int maxell, double ncells, const double *raxis,
                      const KAxes &ka, bool with_k, cudaStream_t s);
  // One (ell, m) term of Correlator::correlate_internal, accumulated into
  // the FP64 subgrids, or (first) written over them.
  // Returns the number of full-grid transforms run (1 or 2).
  int term(Cells in, int ell, int m, const double xyz0[3],
            double ncells, double *ksub, double *rsub, const double *raxis,
            const KAxes &ka, cudaStream_t s, PhaseHook *hook, bool first,
            bool g_of_input, bool z_done);
  // PeriodicCorrelator::correlate_internal (correlator.h:273-357): the one P
  // of every multipole, |F|^2 or (cross) F conj(G), left unweighted in the
  // stored subgrids, P itself in ksub and its inverse transform in rsub.
  // The autocorrelation needs the even form.
  void periodic(Cells in, bool cross, double *ksub, double *rsub,
                cudaStream_t s, PhaseHook *hook);
  // Whether two weighted terms can share one z pass (FP32, power-of-two
  // rows).  zfwd_pair runs the z pass of terms a and b (both ell > 0) in
  // one launch: term a's result lands in W, term b's in a second buffer
  // that take_second() swaps into W before term b runs with z_done.
  bool pairs() const;
  // 1 when the last group of B columns holds only the last column (kz =
  // N2/2), which the paired column passes then take for B planes per CTA;
  // with k_extract, only when that column lies outside the k-subgrid.
  template <int B>
  int nyq_group(bool k_extract) const {
    return (g.h - 1) % B == 0 && (!k_extract || g.ks2 / 2 < g.h - 1) ? 1 : 0;
  }
  void zfwd_pair(Cells in, int ell_a, int m_a, int ell_b, int m_b,
                 const double xyz0[3], cudaStream_t s, PhaseHook *hook);
  void take_second() { std::swap(W, W2); }

  // G in the half-complex layout [N0][N1][N2/2+1] with rows g.hp elements
  // apart (FP64 or FP32 complex).
  void *g_data() {
    prepare_product();
    return G.get();
  }
  bool fp64() const { return fp64_; }

  FusedGeom g;

 private:
  template <typename V>
  void upload(DeviceBuffer &dst, const std::vector<V> &v);
  // Shared-memory limits of the kernels that this correlator launches: x's by
  // the pass's mode (k_xcorr_p2).
  template <typename T>
  void set_limits(bool survey);
  template <typename T>
  void x_limits(int mode);
  // What a product with a second grid needs beside the autocorrelation.
  void prepare_product();
  // Whether the z passes are the power-of-two ones (even rows of m pairs).
  bool p2_rows() const;
  // Where the x pass leaves its inverse's rows: in W itself, whose columns a CTA
  // has read before it writes them, unless the r-subgrid has more rows.
  template <typename T>
  typename Vec2<T>::type *inverse_rows() const {
    using C = typename Vec2<T>::type;
    return g.nri > g.n0 ? Wr.as<C>() : W.as<C>();
  }
  // Whether the FP32 passes weight in FP64, cells, k- and r-subgrids alike.
  bool wide() const { return !fp64_ && wide_rows(g.n2); }
  bool reads_as_is(bool f32) const { return fp64_ || f32 || wide(); }
  template <typename T>
  void zfwd(Cells in, bool weight, const YlmParams &p, const double xyz0[3],
            cudaStream_t s);
  template <typename T>
  void yfwd(cudaStream_t s);
  template <typename T>
  void grid2_x(cudaStream_t s);
  template <typename T>
  void xcorr(int mode, double *ksub, const void *ktab, double w00, bool first,
             cudaStream_t s);
  // Weights of the k-subgrid cells for (ell, m), built on first use.
  // (FP64 for the FP64 form and wide rows, else FP32)
  const void *k_table(int ell, int m, const KAxes &ka, cudaStream_t s);
  // Y_lm(r) of the r-subgrid cells for (ell, m), built on first use, in
  // the same type as the k weights.
  const void *r_table(int ell, int m, const double *raxis,
                      const YlmParams &pr, cudaStream_t s);
  template <typename T>
  void yinv(cudaStream_t s);
  template <typename T>
  void zinv(double *rsub, const void *rtab, bool first, cudaStream_t s);

  bool fp64_;
  bool product_ready = false;
  GenAxis gx, gy, gz;  // of the axes that are not powers of two
  DeviceBuffer tabx, taby, tabz;
  DeviceBuffer W, G, Wr, Wry, rho32;  // Wr: see inverse_rows
  DeviceBuffer W2, rowtab2;  // the second term of a paired z pass
  DeviceBuffer kterm, rterm;  // a wide term's subgrids before their weights
  std::map<int, DeviceBuffer> ktabs;
  std::map<int, DeviceBuffer> rtabs;
  DeviceBuffer rowtab;  // per-row z-pass weight coefficients (FP32 form)
};

}  // namespace fc
