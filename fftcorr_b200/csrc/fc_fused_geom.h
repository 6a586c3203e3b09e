// fc_fused_geom.h -- geometry shared by the fused passes' kernels.
#pragma once

namespace fc {

// Passed by value to every kernel.
struct FusedGeom {
  int n0, n1, n2;  // grid shape
  int m;           // N2 / 2
  int h;           // N2 / 2 + 1: half-complex z extent
  int hp;          // row pitch of W, G, Wr, Wry: h rounded up to 16, so
                   // every 16-column group starts on a 128-byte line
  int rs, ro;      // r-subgrid edge and its centre offset (rs / 2)
  int ks0, ks1, ks2;  // k-subgrid shape
  int kp;          // row pitch of the stored half of the k-subgrid (kz >= 0)
  int nri;         // r-subgrid rows along x that are computed: ro + 1 (x >= 0)
                   // in the even form, else rs
};

// What is stored of the subgrids.  Re P is even (P(-k) = conj P(k)), so of
// the k-subgrid only the cells with kz >= 0 are kept: cell (i, j, oz + kz) at
// (i ks1 + j) kp + kz.  In the even form the r-subgrid keeps the rows x >= 0:
// cell (ro + x, j, k) at (x rs + j) rs + k.  The centre of a subgrid of odd
// sides is its middle cell, so the mirror image of linear cell c is n - 1 - c.
__host__ __device__ inline size_t half_k_cell(const FusedGeom &g, size_t c) {
  const int oz = g.ks2 / 2;
  if ((int)(c % g.ks2) < oz) c = (size_t)g.ks0 * g.ks1 * g.ks2 - 1 - c;
  return c / g.ks2 * g.kp + (c % g.ks2 - oz);
}
__host__ __device__ inline size_t half_r_cell(const FusedGeom &g, size_t c) {
  if (g.nri == g.rs) return c;
  const size_t lo = (size_t)g.ro * g.rs * g.rs;
  return (c >= lo ? c : (size_t)g.rs * g.rs * g.rs - 1 - c) - lo;
}

}  // namespace fc
