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
};

}  // namespace fc
