// fc_fused_gen_f32.cu -- the mixed-radix passes in FP32 (fc_fused_gen.cuh), and
// what does not depend on the precision.
#include "fc_fused_gen.cuh"

namespace fc {

FC_GEN(float)

bool gen_supported(int L, bool row) {
  GPlan p;
  if (!gplan_length(L, &p)) return false;
  if (row) return row_smem(L, 1) <= kGenSmem;
  return col_smem(L) <= kGenSmem;
}

void GenAxis::init(int L, bool fp64) {
  FC_REQUIRE(gplan_length(L, &plan), FC_ERR_UNSUPPORTED,
             "grid size has a prime factor above 7");
  auto put = [&](const auto &t) {
    tw.resize(t.size() * sizeof(t[0]));
    FC_CUDA(cudaMemcpy(tw.get(), t.data(), t.size() * sizeof(t[0]),
                       cudaMemcpyHostToDevice));
  };
  if (fp64) put(gplan_twiddles<double2>(plan));
  else put(gplan_twiddles<float2>(plan));
}

}  // namespace fc
