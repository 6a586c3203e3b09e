// fc_fused_gen_f64.cu -- the mixed-radix passes in FP64 (fc_fused_gen.cuh).
#include "fc_fused_gen.cuh"

namespace fc {

FC_GEN(double)

}  // namespace fc
