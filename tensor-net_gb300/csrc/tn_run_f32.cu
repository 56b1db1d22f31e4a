// tn_run_f32.cu -- the executor in MIXED precision.
#include "tn_run.cuh"

namespace tn {

TN_INSTANTIATE_RUN(float, f32)

}  // namespace tn
