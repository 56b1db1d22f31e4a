// tn_run_f64.cu -- the executor in F64 precision.
#include "tn_run.cuh"

namespace tn {

TN_INSTANTIATE_RUN(double, f64)

}  // namespace tn
