// tn_run_df.cu -- the executor in DF precision.
#include "tn_run.cuh"

namespace tn {

TN_INSTANTIATE_RUN(dd, df)

}  // namespace tn
