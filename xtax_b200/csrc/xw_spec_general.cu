// xw_spec_general.cu -- the latency mode's kernels for every objective and
// move set.
#include "xw_spec.cuh"

namespace xw {

const void* anneal_spec_general_fn(int ctas, bool one_zero) { return spec_fn<true>(ctas, one_zero); }

}  // namespace xw
