// The aggregation kernels for one combination of the template switches of spmm_kernels.cuh
// (UNIT = false, HOT = false); a translation unit of its own so that the combinations compile side by side.
#include "spmm_kernels.cuh"

#include <algorithm>

namespace drone {

int spmm_dispatch_plain(const SpmmArgs &a, bool vec4) {
    return vec4 ? dispatch_vectors<false, false>(a) : dispatch_floats<false, false>(a);
}

}  // namespace drone
