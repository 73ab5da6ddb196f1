// The aggregation kernels for one combination of the template switches of spmm_kernels.cuh
// (UNIT = true, HOT = false); a translation unit of its own so that the combinations compile side by side.
#include "spmm_kernels.cuh"

#include <algorithm>

namespace drone {

int spmm_dispatch_unit(const SpmmArgs &a, bool vec4) {
    return vec4 ? dispatch_vectors<true, false>(a) : dispatch_floats<true, false>(a);
}

}  // namespace drone
