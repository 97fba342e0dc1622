// track_kernel_full.cu -- the tracking kernel's instantiations for lattices with any element (KIND_FULL).
#include "track_kernel.cuh"

namespace stg {

STG_KIND(, KIND_FULL)

}  // namespace stg
