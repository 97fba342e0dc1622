// track_kernel_map.cu -- the tracking kernel's instantiations for plain rings with TriCub
// maps (KIND_MAP).
#include "track_kernel.cuh"

namespace stg {

STG_KIND(, KIND_MAP)

}  // namespace stg
