// track_kernel_plain.cu -- the tracking kernel's instantiations for plain-ring lattices with lead blocks (KIND_PLAIN).
#include "track_kernel.cuh"

namespace stg {

STG_KIND(, KIND_PLAIN)

}  // namespace stg
