// vs_resident_fast_tmm.cu -- the resident kernel for two-mass sources, reciprocal form.
#include "vs_resident.cuh"

namespace vsb {

ResidentFn resident_fast_tmm(bool hist) {
    return hist ? resident_kernel<true, false, true> : resident_kernel<false, false, true>;
}

}  // namespace vsb
