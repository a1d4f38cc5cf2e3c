// vs_resident_exact_tmm.cu -- the resident kernel for two-mass sources, reference arithmetic.
#include "vs_resident.cuh"

namespace vsb {

ResidentFn resident_exact_tmm(bool hist) {
    return hist ? resident_kernel<true, true, true> : resident_kernel<false, true, true>;
}

}  // namespace vsb
