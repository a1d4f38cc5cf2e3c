// vs_resident_exact.cu -- the resident kernel for table sources, reference arithmetic.
#include "vs_resident.cuh"

namespace vsb {

ResidentFn resident_exact(bool hist) {
    return hist ? resident_kernel<true, true, false> : resident_kernel<false, true, false>;
}

}  // namespace vsb
