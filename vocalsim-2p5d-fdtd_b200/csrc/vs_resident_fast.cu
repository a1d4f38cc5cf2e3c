// vs_resident_fast.cu -- the resident kernel for table sources, reciprocal form.
#include "vs_resident.cuh"

namespace vsb {

ResidentFn resident_fast(bool hist) {
    return hist ? resident_kernel<true, false, false> : resident_kernel<false, false, false>;
}

}  // namespace vsb
