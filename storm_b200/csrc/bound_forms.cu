// bound_forms.cu -- the score bound's kernels for scores other than the default ones.
#include "bound_kernel.cuh"

namespace sg {

const void* bound_form(const BoundJob& job) { return bound_kernel_of<BandConst>(job); }

}  // namespace sg
