// Association kernels of clouds without labels.
#include "cvo_assoc.cuh"

namespace cvo_gb {

int assoc_kernels_no_labels(int fch, bool gt, AssocKernels *a) { return assoc_kernels<0>(fch, gt, a); }

}  // namespace cvo_gb
