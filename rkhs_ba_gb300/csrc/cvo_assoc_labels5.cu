// Association kernels with labels of 5 chunks (up to 20 classes).
#include "cvo_assoc.cuh"

namespace cvo_gb {

int assoc_kernels_labels5(int fch, bool gt, AssocKernels *a) { return assoc_kernels<5>(fch, gt, a); }

}  // namespace cvo_gb
