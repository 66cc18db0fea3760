// Association kernels with labels of 9 chunks (up to 36 classes).
#include "cvo_assoc.cuh"

namespace cvo_gb {

int assoc_kernels_labels9(int fch, bool gt, AssocKernels *a) { return assoc_kernels<9>(fch, gt, a); }

}  // namespace cvo_gb
