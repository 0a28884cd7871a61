// box_mixed.cu -- one-launch box kernels of the mixed precision mode (see box_launch.cuh).
#include "box_launch.cuh"

namespace ifdm {

const BoxKernels &box_kernels_mixed() { return BoxTable<float, double>::table(); }

}  // namespace ifdm
