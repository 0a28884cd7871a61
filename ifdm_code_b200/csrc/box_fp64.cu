// box_fp64.cu -- one-launch box kernels of the FP64 precision mode (see box_launch.cuh).
#include "box_launch.cuh"

namespace ifdm {

const BoxKernels &box_kernels_fp64() { return BoxTable<double, double>::table(); }

}  // namespace ifdm
