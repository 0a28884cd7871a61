// box_fp32.cu -- one-launch box kernels of the FP32 precision mode (see box_launch.cuh).
#include "box_launch.cuh"

namespace ifdm {

const BoxKernels &box_kernels_fp32() { return BoxTable<float, float>::table(); }

}  // namespace ifdm
