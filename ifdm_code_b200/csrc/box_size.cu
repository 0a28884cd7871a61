// box_size.cu -- the one-launch box kernels of one grid size and precision mode,
// given on the command line: BOX_NAME (fp64, fp32, mixed), BOX_R and BOX_K (storage
// and arithmetic type), BOX_N (see box_launch.cuh).
#include "box_launch.cuh"

namespace ifdm {

#define BOX_FN2(name, n) box_kernels_##name##_##n
#define BOX_FN(name, n) BOX_FN2(name, n)

const BoxKernels &BOX_FN(BOX_NAME, BOX_N)() { return BoxSize<BOX_R, BOX_K, BOX_N>::table(); }

}  // namespace ifdm
