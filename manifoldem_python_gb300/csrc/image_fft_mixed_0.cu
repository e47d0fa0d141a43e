// Image transforms and whole-image rotations of every eighth box size of the mixed-radix table
// (see image_fft_mixed.cu); split over translation units to compile in parallel.
#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {
extern const Kernels kPart0[] = {
    make_kernels<36, 6, 12, 36>(), make_kernels<56, 7, 28, 56>(), make_kernels<88, 11, 22, 44>(),
    make_kernels<112, 8, 28, 112>(), make_kernels<154, 11, 14, 77>(),
    make_kernels<192, 12, 12, 64>(), make_kernels<224, 14, 28, 112>(), make_kernels<264, 12>(),
    make_kernels<320, 16>(), make_kernels<364, 14>(), make_kernels<512, 16>(),
};
extern const int kPart0Count = sizeof(kPart0) / sizeof(kPart0[0]);
}  // namespace mixed
}  // namespace mem
