// Image transforms and whole-image rotations of every tenth box size of the mixed-radix table
// (see image_fft_mixed.cu); split over translation units to compile in parallel.
#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {
extern const Kernels kPart2[] = {
    make_kernels<42, 7, 14, 42>(), make_kernels<72, 9, 18, 72>(), make_kernels<108, 9, 12, 108>(),
    make_kernels<154, 11, 14, 77>(), make_kernels<198, 11, 22, 99>(), make_kernels<250, 25>(),
    make_kernels<308, 14>(), make_kernels<364, 14>(), make_kernels<76, 19, 19, 76>(),
    make_kernels<204, 17, 17, 68>(), make_kernels<340, 17>(),
};
extern const int kPart2Count = sizeof(kPart2) / sizeof(kPart2[0]);
}  // namespace mixed
}  // namespace mem
