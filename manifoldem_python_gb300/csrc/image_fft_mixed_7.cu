// Image transforms and whole-image rotations of every tenth box size of the mixed-radix table
// (see image_fft_mixed.cu); split over translation units to compile in parallel.
#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {
extern const Kernels kPart7[] = {
    make_kernels<54, 9, 27, 54>(), make_kernels<90, 9, 18, 90>(), make_kernels<130, 13, 10, 65>(),
    make_kernels<176, 11, 16, 88>(), make_kernels<220, 10, 10, 44>(), make_kernels<270, 15>(),
    make_kernels<336, 14>(), make_kernels<432, 18>(), make_kernels<138, 23, 23, 138>(),
    make_kernels<272, 17>(),
};
extern const int kPart7Count = sizeof(kPart7) / sizeof(kPart7[0]);
}  // namespace mixed
}  // namespace mem
