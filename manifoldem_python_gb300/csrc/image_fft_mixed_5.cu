// Image transforms and whole-image rotations of every eighth box size of the mixed-radix table
// (see image_fft_mixed.cu); split over translation units to compile in parallel.
#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {
extern const Kernels kPart5[] = {
    make_kernels<50, 5, 10, 50>(), make_kernels<78, 13, 26, 78>(),
    make_kernels<104, 13, 26, 104>(), make_kernels<140, 10, 20, 140>(),
    make_kernels<176, 11, 16, 88>(), make_kernels<210, 15, 15, 70>(), make_kernels<252, 14>(),
    make_kernels<300, 15>(), make_kernels<350, 25>(), make_kernels<432, 18>(),
};
extern const int kPart5Count = sizeof(kPart5) / sizeof(kPart5[0]);
}  // namespace mixed
}  // namespace mem
