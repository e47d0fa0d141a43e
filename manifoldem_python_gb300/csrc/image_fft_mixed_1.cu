// Image transforms and whole-image rotations of every eighth box size of the mixed-radix table
// (see image_fft_mixed.cu); split over translation units to compile in parallel.
#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {
extern const Kernels kPart1[] = {
    make_kernels<40, 5, 10, 40>(), make_kernels<60, 6, 30, 60>(), make_kernels<90, 9, 18, 90>(),
    make_kernels<120, 10, 30, 120>(), make_kernels<156, 13, 26, 156>(),
    make_kernels<196, 14, 28, 98>(), make_kernels<234, 13>(), make_kernels<270, 15>(),
    make_kernels<324, 18>(), make_kernels<384, 16>(),
};
extern const int kPart1Count = sizeof(kPart1) / sizeof(kPart1[0]);
}  // namespace mixed
}  // namespace mem
