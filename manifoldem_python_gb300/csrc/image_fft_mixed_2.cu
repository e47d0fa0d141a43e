// Image transforms and whole-image rotations of every eighth box size of the mixed-radix table
// (see image_fft_mixed.cu); split over translation units to compile in parallel.
#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {
extern const Kernels kPart2[] = {
    make_kernels<42, 7, 14, 42>(), make_kernels<66, 11, 22, 66>(), make_kernels<96, 8, 32, 96>(),
    make_kernels<126, 9, 18, 126>(), make_kernels<160, 10, 32, 160>(),
    make_kernels<198, 11, 22, 99>(), make_kernels<240, 15>(), make_kernels<280, 14>(),
    make_kernels<330, 15>(), make_kernels<390, 15>(),
};
extern const int kPart2Count = sizeof(kPart2) / sizeof(kPart2[0]);
}  // namespace mixed
}  // namespace mem
