// Image transforms and whole-image rotations of every eighth box size of the mixed-radix table
// (see image_fft_mixed.cu); split over translation units to compile in parallel.
#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {
extern const Kernels kPart3[] = {
    make_kernels<44, 11, 22, 44>(), make_kernels<70, 7, 10, 70>(), make_kernels<98, 7, 14, 98>(),
    make_kernels<130, 13, 10, 65>(), make_kernels<162, 9, 27, 162>(),
    make_kernels<200, 10, 20, 100>(), make_kernels<242, 11>(), make_kernels<286, 13>(),
    make_kernels<336, 14>(), make_kernels<396, 18>(),
};
extern const int kPart3Count = sizeof(kPart3) / sizeof(kPart3[0]);
}  // namespace mixed
}  // namespace mem
