// Image transforms and whole-image rotations of every tenth box size of the mixed-radix table
// (see image_fft_mixed.cu); split over translation units to compile in parallel.
#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {
extern const Kernels kPart3[] = {
    make_kernels<44, 11, 22, 44>(), make_kernels<78, 13, 26, 78>(),
    make_kernels<110, 11, 22, 55>(), make_kernels<156, 13, 26, 156>(),
    make_kernels<200, 10, 20, 100>(), make_kernels<252, 14>(), make_kernels<312, 12>(),
    make_kernels<384, 16>(), make_kernels<92, 23, 23, 46>(), make_kernels<228, 19>(),
    make_kernels<342, 19>(),
};
extern const int kPart3Count = sizeof(kPart3) / sizeof(kPart3[0]);
}  // namespace mixed
}  // namespace mem
