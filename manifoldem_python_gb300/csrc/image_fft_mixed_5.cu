// Image transforms and whole-image rotations of every tenth box size of the mixed-radix table
// (see image_fft_mixed.cu); split over translation units to compile in parallel.
#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {
extern const Kernels kPart5[] = {
    make_kernels<50, 5, 10, 50>(), make_kernels<84, 7, 28, 84>(),
    make_kernels<120, 10, 30, 120>(), make_kernels<162, 9, 27, 162>(),
    make_kernels<210, 15, 15, 70>(), make_kernels<260, 13>(), make_kernels<324, 18>(),
    make_kernels<396, 18>(), make_kernels<114, 19, 19, 114>(), make_kernels<238, 17>(),
    make_kernels<374, 17>(),
};
extern const int kPart5Count = sizeof(kPart5) / sizeof(kPart5[0]);
}  // namespace mixed
}  // namespace mem
