// Image transforms and whole-image rotations of every tenth box size of the mixed-radix table
// (see image_fft_mixed.cu); split over translation units to compile in parallel.
#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {
extern const Kernels kPart9[] = {
    make_kernels<60, 6, 30, 60>(), make_kernels<98, 7, 14, 98>(),
    make_kernels<140, 10, 20, 140>(), make_kernels<182, 13, 26, 91>(), make_kernels<234, 13>(),
    make_kernels<286, 13>(), make_kernels<350, 25>(), make_kernels<480, 20>(),
    make_kernels<170, 17, 34, 170>(), make_kernels<304, 19>(),
};
extern const int kPart9Count = sizeof(kPart9) / sizeof(kPart9[0]);
}  // namespace mixed
}  // namespace mem
