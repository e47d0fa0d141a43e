// Image transforms and whole-image rotations of every eighth box size of the mixed-radix table
// (see image_fft_mixed.cu); split over translation units to compile in parallel.
#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {
extern const Kernels kPart7[] = {
    make_kernels<54, 9, 27, 54>(), make_kernels<84, 7, 28, 84>(), make_kernels<110, 11, 22, 55>(),
    make_kernels<150, 15, 25, 150>(), make_kernels<182, 13, 26, 91>(),
    make_kernels<220, 10, 10, 44>(), make_kernels<260, 13>(), make_kernels<312, 12>(),
    make_kernels<360, 15>(), make_kernels<480, 20>(),
};
extern const int kPart7Count = sizeof(kPart7) / sizeof(kPart7[0]);
}  // namespace mixed
}  // namespace mem
