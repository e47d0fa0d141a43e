// Image transforms and whole-image rotations of every tenth box size of the mixed-radix table
// (see image_fft_mixed.cu); split over translation units to compile in parallel.
#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {
extern const Kernels kPart4[] = {
    make_kernels<48, 6, 24, 48>(), make_kernels<80, 8, 20, 80>(), make_kernels<112, 8, 28, 112>(),
    make_kernels<160, 10, 32, 160>(), make_kernels<208, 13, 26, 104>(), make_kernels<256, 16>(),
    make_kernels<320, 16>(), make_kernels<390, 15>(), make_kernels<102, 17, 34, 102>(),
    make_kernels<230, 23>(), make_kernels<368, 23>(),
};
extern const int kPart4Count = sizeof(kPart4) / sizeof(kPart4[0]);
}  // namespace mixed
}  // namespace mem
