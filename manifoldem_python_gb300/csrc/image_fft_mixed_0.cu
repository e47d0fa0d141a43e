// Image transforms and whole-image rotations of every tenth box size of the mixed-radix table
// (see image_fft_mixed.cu); split over translation units to compile in parallel.
#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {
extern const Kernels kPart0[] = {
    make_kernels<36, 6, 12, 36>(), make_kernels<66, 11, 22, 66>(),
    make_kernels<100, 10, 20, 100>(), make_kernels<144, 12, 24, 144>(),
    make_kernels<192, 12, 12, 64>(), make_kernels<240, 15>(), make_kernels<288, 16>(),
    make_kernels<352, 16>(), make_kernels<512, 16>(), make_kernels<184, 23, 23, 92>(),
    make_kernels<306, 17>(),
};
extern const int kPart0Count = sizeof(kPart0) / sizeof(kPart0[0]);
}  // namespace mixed
}  // namespace mem
