// Image transforms and whole-image rotations of every eighth box size of the mixed-radix table
// (see image_fft_mixed.cu); split over translation units to compile in parallel.
#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {
extern const Kernels kPart4[] = {
    make_kernels<48, 6, 24, 48>(), make_kernels<72, 9, 18, 72>(),
    make_kernels<100, 10, 20, 100>(), make_kernels<132, 11, 22, 132>(),
    make_kernels<168, 12, 28, 168>(), make_kernels<208, 13, 26, 104>(), make_kernels<250, 25>(),
    make_kernels<288, 16>(), make_kernels<338, 13>(), make_kernels<400, 20>(),
};
extern const int kPart4Count = sizeof(kPart4) / sizeof(kPart4[0]);
}  // namespace mixed
}  // namespace mem
