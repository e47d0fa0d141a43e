// Image transforms and whole-image rotations of every tenth box size of the mixed-radix table
// (see image_fft_mixed.cu); split over translation units to compile in parallel.
#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {
extern const Kernels kPart6[] = {
    make_kernels<52, 13, 26, 52>(), make_kernels<88, 11, 22, 44>(),
    make_kernels<126, 9, 18, 126>(), make_kernels<168, 12, 28, 168>(),
    make_kernels<216, 12, 24, 108>(), make_kernels<264, 12>(), make_kernels<330, 15>(),
    make_kernels<400, 20>(), make_kernels<136, 17, 34, 136>(), make_kernels<266, 19>(),
    make_kernels<380, 19>(),
};
extern const int kPart6Count = sizeof(kPart6) / sizeof(kPart6[0]);
}  // namespace mixed
}  // namespace mem
