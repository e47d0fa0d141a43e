// Image transforms and whole-image rotations of every eighth box size of the mixed-radix table
// (see image_fft_mixed.cu); split over translation units to compile in parallel.
#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {
extern const Kernels kPart6[] = {
    make_kernels<52, 13, 26, 52>(), make_kernels<80, 8, 20, 80>(),
    make_kernels<108, 9, 12, 108>(), make_kernels<144, 12, 24, 144>(),
    make_kernels<180, 15, 18, 90>(), make_kernels<216, 12, 24, 108>(), make_kernels<256, 16>(),
    make_kernels<308, 14>(), make_kernels<352, 16>(), make_kernels<448, 16>(),
};
extern const int kPart6Count = sizeof(kPart6) / sizeof(kPart6[0]);
}  // namespace mixed
}  // namespace mem
