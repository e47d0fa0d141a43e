// Image transforms and whole-image rotations of every tenth box size of the mixed-radix table
// (see image_fft_mixed.cu); split over translation units to compile in parallel.
#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {
extern const Kernels kPart8[] = {
    make_kernels<56, 7, 28, 56>(), make_kernels<96, 8, 32, 96>(),
    make_kernels<132, 11, 22, 132>(), make_kernels<180, 15, 18, 90>(),
    make_kernels<224, 14, 28, 112>(), make_kernels<280, 14>(), make_kernels<338, 13>(),
    make_kernels<448, 16>(), make_kernels<152, 19, 38, 152>(), make_kernels<276, 23>(),
};
extern const int kPart8Count = sizeof(kPart8) / sizeof(kPart8[0]);
}  // namespace mixed
}  // namespace mem
