// Image-transform kernels of every eighth box size of the mixed-radix table (see
// image_fft_mixed.cu); split over translation units to compile in parallel.
#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {
extern const Kernels kPart6[] = {
    make_kernels<52, 13>(), make_kernels<80, 8>(), make_kernels<108, 9>(),
    make_kernels<144, 12>(), make_kernels<180, 15>(), make_kernels<216, 12>(),
    make_kernels<256, 16>(), make_kernels<308, 14>(), make_kernels<352, 16>(),
    make_kernels<448, 16>(),
};
extern const int kPart6Count = sizeof(kPart6) / sizeof(kPart6[0]);
}  // namespace mixed
}  // namespace mem
