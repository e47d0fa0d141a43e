// Image-transform kernels of every eighth box size of the mixed-radix table (see
// image_fft_mixed.cu); split over translation units to compile in parallel.
#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {
extern const Kernels kPart7[] = {
    make_kernels<54, 9>(), make_kernels<84, 7>(), make_kernels<110, 11>(),
    make_kernels<150, 15>(), make_kernels<182, 13>(), make_kernels<220, 10>(),
    make_kernels<260, 13>(), make_kernels<312, 12>(), make_kernels<360, 15>(),
    make_kernels<480, 20>(),
};
extern const int kPart7Count = sizeof(kPart7) / sizeof(kPart7[0]);
}  // namespace mixed
}  // namespace mem
