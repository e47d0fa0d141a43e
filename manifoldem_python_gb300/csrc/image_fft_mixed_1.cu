// Image transforms and whole-image rotations of every tenth box size of the mixed-radix table
// (see image_fft_mixed.cu); split over translation units to compile in parallel.
#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {
extern const Kernels kPart1[] = {
    make_kernels<40, 5, 10, 40>(), make_kernels<70, 7, 10, 70>(),
    make_kernels<104, 13, 26, 104>(), make_kernels<150, 15, 25, 150>(),
    make_kernels<196, 14, 28, 98>(), make_kernels<242, 11>(), make_kernels<300, 15>(),
    make_kernels<360, 15>(), make_kernels<68, 17, 17, 68>(), make_kernels<190, 19, 38, 190>(),
    make_kernels<322, 23>(),
};
extern const int kPart1Count = sizeof(kPart1) / sizeof(kPart1[0]);
}  // namespace mixed
}  // namespace mem
