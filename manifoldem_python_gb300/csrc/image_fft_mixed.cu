// Box sizes of the mixed-radix image transforms (fft_mixed_kernels.cuh) and their launches.
//
// The table holds even sizes from 36 to 512 px that factor as R1 R2 with R1 up to 20, 23 or 25, R2
// even and up to 32, and prime factors up to 23: two thirds of the even sizes up to 300 and all
// the customary ones.  Other sizes keep cuFFT; 32, 64 and 128 px keep the kernels of image_fft.cu,
// whose warps own their rows and columns (a spectrum of 128 px: 32 us per 1000 images).
#include <algorithm>

#include "fft_mixed_kernels.cuh"

namespace mem {
namespace mixed {

#define MEM_PART(i)                \
    extern const Kernels kPart##i[]; \
    extern const int kPart##i##Count;
MEM_PART(0) MEM_PART(1) MEM_PART(2) MEM_PART(3) MEM_PART(4) MEM_PART(5) MEM_PART(6) MEM_PART(7)
MEM_PART(8) MEM_PART(9)
#undef MEM_PART

namespace {

const Kernels* find(int N) {
    const Kernels* parts[] = {kPart0, kPart1, kPart2, kPart3, kPart4,
                              kPart5, kPart6, kPart7, kPart8, kPart9};
    const int counts[] = {kPart0Count, kPart1Count, kPart2Count, kPart3Count,
                          kPart4Count, kPart5Count, kPart6Count, kPart7Count,
                          kPart8Count, kPart9Count};
    for (int i = 0; i < 10; ++i)
        for (int j = 0; j < counts[i]; ++j)
            if (parts[i][j].N == N) return &parts[i][j];
    return nullptr;
}

template <class Args>
int launch(const Kernels& k, void (*fn)(Args), const Args& args, int64_t images,
           cudaStream_t s) {
    if (images == 0) return MEM_OK;
    MEM_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)k.smem));
    fn<<<(unsigned)images, k.threads, k.smem, s>>>(args);
    MEM_LAUNCH_CHECK();
    return MEM_OK;
}

}  // namespace

bool supported(int N) { return find(N) != nullptr; }

size_t inverse_alignment(int N) {
    const Kernels* k = find(N);
    return k && k->tiled ? sizeof(float2) : sizeof(float);
}

int lowpass(int N, const mem_inputs& in, int64_t images, const float* gtab, const float2* twid,
            float* xbuf, uint32_t* status, cudaStream_t s) {
    const Kernels* k = find(N);
    if (!k) return MEM_ERR_UNSUPPORTED;
    return launch(*k, k->lowpass,
                  LowpassArgs{in.stack, in.num_stack, in.stack_index, in.flip, gtab, twid, xbuf,
                              status},
                  images, s);
}

int spectrum(int N, int64_t images, const float* src, const uint8_t* masks, const int32_t* img_pd,
             const float2* twid, float2* spec, cudaStream_t s) {
    const Kernels* k = find(N);
    if (!k) return MEM_ERR_UNSUPPORTED;
    return launch(*k, k->spectrum, SpectrumArgs{src, masks, img_pd, twid, spec}, images, s);
}

int inverse(int N, int64_t images, const float2* spec, const float2* twid, float* dst,
            const uint64_t* qf, const CtfConst& cc, cudaStream_t s) {
    const Kernels* k = find(N);
    if (!k) return MEM_ERR_UNSUPPORTED;
    return launch(*k, qf ? k->inverse_signed : k->inverse, InverseArgs{spec, twid, dst, qf, cc},
                  images, s);
}

bool rotate_supported(int N) {
    const Kernels* k = find(N);
    return k && k->rotate;
}

int rotate(int N, int64_t images, float* xbuf, float* img_out, const void* rotc, cudaStream_t s) {
    const Kernels* k = find(N);
    if (!k || !k->rotate) return MEM_ERR_UNSUPPORTED;
    if (images == 0) return MEM_OK;
    MEM_CUDA_TRY(cudaFuncSetAttribute(k->rotate, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)k->rot_smem));
    k->rotate<<<(unsigned)images, k->rot_threads, k->rot_smem, s>>>(
            xbuf, img_out, static_cast<const rot::RotConst*>(rotc));
    MEM_LAUNCH_CHECK();
    return MEM_OK;
}

}  // namespace mixed
}  // namespace mem
