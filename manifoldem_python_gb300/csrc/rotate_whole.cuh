// The two periodic cubic B-spline rotations (rotatefill.op, modules/rotatefill.py:21-41, called at
// modules/getDistanceCTF_local_Conj9combinedS2.py:328-330) of images of any compile-time box size
// whose coefficient image fits one CTA's shared memory: the scheme of rotate_fixed.cuh (N = 64,
// 128) without its power-of-two layout.
//
// A line is split into G segments of SEG samples (SEG divides N), one thread per segment holding
// it in registers; LPR lines (LPR divides N) are worked on at a time by LPR G threads.  Each thread
// also samples a run of SEG outputs, the segment that the next prefilter gives it.  Between the
// rotations the samples pass through the image's own global slot (each thread reads back what it
// wrote, lanes on consecutive addresses, L2), not through registers: 36,864 samples of a 192 px
// image would take 56% of the register file.
// Bound by shared-memory wavefronts, 25 tap loads per two samples with about two-way bank conflicts.
//   1000 images of 192 px: 342 us (385 with 32 loads per two samples), 513 with the runtime-size
//   kernel (serial 18-tap segment starts, one sample at a time, integer division in its loops);
//   846 of 100 px: 74 us (88), was 135; 300 of 70 px: 18 us (20), was 31.
#pragma once

#include "rotate_fixed.cuh"

namespace mem {
namespace rot {

// row stride of the coefficient image: 1 mod 32 (a warp's samples along a line then meet about
// two to a bank) where that fits beside the carries, else odd
constexpr size_t kWholeSmem = 225 * 1024;
template <int N, int CARRY>
constexpr int whole_stride() {
    constexpr int p = ((N + kHalo + 30) / 32) * 32 + 1;
    return ((size_t)(N + kHalo) * p + CARRY) * sizeof(float) <= kWholeSmem ? p : ((N + kHalo) | 1);
}

template <int N_, int SEG_, int LPR_>
struct WholeShape {
    static constexpr int N = N_, SEG = SEG_, LPR = LPR_, G = N / SEG, ROUNDS = N / LPR;
    static_assert(N % SEG == 0 && N % LPR == 0, "whole segments and rounds");
    static constexpr int TASKS = LPR * G, NT = (TASKS + 31) / 32 * 32;
    static constexpr int CARRY = 2 * TASKS;                    // floats
    static constexpr int P = whole_stride<N, CARRY>();
    static constexpr size_t SMEM = ((size_t)(N + kHalo) * P + CARRY) * sizeof(float);
    static constexpr int BY_SMEM = (int)(kWholeSmem / SMEM), BY_REGS = 65536 / (NT * 64);
    static constexpr int MINB = BY_SMEM < 1 ? 1 : BY_SMEM < BY_REGS ? BY_SMEM
                                                  : BY_REGS < 1     ? 1
                                                                    : BY_REGS;
};

// One axis of the periodic prefilter.  AXIS 0: lines are rows of s, 1: columns.  FROM: 0 the
// line is in s; 1 sample k of line l is src[k N + l] (global), times the annular mask at (l, k);
// 2 the same without a mask.  The result is in s.  A segment's starting state is the end state
// from zero of the CT previous segments (z1^20 = 4e-12 of the state is left out).
template <class Sh, int AXIS, int FROM>
__device__ __forceinline__ void prefilter_whole(float* s, float* carry, const float* src) {
    constexpr int N = Sh::N, SEG = Sh::SEG, G = Sh::G, LPR = Sh::LPR, P = Sh::P;
    constexpr int CT = (20 + SEG - 1) / SEG < G ? (20 + SEG - 1) / SEG : G;
    constexpr int SK = AXIS == 0 ? 1 : P, SL = AXIS == 0 ? P : 1;
    constexpr float zseg = z1_pow<SEG>();
    constexpr float gain = -6.0f * kZ1;
    const int t = threadIdx.x;
    const bool active = Sh::TASKS == Sh::NT || t < Sh::TASKS;
    const int lw = t % LPR, g = t / LPR;
    float* carry_c = carry;                                    // [G][LPR]
    float* carry_a = carry + Sh::TASKS;
#pragma unroll 1
    for (int l0 = 0; l0 < N; l0 += LPR) {
        const int line = l0 + lw;
        float* b0 = s + line * SL + g * SEG * SK;
        float v[SEG];
        if (active) {
            float e = 0.f;
#pragma unroll
            for (int k = 0; k < SEG; ++k) {
                v[k] = FROM == 0 ? b0[k * SK] : src[(g * SEG + k) * N + line];
                if (FROM == 1) v[k] *= mask_ref(line, g * SEG + k, N);
                e = fmaf(kZ1, e, v[k]);
            }
            carry_c[g * LPR + lw] = e;
        }
        __syncthreads();
        if (active) {
            float c = 0.f;
#pragma unroll
            for (int m = CT; m >= 1; --m) {
                const int q = g - m + (g < m ? G : 0);
                c = fmaf(zseg, c, carry_c[q * LPR + lw]);
            }
#pragma unroll
            for (int k = 0; k < SEG; ++k) {
                c = fmaf(kZ1, c, v[k]);
                v[k] = c;
            }
            float e = 0.f;
#pragma unroll
            for (int k = SEG - 1; k >= 0; --k) e = fmaf(kZ1, e, v[k]);
            carry_a[g * LPR + lw] = e;
        }
        __syncthreads();
        if (active) {
            float c = 0.f;
#pragma unroll
            for (int m = CT; m >= 1; --m) {
                const int q = g + m - (g + m >= G ? G : 0);
                c = fmaf(zseg, c, carry_a[q * LPR + lw]);
            }
#pragma unroll
            for (int k = SEG - 1; k >= 0; --k) {
                c = fmaf(kZ1, c, v[k]);
                b0[k * SK] = gain * c;
            }
        }
        // the next round's first writes are to carry_c, read before the last barrier
    }
    __syncthreads();
}

template <int N>
__device__ __forceinline__ int wrap_any(int i) {               // [-N, 2N) -> [0, N)
    i += (i < 0) ? N : 0;
    return i - ((i >= N) ? N : 0);
}

// One rotation of the coefficient image in s: the thread of (u, g) samples the outputs (g SEG + k,
// u) when the lanes run along output rows, (u, g SEG + k) when they run along columns
// (whichever lane step has components of one sign), into dst[(g SEG + k) N + u].
template <class Sh>
__device__ __forceinline__ bool rotate_whole_once(const float* s, const RotConst& Q, float* dst) {
    constexpr int N = Sh::N, SEG = Sh::SEG, LPR = Sh::LPR;
    constexpr int64_t kOne = 1ll << 32;
    const bool along_cols = (Q.rc > 0) != (Q.rs > 0);
    const int64_t dX = along_cols ? Q.rs : Q.rc, dY = along_cols ? Q.rc : -Q.rs;
    const int lw = threadIdx.x % LPR, v0 = (threadIdx.x / LPR) * SEG;
    if (Sh::TASKS == Sh::NT || (int)threadIdx.x < Sh::TASKS) {
#pragma unroll 1
        for (int l0 = 0; l0 < N; l0 += LPR) {
            const int u = l0 + lw;
            const int r = along_cols ? u : v0, c = along_cols ? v0 : u;
            int64_t X = Q.bx - kOne + (int64_t)r * Q.rc + (int64_t)c * Q.rs;
            int64_t Y = Q.by - kOne - (int64_t)r * Q.rs + (int64_t)c * Q.rc;
            float* d = dst + v0 * N + u;
#pragma unroll 1
            for (int k = 0; k < SEG; k += 2, X += 2 * dX, Y += 2 * dY, d += 2 * N) {
                // an odd SEG's last sample alone: its partner repeats it
                const bool two = SEG % 2 == 0 || k + 1 < SEG;
                const float2 v = sample_pair(
                    X, Y, two ? X + dX : X, two ? Y + dY : Y, Sh::P, [s](int x, int y) {
                        return s + wrap_any<N>(x) * Sh::P + wrap_any<N>(y);
                    });
                d[0] = v.x;
                if (two) d[N] = v.y;
            }
        }
    }
    return along_cols;
}

template <int NT>
__device__ __forceinline__ void store_rows(const float* s, int P, int N, float* out) {
    for (int p = threadIdx.x; p < N * N; p += NT) out[p] = s[(p / N) * P + p % N];
}

// xbuf: the low-passed image in storage orientation, then scratch; out: imgAll
template <class Sh>
__global__ void __launch_bounds__(Sh::NT, Sh::MINB) rotate_whole_kernel(
        float* xbuf, float* img_out, const RotConst* __restrict__ rotc) {
    constexpr int N = Sh::N, P = Sh::P, NT = Sh::NT;
    extern __shared__ float whole_smem[];
    float* carry = whole_smem;
    float* s = whole_smem + Sh::CARRY;
    const int64_t img = blockIdx.x;
    float* xi = xbuf + img * (int64_t)(N * N);
    float* out = img_out + img * (int64_t)(N * N);
    const RotConst q0 = rotc[2 * img];
    prefilter_whole<Sh, 0, 1>(s, carry, xi);
    prefilter_whole<Sh, 1, 0>(s, carry, nullptr);
    fill_halo<NT, kHalo>(s, N, P);
    // every read of xi is behind a barrier: it takes the first rotation's samples; a thread's
    // samples are the prefilter segment it reads back, and the prefilter's barriers separate the
    // sampling from the stores into s
    if (rotate_whole_once<Sh>(s, q0, xi)) {
        prefilter_whole<Sh, 0, 2>(s, carry, xi);
        prefilter_whole<Sh, 1, 0>(s, carry, nullptr);
    } else {
        prefilter_whole<Sh, 1, 2>(s, carry, xi);
        prefilter_whole<Sh, 0, 0>(s, carry, nullptr);
    }
    fill_halo<NT, kHalo>(s, N, P);
    const RotConst q1 = rotc[2 * img + 1];
    const bool turned = (q1.rc > 0) != (q1.rs > 0);
    rotate_whole_once<Sh>(s, q1, turned ? xi : out);
    if (!turned) return;                                       // lanes along rows: in place
    __syncthreads();
    // lanes along columns: xi holds the transposed result, turned through s
    for (int p = threadIdx.x; p < N * N; p += NT) {
        const int v = p / N, u = p - v * N;
        s[u * P + v] = xi[p];
    }
    __syncthreads();
    store_rows<NT>(s, P, N, out);
}

}  // namespace rot
}  // namespace mem
