// RELION branch of the image read (reference modules/getDistanceCTF_local_Conj9combinedS2.py
// :259-264): the particle image as stored in the MRC stack (no transpose), shifted by
// (sh_y - 0.5, sh_x - 0.5) with scipy.ndimage.shift(order=3, mode='wrap').
//
// That scipy call (measured against scipy 1.18 to 1e-15) is a cubic B-spline shift whose
//   * coefficients come from the mirror-boundary prefilter (the 'mirror' spline filter: the
//     signal extended symmetrically, period 2N-2) along each axis;
//   * sample coordinate u = i - s is wrapped with period N-1 into [0, N-1] when it falls outside;
//   * four taps floor(u)-1 .. floor(u)+2 take mirrored indices (k -> -k, N-1+k -> N-1-k).
// A shift has one fractional offset per axis, so the 2D interpolation is two separable passes,
// each a prefilter and 4 taps of constant weight.
//
// Output: the shifted image transposed (out[a][b] = I[b][a]), i.e. laid out as a SPIDER stack
// image is, so the rest of the stage (conjugate flip, normalisation, low-pass, ...) reads it
// unchanged.  One CTA per image, the image in shared memory, N <= 236.
//
// relion_shift_kernel (N >= 40): a line is split into nseg segments of L <= 32 samples, one thread
// per segment holding it in registers; the states between segments go through shared memory (z^20 =
// 4e-12 of a state is left out at a line's start, where the float transforms that follow round at
// 1e-7 of the image's largest value).
// Axis 0 comes first, its lines read from global memory (lanes on consecutive columns), and
// axis 1 last, its results written to global memory (lanes on consecutive rows of the transposed
// output): an image is read and written once, coalesced.  Bound by the latency of the
// segments at a line's ends (their windows are mirrored or wrapped tap by tap, inner segments slide
// theirs along the line): 846 images of 100 px take 98 us, 111 with mirrored taps everywhere and
// two operations per anticausal step; 209 with a whole line per thread (serial chains of 3 N)
// and the taps of every output in FP64.  512 threads: 98, a branch per output: 125.  Smaller boxes keep that form, whose start values are exact for
// any length (relion_small_kernel).
#include <algorithm>
#include <cmath>

#include "mem_internal.cuh"

namespace mem {
namespace {

constexpr float kPole = -0.26794919243112270f;   // sqrt(3) - 2

__device__ __forceinline__ int mirror_index(int k, int N) {
    const int P = 2 * N - 2;
    if (P <= 0) return 0;
    k %= P;
    if (k < 0) k += P;
    return k >= N ? P - k : k;
}

// mirror-boundary cubic B-spline prefilter of one line x[0..N-1] (stride st) in place
__device__ void mirror_prefilter_line(float* x, int N, int st) {
    if (N < 2) return;
    const float z = kPole;
    // causal start: sum over one period of the symmetric extension, / (1 - z^(2N-2))
    float zk = z, s = x[0];
    const int L = 2 * N - 2;
    float zL = 1.f;
    for (int k = 0; k < L; ++k) zL *= z;
    float zLk = zL / z;                     // z^(L-1)
    for (int k = 1; k < N - 1; ++k) {
        s += (zk + zLk) * x[k * st];
        zk *= z;
        zLk /= z;
    }
    s += zk * x[(N - 1) * st];              // z^(N-1) x[N-1]
    float cp = s / (1.f - zL);
    x[0] = cp;
    for (int k = 1; k < N; ++k) {
        cp = x[k * st] + z * cp;
        x[k * st] = cp;
    }
    // anticausal start for the mirror boundary, then c-[k] = z (c-[k+1] - c+[k]); output 6 c-
    float cm = (z / (z * z - 1.f)) * (x[(N - 1) * st] + z * x[(N - 2) * st]);
    x[(N - 1) * st] = 6.f * cm;
    for (int k = N - 2; k >= 0; --k) {
        cm = z * (cm - x[k * st]);
        x[k * st] = 6.f * cm;
    }
}

__device__ __forceinline__ void bspline4(float t, float w[4]) {
    const float u = 1.0f - t;
    const float t2 = t * t, u2 = u * u;
    w[0] = (1.0f / 6.0f) * u2 * u;
    w[3] = (1.0f / 6.0f) * t2 * t;
    w[1] = (2.0f / 3.0f) - t2 * (1.0f - 0.5f * t);
    w[2] = (2.0f / 3.0f) - u2 * (1.0f - 0.5f * u);
}

// the wrapped sample coordinate of output index i for shift s: first tap and fraction
__device__ __forceinline__ void wrap_coord(int i, double s, int N, int* f, float* t) {
    double u = (double)i - s;
    const double per = (double)(N - 1);
    if (per > 0.0 && (u < 0.0 || u > per)) {
        const bool below = u < 0.0;
        u -= per * floor(u / per);
        if (below && u == 0.0) u = per;            // a negative whole period lands on the far end
    }
    const double fu = floor(u);
    *f = (int)fu;
    *t = (float)(u - fu);
}

constexpr int kMaxPer = 2;                         // N < 40: outputs per lane and line

// Interpolation along one axis, one warp per line, in place: lane l computes the outputs
// j = l + 32 q of its line into registers, then writes them (taps and weights per j are the
// same for every line and are computed once).  Lines are rows (axis 1, stride 1 along the line)
// or columns (axis 0, stride P).
__device__ __forceinline__ void shift_lines(float* A, int N, int P, double sh, int line_stride,
                                            int elem_stride, int nwarps) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int tap[kMaxPer][4];
    float w[kMaxPer][4];
#pragma unroll
    for (int q = 0; q < kMaxPer; ++q) {
        const int j = lane + 32 * q;
        int f = 0;
        float t = 0.f;
        if (j < N) wrap_coord(j, sh, N, &f, &t);
        bspline4(t, w[q]);
#pragma unroll
        for (int b = 0; b < 4; ++b) tap[q][b] = mirror_index(f - 1 + b, N) * elem_stride;
    }
    for (int line = warp; line < N; line += nwarps) {
        float* x = A + line * line_stride;
        float v[kMaxPer];
#pragma unroll
        for (int q = 0; q < kMaxPer; ++q) {
            float acc = 0.f;
            if (lane + 32 * q < N) {
#pragma unroll
                for (int b = 0; b < 4; ++b) acc = fmaf(w[q][b], x[tap[q][b]], acc);
            }
            v[q] = acc;
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < kMaxPer; ++q)
            if (lane + 32 * q < N) x[(lane + 32 * q) * elem_stride] = v[q];
        __syncwarp();
    }
}

template <int NT>
__global__ void __launch_bounds__(NT) relion_small_kernel(
        const float* __restrict__ stack, int64_t num_stack, const int64_t* __restrict__ sidx,
        const double* __restrict__ shift_yx, int N, float* __restrict__ out,
        uint32_t* __restrict__ status) {
    extern __shared__ float A[];           // the image, [N][N+1]
    const int P = N + 1;
    const int64_t img = blockIdx.x;
    const int64_t s = sidx[img];
    float* dst = out + img * (int64_t)N * N;
    const int NN = N * N;
    if (s < 0 || s >= num_stack) {
        if (threadIdx.x == 0) atomicOr(status, 2u);
        for (int p = threadIdx.x; p < NN; p += NT) dst[p] = __int_as_float(0x7fc00000);
        return;
    }
    const float* src = stack + s * (int64_t)NN;
    for (int p = threadIdx.x; p < NN; p += NT) {
        const int r = p / N, c = p - r * N;
        A[r * P + c] = src[p];
    }
    __syncthreads();
    for (int r = threadIdx.x; r < N; r += NT) mirror_prefilter_line(A + r * P, N, 1);   // axis 1
    __syncthreads();
    for (int c = threadIdx.x; c < N; c += NT) mirror_prefilter_line(A + c, N, P);       // axis 0
    __syncthreads();
    // axis 1 (shift sh_x - 0.5), then axis 0 (shift sh_y - 0.5)
    shift_lines(A, N, P, shift_yx[2 * img + 1], P, 1, NT / 32);
    __syncthreads();
    shift_lines(A, N, P, shift_yx[2 * img], 1, P, NT / 32);
    __syncthreads();
    // transposed store: out[a][b] = I[b][a]
    for (int p = threadIdx.x; p < NN; p += NT) {
        const int a = p / N, b = p - a * N;
        dst[p] = A[b * P + a];
    }
}

// Segments of one axis of one image (see above): line l, segment g of L samples (the last one
// shorter).
constexpr int kSeg = 32;
struct ShiftAxis {
    int N, L, nseg, lpr;
    float zL;                              // kPole^L
};

// prefilter and shift along one axis.  GLOBAL_IN: sample k of line l is src[k N + l], else
// s[l SL + k SK]; the coefficients go to s; the result to s, or (GLOBAL_OUT) to dst[k N + l].
template <int NT, bool GLOBAL_IN, bool GLOBAL_OUT>
__device__ __forceinline__ void shift_axis(float* s, float* carry, const float* __restrict__ src,
                                           float* __restrict__ dst, double shift, int SL, int SK,
                                           const ShiftAxis& ax) {
    const float z = kPole;
    const int N = ax.N, L = ax.L;
    const int lw = threadIdx.x % ax.lpr, g = threadIdx.x / ax.lpr;
    const int k0 = g * L, len = min(L, N - k0);
    // output k samples at k - shift = k + i0 + t
    const double fl = floor(-shift);
    // far outside, where every sample wraps, the whole part is first reduced by whole periods, to the
    // same side (a sample a whole number of periods away lands on the line's other end)
    const double per = (double)(N - 1);
    const double fr = fabs(fl) > 1.0e6 ? fl - per * floor(fl / per) + copysign(16.0 * per, fl) : fl;
    const int i0 = (int)fmin(fmax(fr, -1.0e9), 1.0e9);       // in range for a NaN or inf shift too
    const float t = (float)(-shift - fl);
    float w[4];
    bspline4(t, w);
    float* carry_c = carry;                // [nseg][lpr] causal, then anticausal end states
    float* carry_a = carry + NT;
    for (int l0 = 0; l0 < N; l0 += ax.lpr) {
        const int line = l0 + lw;
        const bool on = g < ax.nseg && line < N;
        float* x = s + line * SL;
        float v[kSeg], line_end = 0.f;
        if (on) {
            float e = 0.f;
#pragma unroll
            for (int k = 0; k < kSeg; ++k)
                if (k < len) {
                    v[k] = GLOBAL_IN ? __ldg(src + (int64_t)(k0 + k) * N + line)
                                     : x[(k0 + k) * SK];
                    e = fmaf(z, e, v[k]);
                }
            carry_c[g * ax.lpr + lw] = e;
        }
        __syncthreads();
        if (on) {
            // the state before the segment: the two previous end states, or for the first
            // segment the mirrored samples themselves, sum_{j >= 1} z^(j-1) x[j]
            float c;
            if (g == 0) {
                c = 0.f;
#pragma unroll
                for (int k = kSeg - 1; k >= 1; --k)
                    if (k < len) c = fmaf(z, c, v[k]);
            } else {
                c = carry_c[(g - 1) * ax.lpr + lw];
                if (g > 1) c = fmaf(ax.zL, carry_c[(g - 2) * ax.lpr + lw], c);
            }
            float last = 0.f, before = 0.f;            // c+ of the line's last two samples
#pragma unroll
            for (int k = 0; k < kSeg; ++k)
                if (k < len) {
                    c = fmaf(z, c, v[k]);
                    v[k] = -z * c;                 // z (e - c) = fma(z, e, -z c): one step
                    before = last;
                    last = c;
                }
            const float end = (z / (z * z - 1.f)) * (last + z * before);
            float e = 0.f;
            if (g == ax.nseg - 1) {                    // the mirror's closed form at the end
                e = end;
#pragma unroll
                for (int k = kSeg - 1; k >= 0; --k)
                    if (k < len - 1) e = fmaf(z, e, v[k]);
            } else {
#pragma unroll
                for (int k = kSeg - 1; k >= 0; --k)
                    if (k < len) e = fmaf(z, e, v[k]);
            }
            carry_a[g * ax.lpr + lw] = e;
            line_end = end;
        }
        __syncthreads();
        if (on) {
            if (g == ax.nseg - 1) {
                float c = line_end;
#pragma unroll
                for (int k = kSeg - 1; k >= 0; --k)
                    if (k < len) {
                        if (k < len - 1) c = fmaf(z, c, v[k]);
                        x[(k0 + k) * SK] = 6.f * c;
                    }
            } else {
                float c = carry_a[(g + 1) * ax.lpr + lw];
                if (g + 2 < ax.nseg) {
                    // the end state of a segment of L, carried over the one between
                    c = fmaf(ax.zL, carry_a[(g + 2) * ax.lpr + lw], c);
                }
#pragma unroll
                for (int k = kSeg - 1; k >= 0; --k)
                    if (k < len) {
                        c = fmaf(z, c, v[k]);
                        x[(k0 + k) * SK] = 6.f * c;
                    }
            }
        }
        __syncthreads();
        const int f0 = k0 + i0;
        if (on && f0 >= 1 && f0 + len <= N - 2) {
            // every window inside the line: taps f - 1 .. f + 2 slide along it
            const float* q = x + (f0 - 1) * SK;
            float a = q[0], b = q[SK], c = q[2 * SK];
            q += 3 * SK;
#pragma unroll
            for (int k = 0; k < kSeg; ++k)
                if (k < len) {
                    const float d = *q;
                    q += SK;
                    v[k] = fmaf(w[3], d, fmaf(w[2], c, fmaf(w[1], b, w[0] * a)));
                    a = b;
                    b = c;
                    c = d;
                }
        } else if (on) {
#pragma unroll
            for (int k = 0; k < kSeg; ++k)
                if (k < len) {
                    // wrapped with period N - 1 where the sample point lies outside [0, N - 1]
                    int f = f0 + k;
                    if (f < 0 || f > N - 1 || (f == N - 1 && t > 0.f)) {
                        const bool below = f < 0;
                        f %= N - 1;
                        f += f < 0 ? N - 1 : 0;
                        f = below && f == 0 && t == 0.f ? N - 1 : f;     // as scipy wraps
                    }
                    float acc = 0.f;
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        int q = f - 1 + b;             // -1 .. N + 1, mirrored
                        q = q < 0 ? -q : q;
                        q = q > N - 1 ? 2 * (N - 1) - q : q;
                        acc = fmaf(w[b], x[q * SK], acc);
                    }
                    v[k] = acc;
                }
        }
        if (!GLOBAL_OUT) __syncthreads();              // every tap of the lines is read
        if (on) {
#pragma unroll
            for (int k = 0; k < kSeg; ++k)
                if (k < len) {
                    if (GLOBAL_OUT)
                        dst[(int64_t)(k0 + k) * N + line] = v[k];
                    else
                        x[(k0 + k) * SK] = v[k];
                }
        }
    }
    __syncthreads();
}

template <int NT>
__global__ void __launch_bounds__(NT, 3) relion_shift_kernel(
        const float* __restrict__ stack, int64_t num_stack, const int64_t* __restrict__ sidx,
        const double* __restrict__ shift_yx, ShiftAxis ax, float* __restrict__ out,
        uint32_t* __restrict__ status) {
    extern __shared__ float smem[];        // carries [2 NT], the image [N][N | 1]
    const int N = ax.N, P = N | 1, NN = N * N;
    const int64_t img = blockIdx.x;
    const int64_t s = sidx[img];
    float* dst = out + img * (int64_t)NN;
    if (s < 0 || s >= num_stack) {
        if (threadIdx.x == 0) atomicOr(status, 2u);
        for (int p = threadIdx.x; p < NN; p += NT) dst[p] = __int_as_float(0x7fc00000);
        return;
    }
    float* A = smem + 2 * NT;
    // axis 0 (rows r of column l): shift sh_y - 0.5; axis 1 (columns c of row l): sh_x - 0.5,
    // written to out[c][r]
    shift_axis<NT, true, false>(A, smem, stack + s * (int64_t)NN, nullptr, shift_yx[2 * img], 1, P,
                                ax);
    shift_axis<NT, false, true>(A, smem, nullptr, dst, shift_yx[2 * img + 1], P, 1, ax);
}

}  // namespace

namespace kern {
int relion_shift(const mem_plan& P, const mem_inputs& in, float* out, uint32_t* status,
                 cudaStream_t s) {
    if (P.n_images == 0) return MEM_OK;
    const int N = P.N;
    if (N > kMaxSmemN) return MEM_ERR_UNSUPPORTED;         // one image in shared memory
    if (N >= 40) {
        constexpr int NT = 256;
        ShiftAxis ax;
        ax.N = N;
        ax.nseg = (N + kSeg - 1) / kSeg;
        ax.L = (N + ax.nseg - 1) / ax.nseg;            // >= 20: the last segment has >= 13 samples
        ax.lpr = std::min(N, NT / ax.nseg);
        ax.zL = (float)std::pow((double)kPole, (double)ax.L);
        const size_t smem = (2 * NT + (size_t)N * (N | 1)) * sizeof(float);
        MEM_CUDA_TRY(cudaFuncSetAttribute(relion_shift_kernel<NT>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)smem));
        relion_shift_kernel<NT><<<(unsigned)P.n_images, NT, smem, s>>>(
                in.stack, in.num_stack, in.stack_index, in.shift_yx, ax, out, status);
    } else {
        const size_t smem = (size_t)N * (N + 1) * sizeof(float);
        constexpr int NT = 256;
        relion_small_kernel<NT><<<(unsigned)P.n_images, NT, smem, s>>>(
                in.stack, in.num_stack, in.stack_index, in.shift_yx, N, out, status);
    }
    MEM_LAUNCH_CHECK();
    return MEM_OK;
}
}  // namespace kern
}  // namespace mem
