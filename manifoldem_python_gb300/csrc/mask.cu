// Volume mask of the distance stage (reference modules/getDistanceCTF_local_Conj9combinedS2.py
// :303-310, projectMask.op modules/projectMask.py:118-135): the mask volume rotated to the PD's
// direction with scipy.ndimage.affine_transform (order 3, mode 'nearest'), summed along z and
// thresholded at 1 gives the 2D mask msk2 that multiplies every rotated image before its
// spectrum (:344) -- and through the spectra the averages (:366-367).
//
// In the scipy here (1.18) an order-3 'nearest' interpolation is (measured to 3e-15 against
// affine_transform on 3D volumes): the volume padded by 12 samples per side with its edge
// values, the 'reflect' spline prefilter of the padded volume along each axis, then the
// tensor-product cubic B-spline with tap indices clamped to the padded volume.  The 'reflect'
// prefilter of a line is the exact periodic prefilter of its half-sample-symmetric extension
// (period 2M).  Everything here is float64: the mask is a threshold of a sum.
#include <cmath>

#include "mem_internal.cuh"

namespace mem {
namespace {

constexpr int kMaskPad = 12;
constexpr int kMaxM = kMaxSmemN + 2 * kMaskPad;
constexpr double kPoleD = -0.2679491924311227065;   // sqrt(3) - 2

// P[a][b][c] (M^3, M = N + 24) = swapaxes(vol, 0, 2) padded with edge values; vol is (N, N, N)
// as stored (z, y, x), so P[a][b][c] = vol[cc][cb][ca] with (ca, cb, cc) the clamped indices
__global__ void mask_pad_kernel(const float* __restrict__ vol, int N, double* __restrict__ P) {
    const int M = N + 2 * kMaskPad;
    const int64_t total = (int64_t)M * M * M;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int a = (int)(e / ((int64_t)M * M));
        const int b = (int)((e / M) % M), c = (int)(e % M);
        const int ca = min(max(a - kMaskPad, 0), N - 1);
        const int cb = min(max(b - kMaskPad, 0), N - 1);
        const int cc = min(max(c - kMaskPad, 0), N - 1);
        P[e] = (double)vol[((int64_t)cc * N + cb) * N + ca];
    }
}

// 'reflect' cubic B-spline prefilter along one axis of P, one thread per line
__global__ void mask_prefilter_kernel(double* __restrict__ P, int M, int axis) {
    const int64_t line = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (line >= (int64_t)M * M) return;
    const int64_t u = line / M, v = line % M;
    int64_t base, st;
    if (axis == 0) { base = u * M + v; st = (int64_t)M * M; }
    else if (axis == 1) { base = u * M * M + v; st = M; }
    else { base = (u * M + v) * M; st = 1; }
    const int L = 2 * M;
    double y[2 * kMaxM];
    for (int k = 0; k < M; ++k) {
        const double x = P[base + k * st];
        y[k] = x;
        y[L - 1 - k] = x;
    }
    const double z = kPoleD;
    double zL = 1.0;
    for (int k = 0; k < L; ++k) zL *= z;
    // causal: start value = sum_k z^k y[-k mod L] / (1 - z^L)
    double s = y[0], zk = z;
    for (int k = 1; k < L; ++k) {
        s += zk * y[L - k];
        zk *= z;
    }
    y[0] = s / (1.0 - zL);
    for (int k = 1; k < L; ++k) y[k] += z * y[k - 1];
    // anticausal d[k] = c+[k] + z d[k+1], start value sum_j z^j c+[(L-1+j) mod L] / (1 - z^L)
    double t = y[L - 1];
    zk = z;
    for (int j = 1; j < L; ++j) {
        t += zk * y[j - 1];
        zk *= z;
    }
    double d = t / (1.0 - zL);
    y[L - 1] = d;
    for (int k = L - 2; k >= 0; --k) {
        d = y[k] + z * d;
        y[k] = d;
    }
    const double gain = -6.0 * z;
    for (int k = 0; k < M; ++k) P[base + k * st] = gain * y[k];
}

__device__ __forceinline__ void bspline4d(double t, double w[4]) {
    const double u = 1.0 - t;
    const double t2 = t * t, u2 = u * u;
    w[0] = (1.0 / 6.0) * u2 * u;
    w[3] = (1.0 / 6.0) * t2 * t;
    w[1] = (2.0 / 3.0) - t2 * (1.0 - 0.5 * t);
    w[2] = (2.0 / 3.0) - u2 * (1.0 - 0.5 * u);
}

// masks[pd][a][b] = (sum_k rho(b, a, k) > 1), rho(o) = spline(C, R o + offset):
// projectMask's msk = sum(rho, axis=2).reshape(N, N).T > 1
//
// Only the comparison with 1 leaves the kernel, so almost every pixel is decided in float32 with
// a bound on its error, and the pixels whose sum lies within the bound are summed again in FP64:
// the masks are those of an all-FP64 evaluation (which FP64's 2 FMA per clock and SM bound:
// 6250 us for 24 PDs at 96 px, 499 us this way).  A CTA owns 16 x 16 pixels of one PD and walks their z lines in
// slabs of 16 samples.  A slab's samples lie in a box of at most about 30^3 coefficients (a
// rotated cube plus the window), which is staged in shared memory as float once (each
// coefficient serves up to 64 taps; converted per tap from global memory the taps would touch
// 16 lines per warp load).  512 threads: thread t takes pixel t mod 256 and 8 of the 16 samples.
// A slab whose coefficients are all below 1e-6 only adds its bound.  Bound: the staging of the
// boxes from L2 (about 6 coefficients per sample) and the shared-memory taps of the rest.
//
// Error of one float sample against max|c| of its box, eps = 2^-24: the coefficients eps, each
// axis' four weights 4 eps each (fraction to 2^-24, three roundings), three levels of four
// fused multiply-adds 4 eps each: (1 + 48 + 12) eps; kSampleErr doubles it.  Coordinates are
// stepped in fixed point (40 fractional bits, 2^-41 per step).  The samples are added in FP64.
constexpr int kMaskTile = 16, kMaskThreads = 512, kMaskBox = 27008;     // floats: 105.5 KB
constexpr float kSampleErr = 7.3e-6f, kBoxZero = 1e-6f;

__device__ __forceinline__ double mask_sample(const double* __restrict__ C, int M,
                                              const double* __restrict__ T, int i, int j, int k) {
    double uvw[3];
    int f[3];
    double w[3][4];
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        uvw[ax] = T[3 * ax] * i + T[3 * ax + 1] * j + T[3 * ax + 2] * k + T[9 + ax];
        const double fl = floor(uvw[ax]);
        f[ax] = (int)fl;
        bspline4d(uvw[ax] - fl, w[ax]);
    }
    double acc = 0.0;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int64_t ia = min(max(kMaskPad + f[0] - 1 + a, 0), M - 1);
        double accb = 0.0;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int64_t ib = min(max(kMaskPad + f[1] - 1 + b, 0), M - 1);
            const double* row = C + (ia * M + ib) * M;
            double accc = 0.0;
#pragma unroll
            for (int c = 0; c < 4; ++c)
                accc += w[2][c] * row[min(max(kMaskPad + f[2] - 1 + c, 0), M - 1)];
            accb += w[1][b] * accc;
        }
        acc += w[0][a] * accb;
    }
    return acc;
}

__device__ __forceinline__ void bspline4f(float t, float w[4]) {
    const float u = 1.0f - t;
    const float t2 = t * t, u2 = u * u;
    w[0] = (1.0f / 6.0f) * u2 * u;
    w[3] = (1.0f / 6.0f) * t2 * t;
    w[1] = (2.0f / 3.0f) - t2 * (1.0f - 0.5f * t);
    w[2] = (2.0f / 3.0f) - u2 * (1.0f - 0.5f * u);
}

__global__ void __launch_bounds__(kMaskThreads, 2) mask_project_kernel(
        const double* __restrict__ C, int N, const double* __restrict__ xf,
        uint8_t* __restrict__ masks) {
    extern __shared__ __align__(16) float box[];   // kMaskBox floats; FP64 lines at the end
    __shared__ double half_sum[kMaskTile * kMaskTile];
    __shared__ double T[12];
    __shared__ int lo[3], dim[3], n_again;
    __shared__ float wmax[kMaskThreads / 32];
    __shared__ uint8_t again[kMaskTile * kMaskTile];
    const int M = N + 2 * kMaskPad;
    const int pd = blockIdx.y;
    const int tiles = (N + kMaskTile - 1) / kMaskTile;
    const int i0 = ((int)blockIdx.x / tiles) * kMaskTile, j0 = ((int)blockIdx.x % tiles) * kMaskTile;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int px = t & 255, part = t >> 8;
    const int i = i0 + (px >> 4), j = j0 + (px & 15);
    const bool active = i < N && j < N;
    if (t < 12) T[t] = xf[12 * pd + t];
    if (t == 0) n_again = 0;
    __syncthreads();
    // fixed-point coordinates of sample k = 0 of this thread's line, and their step along the line
    long long u0[3], du[3];
    bool in_range = true;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        const double s = 1099511627776.0;          // 2^40
        const double b = T[3 * ax] * i + T[3 * ax + 1] * j + T[9 + ax], d = T[3 * ax + 2];
        in_range = in_range && fabs(b) < 16384.0 && fabs(d) < 64.0;
        u0[ax] = in_range ? __double2ll_rn(b * s) : 0;
        du[ax] = in_range ? __double2ll_rn(d * s) : 0;
    }
    double sum = 0.0;
    float err = 1e-9f;                             // the same in every thread of the CTA
    bool staged = __syncthreads_and(in_range || !active);
    for (int k0 = 0; staged && k0 < N; k0 += kMaskTile) {
        const int kn = min(kMaskTile, N - k0);
        if (t < 3) {                               // the slab's box along axis t
            const int in = min(kMaskTile, N - i0) - 1, jn = min(kMaskTile, N - j0) - 1;
            const double a = T[3 * t], b = T[3 * t + 1], c = T[3 * t + 2];
            const double base = a * i0 + b * j0 + c * k0 + T[9 + t];
            const double dn = fmin(0.0, a * in) + fmin(0.0, b * jn) + fmin(0.0, c * (kn - 1));
            const double up = fmax(0.0, a * in) + fmax(0.0, b * jn) + fmax(0.0, c * (kn - 1));
            const int l = (int)floor(base + dn - 1e-6) - 1;
            lo[t] = l;
            dim[t] = (int)floor(base + up + 1e-6) + 2 - l + 1;
        }
        __syncthreads();                           // also: the last slab's box is done with
        const int l0 = lo[0], l1 = lo[1], l2 = lo[2];
        const int n0 = dim[0], n1 = dim[1], n2 = dim[2] | 1;       // odd row length
        if (n0 > 256 || n1 > 256 || n2 > 256 || n0 * n1 * n2 > kMaskBox) {
            staged = false;                        // not a rotation: every pixel in FP64
            break;
        }
        float mx = 0.f;
        const int rows = n0 * n1;
        for (int z = lane; z < n2; z += 32) {
            const int iz = min(max(kMaskPad + l2 + z, 0), M - 1);
#pragma unroll 8
            for (int r = warp; r < rows; r += kMaskThreads / 32) {
                const int a = r / n1, b = r - a * n1;
                const int64_t ia = min(max(kMaskPad + l0 + a, 0), M - 1);
                const int64_t ib = min(max(kMaskPad + l1 + b, 0), M - 1);
                const float v = (float)C[(ia * M + ib) * M + iz];
                box[r * n2 + z] = v;
                mx = v == v ? fmaxf(mx, fabsf(v)) : __int_as_float(0x7f800000);
            }
        }
        mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx)));
        if (lane == 0) wmax[warp] = mx;
        __syncthreads();
        mx = wmax[0];
#pragma unroll
        for (int w = 1; w < kMaskThreads / 32; ++w) mx = fmaxf(mx, wmax[w]);
        if (mx < kBoxZero) {
            err += (float)kn * mx;
            continue;
        }
        err += (float)kn * kSampleErr * mx;
        const int ka = k0 + 8 * part, kb = min(ka + 8, k0 + kn);
        if (active) {
            long long x = u0[0] + ka * du[0], y = u0[1] + ka * du[1], z = u0[2] + ka * du[2];
#pragma unroll 1
            for (int k = ka; k < kb; ++k) {
                float wx[4], wy[4], wz[4];
                const float q = 2.3283064365386963e-10f;            // 2^-32
                bspline4f((float)(uint32_t)(x >> 8) * q, wx);
                bspline4f((float)(uint32_t)(y >> 8) * q, wy);
                bspline4f((float)(uint32_t)(z >> 8) * q, wz);
                // inside the box up to the rounding of the coordinates; clamped all the same
                const int a0 = min(max((int)(x >> 40) - 1 - l0, 0), n0 - 4);
                const int b0 = min(max((int)(y >> 40) - 1 - l1, 0), n1 - 4);
                const int c0 = min(max((int)(z >> 40) - 1 - l2, 0), n2 - 4);
                float acc = 0.f;
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    float accb = 0.f;
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        const float* row = box + ((a0 + a) * n1 + b0 + b) * n2 + c0;
                        float accc = wz[0] * row[0];
                        accc = fmaf(wz[1], row[1], accc);
                        accc = fmaf(wz[2], row[2], accc);
                        accc = fmaf(wz[3], row[3], accc);
                        accb = fmaf(wy[b], accc, accb);
                    }
                    acc = fmaf(wx[a], accb, acc);
                }
                sum += (double)acc;
                x += du[0];
                y += du[1];
                z += du[2];
            }
        }
    }
    if (part == 1) half_sum[px] = sum;
    __syncthreads();
    if (part == 0 && active) {
        sum += half_sum[px];
        const bool sure = staged && fabs(sum - 1.0) > (double)err;  // false for NaN sums and bounds
        if (sure)
            masks[(int64_t)pd * N * N + (int64_t)j * N + i] = sum > 1.0 ? 1 : 0;
        else
            again[atomicAdd(&n_again, 1)] = (uint8_t)px;
    }
    __syncthreads();
    // the undecided pixels: a warp per pixel, a lane per sample, the sum in order of k
    static_assert(kMaskThreads / 32 * kMaxSmemN * sizeof(double) <= kMaskBox * sizeof(float), "");
    double* line = reinterpret_cast<double*>(box) + warp * kMaxSmemN;
    for (int q = warp; q < n_again; q += kMaskThreads / 32) {
        const int p = again[q], pi = i0 + (p >> 4), pj = j0 + (p & 15);
        for (int k = lane; k < N; k += 32) line[k] = mask_sample(C, M, T, pi, pj, k);
        __syncwarp();
        if (lane == 0) {
            double s = 0.0;
            for (int k = 0; k < N; ++k) s += line[k];
            masks[(int64_t)pd * N * N + (int64_t)pj * N + pi] = s > 1.0 ? 1 : 0;
        }
        __syncwarp();
    }
}

// dst[img] = src[img] * mask of the image's PD (in place when dst == src)
__global__ void apply_pd_mask_kernel(const float* __restrict__ src, float* __restrict__ dst,
                                     const uint8_t* __restrict__ masks,
                                     const int32_t* __restrict__ img_pd, int NN) {
    const int64_t img = blockIdx.y;
    const uint8_t* m = masks + (int64_t)img_pd[img] * NN;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < NN; p += gridDim.x * blockDim.x)
        dst[img * NN + p] = m[p] ? src[img * NN + p] : 0.0f;
}

}  // namespace

namespace kern {
int apply_pd_mask(const mem_plan& P, const float* src, float* dst, const uint8_t* masks,
                  const int32_t* img_pd, cudaStream_t s) {
    if (P.n_images == 0) return MEM_OK;
    const int NN = P.N * P.N;
    dim3 grid((unsigned)std::min(64, (NN + 255) / 256), (unsigned)P.n_images);
    apply_pd_mask_kernel<<<grid, 256, 0, s>>>(src, dst, masks, img_pd, NN);
    MEM_LAUNCH_CHECK();
    return MEM_OK;
}
}  // namespace kern
}  // namespace mem

using namespace mem;

extern "C" {

int mem_mask_coefficients_size(int32_t N, size_t* bytes) {
    if (!bytes || N < 1 || N > kMaxSmemN) return MEM_ERR_INVALID;
    const size_t M = (size_t)N + 2 * kMaskPad;
    *bytes = M * M * M * sizeof(double);
    return MEM_OK;
}

int mem_mask_prepare(const float* volume, int32_t N, double* coeffs, void* stream) {
    if (!volume || !coeffs || N < 2) return MEM_ERR_INVALID;
    if (N > kMaxSmemN) return MEM_ERR_UNSUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
    const int M = N + 2 * kMaskPad;
    mask_pad_kernel<<<1024, 256, 0, s>>>(volume, N, coeffs);
    MEM_LAUNCH_CHECK();
    const unsigned nb = (unsigned)(((int64_t)M * M + 127) / 128);
    for (int axis = 0; axis < 3; ++axis) {
        mask_prefilter_kernel<<<nb, 128, 0, s>>>(coeffs, M, axis);
        MEM_LAUNCH_CHECK();
    }
    return MEM_OK;
}

int mem_mask_project(const double* coeffs, int32_t N, int32_t n_pd, const double* transforms,
                     uint8_t* masks, void* stream) {
    if (!coeffs || !transforms || !masks || N < 2 || n_pd < 0) return MEM_ERR_INVALID;
    if (N > kMaxSmemN) return MEM_ERR_UNSUPPORTED;
    if (n_pd == 0) return MEM_OK;
    const int tiles = (N + kMaskTile - 1) / kMaskTile;
    constexpr size_t smem = kMaskBox * sizeof(float);
    MEM_CUDA_TRY(cudaFuncSetAttribute(mask_project_kernel,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    dim3 grid((unsigned)(tiles * tiles), (unsigned)n_pd);
    mask_project_kernel<<<grid, kMaskThreads, smem, (cudaStream_t)stream>>>(coeffs, N, transforms,
                                                                            masks);
    MEM_LAUNCH_CHECK();
    return MEM_OK;
}

}  // extern "C"
