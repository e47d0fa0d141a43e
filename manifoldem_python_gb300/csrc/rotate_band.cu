// The two periodic cubic B-spline rotations of rotatefill.op (modules/rotatefill.py:21-41,
// called at modules/getDistanceCTF_local_Conj9combinedS2.py:328-330) for boxes whose
// coefficient image does not fit one CTA's shared memory (64 <= N <= 512).
//
// One launch per rotation, one CTA per image and band of h consecutive layout rows:
//   1. the prefilter along layout columns for the band's rows and the 3 below them (the 4x4
//      window), straight from the input image in global memory: the recursions start kWarm rows
//      outside (periodic; z1^20 = 4e-12 of a state is left out, where the float transforms that
//      the image comes from round at 1e-7 of its largest value), so a band needs no other
//      band's coefficients and no scratch; lanes on consecutive columns, segments of up to 32
//      rows in registers;
//   2. the prefilter along each of the band's rows in shared memory, and the 3-column halo;
//   3. every output sample whose window starts in the band: along an output row the window's
//      first layout row is linear in the column, so the samples in the band are up to three
//      intervals of columns (the band and its periodic copies).  A warp owns every 16th pair of
//      output rows; its lanes find the intervals of one row each, then walk the pairs' intervals
//      together, 32 columns of both rows (paired FP32): stores are coalesced and few lanes idle.
// The first rotation reads the low-passed image in its storage orientation (transposed), so its
// layout rows are reference columns: it samples at (Y, X) and filters the reference rows first,
// as the other rotation kernels do; its result goes to the image's spectrum slot (free at this
// point) in the reference orientation, where the second rotation reads it.
//
// Bound by issue slots, then shared-memory wavefronts (16 tap loads per sample, about two-way
// conflicts; one 5x5 window for two samples, rot::sample_pair, has fewer loads but more
// instructions and took 1016 us).  Three bands of 84 rows at 250 px, two CTAs of 512 threads per
// SM.  1198 images of 250 px: 961 us; 1032 with the paired rows 16 apart (coordinates, column
// counters and bounds of their own); 1453 with one CTA per image working through the bands of
// both rotations, which was bound by its barriers (one CTA per SM, the column coefficients
// through global scratch) and by the sampling loops' idle lanes.
#include <algorithm>
#include <cmath>

#include "mem_internal.cuh"
#include "rotate_fixed.cuh"

namespace mem {
namespace {

using rot::kZ1;
using rot::RotConst;

constexpr int kBandThreads = 512, kBandWarps = kBandThreads / 32;
constexpr int kBandSeg = 32;                  // prefilter segment held in registers
constexpr int kWarm = 20;                     // rows before and after a band in the column pass
constexpr int kMaxBandN = 512;                // a lane per output row of a warp: 16 x 32

struct BandShape {
    int N, P1, Pm1;                           // row strides = 1 and -1 mod 32
    int H0, nb;                               // rows per band, bands
    int cseg;                                 // column pass: segments of kBandSeg rows
    int rseg;                                 // row pass: segments, the last one shorter
    float zrlast;                             // z1^(length of the last row segment)
};

__device__ __forceinline__ int wrap_n(int i, int N) {      // i in [-N, 2N) -> [0, N)
    i += (i < 0) ? N : 0;
    return i - ((i >= N) ? N : 0);
}

// The phases of one segment's prefilter in registers: the end state of the causal recursion
// from zero; the causal recursion from state c and the anticausal end state from zero; the
// anticausal recursion from state c.  FULL: kBandSeg samples, else len of them.
template <bool FULL>
__device__ __forceinline__ float seg_end(const float* v, int len) {
    float e = 0.f;
#pragma unroll
    for (int k = 0; k < kBandSeg; ++k)
        if (FULL || k < len) e = fmaf(kZ1, e, v[k]);
    return e;
}
template <bool FULL>
__device__ __forceinline__ float seg_causal(float* v, int len, float c) {
#pragma unroll
    for (int k = 0; k < kBandSeg; ++k)
        if (FULL || k < len) {
            c = fmaf(kZ1, c, v[k]);
            v[k] = c;
        }
    float e = 0.f;
#pragma unroll
    for (int k = kBandSeg - 1; k >= 0; --k)
        if (FULL || k < len) e = fmaf(kZ1, e, v[k]);
    return e;
}
// sample k goes to x[k]
template <bool FULL>
__device__ __forceinline__ void seg_anticausal(const float* v, int len, float c, float* x) {
    constexpr float gain = -6.0f * kZ1;
#pragma unroll
    for (int k = kBandSeg - 1; k >= 0; --k)
        if (FULL || k < len) {
            c = fmaf(kZ1, c, v[k]);
            x[k] = gain * c;
        }
}

// Two output samples a, b from the band with paired FP32 instructions: fixed-point layout
// coordinates (U, V) and the first coefficient of each window
__device__ __forceinline__ float2 sample_band2(const float* a, const float* b, int P, int64_t Ua,
                                               int64_t Va, int64_t Ub, int64_t Vb) {
    const float2 k32 = make_float2(2.3283064365386963e-10f, 2.3283064365386963e-10f);
    const float2 tu = __fmul2_rn(make_float2((float)(uint32_t)(Ua & 0xffffffffll),
                                             (float)(uint32_t)(Ub & 0xffffffffll)), k32);
    const float2 tv = __fmul2_rn(make_float2((float)(uint32_t)(Va & 0xffffffffll),
                                             (float)(uint32_t)(Vb & 0xffffffffll)), k32);
    float2 wu[4], wv[4];
    rot::bspline_w2(tu, wu);
    rot::bspline_w2(tv, wv);
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float2 v = __fmul2_rn(wv[0], make_float2(a[i * P], b[i * P]));
        v = __ffma2_rn(wv[1], make_float2(a[i * P + 1], b[i * P + 1]), v);
        v = __ffma2_rn(wv[2], make_float2(a[i * P + 2], b[i * P + 2]), v);
        v = __ffma2_rn(wv[3], make_float2(a[i * P + 3], b[i * P + 3]), v);
        acc = __ffma2_rn(wu[i], v, acc);
    }
    return acc;
}

// TRANS: the first rotation (input transposed and masked on load, see above)
template <bool TRANS>
__global__ void __launch_bounds__(kBandThreads, 2) rotate_band_kernel(
        const float* __restrict__ in, int64_t in_stride, float* __restrict__ out,
        int64_t out_stride, const RotConst* __restrict__ rotc, const BandShape B) {
    extern __shared__ float sm[];
    float* carry_c = sm;                          // causal / anticausal segment end states
    float* carry_a = sm + kBandThreads;
    float* s = sm + 2 * kBandThreads;             // (H0 + 3) x P band
    const int N = B.N, t = threadIdx.x;
    const int64_t img = blockIdx.x / B.nb;
    const int b0 = (int)(blockIdx.x % B.nb) * B.H0;
    const int h = min(B.H0, N - b0), rows = h + 3;
    const RotConst Q = rotc[2 * img + (TRANS ? 0 : 1)];
    // A warp's lanes sample along an output row, a layout step of (rc, rs) (TRANS) or (rs, rc)
    // per lane; tap (rho, iv) sits in bank (rho P + iv) mod 32, so P = 1 mod 32 keeps the bank
    // index monotone across the lanes when the two components have one sign and P = -1 mod 32
    // when they have opposite signs (about two wavefronts per tap instruction).
    const int P = (Q.rc > 0) == (Q.rs > 0) ? B.P1 : B.Pm1;
    const float* src = in + img * in_stride;
    constexpr float zseg = rot::z1_pow<kBandSeg>();
    // 1. layout columns: line v, sample i = layout row b0 - kWarm + i, cseg whole segments (the
    // rows after the band's last warm the anticausal recursion up)
    {
        const int lpr = 32 * (kBandThreads / (32 * B.cseg));
        const int lw = t % lpr, g = t / lpr;
        const int i0 = g * kBandSeg - kWarm;                   // first row, counted from b0
        const int u0 = wrap_n(b0 + i0, N);
        const bool wraps = u0 + kBandSeg > N;                  // the same in a whole warp
        for (int l0 = 0; l0 < N; l0 += lpr) {
            const int line = l0 + lw;
            const bool on = g < B.cseg && line < N;
            float v[kBandSeg];
            if (on) {
                const float* p = src + u0 * N + line;
                if (!wraps) {
#pragma unroll
                    for (int k = 0; k < kBandSeg; ++k, p += N) v[k] = __ldg(p);
                } else {
                    int u = u0;
#pragma unroll
                    for (int k = 0; k < kBandSeg; ++k) {
                        v[k] = __ldg(p);
                        const bool end = ++u == N;
                        u = end ? 0 : u;
                        p += end ? N - N * N : N;
                    }
                }
                if (TRANS) {
                    // mask_ref(line, u): (line - N/2 + 1)^2 + (u - N/2)^2 < (N/2)^2, exact in float
                    const float hf = 0.5f * (float)N, x = (float)line - hf + 1.0f;
                    const float d = hf * hf - x * x;
                    float y = (float)u0 - hf;
#pragma unroll
                    for (int k = 0; k < kBandSeg; ++k) {
                        v[k] = y * y < d ? v[k] : 0.f * v[k];
                        y += 1.0f;
                        if (wraps && y >= hf) y -= (float)N;
                    }
                }
                carry_c[g * lpr + lw] = seg_end<true>(v, kBandSeg);
            }
            __syncthreads();
            if (on) {
                float c = g > 0 ? carry_c[(g - 1) * lpr + lw] : 0.f;
                if (g > 1) c = fmaf(zseg, carry_c[(g - 2) * lpr + lw], c);
                carry_a[g * lpr + lw] = seg_causal<true>(v, kBandSeg, c);
            }
            __syncthreads();
            if (on) {
                float c = g + 1 < B.cseg ? carry_a[(g + 1) * lpr + lw] : 0.f;
                if (g + 2 < B.cseg) c = fmaf(zseg, carry_a[(g + 2) * lpr + lw], c);
                constexpr float gain = -6.0f * kZ1;
                float* x = s + (i0 + kBandSeg - 1) * P + line;
#pragma unroll
                for (int k = kBandSeg - 1; k >= 0; --k, x -= P) {
                    c = fmaf(kZ1, c, v[k]);
                    if ((unsigned)(i0 + k) < (unsigned)rows) *x = gain * c;
                }
            }
        }
        __syncthreads();
    }
    // 2. layout rows, complete lines, in place (lanes on consecutive rows: the row stride is +-1
    // mod 32, so a warp's accesses fall in 32 banks)
    {
        const int lpr = 32 * (kBandThreads / (32 * B.rseg));
        const int lw = t % lpr, g = t / lpr;
        const int k0 = g * kBandSeg, len = min(kBandSeg, N - k0);
        const bool full = len == kBandSeg;                     // the same in a whole warp
        const int g1 = g == 0 ? B.rseg - 1 : g - 1, g2 = g1 == 0 ? B.rseg - 1 : g1 - 1;
        const int h1 = g == B.rseg - 1 ? 0 : g + 1, h2 = h1 == B.rseg - 1 ? 0 : h1 + 1;
        const float zg1 = g1 == B.rseg - 1 ? B.zrlast : zseg;
        const float zh1 = h1 == B.rseg - 1 ? B.zrlast : zseg;
        for (int l0 = 0; l0 < rows; l0 += lpr) {
            const int line = l0 + lw;
            const bool on = g < B.rseg && line < rows;
            float* x = s + line * P + k0;
            float v[kBandSeg];
            if (on) {
#pragma unroll
                for (int k = 0; k < kBandSeg; ++k)
                    if (full || k < len) v[k] = x[k];
                carry_c[g * lpr + lw] = full ? seg_end<true>(v, len) : seg_end<false>(v, len);
            }
            __syncthreads();
            if (on) {
                const float c = fmaf(zg1, carry_c[g2 * lpr + lw], carry_c[g1 * lpr + lw]);
                carry_a[g * lpr + lw] =
                        full ? seg_causal<true>(v, len, c) : seg_causal<false>(v, len, c);
            }
            __syncthreads();
            if (on) {
                const float c = fmaf(zh1, carry_a[h2 * lpr + lw], carry_a[h1 * lpr + lw]);
                if (full)
                    seg_anticausal<true>(v, len, c, x);
                else
                    seg_anticausal<false>(v, len, c, x);
            }
        }
        __syncthreads();
        for (int p = t; p < rows * 3; p += kBandThreads) {
            const int rho = p / 3, j = p - rho * 3;
            s[rho * P + N + j] = s[rho * P + j];
        }
        __syncthreads();
    }
    // 3. the samples.  Lane l finds the column intervals of row l % 2 of the warp's pair l / 2
    constexpr int64_t kOne = 1ll << 32;
    float* dst = out + img * out_stride;
    const int warp = t >> 5, lane = t & 31;
    const int64_t dXr = Q.rc, dYr = -Q.rs, dXc = Q.rs, dYc = Q.rc;     // steps per row, column
    const int64_t dUr = TRANS ? dYr : dXr, dUc = TRANS ? dYc : dXc;
    const int64_t dVr = TRANS ? dXr : dYr, dVc = TRANS ? dXc : dYc;
    const int64_t U00 = (TRANS ? Q.by : Q.bx) - kOne, V00 = (TRANS ? Q.bx : Q.by) - kOne;
    int lo[3], hi[3];
    {
        const int r = 2 * warp + 2 * kBandWarps * (lane >> 1) + (lane & 1);
        const int64_t Ur = U00 + (int64_t)r * dUr;
        const float inv = 1.0f / (float)dUc;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int base = b0 + (k - 1) * N;
            lo[k] = 0;
            hi[k] = N;
            if (dUc != 0) {
                // The distances to the band are formed in fixed point, so that the bounds are good to
                // 2^-22 of themselves at any slope (from coordinates rounded to float they were
                // many columns off where a row is almost level, near multiples of 90 degrees).
                // Widened by a column each way; every sample checks its row
                const float ea = (float)((int64_t)base * kOne - Ur) * inv;
                const float eb = (float)((int64_t)(base + h) * kOne - Ur) * inv;
                const float a = fminf(fmaxf(fminf(ea, eb), -2.f), (float)N + 2.f);
                const float b = fminf(fmaxf(fmaxf(ea, eb), -2.f), (float)N + 2.f);
                lo[k] = max(0, (int)floorf(a) - 1);
                hi[k] = min(N, (int)ceilf(b) + 1);
            } else {
                const int f = (int)(Ur >> 32) - base;                  // a constant row
                if (f < 0 || f >= h) hi[k] = 0;
            }
            if (r >= N) hi[k] = 0;
            // both rows of the pair: the even lane's interval covers the two
            if (lo[k] >= hi[k]) {
                lo[k] = N;
                hi[k] = 0;
            }
            lo[k] = min(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], 1));
            hi[k] = max(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], 1));
        }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int base = b0 + (k - 1) * N;
        unsigned todo = __ballot_sync(0xffffffffu, lo[k] < hi[k]) & 0x55555555u;
        while (todo) {                         // two rows r, r + 1 at a time
            const int q = __ffs(todo) - 1;
            todo &= todo - 1;
            int c = __shfl_sync(0xffffffffu, lo[k], q);
            int left = __shfl_sync(0xffffffffu, hi[k], q) - c;     // the same in every lane
            const int r = 2 * warp + kBandWarps * q;
            const bool two = r + 1 < N;
            int64_t U = U00 + (int64_t)r * dUr + (int64_t)(c + lane) * dUc;
            int64_t V = V00 + (int64_t)r * dVr + (int64_t)(c + lane) * dVc;
            float* d = dst + r * N + c + lane;
#pragma unroll 1
            for (; left > 0; left -= 32, d += 32, U += 32 * dUc, V += 32 * dVc) {
                const int64_t Ub = U + dUr, Vb = V + dVr;
                const bool in_a = lane < left && (unsigned)((int)(U >> 32) - base) < (unsigned)h;
                const bool in_b = two && lane < left &&
                                  (unsigned)((int)(Ub >> 32) - base) < (unsigned)h;
                // a valid address for an unused half
                const float* a = s, *b = s;
                if (in_a) a += ((int)(U >> 32) - base) * P + wrap_n((int)(V >> 32), N);
                if (in_b) b += ((int)(Ub >> 32) - base) * P + wrap_n((int)(Vb >> 32), N);
                const float2 v = sample_band2(a, b, P, U, V, Ub, Vb);
                if (in_a) d[0] = v.x;
                if (in_b) d[N] = v.y;
            }
        }
    }
}

}  // namespace

namespace kern {

bool rotate_band_supported(int N) { return N >= 64 && N <= kMaxBandN; }

int rotate_band(const mem_plan& P, float* xbuf, float2* spec, float* img_out, const void* rotc,
                cudaStream_t s) {
    if (P.n_images == 0) return MEM_OK;
    const int N = P.N;
    if (!rotate_band_supported(N) || P.Kc * 2 < (int64_t)N * N) return MEM_ERR_UNSUPPORTED;
    BandShape B;
    B.N = N;
    // row strides >= N + 3 (the 3-column halo)
    B.P1 = ((N + 3 + 30) / 32) * 32 + 1;
    B.Pm1 = ((N + 3 + 32) / 32) * 32 - 1;
    const int Pst = std::max(B.P1, B.Pm1);
    // the fewest bands with two CTAs per SM (MEM_ROT_BANDS asks for more)
    const size_t budget = 110 * 1024 - 2 * kBandThreads * sizeof(float);
    B.nb = 1;
    while ((size_t)((N + B.nb - 1) / B.nb + 3) * Pst * sizeof(float) > budget) ++B.nb;
    if (const char* e = std::getenv("MEM_ROT_BANDS")) B.nb = std::max(B.nb, std::atoi(e));
    B.H0 = (N + B.nb - 1) / B.nb;
    B.nb = (N + B.H0 - 1) / B.H0;
    B.cseg = (B.H0 + 3 + 2 * kWarm + kBandSeg - 1) / kBandSeg;
    B.rseg = (N + kBandSeg - 1) / kBandSeg;
    B.zrlast = (float)std::pow((double)kZ1, (double)(N - kBandSeg * (B.rseg - 1)));
    const size_t smem = (2 * kBandThreads + (size_t)(B.H0 + 3) * Pst) * sizeof(float);
    if (smem > 227 * 1024 || B.cseg > kBandWarps || B.rseg > kBandWarps)
        return MEM_ERR_UNSUPPORTED;
    const RotConst* rc = static_cast<const RotConst*>(rotc);
    float* first = reinterpret_cast<float*>(spec);         // the first rotation's results
    const int64_t NN = (int64_t)N * N;
    const unsigned grid = (unsigned)(P.n_images * B.nb);
    MEM_CUDA_TRY(cudaFuncSetAttribute(rotate_band_kernel<true>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    MEM_CUDA_TRY(cudaFuncSetAttribute(rotate_band_kernel<false>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    rotate_band_kernel<true><<<grid, kBandThreads, smem, s>>>(xbuf, NN, first, 2 * P.Kc, rc, B);
    MEM_LAUNCH_CHECK();
    rotate_band_kernel<false><<<grid, kBandThreads, smem, s>>>(first, 2 * P.Kc, img_out, NN, rc, B);
    MEM_LAUNCH_CHECK();
    return MEM_OK;
}

}  // namespace kern
}  // namespace mem
