// Diffusion-map embedding of one PD's distance matrix on the GPU: the dense-matrix work of
// DMembeddingII.op (reference modules/DMembeddingII.py:86-185) with fergusonE.op
// (modules/fergusonE.py:33-58) and slaplacianonFly.op (modules/slaplacianonFly.py:42-81).
//
//   1. symmetrised squared distances (DMembeddingII.py:112-139, construct_matrix0/1 :72-84):
//        s_ij = sqrt(D_ji) if j is among the k nearest of point i (column i of D, the point itself
//               first), D_ji >= 1e-6 and j != i; else 0
//        Y_ij = s_ij^2 + s_ji^2 - s_ij s_ji
//      entry (i, j) is an edge if Y_ij != 0 or if j is a listed neighbour of i with D_ji < 1e-6
//      (or j = i); non-edges are stored as -1;
//   2. bandwidth sweep (fergusonE.py:36-44): for every log eps,
//        sum over edges of exp(-Y/(2 eps)) for the terms with Y/(2 eps) < thr;
//   3. normalised kernel (slaplacianonFly.py:55-80, alpha = 1):
//        W = exp(-Y/sigma^2) on edges; W'_ij = W_ij/(d_i d_j), d = column sums of W;
//        L_ij = W'_ij/(e_i e_j), e = sqrt(column sums of W'); L = |L + L^T|/2.
// The eigen-decomposition of L, the tanh fit of the sweep and the neighbour lists (a sort per
// column) stay with the caller.  The sweep evaluates exp in float32 and sums in float64 per
// block; everything else is float64.
#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "mem_internal.cuh"

namespace mem {
namespace {

constexpr double kZeroDist = 1e-6;
constexpr int kTile = 32;

// 1. Y from D (row-major n x n); listed = nullptr: every entry is a listed neighbour (k = n).
// s_ij^2 and s_ji^2 are D_ji and D_ij themselves, so square roots are left for the product of two
// different entries; where they are equal, as in every D of the distance stage, Y_ij = D_ij.
// One CTA per unordered pair of 32 x 32 tiles (bi, bj), bi <= bj: it reads both tiles once and
// writes both.  Bound by memory for a symmetric D: n = 3000 takes 36 us; 152 with a square root
// per pair, where FP64 (2 FMA per clock and SM) bounded it, and 387 with four.
// Comparisons are on the bit patterns (positive doubles sort as integers), off the FP64 unit.
constexpr long long kInfBits = 0x7ff0000000000000ll;
// kZeroDist <= d <= inf
__device__ __forceinline__ bool dm_far(double d) {
    // unsigned: a negative d's pattern lies above all positive ones
    const unsigned long long zero = (unsigned long long)__double_as_longlong(kZeroDist);
    return (unsigned long long)__double_as_longlong(d) - zero <=
           (unsigned long long)kInfBits - zero;
}
__device__ __forceinline__ bool dm_nan(double d) {
    return (__double_as_longlong(d) & 0x7fffffffffffffffll) > kInfBits;
}
// Y of a pair with at least one of u1 (s_ij = sqrt(D_ji) counts) and u2 (s_ji); NaN where an
// infinite distance counts
__device__ __forceinline__ double dm_pair_value(double dij, double dji, bool u1, bool u2) {
    const long long a = __double_as_longlong(dij), b = __double_as_longlong(dji);
    if (u1 && u2 && a != b) return dji + dij - sqrt(dji) * sqrt(dij);
    const long long v = u1 ? b : a;
    return __longlong_as_double(v == kInfBits ? 0x7ff8000000000000ll : v);
}

__global__ void __launch_bounds__(256) dm_sym_kernel(
        const double* __restrict__ D, int64_t n, const uint8_t* __restrict__ listed,
        double* __restrict__ Y) {
    __shared__ double tY[kTile][kTile + 1];      // D block (bj, bi), then its Y block
    __shared__ uint8_t tL[kTile][kTile + 1];
    const int64_t bi = (int64_t)blockIdx.y * kTile, bj = (int64_t)blockIdx.x * kTile;
    if (bj < bi) return;
    const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8 threads
    double dij[kTile / 8];
    uint8_t lij[kTile / 8];
#pragma unroll
    for (int q = 0; q < kTile / 8; ++q) {
        const int r = ty + 8 * q;
        const int64_t gi = bj + r, gj = bi + tx;   // D[bj + r][bi + tx]
        const bool in = gi < n && gj < n;
        tY[r][tx] = in ? D[gi * n + gj] : 0.0;
        tL[r][tx] = in ? (listed ? listed[gi * n + gj] : (uint8_t)1) : (uint8_t)0;
        const int64_t i = bi + r, j = bj + tx;
        const bool in2 = i < n && j < n;
        dij[q] = in2 ? D[i * n + j] : 0.0;
        lij[q] = in2 ? (listed ? listed[i * n + j] : (uint8_t)1) : (uint8_t)0;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kTile / 8; ++q) {
        const int r = ty + 8 * q;
        const int64_t i = bi + r, j = bj + tx;
        if (i >= n || j >= n) continue;
        const double dji = tY[tx][r];                          // D_ji
        const bool l1 = lij[q] != 0, l2 = tL[tx][r] != 0;      // j listed for i, i listed for j
        const bool far1 = i != j && dm_far(dji), far2 = i != j && dm_far(dij[q]);
        const bool u1 = l1 && far1, u2 = l2 && far2;           // s_ij, s_ji are not 0
        const double y = u1 || u2 ? dm_pair_value(dij[q], dji, u1, u2) : -1.0;
        // a pair of s = 0 is an edge where a listed distance is below kZeroDist
        const bool z1 = l1 && (i == j || !(far1 || dm_nan(dji)));
        const bool z2 = l2 && (i == j || !(far2 || dm_nan(dij[q])));
        Y[i * n + j] = u1 || u2 || !z1 ? y : 0.0;
        // this thread alone reads and writes element (tx, r) of the shared tile
        tY[tx][r] = u1 || u2 || !z2 ? y : 0.0;
    }
    if (bi == bj) return;                          // the diagonal tile is complete
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kTile / 8; ++q) {
        const int r = ty + 8 * q;
        if (bj + r < n && bi + tx < n) Y[(bj + r) * n + bi + tx] = tY[r][tx];
    }
}

// 2. Sweep.  Every thread holds kPer entries of Y and would walk all the log eps values, but for
// most of them a warp's 256 entries are all beyond the threshold (a term is 0, except a zero
// distance's 1) or all so close that exp rounds to 1: a term lies strictly between only while
// d = Y/(2 eps) runs from the threshold down to 2^-26, about 20 of the sweep's 300 in ln eps.  So
// per chunk of entries the CTA first classifies every log eps from each warp's smallest positive
// and largest Y, adds the exact counts where all its warps are trivial, and evaluates the listed
// rest.  Float sums per warp and their order are those of a full evaluation; a block keeps the
// FP64 sums of all its chunks in shared memory and adds them to global memory once.
// NT: 256 threads (2048 entries per chunk), or 64 while there are fewer than two such chunks per
// SM, so that n = 300 runs on 152 SMs instead of 44.
constexpr int kPer = 8, kMaxEps = 2048;
constexpr int kSweepList = 256;                   // listed scales evaluated between two barriers
constexpr float kExpOne = 1.4901161193847656e-8f; // 2^-26: exp2f(-d) = 1 for 0 <= d <= 2^-26

// exp2(-d); PLAIN, for 0 <= d < 126 (normal results): the ex2.approx instruction alone.  With one
// comparison per term and non-edges folded into +inf this takes the sweep's inner loop, which the
// issue slots bound, from 600 to 296 us at n = 3000 and from 45 to 28 us at n = 300.
template <bool PLAIN>
__device__ __forceinline__ float exp2_neg(float d) {
    if (!PLAIN) return exp2f(-d);
    float v;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(v) : "f"(-d));
    return v;
}

template <int NT>
__global__ void __launch_bounds__(NT) dm_sweep_kernel(
        const double* __restrict__ Y, int64_t total, const float* __restrict__ scale,
        int n_eps, float thr, int aligned, double* __restrict__ sums) {
    constexpr int NW = NT / 32;
    __shared__ double part[kMaxEps];
    __shared__ uint16_t list[kMaxEps];
    __shared__ float wsum[kSweepList][NW];
    __shared__ float wmin[NW], wmax[NW];
    __shared__ int wzero[NW], wedge[NW], n_list, n_odd;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (int e = t; e < n_eps; e += NT) part[e] = 0.0;
    const float tl = thr * 1.4426950408889634f;   // the threshold on d = Y/(2 eps), base 2
    constexpr int64_t per_block = (int64_t)NT * kPer;
    const int64_t chunks = (total + per_block - 1) / per_block;
    for (int64_t ch = blockIdx.x; ch < chunks; ch += gridDim.x) {
        float y[kPer];
        const int64_t base = ch * per_block + (int64_t)t * kPer;
        if (aligned && base + kPer <= total) {    // Y on a 16-byte boundary
            const double2* p = reinterpret_cast<const double2*>(Y + base);
#pragma unroll
            for (int u = 0; u < kPer / 2; ++u) {
                const double2 v = p[u];
                y[2 * u] = (float)v.x;
                y[2 * u + 1] = (float)v.y;
            }
        } else {
#pragma unroll
            for (int u = 0; u < kPer; ++u)
                y[u] = base + u < total ? (float)Y[base + u] : -1.0f;    // -1: not an edge
        }
        float lo = __int_as_float(0x7f800000), hi = 0.f;
        int zero = 0, edge = 0;
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            if (y[u] > 0.f) {
                lo = fminf(lo, y[u]);
                hi = fmaxf(hi, y[u]);
            }
            zero += y[u] == 0.f;
            edge += y[u] >= 0.f;
        }
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        zero = __reduce_add_sync(0xffffffffu, zero);
        edge = __reduce_add_sync(0xffffffffu, edge);
        __syncthreads();                          // the last chunk's lists and sums are done with
        if (lane == 0) {
            wmin[warp] = lo;
            wmax[warp] = hi;
            wzero[warp] = zero;
            wedge[warp] = edge;
        }
        if (t == 0) n_list = n_odd = 0;
#pragma unroll
        for (int u = 0; u < kPer; ++u)
            if (!(y[u] >= 0.f)) y[u] = __int_as_float(0x7f800000);
        __syncthreads();
        for (int e = t; e < n_eps; e += NT) {
            const float c = scale[e];             // log2(e) / (2 eps)
            int ones = 0;
            bool todo = false;
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                const bool none = wedge[w] == wzero[w];         // no positive entry
                const float dmax = wmax[w] * c;
                if (none || wmin[w] * c >= tl)
                    ones += 0.f < tl ? wzero[w] : 0;
                else if (dmax >= 0.f && dmax <= kExpOne && dmax < tl)
                    ones += wedge[w];
                else
                    todo = true;
            }
            if (todo) {
                list[atomicAdd(&n_list, 1)] = (uint16_t)e;
                if (!(c > 0.f && c < __int_as_float(0x7f800000))) n_odd = 1;
            }
            if (!todo && ones) part[e] += (double)ones;
        }
        __syncthreads();
        const int nl = n_list;
        const bool finite = n_odd == 0;
        for (int l0 = 0; l0 < nl; l0 += kSweepList) {
            const int l1 = min(nl, l0 + kSweepList);
            // A term is exp2(-d log2(e)); beyond the threshold, and for a non-edge (kept as +inf
            // here), 0.  scale is +inf for the smallest eps (beyond float range): zero-distance
            // edges still give exp(0) = 1 there, all others are beyond the threshold.
            auto evaluate = [&](auto plain) {
#pragma unroll 2
                for (int l = l0; l < l1; ++l) {
                    const float c = scale[list[l]];
                    float acc = 0.f;
#pragma unroll
                    for (int u = 0; u < kPer; ++u) {
                        const float d2 = decltype(plain)::value || y[u] != 0.f ? y[u] * c : 0.f;
                        acc += d2 < tl ? exp2_neg<decltype(plain)::value>(d2) : 0.f;
                    }
                    for (int o = 16; o > 0; o >>= 1)
                        acc += __shfl_xor_sync(0xffffffffu, acc, o);
                    if (lane == 0) wsum[l - l0][warp] = acc;
                }
            };
            // the short form needs a finite scale in the whole list and a threshold that keeps
            // the exponent out of the denormals
            if (finite && tl <= 120.f)
                evaluate(std::true_type{});
            else
                evaluate(std::false_type{});
            __syncthreads();
            for (int i = t; i < l1 - l0; i += NT) {
                double s = 0.0;
#pragma unroll
                for (int w = 0; w < NW; ++w) s += (double)wsum[i][w];
                part[list[l0 + i]] += s;
            }
            __syncthreads();
        }
    }
    __syncthreads();
    for (int e = t; e < n_eps; e += NT)
        if (part[e] != 0.0) atomicAdd(&sums[e], part[e]);
}

// 3. The normalised kernel, four launches over W (in L2 up to n = 4000):
//   a. W = exp(-Y / sigma^2) on edges, in place, tile pairs as in dm_sym_kernel: one FP64 exp
//      for both entries of a pair where Y_ij = Y_ji;
//   b. d = column sums of W;
//   c. e_j = sqrt(sum_i W_ij / (d_i d_j)), from reciprocals 1/d kept per row;
//   d. L_ij = W_ij f_i f_j with f = 1 / (d e), L = |L + L^T| / 2, tile pairs.
// A column sum is split over the rows of a 16-column slice (64 row threads, added in a fixed
// order), so that n = 300 already fills 19 SMs and n = 3000 all of them; one thread per column
// walking all rows took 2498 + 1564 us at n = 3000 (now 153 + 34 + 30) and 249 + 148 us at
// n = 300 (the whole embedding work there: 65 us now, 918 us before).
// y >= 0 by the bit pattern (-0 included, a NaN not)
__device__ __forceinline__ bool dm_edge(double y) {
    const long long v = __double_as_longlong(y);
    return v >= 0 ? v <= kInfBits : (v << 1) == 0;
}

__global__ void __launch_bounds__(256) dm_weights_kernel(double* __restrict__ W, int64_t n,
                                                         double inv_s2) {
    __shared__ double tb[kTile][kTile + 1];
    const int64_t bi = (int64_t)blockIdx.y * kTile, bj = (int64_t)blockIdx.x * kTile;
    if (bj < bi) return;
    const int tx = threadIdx.x, ty = threadIdx.y;
    double a[kTile / 8];
#pragma unroll
    for (int q = 0; q < kTile / 8; ++q) {
        const int r = ty + 8 * q;
        tb[r][tx] = (bj + r < n && bi + tx < n) ? W[(bj + r) * n + bi + tx] : -1.0;
        a[q] = (bi + r < n && bj + tx < n) ? W[(bi + r) * n + bj + tx] : -1.0;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kTile / 8; ++q) {
        const int r = ty + 8 * q;
        const double yij = a[q], yji = tb[tx][r];
        const bool same = __double_as_longlong(yij) == __double_as_longlong(yji);
        const double wij = dm_edge(yij) ? exp(-yij * inv_s2) : 0.0;
        const double wji = same ? wij : (dm_edge(yji) ? exp(-yji * inv_s2) : 0.0);
        if (bi + r < n && bj + tx < n) W[(bi + r) * n + bj + tx] = wij;
        tb[tx][r] = wji;
    }
    if (bi == bj) return;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kTile / 8; ++q) {
        const int r = ty + 8 * q;
        if (bj + r < n && bi + tx < n) W[(bj + r) * n + bi + tx] = tb[r][tx];
    }
}

// column sums of a 16-column slice: first = d (PASS 0: 1 / d to out), then e (PASS 1: out = f)
constexpr int kColW = 16, kColRows = 64;
template <int PASS>
__global__ void __launch_bounds__(kColW* kColRows) dm_colsum_kernel(
        const double* __restrict__ W, int64_t n, const double* __restrict__ rd,
        double* __restrict__ out) {
    __shared__ double part[kColRows][kColW + 1];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int64_t j = (int64_t)blockIdx.x * kColW + tx;
    double s = 0.0;
    if (j < n) {
#pragma unroll 4
        for (int64_t i = ty; i < n; i += kColRows) {
            const double w = W[i * n + j];
            s = PASS == 0 ? s + w : fma(w, rd[i], s);
        }
    }
    part[ty][tx] = s;
    __syncthreads();
    for (int h = kColRows / 2; h > 0; h >>= 1) {
        if (ty < h) part[ty][tx] += part[ty + h][tx];
        __syncthreads();
    }
    if (ty == 0 && j < n)
        out[j] = PASS == 0 ? 1.0 / part[0][tx] : rd[j] / sqrt(part[0][tx] * rd[j]);
}

// L_ij = W_ij f_i f_j, then L = |L + L^T| / 2 (tile pairs (bi, bj), (bj, bi))
__global__ void __launch_bounds__(256) dm_finish_kernel(double* __restrict__ W, int64_t n,
                                                        const double* __restrict__ f) {
    __shared__ double tb[kTile][kTile + 1];
    const int64_t bi = (int64_t)blockIdx.y * kTile, bj = (int64_t)blockIdx.x * kTile;
    if (bj < bi) return;                           // each unordered tile pair once
    const int tx = threadIdx.x, ty = threadIdx.y;
    double a[kTile / 8];
#pragma unroll
    for (int q = 0; q < kTile / 8; ++q) {
        const int r = ty + 8 * q;
        tb[r][tx] = (bj + r < n && bi + tx < n) ? W[(bj + r) * n + bi + tx] : 0.0;
        a[q] = (bi + r < n && bj + tx < n) ? W[(bi + r) * n + bj + tx] : 0.0;
    }
    __syncthreads();
    const double fj = bj + tx < n ? f[bj + tx] : 0.0;
#pragma unroll
    for (int q = 0; q < kTile / 8; ++q) {
        const int r = ty + 8 * q;
        const double fi = bi + r < n ? f[bi + r] : 0.0;
        const double v = fabs((a[q] + tb[tx][r]) * (fi * fj)) / 2.0;
        if (bi + r < n && bj + tx < n) W[(bi + r) * n + bj + tx] = v;
        tb[tx][r] = v;
    }
    if (bi == bj) return;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kTile / 8; ++q) {
        const int r = ty + 8 * q;
        if (bj + r < n && bi + tx < n) W[(bj + r) * n + bi + tx] = tb[r][tx];
    }
}

}  // namespace
}  // namespace mem

using namespace mem;

extern "C" {

int mem_dm_symmetrise(const double* D, int64_t n, const uint8_t* listed, double* Y,
                      void* stream) {
    if (!D || !Y || n < 1) return MEM_ERR_INVALID;
    const unsigned nb = (unsigned)((n + kTile - 1) / kTile);
    dm_sym_kernel<<<dim3(nb, nb), dim3(kTile, 8), 0, (cudaStream_t)stream>>>(D, n, listed, Y);
    MEM_LAUNCH_CHECK();
    return MEM_OK;
}

int mem_dm_sweep(const double* Y, int64_t n, const float* scale, int32_t n_eps, double thr,
                 double* sums, void* stream) {
    if (!Y || !scale || !sums || n < 1 || n_eps < 1 || n_eps > kMaxEps) return MEM_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    MEM_CUDA_TRY(cudaMemsetAsync(sums, 0, sizeof(double) * n_eps, s));
    const int64_t total = n * n;
    // persistent: as many CTAs as fit the SMs at most, each adding its sums to global memory once
    const int aligned = (reinterpret_cast<uintptr_t>(Y) & 15) == 0;
    const int64_t wide = (total + 256 * kPer - 1) / (256 * kPer);
    const int64_t narrow = (total + 64 * kPer - 1) / (64 * kPer);
    if (wide >= 2 * 152)
        dm_sweep_kernel<256><<<(unsigned)std::min<int64_t>(wide, 4 * 152), 256, 0, s>>>(
                Y, total, scale, n_eps, (float)thr, aligned, sums);
    else
        dm_sweep_kernel<64><<<(unsigned)std::min<int64_t>(narrow, 8 * 152), 64, 0, s>>>(
                Y, total, scale, n_eps, (float)thr, aligned, sums);
    MEM_LAUNCH_CHECK();
    return MEM_OK;
}

int mem_dm_laplacian(double* Y, int64_t n, double sigma, double* scratch, void* stream) {
    if (!Y || !scratch || n < 1 || !(sigma > 0.0)) return MEM_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    const unsigned nb = (unsigned)((n + kTile - 1) / kTile);
    const unsigned nc = (unsigned)((n + kColW - 1) / kColW);
    double *rd = scratch, *f = scratch + n;
    dm_weights_kernel<<<dim3(nb, nb), dim3(kTile, 8), 0, s>>>(Y, n, 1.0 / (sigma * sigma));
    MEM_LAUNCH_CHECK();
    dm_colsum_kernel<0><<<nc, dim3(kColW, kColRows), 0, s>>>(Y, n, nullptr, rd);
    MEM_LAUNCH_CHECK();
    dm_colsum_kernel<1><<<nc, dim3(kColW, kColRows), 0, s>>>(Y, n, rd, f);
    MEM_LAUNCH_CHECK();
    dm_finish_kernel<<<dim3(nb, nb), dim3(kTile, 8), 0, s>>>(Y, n, f);
    MEM_LAUNCH_CHECK();
    return MEM_OK;
}

}  // extern "C"
