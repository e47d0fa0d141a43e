// The image-transform kernels for N = R1 R2 (fft_mixed.cuh).  As in image_fft.cu (N = 32, 64, 128):
//   lowpass    gather + conjugate flip + background normalisation + low-pass (reference
//              modules/getDistanceCTF_local_Conj9combinedS2.py:245-293);
//   spectrum   image (times the PD's volume mask, :344) -> half-plane spectrum [N][N/2+1];
//   inverse    half-plane spectrum (times sign(C) / N^2) -> image (:375-389).
// Layout and scaling are those of a cuFFT R2C / C2R pair.  Two forms, by where an image fits:
//
// Whole (N <= 228): one image per CTA, the N x N / 2 complex buffer in shared memory; an image is
// read and written once.  Bound by the latency of its 8 (low-pass 12) shared-memory passes at the
// 12 to 20 warps that the buffer and about 100 registers per thread leave on an SM.
//
// Tiled (larger N): one image per CTA too, rows in chunks of PC pair-rows and columns in tiles of
// CT columns through a buffer of up to 108 KB, two CTAs per SM.  Between rows and columns the
// spectra go through the image's own output slot (in L2: 304 slots of 250 KB at 250 px, read back
// right after they are written).  Keeping the rows of an image in the shared memories of a
// cluster of two CTAs instead measured 1758 us for the low-pass of 1198 images of 250 px, against
// 583 us for this form: the column passes' 8-byte accesses are slow over distributed shared memory.
//
// Against cuFFT (a row pass and a column pass over HBM for every transform, the gather and the
// filter in passes of their own):
//   1000 images of 192 px:  low-pass 217 us, was 465; spectrum 108, was 150; flip 103, was 153
//   1198 images of 250 px:  low-pass 583 us, was 1240; spectrum 252, was 434; flip 289, was 451
#pragma once

#include "fft_mixed.cuh"
#include "mem_internal.cuh"
#include "rotate_whole.cuh"

namespace mem {
namespace mixed {

struct LowpassArgs {
    const float* stack;
    int64_t num_stack;
    const int64_t* sidx;
    const uint8_t* flip;
    const float* gtab;
    const float2* twid;
    float* xbuf;
    uint32_t* status;
};
struct SpectrumArgs {
    const float* images;
    const uint8_t* masks;        // null, or [n_pd][N][N]
    const int32_t* img_pd;
    const float2* twid;
    float2* spec;
};
struct InverseArgs {
    const float2* spec;
    const float2* twid;
    float* images;
    const uint64_t* qfix;
    CtfConst cc;
};

// the kernels of one box size
struct Kernels {
    int N, threads;
    bool tiled;                  // the inverse keeps pairs of floats in its output
    size_t smem;
    void (*lowpass)(LowpassArgs);
    void (*spectrum)(SpectrumArgs);
    void (*inverse)(InverseArgs);
    void (*inverse_signed)(InverseArgs);
    // rotation of whole images in shared memory (null where a coefficient image does not fit)
    void (*rotate)(float*, float*, const rot::RotConst*);
    int rot_threads;
    size_t rot_smem;
};

struct KSumM {                    // Kahan-compensated float accumulator
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float x) {
        const float y = x - c;
        const float t = s + y;
        c = (t - s) - y;
        s = t;
    }
    __device__ __forceinline__ float value() const { return s - c; }
};

// the pair-rows in shared memory
template <class Sh>
struct SmemBuf {
    float2* s;
    __device__ __forceinline__ float2& at(int p, int i) const { return s[p * Sh::S + i]; }
};

// 1 - annularMask.op(0, N/2, N, N) at (r, c): centre (N/2 - 1, N/2), radius N/2
template <int N>
__device__ __forceinline__ float background(float x, int r, int c) {
    const float h = 0.5f * (float)N;
    const float u = (float)r - h + 1.0f, v = (float)c - h;
    return (u * u + v * v < h * h) ? 0.f : x;
}

// background mean and 1/std over the image from the threads' sums (:277-281)
template <int NT>
__device__ __forceinline__ void image_stats(double a, double b, double (&red)[2][NT / 32],
                                            float (&stat)[2], int NN, float* mean, float* inv) {
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = a;
        red[1][threadIdx.x >> 5] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0, t2 = 0.0;
#pragma unroll
        for (int i = 0; i < NT / 32; ++i) {
            t += red[0][i];
            t2 += red[1][i];
        }
        const double m = t / NN;
        stat[0] = (float)m;
        stat[1] = (float)(1.0 / sqrt(fmax(t2 / NN - m * m, 0.0)));
    }
    __syncthreads();
    *mean = stat[0];
    *inv = stat[1];
}

// W[k] = exp(-2 pi i k / N), k < N, from the table k <= N/2
template <class Sh, int NT>
__device__ __forceinline__ void load_twiddles(float2* W, const float2* __restrict__ twid) {
    for (int k = threadIdx.x; k < Sh::N; k += NT) {
        const float2 v = twid[k <= Sh::H ? k : Sh::N - k];
        W[k] = k <= Sh::H ? v : make_float2(v.x, -v.y);
    }
}

// ------------------------------------------------------------------------- whole images
template <class Sh>
constexpr size_t whole_bytes() {
    return (size_t)Sh::H * Sh::S * sizeof(float2);
}
// Threads and CTAs per SM: 128 x 5 while five buffers fit, 320 x 2 while two do (the load of one
// image then overlaps the passes of another), else 384 threads alone; measured against 256 x 2,
// 256 x 3, 512 x 1, 768 x 1 (low-pass of 1000 images: 120 px 97 us, 256 x 2 the same; 150 px 137,
// 512 x 1 190; 192 px 217, 512 x 1 235; 846 of 100 px 53, 256 x 2 60)
template <class Sh>
constexpr int whole_blocks() {
    return whole_bytes<Sh>() <= 44 * 1024 ? 5 : whole_bytes<Sh>() <= 108 * 1024 ? 2 : 1;
}
template <class Sh>
constexpr int whole_threads() {
    return whole_blocks<Sh>() == 5 ? 128 : whole_blocks<Sh>() == 2 ? 320 : 384;
}

template <class Sh, int NT>
__device__ __forceinline__ void rows_to_columns(const SmemBuf<Sh>& S, const float2* W) {
    constexpr int H = Sh::H;
    for (int e = threadIdx.x; e < H * Sh::R1; e += NT) Sh::rows_fwd2(S, e % H, e / H);
    __syncthreads();
    if constexpr (!Sh::DUAL) {
        for (int e = threadIdx.x; e < H * H; e += NT) Sh::cols_split(S, e / H, e % H);
        __syncthreads();
    }
    for (int e = threadIdx.x; e < H * Sh::kColTasks; e += NT) Sh::cols_fwd1(S, W, e % H, e / H);
    __syncthreads();
}

// from inverse pass 1 of the columns to the image rows in global memory
template <class Sh, int NT>
__device__ __forceinline__ void columns_to_image(const SmemBuf<Sh>& S, const float2* W,
                                                 float* __restrict__ dst) {
    constexpr int N = Sh::N, R1 = Sh::R1, R2 = Sh::R2, H = Sh::H;
    __syncthreads();
    for (int e = threadIdx.x; e < H * Sh::kColTasks; e += NT) Sh::cols_inv2(S, e % H, e / H);
    __syncthreads();
    if constexpr (!Sh::DUAL) {
        for (int e = threadIdx.x; e < H * H; e += NT) Sh::cols_merge(S, e / H, e % H);
        __syncthreads();
    }
    for (int e = threadIdx.x; e < H * R1; e += NT) Sh::rows_inv1(S, W, e % H, e / H);
    __syncthreads();
    for (int e = threadIdx.x; e < H * R2; e += NT) {
        const int p = e / R2, t = e - p * R2;
        float2 v[R1];
        Sh::rows_inv2(S, p, t, v);
        float* d = dst + 2 * p * N + t;
#pragma unroll
        for (int m = 0; m < R1; ++m) {
            d[R2 * m] = v[m].x;
            d[N + R2 * m] = v[m].y;
        }
    }
}

template <class Sh, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) whole_lowpass_kernel(LowpassArgs a) {
    constexpr int N = Sh::N, R1 = Sh::R1, R2 = Sh::R2, HS = Sh::HS, H = Sh::H;
    extern __shared__ float2 mixed_smem[];
    __shared__ float2 W[N];
    __shared__ double red[2][NT / 32];
    __shared__ float stat[2];
    const int64_t img = blockIdx.x;
    const int64_t s = a.sidx[img];
    float* dst = a.xbuf + img * (int64_t)N * N;
    if (s < 0 || s >= a.num_stack) {
        if (threadIdx.x == 0) atomicOr(a.status, kStatusBadIndex);
        for (int e = threadIdx.x; e < N * N; e += NT) dst[e] = __int_as_float(0x7fc00000);
        return;
    }
    load_twiddles<Sh, NT>(W, a.twid);
    const bool f = a.flip[img] != 0;
    const float* src = a.stack + s * (int64_t)N * N;
    const SmemBuf<Sh> S{mixed_smem};
    // rows (2p, 2p+1) -> Z_p; background statistics
    KSumM sum, sq;
#pragma unroll 8
    for (int e = threadIdx.x; e < H * N; e += NT) {
        const int p = e / N, b = e - p * N;
        const float* r = src + 2 * p * N + (f ? N - 1 - b : b);
        const float x0 = __ldg(r), x1 = __ldg(r + N);
        const float g0 = background<N>(x0, b, 2 * p), g1 = background<N>(x1, b, 2 * p + 1);
        sum.add(g0);
        sq.add(g0 * g0);
        sum.add(g1);
        sq.add(g1 * g1);
        S.at(p, Sh::nat(b)) = make_float2(x0, x1);
    }
    float mean, inv;
    image_stats<NT>((double)sum.value(), (double)sq.value(), red, stat, N * N, &mean, &inv);
    for (int e = threadIdx.x; e < H * R2; e += NT)
        Sh::template rows_fwd1<true>(S, W, e % H, e / H, mean, inv);
    __syncthreads();
    rows_to_columns<Sh, NT>(S, W);
    for (int e = threadIdx.x; e < H * R1; e += NT) {
        const int c = e % H, k1 = e / H;
        float2 v[R2];
        Sh::cols_fwd2(S, c, k1, v);
        if (c == 0) {                              // packed: filtered below, once complete
            Sh::cols_put(S, c, k1, v);
            continue;
        }
#pragma unroll
        for (int i = 0; i < R2; ++i) {
            const int j = k1 + R1 * i;
            const float g = __ldg(a.gtab + min(j, N - j) * HS + c);
            v[i] = make_float2(v[i].x * g, v[i].y * g);
        }
        Sh::cols_inv1(S, W, c, k1, v);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        for (int j = threadIdx.x; j <= N / 2; j += 32)
            Sh::packed_filter(S, j, __ldg(a.gtab + j * HS), __ldg(a.gtab + j * HS + H));
        __syncwarp();
        static_assert(R1 <= 32, "a lane per group of the packed column");
        if ((int)threadIdx.x < R1) {
            float2 v[R2];
            Sh::cols_get(S, 0, threadIdx.x, v);
            Sh::cols_inv1(S, W, 0, threadIdx.x, v);
        }
    }
    columns_to_image<Sh, NT>(S, W, dst);
}

// v[m] = rows (2p, 2p+1) of an image at element t + R2 m, times its mask
template <class Sh>
__device__ __forceinline__ void load_pair(const float* __restrict__ src,
                                          const uint8_t* __restrict__ mask, int p, int t,
                                          float2* v) {
    constexpr int N = Sh::N, R1 = Sh::R1, R2 = Sh::R2;
    const int o = 2 * p * N + t;
#pragma unroll
    for (int m = 0; m < R1; ++m)
        v[m] = make_float2(__ldg(src + o + R2 * m), __ldg(src + o + N + R2 * m));
    if (mask) {
#pragma unroll
        for (int m = 0; m < R1; ++m) {
            v[m].x = mask[o + R2 * m] ? v[m].x : 0.f;
            v[m].y = mask[o + N + R2 * m] ? v[m].y : 0.f;
        }
    }
}

template <class Sh, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) whole_spectrum_kernel(SpectrumArgs a) {
    constexpr int N = Sh::N, R1 = Sh::R1, R2 = Sh::R2, HS = Sh::HS, H = Sh::H;
    extern __shared__ float2 mixed_smem[];
    __shared__ float2 W[N];
    const int64_t img = blockIdx.x;
    const SmemBuf<Sh> S{mixed_smem};
    load_twiddles<Sh, NT>(W, a.twid);
    const float* src = a.images + img * (int64_t)N * N;
    const uint8_t* mask = a.masks ? a.masks + a.img_pd[img] * (int64_t)N * N : nullptr;
    __syncthreads();
    for (int e = threadIdx.x; e < H * R2; e += NT) {
        const int p = e / R2, t = e - p * R2;
        float2 v[R1];
        load_pair<Sh>(src, mask, p, t, v);
        Sh::rows_fwd1_store(S, W, p, t, v);
    }
    __syncthreads();
    rows_to_columns<Sh, NT>(S, W);
    float2* spec = a.spec + img * (int64_t)N * HS;
    for (int e = threadIdx.x; e < H * R1; e += NT) {
        const int c = e % H, k1 = e / H;
        float2 v[R2];
        Sh::cols_fwd2(S, c, k1, v);
        if (c == 0) {
            Sh::cols_put(S, c, k1, v);
            continue;
        }
#pragma unroll
        for (int i = 0; i < R2; ++i) spec[(k1 + R1 * i) * HS + c] = v[i];
    }
    __syncthreads();
    for (int j = threadIdx.x; j < N; j += NT)
        Sh::packed_split(S, j, spec + j * HS, spec + j * HS + H);
}

// element (j, c) of a half-plane spectrum, times sign(C) / N^2 when SIGNED
template <class Sh, bool SIGNED>
__device__ __forceinline__ float2 spectrum_value(const float2* __restrict__ spec, int j, int c,
                                                 uint64_t qf, const CtfConst& cc) {
    constexpr int N = Sh::N;
    const float2 y = spec[j * Sh::HS + c];
    if (!SIGNED) return y;
    const int fa = min(j, N - j);
    const float g = (float)ctf_sign(fa * fa + c * c, qf, cc) * (1.0f / ((float)N * (float)N));
    return make_float2(g * y.x, g * y.y);
}

template <class Sh, int NT, int MINB, bool SIGNED>
__global__ void __launch_bounds__(NT, MINB) whole_inverse_kernel(InverseArgs a) {
    constexpr int N = Sh::N, R1 = Sh::R1, R2 = Sh::R2, HS = Sh::HS, H = Sh::H;
    extern __shared__ float2 mixed_smem[];
    __shared__ float2 W[N];
    const int64_t img = blockIdx.x;
    const SmemBuf<Sh> S{mixed_smem};
    load_twiddles<Sh, NT>(W, a.twid);
    const float2* spec = a.spec + img * (int64_t)N * HS;
    const uint64_t qf = SIGNED ? a.qfix[img] : 0ull;
    __syncthreads();
    for (int e = threadIdx.x; e < H * R1; e += NT) {
        const int c = e % H, k1 = e / H;
        float2 v[R2];
#pragma unroll
        for (int i = 0; i < R2; ++i)
            v[i] = spectrum_value<Sh, SIGNED>(spec, k1 + R1 * i, c, qf, a.cc);
        if (c == 0) {                              // S_0 + i S_{N/2}
#pragma unroll
            for (int i = 0; i < R2; ++i) {
                const float2 h = spectrum_value<Sh, SIGNED>(spec, k1 + R1 * i, H, qf, a.cc);
                v[i] = make_float2(v[i].x - h.y, v[i].y + h.x);
            }
        }
        Sh::cols_inv1(S, W, c, k1, v);
    }
    columns_to_image<Sh, NT>(S, W, a.images + img * (int64_t)N * N);
}

// ------------------------------------------------------------------------- tiled images
// Rows: PC pair-rows at a time, as in the whole-image form.  Columns: CT at a time, element i of
// column c at [i][c] of the buffer; pass 1 reads its elements straight from global memory (lanes
// on consecutive columns), pass 2 the buffer.  The columns 0 and N/2 of the row spectra are real;
// between rows and columns a slot [N][H] keeps their real parts in one element.
// Up to 42 pair-rows and columns at a time, fewer where two buffers of that would not fit an SM:
// wide tiles keep the columns' global accesses long (1198 images of 250 px, low-pass / spectrum /
// flip: 583 / 252 / 289 us; 25 at a time with 128 threads, three CTAs per SM: 707 / 289 / 360;
// 16 with five CTAs: 578 / 291 / 346; 63 with one: 755 / 287 / 317).
template <class Sh>
struct Tile {
    static constexpr int NT = 288, MINB = 2;
    static constexpr size_t kRoom = 108 * 1024;
    static constexpr int cut(int lines, size_t line_bytes) {           // lines per buffer
        const int most = (int)(kRoom / line_bytes) < 42 ? (int)(kRoom / line_bytes) : 42;
        const int parts = (lines + most - 1) / most;
        return (lines + parts - 1) / parts;
    }
    static constexpr int PC = cut(Sh::H, Sh::S * sizeof(float2));
    static constexpr int CT = cut(Sh::HS, Sh::N * sizeof(float2));
    static constexpr size_t kRowBytes = (size_t)PC * Sh::S * sizeof(float2);
    static constexpr size_t kColBytes = (size_t)Sh::N * CT * sizeof(float2);
    static constexpr size_t bytes = kRowBytes > kColBytes ? kRowBytes : kColBytes;
};

// the chunk's row spectra (Z in the buffer, pass 1 done) split and handed to put(row, c, value),
// c = 0 .. H - 1, the columns 0 and H as (real part of 0, real part of H)
template <class Sh, class Put>
__device__ __forceinline__ void tiled_rows_out(const SmemBuf<Sh>& S, int p0, int np, Put put) {
    constexpr int NT = Tile<Sh>::NT, H = Sh::H, PC = Tile<Sh>::PC;
    for (int e = threadIdx.x; e < PC * Sh::R1; e += NT)
        if (e % PC < np) Sh::rows_fwd2(S, e % PC, e / PC);
    __syncthreads();
#pragma unroll 4
    for (int e = threadIdx.x; e < np * H; e += NT) {
        const int pl = e / H, c = e - pl * H;
        float2 x, y;
        Sh::split(c == 0, S.at(pl, Sh::pos(c)), S.at(pl, Sh::pos(Sh::odd_col(c))), &x, &y);
        put(2 * (p0 + pl), c, x);
        put(2 * (p0 + pl) + 1, c, y);
    }
    __syncthreads();
}

// the packed row spectra in the image's slot -> the image, in place: rows 2p and 2p + 1 of the slot
// are read before they are written
template <class Sh>
__device__ __forceinline__ void tiled_image_out(const SmemBuf<Sh>& S, const float2* W,
                                                float* slot) {
    constexpr int NT = Tile<Sh>::NT, N = Sh::N, H = Sh::H, R1 = Sh::R1, R2 = Sh::R2;
    constexpr int PC = Tile<Sh>::PC;
#pragma unroll 1
    for (int p0 = 0; p0 < H; p0 += PC) {
        const int np = min(PC, H - p0);
        const float2* rows = reinterpret_cast<const float2*>(slot) + (int64_t)2 * p0 * H;
#pragma unroll 4
        for (int e = threadIdx.x; e < np * H; e += NT) {
            const int pl = e / H, c = e - pl * H;
            Sh::merge(c == 0, rows[2 * pl * H + c], rows[(2 * pl + 1) * H + c],
                      &S.at(pl, Sh::pos(c)), &S.at(pl, Sh::pos(Sh::odd_col(c))));
        }
        __syncthreads();
        for (int e = threadIdx.x; e < PC * R1; e += NT)
            if (e % PC < np) Sh::rows_inv1(S, W, e % PC, e / PC);
        __syncthreads();
        for (int e = threadIdx.x; e < np * R2; e += NT) {
            const int pl = e / R2, t = e - pl * R2;
            float2 v[R1];
            Sh::rows_inv2(S, pl, t, v);
            float* d = slot + 2 * (p0 + pl) * N + t;
#pragma unroll
            for (int m = 0; m < R1; ++m) {
                d[R2 * m] = v[m].x;
                d[N + R2 * m] = v[m].y;
            }
        }
        __syncthreads();
    }
}

template <class Sh>
__global__ void __launch_bounds__(Tile<Sh>::NT, Tile<Sh>::MINB) tiled_lowpass_kernel(
        LowpassArgs a) {
    constexpr int NT = Tile<Sh>::NT, N = Sh::N, R1 = Sh::R1, R2 = Sh::R2, HS = Sh::HS, H = Sh::H;
    constexpr int PC = Tile<Sh>::PC, CT = Tile<Sh>::CT;
    extern __shared__ float2 mixed_smem[];
    __shared__ float2 W[N];
    __shared__ double red[2][NT / 32];
    __shared__ float stat[2];
    const int64_t img = blockIdx.x;
    const int64_t s = a.sidx[img];
    float* dst = a.xbuf + img * (int64_t)N * N;
    if (s < 0 || s >= a.num_stack) {
        if (threadIdx.x == 0) atomicOr(a.status, kStatusBadIndex);
        for (int e = threadIdx.x; e < N * N; e += NT) dst[e] = __int_as_float(0x7fc00000);
        return;
    }
    load_twiddles<Sh, NT>(W, a.twid);
    const bool f = a.flip[img] != 0;
    const float* src = a.stack + s * (int64_t)N * N;
    const SmemBuf<Sh> S{mixed_smem};
    KSumM sum, sq;
    auto stat_add = [&](float x, int r, int bs) {
        const float g = background<N>(x, f ? N - 1 - bs : bs, r);
        sum.add(g);
        sq.add(g * g);
    };
    if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {        // N N is a multiple of 4
#pragma unroll 4
        for (int q = threadIdx.x; q < N * N / 4; q += NT) {
            const float4 x = __ldg(reinterpret_cast<const float4*>(src) + q);
            const int r = 4 * q / N, b = 4 * q - r * N;        // N is even: pairs share a row
            const int r2 = b + 2 < N ? r : r + 1, b2 = b + 2 < N ? b + 2 : 0;
            stat_add(x.x, r, b);
            stat_add(x.y, r, b + 1);
            stat_add(x.z, r2, b2);
            stat_add(x.w, r2, b2 + 1);
        }
    } else {
#pragma unroll 8
        for (int e = threadIdx.x; e < N * N; e += NT) stat_add(__ldg(src + e), e / N, e % N);
    }
    float mean, inv;
    image_stats<NT>((double)sum.value(), (double)sq.value(), red, stat, N * N, &mean, &inv);
    float2* slot = reinterpret_cast<float2*>(dst);             // [N][H]
#pragma unroll 1
    for (int p0 = 0; p0 < H; p0 += PC) {
        const int np = min(PC, H - p0);
        for (int e = threadIdx.x; e < np * R2; e += NT) {
            const int pl = e / R2, t = e - pl * R2;
            const float* r = src + 2 * (p0 + pl) * N;
            float2 v[R1];
#pragma unroll
            for (int m = 0; m < R1; ++m) {
                const int b = f ? N - 1 - (t + R2 * m) : t + R2 * m;
                v[m] = make_float2((__ldg(r + b) - mean) * inv, (__ldg(r + N + b) - mean) * inv);
            }
            Sh::rows_fwd1_store(S, W, pl, t, v);
        }
        __syncthreads();
        tiled_rows_out<Sh>(S, p0, np, [&](int row, int c, float2 x) { slot[row * H + c] = x; });
    }
    float2* C = mixed_smem;                                    // [N][CT]
#pragma unroll 1
    for (int c0 = 0; c0 < HS; c0 += CT) {
        for (int e = threadIdx.x; e < CT * R2; e += NT) {
            const int cl = e % CT, t = e / CT, c = min(c0 + cl, H);
            float2 v[R1];
#pragma unroll
            for (int m = 0; m < R1; ++m) {
                v[m] = slot[(t + R2 * m) * H + (c == H ? 0 : c)];
                if (c == 0) v[m].y = 0.f;
                if (c == H) v[m] = make_float2(v[m].y, 0.f);
            }
            fft::dft_any<R1, 1>(v);
#pragma unroll
            for (int k = 0; k < R1; ++k)
                C[(R2 * k + t) * CT + cl] = k ? fft::cmul(v[k], W[t * k]) : v[k];
        }
        __syncthreads();
        for (int e = threadIdx.x; e < CT * R1; e += NT) {
            const int cl = e % CT, k1 = e / CT, c = min(c0 + cl, H);
            float2 v[R2];
#pragma unroll
            for (int t = 0; t < R2; ++t) v[t] = C[(R2 * k1 + t) * CT + cl];
            fft::dft_any<R2, 1>(v);
#pragma unroll
            for (int i = 0; i < R2; ++i) {
                const int j = k1 + R1 * i;
                const float g = __ldg(a.gtab + min(j, N - j) * HS + c);
                v[i] = make_float2(v[i].x * g, v[i].y * g);
            }
            fft::dft_any<R2, -1>(v);
#pragma unroll
            for (int t = 0; t < R2; ++t)
                C[(R2 * k1 + t) * CT + cl] = t ? fft::cmulc(v[t], W[t * k1]) : v[t];
        }
        __syncthreads();
        for (int e = threadIdx.x; e < CT * R2; e += NT) {
            const int cl = e % CT, t = e / CT, c = c0 + cl;
            float2 v[R1];
#pragma unroll
            for (int k = 0; k < R1; ++k) v[k] = C[(R2 * k + t) * CT + cl];
            fft::dft_any<R1, -1>(v);
            if (c > H) continue;
#pragma unroll
            for (int m = 0; m < R1; ++m) {
                float2* o = slot + (t + R2 * m) * H;
                if (c == 0) o[0].x = v[m].x;
                else if (c == H) o[0].y = v[m].x;
                else o[c] = v[m];
            }
        }
        __syncthreads();
    }
    tiled_image_out<Sh>(S, W, dst);
}

template <class Sh>
__global__ void __launch_bounds__(Tile<Sh>::NT, Tile<Sh>::MINB) tiled_spectrum_kernel(
        SpectrumArgs a) {
    constexpr int NT = Tile<Sh>::NT, N = Sh::N, R1 = Sh::R1, R2 = Sh::R2, HS = Sh::HS, H = Sh::H;
    constexpr int PC = Tile<Sh>::PC, CT = Tile<Sh>::CT;
    extern __shared__ float2 mixed_smem[];
    __shared__ float2 W[N];
    const int64_t img = blockIdx.x;
    const SmemBuf<Sh> S{mixed_smem};
    load_twiddles<Sh, NT>(W, a.twid);
    const float* src = a.images + img * (int64_t)N * N;
    const uint8_t* mask = a.masks ? a.masks + a.img_pd[img] * (int64_t)N * N : nullptr;
    float2* spec = a.spec + img * (int64_t)N * HS;
    __syncthreads();
#pragma unroll 1
    for (int p0 = 0; p0 < H; p0 += PC) {
        const int np = min(PC, H - p0);
        for (int e = threadIdx.x; e < np * R2; e += NT) {
            const int pl = e / R2, t = e - pl * R2;
            float2 v[R1];
            load_pair<Sh>(src, mask, p0 + pl, t, v);
            Sh::rows_fwd1_store(S, W, pl, t, v);
        }
        __syncthreads();
        tiled_rows_out<Sh>(S, p0, np, [&](int row, int c, float2 x) {
            if (c == 0) {
                spec[row * HS] = make_float2(x.x, 0.f);
                spec[row * HS + H] = make_float2(x.y, 0.f);
            } else {
                spec[row * HS + c] = x;
            }
        });
    }
    float2* C = mixed_smem;                                    // [N][CT]
#pragma unroll 1
    for (int c0 = 0; c0 < HS; c0 += CT) {
        for (int e = threadIdx.x; e < CT * R2; e += NT) {
            const int cl = e % CT, t = e / CT, c = min(c0 + cl, H);
            float2 v[R1];
#pragma unroll
            for (int m = 0; m < R1; ++m) v[m] = spec[(t + R2 * m) * HS + c];
            fft::dft_any<R1, 1>(v);
#pragma unroll
            for (int k = 0; k < R1; ++k)
                C[(R2 * k + t) * CT + cl] = k ? fft::cmul(v[k], W[t * k]) : v[k];
        }
        __syncthreads();
        for (int e = threadIdx.x; e < CT * R1; e += NT) {
            const int cl = e % CT, k1 = e / CT, c = c0 + cl;
            float2 v[R2];
#pragma unroll
            for (int t = 0; t < R2; ++t) v[t] = C[(R2 * k1 + t) * CT + cl];
            fft::dft_any<R2, 1>(v);
            if (c > H) continue;
#pragma unroll
            for (int i = 0; i < R2; ++i) spec[(k1 + R1 * i) * HS + c] = v[i];
        }
        __syncthreads();
    }
}

template <class Sh, bool SIGNED>
__global__ void __launch_bounds__(Tile<Sh>::NT, Tile<Sh>::MINB) tiled_inverse_kernel(
        InverseArgs a) {
    constexpr int NT = Tile<Sh>::NT, N = Sh::N, R1 = Sh::R1, R2 = Sh::R2, HS = Sh::HS, H = Sh::H;
    constexpr int CT = Tile<Sh>::CT;
    extern __shared__ float2 mixed_smem[];
    __shared__ float2 W[N];
    const int64_t img = blockIdx.x;
    const SmemBuf<Sh> S{mixed_smem};
    load_twiddles<Sh, NT>(W, a.twid);
    const float2* spec = a.spec + img * (int64_t)N * HS;
    const uint64_t qf = SIGNED ? a.qfix[img] : 0ull;
    float* dst = a.images + img * (int64_t)N * N;
    float2* slot = reinterpret_cast<float2*>(dst);             // [N][H]
    float2* C = mixed_smem;                                    // [N][CT]
    __syncthreads();
#pragma unroll 1
    for (int c0 = 0; c0 < HS; c0 += CT) {
        for (int e = threadIdx.x; e < CT * R1; e += NT) {
            const int cl = e % CT, k1 = e / CT, c = min(c0 + cl, H);
            float2 v[R2];
#pragma unroll
            for (int i = 0; i < R2; ++i)
                v[i] = spectrum_value<Sh, SIGNED>(spec, k1 + R1 * i, c, qf, a.cc);
            fft::dft_any<R2, -1>(v);
#pragma unroll
            for (int t = 0; t < R2; ++t)
                C[(R2 * k1 + t) * CT + cl] = t ? fft::cmulc(v[t], W[t * k1]) : v[t];
        }
        __syncthreads();
        for (int e = threadIdx.x; e < CT * R2; e += NT) {
            const int cl = e % CT, t = e / CT, c = c0 + cl;
            float2 v[R1];
#pragma unroll
            for (int k = 0; k < R1; ++k) v[k] = C[(R2 * k + t) * CT + cl];
            fft::dft_any<R1, -1>(v);
            if (c > H) continue;
#pragma unroll
            for (int m = 0; m < R1; ++m) {
                float2* o = slot + (t + R2 * m) * H;
                if (c == 0) o[0].x = v[m].x;
                else if (c == H) o[0].y = v[m].x;
                else o[c] = v[m];
            }
        }
        __syncthreads();
    }
    tiled_image_out<Sh>(S, W, dst);
}

template <int N, int R1>
constexpr Kernels make_kernels() {
    using Sh = fft::MixShape<N, R1, N / R1>;
    if constexpr (whole_bytes<Sh>() + sizeof(float2) * N + 1024 <= 227 * 1024) {
        constexpr int NT = whole_threads<Sh>(), MB = whole_blocks<Sh>();
        return Kernels{N, NT, false, whole_bytes<Sh>(), whole_lowpass_kernel<Sh, NT, MB>,
                       whole_spectrum_kernel<Sh, NT, MB>, whole_inverse_kernel<Sh, NT, MB, false>,
                       whole_inverse_kernel<Sh, NT, MB, true>, nullptr, 0, 0};
    } else {
        return Kernels{N, Tile<Sh>::NT, true, Tile<Sh>::bytes, tiled_lowpass_kernel<Sh>,
                       tiled_spectrum_kernel<Sh>, tiled_inverse_kernel<Sh, false>,
                       tiled_inverse_kernel<Sh, true>, nullptr, 0, 0};
    }
}

// with the rotation in segments of SEG samples, LPR lines at a time (rotate_whole.cuh); the pair of
// each size was picked for 512 to 1024 resident threads of 64 registers and few rounds
template <int N, int R1, int SEG, int LPR>
constexpr Kernels make_kernels() {
    using Sh = rot::WholeShape<N, SEG, LPR>;
    Kernels k = make_kernels<N, R1>();
    k.rotate = rot::rotate_whole_kernel<Sh>;
    k.rot_threads = Sh::NT;
    k.rot_smem = Sh::SMEM;
    return k;
}

}  // namespace mixed
}  // namespace mem
