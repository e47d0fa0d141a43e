// Plain FP32 form of the all-pairs CTF distance (reference :391-397):
//   D_ij = a_i + a_j + E_ij,   E_ij = u'_i.v'_j + v'_i.u'_j - r'_i.r'_j - s'_i.s'_j
// over the centred half-plane features written by features_kernel (prologue.cu).
// One CTA per upper-triangle tile of a PD (128 x 128, or 64 x 64 and 32 x 32 parts of it where there
// are few), FP32 FMA accumulation over k in order, FP64 epilogue, mirrored store (D exactly
// symmetric, zero diagonal).
#include "mem_internal.cuh"

namespace mem {
namespace {

// T x T tile of D: a warp's lanes form 4 (rows) x 8 (columns) thread tiles of RB x HB runs of 4
template <int T>
struct Shape {
    static constexpr int BK = 16, RB = T == 128 ? 2 : 1, HB = RB;
    static constexpr int NT = T == 32 ? 64 : 256, WM = T == 32 ? 2 : 4;      // warps along the rows
    static constexpr int LR = T * (BK / 4) / NT;       // operand rows a thread loads per stage
    static constexpr int LD = T + 4;                   // padded: the transposing stores
    static constexpr size_t SMEM = 4 * (size_t)BK * LD * sizeof(float);
    static_assert(WM * 16 * RB == T && NT / 32 / WM * 32 * HB == T, "warps cover the tile");
};

// Paired FP32 FMAs (fma.rn.f32x2: two columns of D per instruction, each rounded as a scalar FMA,
// so every element keeps its sum over k in order): with scalar FMAs the 64 of a k step need every
// issue slot of the SM and the loads beside them stall it.  A warp's lanes form 4 x 8 thread
// tiles: a half-warp's 16-byte operand loads then touch 128 bytes at most, one wavefront; as 2 x
// 16 they touched 256 and shared memory bound the kernel.  Three stages of loads travel in
// registers: an operand row is 80 KB from the next, and with one stage ahead the warps waited for
// the loads a fifth of their time.  2000 images of 128 px (136 tiles): 1797 us, 2493 with scalar
// FMAs and one stage ahead; 16 warps per SM (512 threads, or 128 x 64 tiles) took 2021 and 2129.
// A plan of few tiles leaves most SMs idle for a time that does not shrink with the tiles (1750 us
// for one tile): below 100 tiles each is split into 4 CTAs, below 25 into 16.  100 images of
// 128 px: 516 us, was 2305; 900 (36 tiles): 840 us, was 2493.
template <int T>
__global__ void __launch_bounds__(Shape<T>::NT, 1) gemm_fp32_kernel(
        const float* __restrict__ X, const double* __restrict__ pair_norm,
        const uint32_t* __restrict__ scale_bits, const Tile* __restrict__ tiles,
        const PdDev* __restrict__ pds, const int4* __restrict__ chunks, double* __restrict__ D,
        int64_t Kf) {
    using S = Shape<T>;
    constexpr int BK = S::BK, NT = S::NT, LD = S::LD, LR = S::LR, RB = S::RB, HB = S::HB;
    constexpr int JP = 2 * HB, PARTS = 128 / T;
    extern __shared__ __align__(16) float smem[];
    const Tile t = tiles[blockIdx.x / (PARTS * PARTS)];
    const int part = blockIdx.x % (PARTS * PARTS);
    const int r0 = t.I * 128 + part / PARTS * T, c0 = t.J * 128 + part % PARTS * T;
    const PdDev pd = pds[t.pd];
    if (c0 < r0 || r0 >= pd.n || c0 >= pd.n) return;       // below the diagonal or padding
    const int64_t K4 = Kf;
    const int tid = threadIdx.x;
    const int lrow = tid >> 2, lk = (tid & 3) * 4;
    const float* Abase = X + (pd.row_off + r0) * K4;
    const float* Bbase = X + (pd.row_off + c0) * K4;
    const int nstage = (int)(K4 / BK);
    auto As = [&](int buf, int k) { return smem + (buf * BK + k) * LD; };
    auto Bs = [&](int buf, int k) { return smem + (2 * BK + buf * BK + k) * LD; };

    // stage st is the 16-column slice (st & 3) of 64-wide chunk st >> 2 of the plan's chunk
    // schedule (A column, B column, sign), which interleaves the feature blocks so that the
    // dominant low-frequency columns are accumulated last; the schedule's entry is read a stage
    // ahead of the loads that need it
    constexpr int AHEAD = 3;        // stages in registers on their way to smem
    float4 ra[AHEAD][LR], rb[AHEAD][LR];
    int4 ch = chunks[0];
    float sg[AHEAD];
    auto gload = [&](int st, int u) {
        const int64_t ka = ch.x + (st & 3) * BK, kb = ch.y + (st & 3) * BK;
        sg[u] = ch.z ? -1.0f : 1.0f;
#pragma unroll
        for (int h = 0; h < LR; ++h) {
            const int r = lrow + h * (NT / 4);
            ra[u][h] = *reinterpret_cast<const float4*>(Abase + (int64_t)r * K4 + ka + lk);
            rb[u][h] = *reinterpret_cast<const float4*>(Bbase + (int64_t)r * K4 + kb + lk);
        }
        if ((st & 3) == 3 && st + 1 < nstage) ch = chunks[(st + 1) >> 2];
    };
    auto sstore = [&](int buf, int u) {
#pragma unroll
        for (int h = 0; h < LR; ++h) {
            const int r = lrow + h * (NT / 4);
            const float va[4] = {sg[u] * ra[u][h].x, sg[u] * ra[u][h].y, sg[u] * ra[u][h].z,
                                 sg[u] * ra[u][h].w};
#pragma unroll
            for (int q = 0; q < 4; ++q) As(buf, lk + q)[r] = va[q];
            const float vb[4] = {rb[u][h].x, rb[u][h].y, rb[u][h].z, rb[u][h].w};
#pragma unroll
            for (int q = 0; q < 4; ++q) Bs(buf, lk + q)[r] = vb[q];
        }
    };

    float2 acc[4 * RB][JP];                        // rows i, column pairs j
#pragma unroll
    for (int i = 0; i < 4 * RB; ++i)
#pragma unroll
        for (int j = 0; j < JP; ++j) acc[i][j] = make_float2(0.f, 0.f);

    // the thread's rows are RB runs of 4, 16 apart, its columns HB runs of 4, 32 apart
    const int ty = (tid >> 3) & 3, tx = tid & 7, warp = tid >> 5;
    const int row0 = (warp % S::WM) * (16 * RB) + ty * 4, cl0 = (warp / S::WM) * (32 * HB) + tx * 4;
    auto compute = [&](int buf) {
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            const float* pa = As(buf, kk) + row0;
            const float* pb = Bs(buf, kk) + cl0;
            float2 a[4 * RB];
#pragma unroll
            for (int h = 0; h < RB; ++h) {
                const float4 v = *reinterpret_cast<const float4*>(pa + 16 * h);
                a[4 * h] = make_float2(v.x, v.x);
                a[4 * h + 1] = make_float2(v.y, v.y);
                a[4 * h + 2] = make_float2(v.z, v.z);
                a[4 * h + 3] = make_float2(v.w, v.w);
            }
            float2 b[JP];
#pragma unroll
            for (int h = 0; h < HB; ++h) {
                const float4 v = *reinterpret_cast<const float4*>(pb + 32 * h);
                b[2 * h] = make_float2(v.x, v.y);
                b[2 * h + 1] = make_float2(v.z, v.w);
            }
#pragma unroll
            for (int i = 0; i < 4 * RB; ++i)
#pragma unroll
                for (int j = 0; j < JP; ++j) acc[i][j] = __ffma2_rn(a[i], b[j], acc[i][j]);
        }
    };
    // stage st is computed from buffer st & 1 while stage st + 1 is stored into the other and
    // stages up to st + 1 + AHEAD travel
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
        if (u < nstage) gload(u, u);
    sstore(0, 0);
    if (AHEAD < nstage) gload(AHEAD, 0);
    __syncthreads();
    int st = 0;
    for (; st < nstage;) {
        // AHEAD stages per turn, so that the register sets have constant indices
#pragma unroll
        for (int u = 0; u < AHEAD; ++u, ++st) {
            if (st >= nstage) break;
            compute(st & 1);
            if (st + 1 < nstage) {
                sstore((st + 1) & 1, (u + 1) % AHEAD);
                if (st + 1 + AHEAD < nstage) gload(st + 1 + AHEAD, (u + 1) % AHEAD);
                __syncthreads();
            }
        }
    }

    // epilogue: D = a_i + a_j + E / scale^2 in FP64, upper triangle + mirror
    const double sc = (double)feature_scale_from_bits(scale_bits[t.pd]);
    const double inv_sc2 = 1.0 / (sc * sc);
    const int n = pd.n;
    double* Dp = D + pd.d_off;
    const double* an = pair_norm + pd.img_off;
#pragma unroll
    for (int i = 0; i < 4 * RB; ++i) {
        const int gi = r0 + row0 + (i < 4 ? i : 16 + i - 4);
        if (gi >= n) continue;
        const double ai = an[gi];
#pragma unroll
        for (int j = 0; j < 2 * JP; ++j) {
            const int gj = c0 + cl0 + (j < 4 ? j : 32 + j - 4);
            if (gj >= n || gj < gi) continue;
            if (gj == gi) {
                Dp[(int64_t)gi * n + gi] = 0.0;
                continue;
            }
            const float e = (j & 1) ? acc[i][j >> 1].y : acc[i][j >> 1].x;
            const double v = ai + an[gj] + (double)e * inv_sc2;
            Dp[(int64_t)gi * n + gj] = v;
            Dp[(int64_t)gj * n + gi] = v;
        }
    }
}

}  // namespace

namespace kern {
int gemm_fp32(const mem_plan& P, const float* feat, const double* pair_norm,
              const uint32_t* scale_bits, const Tile* tiles, const PdDev* pds,
              const int4* chunks, double* D, cudaStream_t s) {
    if (P.tiles.empty() || !D) return MEM_OK;
    if ((int64_t)P.n_chunks * 64 != P.Kf) return MEM_ERR_INVALID;
    const unsigned tiles_n = (unsigned)P.tiles.size();
    if (tiles_n >= 100)
        gemm_fp32_kernel<128><<<tiles_n, Shape<128>::NT, Shape<128>::SMEM, s>>>(
                feat, pair_norm, scale_bits, tiles, pds, chunks, D, P.Kf);
    else if (tiles_n >= 25)
        gemm_fp32_kernel<64><<<4 * tiles_n, Shape<64>::NT, Shape<64>::SMEM, s>>>(
                feat, pair_norm, scale_bits, tiles, pds, chunks, D, P.Kf);
    else
        gemm_fp32_kernel<32><<<16 * tiles_n, Shape<32>::NT, Shape<32>::SMEM, s>>>(
                feat, pair_norm, scale_bits, tiles, pds, chunks, D, P.Kf);
    MEM_LAUNCH_CHECK();
    return MEM_OK;
}
}  // namespace kern
}  // namespace mem
