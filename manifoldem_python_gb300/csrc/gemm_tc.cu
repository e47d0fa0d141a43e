// Split-BF16 tcgen05 form of the all-pairs CTF distance (reference :391-397).
//
//   D_ij = a_i + a_j + E_ij,  E_ij = u'_i.v'_j + v'_i.u'_j - r'_i.r'_j - s'_i.s'_j
//
// Each feature x is stored as x_hi = bf16(x), x_lo = bf16(x - x_hi); E is accumulated as
// A_hi.B_hi + A_hi.B_lo + A_lo.B_hi (the lo.lo term, ~2^-16 relative, is dropped except in the
// chunks the schedule marks, the low-frequency ring-sum chunks of U', V') on the 5th-gen
// tensor cores: tcgen05.mma kind::f16 (BF16 in, FP32 accumulate in TMEM), operands staged in
// shared memory by TMA (128-byte swizzle).  B reads the same feature matrix as A with its first
// two column blocks swapped: each 64-wide K chunk takes its A and B columns from the plan's
// chunk schedule (TMA coordinates); the r', s' chunks use the instruction descriptor's
// negate-B bit, so one accumulator holds E.
//
// One CTA per upper-triangle 128 x 128 tile (pd, I, J); 10 warps:
//   warps 0-7  epilogue: warp w reads TMEM lanes 32*(w%4).. and columns 64*(w/4)..;
//   warp 8     TMA producer (3-stage ring of 64 KB stages: A_hi, A_lo, B_hi, B_lo, K = 64);
//   warp 9     TMEM allocator and MMA issuer.
// The K loop is cut into groups of `group_chunks` 64-wide chunks; each group accumulates into
// one of two TMEM buffers and the epilogue warps add the finished group into FP32 register sums
// (compensated), so the tensor core's FP32 accumulation only ever spans one group.
// Every mbarrier wait is bounded: on expiry the CTA sets the status word's timeout bit, stops
// issuing, waits (bounded) for its own TMA copies and MMAs, frees its TMEM and returns.
#include <algorithm>
#include <type_traits>

#include "tcgen05.cuh"

namespace mem {
namespace {

using namespace tc;

constexpr int TC_M = 128, TC_BK = 64;
constexpr int TC_EPI_WARPS = 8;
constexpr int TC_THREADS = (TC_EPI_WARPS + 2) * 32;
constexpr int TC_OPB = TC_M * TC_BK * 2;          // one 128-row operand box: 16 KB
constexpr int TC_MAX_STAGES = 3;

// Tile shape 128 x BN (BN = 128 or 256 columns of D): a stage holds A_hi, A_lo (128 rows each)
// and B_hi, B_lo (BN rows each, BN / 128 boxes) of one 64-wide K chunk; three 64 KB stages
// at BN = 128, two 96 KB stages at BN = 256
template <int BN>
struct TcShape {
    static constexpr int B_BOXES = BN / 128;
    static constexpr int STAGE_BYTES = (2 + 2 * B_BOXES) * TC_OPB;
    static constexpr int STAGES = BN == 256 ? 2 : 3;
    static constexpr size_t SMEM = (size_t)STAGES * STAGE_BYTES + 1024 + 256;
    // epilogue warps: 4 lane quadrants x BN / 64 column blocks of 64, so that every epilogue
    // thread keeps 64 running sums (BN = 256 with 8 warps would keep 128 and spill)
    static constexpr int EPI_WARPS = BN / 16;
    static constexpr int THREADS = (EPI_WARPS + 2) * 32;
    static_assert(STAGES <= TC_MAX_STAGES, "stage ring");
};

// instruction descriptor, kind::f16: D f32 (bits 4-5 = 1), A bf16 (7-9 = 1), B bf16 (10-12 = 1),
// K-major A and B (bits 15, 16 = 0), N >> 3 at bits 17-22, M >> 4 at bits 24-28, negate B bit 14
template <int BN>
__host__ __device__ constexpr uint32_t idesc_f16() {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) |
           ((uint32_t)(TC_M >> 4) << 24);
}

constexpr int TC_MAX_BUFS = 4;

struct TcShared {
    uint64_t full[TC_MAX_STAGES];
    uint64_t empty[TC_MAX_STAGES];
    uint64_t acc_full[TC_MAX_BUFS];
    uint64_t acc_empty[TC_MAX_BUFS];
    uint64_t mma_done;
    uint32_t tmem_base;
    int abort_flag;
    int ticket;
};

// Where tile x of the `rest` tiles of the last wave of S CTAs is cut (chunks of its head).  Tile x's
// head goes to CTA x and its tail to CTA x + d, d = S - rest.  So the CTAs x, x + d, x + 2d, ..
// form a chain, m tiles on m + 1 CTAs: the k-th tile's head takes (m - k) / (m + 1) of its chunks, and
// every CTA of the chain gets m / (m + 1) of a tile beside its whole ones.
__host__ __device__ inline int tc_cut_of(int x, int rest, int S, int nchunks) {
    const int d = S - rest, k = x / d, m = (rest - x % d + d - 1) / d;
    return (int)((int64_t)nchunks * (m - k) / (m + 1));
}

// bounded wait for a flag that another CTA sets; as mbar_wait
__device__ __forceinline__ bool flag_wait(const unsigned* flag, volatile int* abort_flag,
                                          uint32_t* status, long long limit) {
    const long long t0 = clock64();
    for (;;) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
        if (v) return true;
        if (*abort_flag) return false;
        if (clock64() - t0 > limit) {
            *abort_flag = 1;
            atomicOr(status, kStatusTimeout);
            return false;
        }
    }
}

// The contraction over the tiles [tile_begin, tile_begin + tile_count) of the plan's tile list:
// CTA b takes tiles tile_begin + b + k gridDim.x (a persistent CTA when the grid is smaller
// than the tile count; one tile per CTA when it is as large).  The producer, the MMA issuer and
// the epilogue each walk the CTA's tiles in the same order; the stage ring and the NBUF TMEM
// accumulators (NBUF x 128 columns) continue from one tile to the next, so a tile's first
// groups are loaded and multiplied while the epilogue still adds and stores the previous tile.
//
// SPLIT: as many CTAs as SMs (T tiles on S of them, S < T): each CTA computes T / S whole tiles, and
// every tile of the last, partial wave is cut in two at a chunk: one CTA computes its first chunks
// before its whole tiles and leaves the running sums in `carry`, another continues from them after
// its own, so that the sums are the same, chunk by chunk.  See tc_cut_of for the cuts.  A continuing
// warp waits (bounded) for the flag of the warp it follows, which was set about a tile's time
// before.  CTA b is the b-th to start (a ticket): it only waits for CTAs that started before it, and
// only for what they do first and without waiting, so that the waits end also where the CTAs do not
// all fit at once (SMs held by other work, a context with fewer of them).
template <bool KAHAN, bool LOLO, int NBUF, int BN, bool SPLIT>
__global__ void __launch_bounds__(TcShape<BN>::THREADS, 1) gemm_tc_kernel(
        const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo,
        const double* __restrict__ pair_norm, const uint32_t* __restrict__ scale_bits,
        const Tile* __restrict__ tiles, const PdDev* __restrict__ pds, double* __restrict__ D,
        uint32_t* __restrict__ status, const int4* __restrict__ chunks, int nchunks,
        int group_chunks, long long wait_limit, int withhold, int tile_begin, int tile_count,
        float* __restrict__ carry, unsigned* __restrict__ carry_flags,
        unsigned* __restrict__ tickets) {
    static_assert(NBUF == 2 || NBUF == 4, "two or four TMEM accumulators");
    static_assert(BN == 128 || BN == 256, "tile widths");
    static_assert(NBUF * BN <= 512, "TMEM holds 512 columns");
    using S = TcShape<BN>;
    constexpr int TC_STAGES = S::STAGES, TC_STAGE_BYTES = S::STAGE_BYTES;
    constexpr uint32_t IDESC = idesc_f16<BN>(), IDESC_NEG = IDESC | (1u << 14);
    constexpr int EPI = S::EPI_WARPS;              // epilogue warps (warps 0 .. EPI - 1)
    constexpr int EC = 64;                         // epilogue columns per thread
    constexpr uint32_t TMEM_COLS = NBUF * BN;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    TcShared* sh = (TcShared*)(smem + TC_STAGES * TC_STAGE_BYTES);
    volatile int* abort_flag = &sh->abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gsize = (group_chunks > 0 && group_chunks < nchunks) ? group_chunks : nchunks;
    const int ngroups = (nchunks + gsize - 1) / gsize;

    if (threadIdx.x == 0) {
        for (int s = 0; s < TC_STAGES; ++s) {
            mbar_init(&sh->full[s], 1);
            mbar_init(&sh->empty[s], 1);
        }
        for (int b = 0; b < NBUF; ++b) {
            mbar_init(&sh->acc_full[b], 1);
            mbar_init(&sh->acc_empty[b], EPI);
        }
        mbar_init(&sh->mma_done, 1);
        sh->abort_flag = 0;
        if (SPLIT) sh->ticket = (int)atomicAdd(tickets, 1u);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == EPI + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&sh->tmem_base)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    const int cta = SPLIT ? sh->ticket : (int)blockIdx.x;
    // SPLIT: this CTA's parts are [head of tile cta], whole tiles, [tail of tile tail]
    const int rest = SPLIT ? tile_count % (int)gridDim.x : 0;
    const int tail = SPLIT ? cta - ((int)gridDim.x - rest) : -1;
    const int heads = SPLIT && cta < rest ? 1 : 0;
    const int whole = SPLIT ? tile_count / (int)gridDim.x
                      : cta < tile_count
                          ? (tile_count - cta + (int)gridDim.x - 1) / (int)gridDim.x
                          : 0;
    const int my_tiles = heads + whole + (tail >= 0 ? 1 : 0);
    struct Part {
        Tile t;
        int c0, c1;                                // its chunks
    };
    auto part_of = [&](int lt) {
        Part p;
        const int k = lt - heads;
        const int i = !SPLIT           ? cta + lt * (int)gridDim.x
                      : k < 0          ? cta
                      : k < whole      ? rest + cta + k * (int)gridDim.x
                                       : tail;
        p.t = tiles[tile_begin + i];
        p.c0 = SPLIT && k == whole ? tc_cut_of(tail, rest, (int)gridDim.x, nchunks) : 0;
        p.c1 = SPLIT && k < 0 ? tc_cut_of(i, rest, (int)gridDim.x, nchunks) : nchunks;
        return p;
    };

    if (warp == EPI) {
        // ---------------------------------------------------------------- TMA producer
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&map_hi) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&map_lo) : "memory");
            long long gc = 0, withheld = -1;     // chunks issued by this CTA (all its tiles)
            bool stop = false;
            for (int lt = 0; lt < my_tiles && !stop; ++lt) {
                const Part part = part_of(lt);
                const Tile t = part.t;
                const PdDev pd = pds[t.pd];
                const int rowA = (int)(pd.row_off + (int64_t)t.I * TC_M);
                const int rowB = (int)(pd.row_off + (int64_t)t.J * BN);
                for (int c = part.c0; c < part.c1; ++c, ++gc) {
                    const int st = (int)(gc % TC_STAGES);
                    const uint32_t ph = (uint32_t)(gc / TC_STAGES) & 1u;
                    if (gc >= TC_STAGES &&
                        !mbar_wait(&sh->empty[st], ph ^ 1u, abort_flag, status, wait_limit)) {
                        stop = true;
                        break;
                    }
                    // a withheld chunk (test of the timeout path; first tile only) is never
                    // loaded, so the MMA issuer's wait for it can only end by its limit
                    if (lt == 0 && c == withhold) {
                        withheld = gc;
                        continue;
                    }
                    // the chunk schedule interleaves the feature blocks so that the dominant
                    // low-frequency columns of every block are accumulated last
                    const int4 ch = chunks[c];
                    uint8_t* sb = smem + st * TC_STAGE_BYTES;
                    mbar_expect_tx(&sh->full[st], TC_STAGE_BYTES);
                    tma_load_2d(sb + 0 * TC_OPB, &map_hi, &sh->full[st], ch.x, rowA);
                    tma_load_2d(sb + 1 * TC_OPB, &map_lo, &sh->full[st], ch.x, rowA);
#pragma unroll
                    for (int q = 0; q < S::B_BOXES; ++q) {
                        tma_load_2d(sb + (2 + q) * TC_OPB, &map_hi, &sh->full[st], ch.y,
                                    rowB + 128 * q);
                        tma_load_2d(sb + (2 + S::B_BOXES + q) * TC_OPB, &map_lo, &sh->full[st],
                                    ch.y, rowB + 128 * q);
                    }
                }
            }
            if (*abort_flag) {   // let the copies already issued land before the CTA exits
                for (long long c = (gc > TC_STAGES ? gc - TC_STAGES : 0); c < gc; ++c)
                    if (c != withheld)
                        mbar_drain(&sh->full[c % TC_STAGES], (uint32_t)(c / TC_STAGES) & 1u,
                                   wait_limit);
            }
        }
    } else if (warp == EPI + 1) {
        // ---------------------------------------------------------------- MMA issuer
        if (lane == 0) {
            bool issued_any = false, stop = false;
            long long gc = 0, gg = 0;            // chunks and accumulation groups of this CTA
            for (int lt = 0; lt < my_tiles && !stop; ++lt) {
                const Part part = part_of(lt);
                int4 ch_next = chunks[part.c0];  // schedule entry, read one chunk ahead
                for (int c = part.c0; c < part.c1; ++c, ++gc) {
                    const int4 ch = ch_next;
                    if (c + 1 < nchunks) ch_next = chunks[c + 1];
                    const int st = (int)(gc % TC_STAGES);
                    const uint32_t ph = (uint32_t)(gc / TC_STAGES) & 1u;
                    const int b = (int)(gg % NBUF);
                    const long long use = gg / NBUF;        // earlier uses of buffer b
                    const bool first = (c % gsize) == 0;
                    const bool last = ((c % gsize) == gsize - 1) || c == nchunks - 1;
                    if (first && use >= 1 &&
                        !mbar_wait(&sh->acc_empty[b], (uint32_t)((use - 1) & 1), abort_flag,
                                   status, wait_limit)) {
                        stop = true;
                        break;
                    }
                    if (!mbar_wait(&sh->full[st], ph, abort_flag, status, wait_limit)) {
                        stop = true;
                        break;
                    }
                    tc_fence_after();
                    const bool neg = ch.z != 0;             // r', s' blocks (chunk schedule)
                    const uint32_t idesc = neg ? IDESC_NEG : IDESC;
                    const uint32_t d = tmem + (uint32_t)(b * BN);
                    const uint32_t sa = smem_u32(smem + st * TC_STAGE_BYTES);
                    // three products per K step; the lo.lo product too for marked chunks (one
                    // branch per chunk, both bodies fully unrolled)
                    auto mma_chunk = [&](auto four) {
#pragma unroll
                        for (int k = 0; k < TC_BK / 16; ++k) {
                            const uint64_t ahi = sdesc_sw128(sa + 0 * TC_OPB + k * 32);
                            const uint64_t alo = sdesc_sw128(sa + 1 * TC_OPB + k * 32);
                            const uint64_t bhi = sdesc_sw128(sa + 2 * TC_OPB + k * 32);
                            const uint64_t blo =
                                sdesc_sw128(sa + (2 + S::B_BOXES) * TC_OPB + k * 32);
                            umma_bf16(d, ahi, bhi, idesc, (first && k == 0) ? 0u : 1u);
                            umma_bf16(d, ahi, blo, idesc, 1u);
                            umma_bf16(d, alo, bhi, idesc, 1u);
                            if (decltype(four)::value) umma_bf16(d, alo, blo, idesc, 1u);
                        }
                    };
                    if (LOLO || ch.w != 0)
                        mma_chunk(std::true_type{});
                    else
                        mma_chunk(std::false_type{});
                    issued_any = true;
                    umma_commit(&sh->empty[st]);
                    if (last) {
                        umma_commit(&sh->acc_full[b]);
                        ++gg;
                    }
                }
            }
            if (*abort_flag && issued_any) {   // wait for the MMAs in flight
                umma_commit(&sh->mma_done);
                mbar_drain(&sh->mma_done, 0, wait_limit);
            }
        }
    } else {
        // ---------------------------------------------------------------- epilogue
        const int q = warp & 3, h = warp >> 2;
        const int row = q * 32 + lane;
        bool ok = true;
        long long gg = 0;
        for (int lt = 0; lt < my_tiles && ok; ++lt) {
            const Part part = part_of(lt);
            const Tile t = part.t;
            float acc[EC], cmp[KAHAN ? EC : 1];
            const int groups = SPLIT ? part.c1 - part.c0 : ngroups;      // SPLIT: gsize is 1
            if (SPLIT && part.c0 > 0) {            // from the sums that the tile's head left
                const int64_t at = (int64_t)tail * EPI + warp;
                ok = flag_wait(carry_flags + at, abort_flag, status, wait_limit);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                const float* from = carry + at * (EC * 32) + lane;
#pragma unroll
                for (int j = 0; j < EC; ++j) acc[j] = __ldcg(from + 32 * j);
            } else {
#pragma unroll
                for (int j = 0; j < EC; ++j) acc[j] = 0.f;
            }
#pragma unroll
            for (int j = 0; j < (KAHAN ? EC : 1); ++j) cmp[j] = 0.f;
            for (int g = 0; g < groups; ++g, ++gg) {
                const int b = (int)(gg % NBUF);
                const long long use = gg / NBUF;
                ok = mbar_wait(&sh->acc_full[b], (uint32_t)(use & 1), abort_flag, status,
                               wait_limit);
                __syncwarp();
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                const uint32_t taddr =
                    tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * BN + h * EC);
                // BN = 256 (16 epilogue warps, 112 registers each): 16-column loads, so that
                // the 64 running sums and the loaded columns fit without spilling
                constexpr int LDC = BN == 256 ? 16 : 32;
#pragma unroll
                for (int half = 0; half < EC / LDC; ++half) {
                    uint32_t r[LDC];
                    if constexpr (LDC == 16)
                        tmem_ld16(taddr + half * LDC, r);
                    else
                        tmem_ld32(taddr + half * LDC, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < LDC; ++j) {
                        const float x = __uint_as_float(r[j]);
                        float& s = acc[half * LDC + j];
                        if (KAHAN) {
                            float& c = cmp[KAHAN ? half * LDC + j : 0];
                            const float y = x - c;
                            const float tt = s + y;
                            c = (tt - s) - y;
                            s = tt;
                        } else {
                            s += x;
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh->acc_empty[b]);
            }
            if (!ok || *abort_flag) break;
            if (SPLIT && part.c1 < nchunks) {      // a head: leave the sums, then the flag
                const int64_t at = (int64_t)cta * EPI + warp;
                float* to = carry + at * (EC * 32) + lane;
#pragma unroll
                for (int j = 0; j < EC; ++j) __stcg(to + 32 * j, acc[j]);
                __threadfence();
                __syncwarp();
                if (lane == 0)
                    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(carry_flags + at),
                                 "r"(1u)
                                 : "memory");
                continue;
            }
            const PdDev pd = pds[t.pd];
            const double sc = (double)feature_scale_from_bits(scale_bits[t.pd]);
            const double inv_sc2 = 1.0 / (sc * sc);
            const int n = pd.n;
            const int gi = t.I * TC_M + row;
            double* Dp = D + pd.d_off;
            const double* an = pair_norm + pd.img_off;
            if (gi < n) {
                const double ai = an[gi];
                const int j0 = t.J * BN + h * EC;
#pragma unroll
                for (int j = 0; j < EC; ++j) {
                    const int gj = j0 + j;
                    // blocks of 8 columns: keeps the compiler from hoisting all 64 norm loads
                    // ahead of the stores (their registers would spill the running sums)
                    if ((j & 7) == 0) asm volatile("" ::: "memory");
                    if (gj >= n || gj < gi) continue;
                    if (gj == gi) {
                        Dp[(int64_t)gi * n + gi] = 0.0;
                        continue;
                    }
                    const float e = KAHAN ? (acc[j] - cmp[KAHAN ? j : 0]) : acc[j];
                    const double v = ai + an[gj] + (double)e * inv_sc2;
                    Dp[(int64_t)gi * n + gj] = v;
                    Dp[(int64_t)gj * n + gi] = v;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == EPI + 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(TMEM_COLS)
                     : "memory");
    }
}

// ---- the CTA-pair form: 256 x 128 tiles on two SMs (cta_group::2) --------------------------
// A cluster of two CTAs on two SMs computes a 256 x 128 tile with one MMA stream: the even
// CTA issues tcgen05.mma.cta_group::2 (M = 256, N = 128); each CTA holds 128 rows of A and 64
// of the 128 B rows of every stage in its own shared memory, and 128 accumulator rows in its
// own tensor memory.  Per SM a 64-wide K chunk moves 48 KB (A 32 KB, half of B 16 KB) instead
// of the 64 KB of a 128 x 128 tile on one SM, and four stages fit in shared memory.
//   loads:  both CTAs' TMA copies count on the even CTA's full barrier (the even CTA arms it
//           with both CTAs' bytes);
//   MMA:    one thread of the even CTA; its commits arrive on the stage's empty barrier and
//           the accumulator's full barrier of both CTAs (multicast);
//   epilogue: each CTA drains its own tensor memory and arrives on the even CTA's
//           accumulator-empty barrier (16 arrivals per group).
// Waits are bounded as in the one-SM kernel.  After an abort the even CTA waits (bounded) for
// the stages it armed; the odd CTA, whose copies count on the even CTA's barriers, waits a
// bounded time far longer than a copy takes before both CTAs meet at the final cluster barrier.
constexpr int TP_STAGES = 4;
constexpr int TP_OPB_B = 64 * TC_BK * 2;                      // one 64-row box: 8 KB
constexpr int TP_STAGE_BYTES = 2 * TC_OPB + 2 * TP_OPB_B;      // 48 KB per CTA
constexpr size_t TP_SMEM = (size_t)TP_STAGES * TP_STAGE_BYTES + 1024 + 512;

struct TpShared {
    uint64_t full[TP_STAGES];
    uint64_t empty[TP_STAGES];
    uint64_t acc_full[TC_MAX_BUFS];
    uint64_t acc_empty[TC_MAX_BUFS];
    uint64_t mma_done;
    uint32_t tmem_base;
    int abort_flag;
};

template <bool LOLO, int NBUF>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TC_THREADS, 1) gemm_tc_pair_kernel(
        const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo,
        const __grid_constant__ CUtensorMap mapb_hi, const __grid_constant__ CUtensorMap mapb_lo,
        const double* __restrict__ pair_norm, const uint32_t* __restrict__ scale_bits,
        const Tile* __restrict__ tiles, const PdDev* __restrict__ pds, double* __restrict__ D,
        uint32_t* __restrict__ status, const int4* __restrict__ chunks, int nchunks,
        int group_chunks, long long wait_limit, int withhold, int tile_begin, int tile_count) {
    static_assert(NBUF == 2 || NBUF == 4, "two or four TMEM accumulators");
    constexpr int BN = 128, EC = 64;
    constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) |
                               ((uint32_t)(256 >> 4) << 24);
    constexpr uint32_t IDESC_NEG = IDESC | (1u << 14);
    constexpr uint32_t TMEM_COLS = NBUF * BN;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    TpShared* sh = (TpShared*)(smem + TP_STAGES * TP_STAGE_BYTES);
    volatile int* abort_flag = &sh->abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const bool even = rank == 0;
    const int pair = (int)(blockIdx.x >> 1), npairs = (int)(gridDim.x >> 1);
    const int my_tiles = pair < tile_count ? (tile_count - pair + npairs - 1) / npairs : 0;
    auto tile_of = [&](int lt) { return tiles[tile_begin + pair + lt * npairs]; };
    const int gsize = (group_chunks > 0 && group_chunks < nchunks) ? group_chunks : nchunks;
    const int ngroups = (nchunks + gsize - 1) / gsize;

    if (threadIdx.x == 0) {
        for (int s = 0; s < TP_STAGES; ++s) {
            mbar_init(&sh->full[s], 1);
            mbar_init(&sh->empty[s], 1);
        }
        for (int b = 0; b < NBUF; ++b) {
            mbar_init(&sh->acc_full[b], 1);
            mbar_init(&sh->acc_empty[b], 2 * TC_EPI_WARPS);
        }
        mbar_init(&sh->mma_done, 1);
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == TC_EPI_WARPS + 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&sh->tmem_base)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    cluster_sync();              // both CTAs' barriers and tensor memory are ready
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    // the even CTA's full and accumulator-empty barriers, as cluster addresses
    const uint32_t full_even = map_to_cta(smem_u32(&sh->full[0]), 0);
    const uint32_t acc_empty_even = map_to_cta(smem_u32(&sh->acc_empty[0]), 0);

    if (warp == TC_EPI_WARPS) {
        // ---------------------------------------------------------------- TMA producer
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&map_hi) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&map_lo) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&mapb_hi) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&mapb_lo) : "memory");
            long long gc = 0, withheld = -1;
            bool stop = false;
            for (int lt = 0; lt < my_tiles && !stop; ++lt) {
                const Tile t = tile_of(lt);
                const PdDev pd = pds[t.pd];
                const int rowA = (int)(pd.row_off + (int64_t)t.I * 256 + rank * 128);
                const int rowB = (int)(pd.row_off + (int64_t)t.J * BN + rank * 64);
                for (int c = 0; c < nchunks; ++c, ++gc) {
                    const int st = (int)(gc % TP_STAGES);
                    const uint32_t ph = (uint32_t)(gc / TP_STAGES) & 1u;
                    if (gc >= TP_STAGES &&
                        !mbar_wait(&sh->empty[st], ph ^ 1u, abort_flag, status, wait_limit)) {
                        stop = true;
                        break;
                    }
                    if (lt == 0 && c == withhold) {      // test of the timeout path
                        withheld = gc;
                        continue;
                    }
                    const int4 ch = chunks[c];
                    uint8_t* sb = smem + st * TP_STAGE_BYTES;
                    if (even) mbar_expect_tx(&sh->full[st], 2 * TP_STAGE_BYTES);
                    const uint32_t bar = full_even + 8u * (uint32_t)st;
                    tma_load_2d_pair(sb, &map_hi, bar, ch.x, rowA);
                    tma_load_2d_pair(sb + TC_OPB, &map_lo, bar, ch.x, rowA);
                    tma_load_2d_pair(sb + 2 * TC_OPB, &mapb_hi, bar, ch.y, rowB);
                    tma_load_2d_pair(sb + 2 * TC_OPB + TP_OPB_B, &mapb_lo, bar, ch.y, rowB);
                }
            }
            if (*abort_flag) {
                if (even) {      // the stages this CTA armed: both CTAs' copies have landed
                    for (long long c = (gc > TP_STAGES ? gc - TP_STAGES : 0); c < gc; ++c)
                        if (c != withheld)
                            mbar_drain(&sh->full[c % TP_STAGES],
                                       (uint32_t)(c / TP_STAGES) & 1u, wait_limit);
                } else {         // copies count on the even CTA's barriers: a bounded pause
                    const long long t0 = clock64();
                    const long long pause = wait_limit < (1ll << 22) ? wait_limit : (1ll << 22);
                    while (clock64() - t0 < pause) __nanosleep(1000);
                }
            }
        }
    } else if (warp == TC_EPI_WARPS + 1) {
        // ---------------------------------------------------------------- MMA issuer
        if (lane == 0 && even) {
            bool issued_any = false, stop = false;
            long long gc = 0, gg = 0;
            for (int lt = 0; lt < my_tiles && !stop; ++lt) {
                int4 ch_next = chunks[0];
                for (int c = 0; c < nchunks; ++c, ++gc) {
                    const int4 ch = ch_next;
                    if (c + 1 < nchunks) ch_next = chunks[c + 1];
                    const int st = (int)(gc % TP_STAGES);
                    const uint32_t ph = (uint32_t)(gc / TP_STAGES) & 1u;
                    const int b = (int)(gg % NBUF);
                    const long long use = gg / NBUF;
                    const bool first = (c % gsize) == 0;
                    const bool last = ((c % gsize) == gsize - 1) || c == nchunks - 1;
                    if (first && use >= 1 &&
                        !mbar_wait(&sh->acc_empty[b], (uint32_t)((use - 1) & 1), abort_flag,
                                   status, wait_limit)) {
                        stop = true;
                        break;
                    }
                    if (!mbar_wait(&sh->full[st], ph, abort_flag, status, wait_limit)) {
                        stop = true;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t idesc = ch.z != 0 ? IDESC_NEG : IDESC;
                    const uint32_t d = tmem + (uint32_t)(b * BN);
                    const uint32_t sa = smem_u32(smem + st * TP_STAGE_BYTES);
                    auto mma_chunk = [&](auto four) {
#pragma unroll
                        for (int k = 0; k < TC_BK / 16; ++k) {
                            const uint64_t ahi = sdesc_sw128(sa + k * 32);
                            const uint64_t alo = sdesc_sw128(sa + TC_OPB + k * 32);
                            const uint64_t bhi = sdesc_sw128(sa + 2 * TC_OPB + k * 32);
                            const uint64_t blo = sdesc_sw128(sa + 2 * TC_OPB + TP_OPB_B + k * 32);
                            umma_bf16_pair(d, ahi, bhi, idesc, (first && k == 0) ? 0u : 1u);
                            umma_bf16_pair(d, ahi, blo, idesc, 1u);
                            umma_bf16_pair(d, alo, bhi, idesc, 1u);
                            if (decltype(four)::value) umma_bf16_pair(d, alo, blo, idesc, 1u);
                        }
                    };
                    if (LOLO || ch.w != 0)
                        mma_chunk(std::true_type{});
                    else
                        mma_chunk(std::false_type{});
                    issued_any = true;
                    umma_commit_pair(&sh->empty[st], (uint16_t)3);
                    if (last) {
                        umma_commit_pair(&sh->acc_full[b], (uint16_t)3);
                        ++gg;
                    }
                }
            }
            if (*abort_flag && issued_any) {   // wait for the MMAs in flight
                umma_commit_pair(&sh->mma_done, (uint16_t)1);
                mbar_drain(&sh->mma_done, 0, wait_limit);
            }
        }
    } else {
        // ---------------------------------------------------------------- epilogue
        const int q = warp & 3, h = warp >> 2;
        const int row = q * 32 + lane;
        bool ok = true;
        long long gg = 0;
        for (int lt = 0; lt < my_tiles && ok; ++lt) {
            const Tile t = tile_of(lt);
            float acc[EC];
#pragma unroll
            for (int j = 0; j < EC; ++j) acc[j] = 0.f;
            for (int g = 0; g < ngroups; ++g, ++gg) {
                const int b = (int)(gg % NBUF);
                const long long use = gg / NBUF;
                ok = mbar_wait(&sh->acc_full[b], (uint32_t)(use & 1), abort_flag, status,
                               wait_limit);
                __syncwarp();
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                const uint32_t taddr =
                    tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * BN + h * EC);
#pragma unroll
                for (int half = 0; half < EC / 32; ++half) {
                    uint32_t r[32];
                    tmem_ld32(taddr + half * 32, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) acc[half * 32 + j] += __uint_as_float(r[j]);
                }
                tc_fence_before();
                __syncwarp();
                // the accumulator's columns are in registers (tcgen05.wait::ld above): a relaxed
                // arrive suffices, and a release at cluster scope cost a memory barrier per
                // warp and group (the kernel's top stall)
                if (lane == 0) mbar_arrive_cluster_relaxed(acc_empty_even + 8u * (uint32_t)b);
            }
            if (!ok || *abort_flag) break;
            const PdDev pd = pds[t.pd];
            const double sc = (double)feature_scale_from_bits(scale_bits[t.pd]);
            const double inv_sc2 = 1.0 / (sc * sc);
            const int n = pd.n;
            const int gi = t.I * 256 + (int)rank * 128 + row;
            double* Dp = D + pd.d_off;
            const double* an = pair_norm + pd.img_off;
            if (gi < n) {
                const double ai = an[gi];
                const int j0 = t.J * BN + h * EC;
#pragma unroll
                for (int j = 0; j < EC; ++j) {
                    const int gj = j0 + j;
                    if (gj >= n || gj < gi) continue;
                    if (gj == gi) {
                        Dp[(int64_t)gi * n + gi] = 0.0;
                        continue;
                    }
                    const double v = ai + an[gj] + (double)acc[j] * inv_sc2;
                    Dp[(int64_t)gi * n + gj] = v;
                    Dp[(int64_t)gj * n + gi] = v;
                }
            }
        }
    }
    tc_fence_before();
    cluster_sync();              // the pair's MMAs, copies and remote arrivals are done
    if (warp == TC_EPI_WARPS + 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(TMEM_COLS)
                     : "memory");
    }
}

// ---- few tiles: every K chunk its own CTA ---------------------------------------------------
// One CTA walks a tile's chunks in about 1 us each (the MMA and its shared-memory traffic), so a
// plan of few tiles leaves most SMs idle: 102 us for the 6 tiles of 300 images of 70 px.  Here unit
// (tile, chunk) is a CTA of its own, which stores the chunk's accumulator -- the very value that the
// epilogue of gemm_tc_kernel adds for the chunk -- and gemm_tc_join_kernel adds a tile's chunks in
// their order: D is bit-identical.  Units go in rounds of what the scratch holds, the running sums
// between rounds in the scratch too.  Bound by writing and reading the 64 KB of a unit in L2.
// 300 images of 70 px: 28 us; 100 of 128 px: 17 us, was 268; see tc_split_units for the line between the two.
constexpr int TS_THREADS = 128;
constexpr int TS_ELEMS = TC_M * 128;
constexpr size_t TS_SMEM = (size_t)4 * TC_OPB + 1024;

template <bool LOLO>
__global__ void __launch_bounds__(TS_THREADS) gemm_tc_chunk_kernel(
        const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo,
        const Tile* __restrict__ tiles, const PdDev* __restrict__ pds, float* __restrict__ part,
        uint32_t* __restrict__ status, const int4* __restrict__ chunks, int c_begin, int c_count,
        long long wait_limit, int withhold) {
    constexpr uint32_t IDESC = idesc_f16<128>(), IDESC_NEG = IDESC | (1u << 14);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sb = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full, done;
    __shared__ uint32_t tmem_base;
    __shared__ int abort_word;
    volatile int* abort_flag = &abort_word;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const Tile t = tiles[blockIdx.x / c_count];
    const int c = c_begin + (int)(blockIdx.x % c_count);
    if (threadIdx.x == 0) {
        mbar_init(&full, 1);
        mbar_init(&done, 1);
        abort_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&tmem_base)),
                     "r"(128u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    if (threadIdx.x == 0) {
        const int4 ch = chunks[c];
        const bool load = c != withhold;           // a withheld chunk: test of the timeout path
        if (load) {
            const PdDev pd = pds[t.pd];
            const int rowA = (int)(pd.row_off + (int64_t)t.I * TC_M);
            const int rowB = (int)(pd.row_off + (int64_t)t.J * 128);
            mbar_expect_tx(&full, 4 * TC_OPB);
            tma_load_2d(sb + 0 * TC_OPB, &map_hi, &full, ch.x, rowA);
            tma_load_2d(sb + 1 * TC_OPB, &map_lo, &full, ch.x, rowA);
            tma_load_2d(sb + 2 * TC_OPB, &map_hi, &full, ch.y, rowB);
            tma_load_2d(sb + 3 * TC_OPB, &map_lo, &full, ch.y, rowB);
        }
        if (mbar_wait(&full, 0, abort_flag, status, wait_limit)) {
            tc_fence_after();
            const uint32_t idesc = ch.z != 0 ? IDESC_NEG : IDESC;
            const uint32_t sa = smem_u32(sb);
            const bool four = LOLO || ch.w != 0;
#pragma unroll
            for (int k = 0; k < TC_BK / 16; ++k) {
                const uint64_t ahi = sdesc_sw128(sa + 0 * TC_OPB + k * 32);
                const uint64_t alo = sdesc_sw128(sa + 1 * TC_OPB + k * 32);
                const uint64_t bhi = sdesc_sw128(sa + 2 * TC_OPB + k * 32);
                const uint64_t blo = sdesc_sw128(sa + 3 * TC_OPB + k * 32);
                umma_bf16(tmem, ahi, bhi, idesc, k == 0 ? 0u : 1u);
                umma_bf16(tmem, ahi, blo, idesc, 1u);
                umma_bf16(tmem, alo, bhi, idesc, 1u);
                if (four) umma_bf16(tmem, alo, blo, idesc, 1u);
            }
            umma_commit(&done);
            // an expired wait below does not end before the MMAs have
            if (!mbar_wait(&done, 0, abort_flag, status, wait_limit))
                mbar_drain(&done, 0, wait_limit);
        } else if (load) {
            mbar_drain(&full, 0, wait_limit);      // the copies land before the CTA exits
        }
    }
    __syncwarp();
    const bool ok = __all_sync(0xffffffffu,
                               mbar_wait(&done, 0, abort_flag, status, wait_limit));
    if (ok) {
        tc_fence_after();
        // [column][row]: a column's 32 lanes store 128 consecutive bytes
        float* out = part + (int64_t)blockIdx.x * TS_ELEMS + warp * 32 + lane;
#pragma unroll 1
        for (int q = 0; q < 4; ++q) {
            uint32_t r[32];
            tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(q * 32), r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) out[(q * 32 + j) * TC_M] = __uint_as_float(r[j]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(128u)
                     : "memory");
    }
}

// adds the round's chunks to the tiles' running sums; the last round stores D
__global__ void __launch_bounds__(TS_THREADS) gemm_tc_join_kernel(
        const float* __restrict__ part, float* __restrict__ run, int c_count, int first, int last,
        const double* __restrict__ pair_norm, const uint32_t* __restrict__ scale_bits,
        const Tile* __restrict__ tiles, const PdDev* __restrict__ pds, double* __restrict__ D) {
    constexpr int kPerTile = TS_ELEMS / TS_THREADS;
    const int tile = blockIdx.x / kPerTile;
    const int e = (int)(blockIdx.x % kPerTile) * TS_THREADS + (int)threadIdx.x;
    const Tile t = tiles[tile];
    const PdDev pd = pds[t.pd];
    const int gi = t.I * TC_M + e % TC_M, gj = t.J * 128 + e / TC_M, n = pd.n;
    if (gi >= n || gj >= n || gj < gi) return;
    float* r = run + (int64_t)tile * TS_ELEMS + e;
    float acc = first ? 0.f : *r;
    const float* p = part + (int64_t)tile * c_count * TS_ELEMS + e;
    constexpr int B = 16;                          // loads in flight per element
    float v[B];
    auto load = [&](int c0) {
#pragma unroll
        for (int u = 0; u < B; ++u) v[u] = p[(int64_t)min(c0 + u, c_count - 1) * TS_ELEMS];
    };
    load(0);
    int c = 0;
    for (; c + B <= c_count; c += B) {
        float w[B];
#pragma unroll
        for (int u = 0; u < B; ++u) w[u] = v[u];
        load(c + B);
#pragma unroll
        for (int u = 0; u < B; ++u) acc += w[u];
    }
#pragma unroll
    for (int u = 0; u < B; ++u)
        if (c + u < c_count) acc += v[u];
    if (!last) {
        *r = acc;
        return;
    }
    double* Dp = D + pd.d_off;
    if (gj == gi) {
        Dp[(int64_t)gi * n + gi] = 0.0;
        return;
    }
    const double sc = (double)feature_scale_from_bits(scale_bits[t.pd]);
    const double inv_sc2 = 1.0 / (sc * sc);
    const double* an = pair_norm + pd.img_off;
    const double d = an[gi] + an[gj] + (double)acc * inv_sc2;
    Dp[(int64_t)gi * n + gj] = d;
    Dp[(int64_t)gj * n + gi] = d;
}

}  // namespace

// Scratch units (64 KB each) with which the contraction of `tiles` tiles is split by chunks, at most
// `most`; 0: one CTA per tile is the faster.  Measured: about 1 us per chunk for a tile of its own
// CTA whatever the number of tiles up to one per SM, against 20 to 27 ns per unit and 8 us per round.
int64_t tc_split_units(int64_t tiles, int64_t chunks, int64_t most) {
    if (tiles < 1 || tiles > 64) return 0;
    const int64_t per_round = std::min(chunks, most / tiles);    // chunks
    if (per_round < 1) return 0;
    const int64_t rounds = (chunks + per_round - 1) / per_round;
    if (8.0 * rounds + 0.02 * (double)(tiles * chunks) > 0.7 * (double)chunks) return 0;
    return per_round * tiles;
}

// Whether the last wave's tiles of a launch of `tiles` on `sms` SMs are cut in two (gemm_tc_kernel,
// SPLIT): one to four whole waves before them, beyond which the wave is a small part (and
// without one a tail would wait for its head).  24 PDs of 400 images of 128 px (250 tiles): 551 us
// whole, 469 cut; of 64 px 179 and 155; 6 PDs of 1500 at 64 px (347 wide tiles): 408 and 330.
bool tc_cut_pays(int64_t tiles, int64_t sms) {
    return tiles > sms && tiles < 5 * sms && tiles % sms != 0 && sms <= kTcFlagBytes / 64;
}

// waves of `tiles` tiles on `sms` SMs, a cut wave as the longest of its chains (tc_cut_of)
double tc_waves(int64_t tiles, int64_t sms) {
    if (!tc_cut_pays(tiles, sms)) return (double)((tiles + sms - 1) / sms);
    const int64_t rest = tiles % sms, d = sms - rest, m = (rest + d - 1) / d;
    return (double)(tiles / sms) + (double)m / (double)(m + 1);
}

namespace kern {
int gemm_split_bf16(const mem_plan& P, const void* feat_hi, const void* feat_lo,
                    const double* pair_norm, const uint32_t* scale_bits, const Tile* tiles,
                    const PdDev* pds, const int4* chunks, double* D, uint32_t* status,
                    float* part, int64_t part_units, bool cut, cudaStream_t s) {
    if (P.tiles.empty() || !D) return MEM_OK;
    // every chunk starts on a 64-column boundary: TMA x offsets are multiples of 8 bf16
    if (P.Kf % TC_BK != 0 || P.n_rows % TC_M != 0 || (int64_t)P.n_chunks * TC_BK != P.Kf)
        return MEM_ERR_INVALID;
    CUtensorMap mhi, mlo;
    int st = tc::make_map(&mhi, feat_hi, P.Kf, P.n_rows);
    if (st != MEM_OK) return st;
    st = tc::make_map(&mlo, feat_lo, P.Kf, P.n_rows);
    if (st != MEM_OK) return st;
    // the default schedule of a plan of few tiles: chunks spread over the SMs
    const mem_contraction_config& c0 = P.tc_classes[0];
    const int T = (int)P.tc_tiles.size();
    if (part_units >= T && P.tc_ranges.size() == 1 && !c0.persistent && c0.accumulators == 2 &&
        c0.tile_n == 128 && c0.tile_m == 128 && P.tc_group_chunks == 1 && !P.tc_kahan) {
        float* run = part + part_units * TS_ELEMS;
        const int per_round = (int)std::min<int64_t>(P.n_chunks, part_units / T);
        auto kfn = P.tc_lolo ? gemm_tc_chunk_kernel<true> : gemm_tc_chunk_kernel<false>;
        MEM_CUDA_TRY(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)TS_SMEM));
        for (int c = 0; c < P.n_chunks; c += per_round) {
            const int count = std::min(per_round, P.n_chunks - c);
            kfn<<<(unsigned)(T * count), TS_THREADS, TS_SMEM, s>>>(
                    mhi, mlo, tiles, pds, part, status, chunks, c, count, P.wait_cycles,
                    P.test_withhold_chunk);
            MEM_LAUNCH_CHECK();
            gemm_tc_join_kernel<<<(unsigned)(T * (TS_ELEMS / TS_THREADS)), TS_THREADS, 0, s>>>(
                    part, run, count, c == 0 ? 1 : 0, c + count == P.n_chunks ? 1 : 0, pair_norm,
                    scale_bits, tiles, pds, D);
            MEM_LAUNCH_CHECK();
        }
        return MEM_OK;
    }
    const int sms = P.num_sms > 0 ? P.num_sms : 1;
    // the default schedule where the last wave is partial: its tiles cut in two (no gain beside the load
    // stream of a split execute, whose CTAs hold some SMs)
    if (cut && P.tc_carry >= sms && P.tc_ranges.size() == 1 && !c0.persistent && c0.accumulators == 2 &&
        c0.tile_m == 128 && P.tc_group_chunks == 1 && !P.tc_kahan && P.test_withhold_chunk < 0 &&
        tc_cut_pays(T, sms)) {
        const int rest = T % sms;
        auto kfn = c0.tile_n == 256
                       ? (P.tc_lolo ? gemm_tc_kernel<false, true, 2, 256, true>
                                    : gemm_tc_kernel<false, false, 2, 256, true>)
                       : (P.tc_lolo ? gemm_tc_kernel<false, true, 2, 128, true>
                                    : gemm_tc_kernel<false, false, 2, 128, true>);
        const size_t smem = c0.tile_n == 256 ? TcShape<256>::SMEM : TcShape<128>::SMEM;
        const int threads = c0.tile_n == 256 ? TcShape<256>::THREADS : TcShape<128>::THREADS;
        unsigned* tickets = reinterpret_cast<unsigned*>(part);    // one, then the flags
        unsigned* flags = tickets + 16;
        float* carry = part + kTcFlagBytes / sizeof(float);
        MEM_CUDA_TRY(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)smem));
        MEM_CUDA_TRY(cudaMemsetAsync(tickets, 0, sizeof(unsigned) * (16 + 16 * rest), s));
        kfn<<<(unsigned)sms, threads, smem, s>>>(mhi, mlo, pair_norm, scale_bits, tiles, pds, D,
                                                 status, chunks, P.n_chunks, P.tc_group_chunks,
                                                 P.wait_cycles, P.test_withhold_chunk, 0, T, carry,
                                                 flags, tickets);
        MEM_LAUNCH_CHECK();
        return MEM_OK;
    }
    CUtensorMap bhi, blo;                // 64-row boxes: the CTA pairs' halves of B
    bool have_b64 = false;
    // one launch per size class of the plan's contraction configuration (tiles sorted by class)
    for (size_t k = 0; k < P.tc_ranges.size(); ++k) {
        const int begin = P.tc_ranges[k].first, count = P.tc_ranges[k].second;
        if (count <= 0) continue;
        const mem_contraction_config& cfg = P.tc_classes[k];
        if (cfg.tile_m == 256) {
            if (!have_b64) {
                st = tc::make_map(&bhi, feat_hi, P.Kf, P.n_rows, 64);
                if (st != MEM_OK) return st;
                st = tc::make_map(&blo, feat_lo, P.Kf, P.n_rows, 64);
                if (st != MEM_OK) return st;
                have_b64 = true;
            }
            const unsigned pgrid =
                2u * (unsigned)(cfg.persistent ? std::min(count, std::max(1, sms / 2)) : count);
#define MEM_TP_LAUNCH(LOLO, NB)                                                                \
    do {                                                                                       \
        MEM_CUDA_TRY(cudaFuncSetAttribute(gemm_tc_pair_kernel<LOLO, NB>,                       \
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,         \
                                          (int)TP_SMEM));                                      \
        gemm_tc_pair_kernel<LOLO, NB><<<pgrid, TC_THREADS, TP_SMEM, s>>>(                      \
            mhi, mlo, bhi, blo, pair_norm, scale_bits, tiles, pds, D, status, chunks,          \
            P.n_chunks, P.tc_group_chunks, P.wait_cycles, P.test_withhold_chunk, begin,        \
            count);                                                                            \
    } while (0)
            if (P.tc_lolo) {
                if (cfg.accumulators == 4) MEM_TP_LAUNCH(true, 4); else MEM_TP_LAUNCH(true, 2);
            } else {
                if (cfg.accumulators == 4) MEM_TP_LAUNCH(false, 4); else MEM_TP_LAUNCH(false, 2);
            }
#undef MEM_TP_LAUNCH
            MEM_LAUNCH_CHECK();
            continue;
        }
        const unsigned grid = cfg.persistent ? (unsigned)std::min(count, sms) : (unsigned)count;
#define MEM_TC_LAUNCH(KAHAN, LOLO, NB, BN)                                                     \
    do {                                                                                       \
        MEM_CUDA_TRY(cudaFuncSetAttribute(gemm_tc_kernel<KAHAN, LOLO, NB, BN, false>,          \
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,         \
                                          (int)TcShape<BN>::SMEM));                            \
        gemm_tc_kernel<KAHAN, LOLO, NB, BN, false>                                             \
            <<<grid, TcShape<BN>::THREADS, TcShape<BN>::SMEM, s>>>(                            \
                mhi, mlo, pair_norm, scale_bits, tiles, pds, D, status, chunks, P.n_chunks,    \
                P.tc_group_chunks, P.wait_cycles, P.test_withhold_chunk, begin, count,         \
                nullptr, nullptr, nullptr);                                                    \
    } while (0)
#define MEM_TC_SHAPE(KAHAN, LOLO)                                                              \
    do {                                                                                       \
        if (cfg.tile_n == 256) MEM_TC_LAUNCH(KAHAN, LOLO, 2, 256);                             \
        else if (cfg.accumulators == 4) MEM_TC_LAUNCH(KAHAN, LOLO, 4, 128);                    \
        else MEM_TC_LAUNCH(KAHAN, LOLO, 2, 128);                                               \
    } while (0)
        // the compensated sums of the 256-wide tile would not fit the register file: its
        // classes keep the 128-wide kernel (apply_contraction) when MEM_TC_KAHAN is set
        if (P.tc_kahan) {
            if (P.tc_lolo) MEM_TC_LAUNCH(true, true, 2, 128); else MEM_TC_LAUNCH(true, false, 2, 128);
        } else {
            if (P.tc_lolo) MEM_TC_SHAPE(false, true); else MEM_TC_SHAPE(false, false);
        }
#undef MEM_TC_SHAPE
#undef MEM_TC_LAUNCH
        MEM_LAUNCH_CHECK();
    }
    return MEM_OK;
}
}  // namespace kern
}  // namespace mem
