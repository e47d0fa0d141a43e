// Sums that round to the float that FP64 gives, kept as pairs of floats.
//
// The NLSA kernels round two FP64 sums to float: the Wiener denominators and the sums over the parts
// of a correlation.  FP64 runs at 1/64 of the FP32 rate on this part, so the sums are kept as an
// unevaluated pair hi + lo (about 48 bits) with a bound on its distance from the FP64 sum, and the
// pair is taken only where every value within the bound rounds to the same float (or where both
// sums are exact).  Where that is not so, the caller repeats the sum in FP64, in its order: the
// floats are those of FP64 sums without exception.
//
// In the bounds eps = 2^-24 and b is at least every |hi| on the way: a float rounding of a value up
// to x errs by at most eps x, the two-sum and the FMA's remainder of a product are exact, and lo, at
// most eps b after settle(), grows by eps b with every term added.  Products near the end of the
// float range lose at most 2^-148 more, far below the bounds' slack.
//
// Host-compilable, so that both sums can be compared with FP64 bit for bit without a GPU.
#pragma once

#include <cmath>
#include <cstdint>

#if defined(__CUDACC__)
#define MEM_SUM_HD __host__ __device__ __forceinline__
#else
#define MEM_SUM_HD inline
#endif
#if !defined(__CUDA_ARCH__)
#include <cfenv>
#endif

namespace mem {

constexpr float kEps2 = 3.552713678800501e-15f;    // eps^2 = 2^-48

// a - x rounded down and a + x rounded up
MEM_SUM_HD float below(float a, float x) {
#if defined(__CUDA_ARCH__)
    return __fsub_rd(a, x);
#else
    std::fesetround(FE_DOWNWARD);
    const volatile float va = a, vx = x;
    const volatile float r = va - vx;
    std::fesetround(FE_TONEAREST);
    return r;
#endif
}
MEM_SUM_HD float above(float a, float x) {
#if defined(__CUDA_ARCH__)
    return __fadd_ru(a, x);
#else
    std::fesetround(FE_UPWARD);
    const volatile float va = a, vx = x;
    const volatile float r = va + vx;
    std::fesetround(FE_TONEAREST);
    return r;
#endif
}
#if defined(__CUDA_ARCH__)
#define MEM_ADD(a, b) __fadd_rn(a, b)
#define MEM_SUB(a, b) __fsub_rn(a, b)
#define MEM_MUL(a, b) __fmul_rn(a, b)
#define MEM_FMA(a, b, c) __fmaf_rn(a, b, c)
#else
#define MEM_ADD(a, b) ((a) + (b))
#define MEM_SUB(a, b) ((a) - (b))
#define MEM_MUL(a, b) ((a) * (b))
#define MEM_FMA(a, b, c) std::fmaf(a, b, c)
#endif

struct Pair {
    float hi = 0.f, lo = 0.f;
    MEM_SUM_HD void add(float x) {                               // Knuth's two-sum of hi and x
        const float s = MEM_ADD(hi, x);
        const float t = MEM_SUB(s, hi);
        lo = MEM_ADD(lo, MEM_ADD(MEM_SUB(hi, MEM_SUB(s, t)), MEM_SUB(x, t)));
        hi = s;
    }
    MEM_SUM_HD void add_square(float x) {                        // + x^2
        const float p = MEM_MUL(x, x);
        add(p);
        lo = MEM_ADD(lo, MEM_FMA(x, x, -p));
    }
    MEM_SUM_HD void sub_square(float x) {
        const float p = MEM_MUL(x, x);
        add(-p);
        lo = MEM_SUB(lo, MEM_FMA(x, x, -p));
    }
    MEM_SUM_HD void settle() {                                   // the two-sum of hi and lo
        const float s = MEM_ADD(hi, lo);
        const float t = MEM_SUB(s, hi);
        lo = MEM_ADD(MEM_SUB(hi, MEM_SUB(s, t)), MEM_SUB(lo, t));
        hi = s;
    }
    // the float that every value within err of hi + lo rounds to; false where there are several (or
    // the sum or the bound is not finite)
    MEM_SUM_HD bool rounds(float err, float* v) const {
        const float f = MEM_ADD(hi, below(lo, err));
        *v = f;
        return f == MEM_ADD(hi, above(lo, err));
    }
};

// A sliding sum of squares w (a window of c terms, then k steps w += x^2 - y^2) and the float of
// w + 1/5.  FP64: w starts as c products added one by one, a step adds the rounded x^2 - y^2.
// Pair: 5 eps^2 b per starting term (2 and 3 for the two additions to lo), 14 per step (2 + 3 + 4 + 5),
// 6 for 1/5; FP64: 2^-53 b per operation.  err() holds them with room for (1 + eps) factors.
struct SlidingSquares {
    Pair w;
    float most = 0.f;                              // of hi
    MEM_SUM_HD void start(float x) {
        w.add_square(x);
        w.settle();
    }
    MEM_SUM_HD void started() { most = w.hi; }
    MEM_SUM_HD void step(float x, float y) {
        w.add_square(x);
        most = fmaxf(most, w.hi);
        w.sub_square(y);
        w.settle();
    }
    // c starting terms, k steps so far
    MEM_SUM_HD bool plus_fifth(int c, int k, float* v) const {
        Pair d = w;
        d.add(0.2f);
        d.lo = MEM_ADD(d.lo, (float)(0.2 - (double)0.2f));
        const float err = (most + 0.2f) * kEps2 * (5.25f * (float)c + 14.5f * (float)k + 8.f);
        return d.rounds(err, v);
    }
};
// the FP64 sum itself
struct SlidingSquares64 {
    double w = 0.0;
    MEM_SUM_HD void start(float x) { w += (double)x * (double)x; }
    MEM_SUM_HD void started() {}
    MEM_SUM_HD void step(float x, float y) {
        w += (double)x * (double)x - (double)y * (double)y;
    }
    MEM_SUM_HD float plus_fifth() const { return (float)(w + 0.2); }
};

// The sum of n <= 64 floats in order.  Multiples of g, the last bit of the smallest term but 0, that
// add up to less than 2^42 g (total <= 2^18 smallest) are exact in FP64 and, with lo below 2^24 g, in
// the pair; that takes in the ties, which such sums hit often.  Else, settled after every kRun terms,
// lo is below (kRun + 1) eps total and the pair within (2 + .. + 9) / 8 eps^2 total per term.
struct PartSum {
    static constexpr int kRun = 8;
    Pair s;
    float total = 0.f, smallest = 3.4e38f;         // of the magnitudes
    MEM_SUM_HD void add(float x) {
        s.add(x);
        const float a = fabsf(x);
        total = MEM_ADD(total, a);
        smallest = a == 0.f ? smallest : fminf(smallest, a);
    }
    MEM_SUM_HD bool value(int n, float* v) const {
        if (!(total < 1e38f)) return false;
        const bool one = s.rounds(total * kEps2 * (6.f * (float)n + 16.f), v);
        if (one) return true;
        *v = MEM_ADD(s.hi, s.lo);
        return total <= 131072.f * smallest;
    }
};

#undef MEM_ADD
#undef MEM_SUB
#undef MEM_MUL
#undef MEM_FMA

}  // namespace mem
