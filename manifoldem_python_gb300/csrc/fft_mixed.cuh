// Real 2D transforms of N x N images for N = R1 R2 (R2 even), as passes over one buffer in shared
// memory: the arithmetic and index maps of image_fft_mixed.cu.  Host-compilable, so that the
// passes can be checked against numpy without a GPU.
//
// dft_any<R, DIR>: an in-register DFT of any length with prime factors up to 23 (powers of
// two up to 16 are those of fft_radix.cuh; odd primes sum the half-length cosine and sine
// products; composite lengths are Cooley-Tukey with constant twiddles).
//
// MixShape<N, R1, R2>: the transform.  Two real rows (2p, 2p+1) form one complex row Z_p (H =
// N/2 rows); the row spectra are separated into H columns, the real columns 0 and N/2 packed into
// one.  An N-point DFT is R1 x R2 in two passes: pass 1 takes elements t + R2 m (m < R1), a
// length-R1 DFT and the twiddle W^(t k1), in place; pass 2 takes the R2 consecutive elements of
// group k1 and a length-R2 DFT, in place, which leaves frequency k1 + R1 k2 at place k2 of group
// k1.  The inverse passes read that order.  Element a of column c sits in pair-row a/2 at the
// place of frequency c (a even) or N - c (a odd; N/2 for the packed column), the places of the
// row spectra that it is computed from, so that every pass is in place within a thread.  The
// separation of the paired rows needs both places: for R1 <= 16 a pass-1 thread of the columns
// takes the even and the odd t of a pair (2 R1 values in registers); for longer R1 it is a pass
// of its own.
// Storage: a group of R2 places is padded to LP = R2 + 1 (odd: consecutive columns, which differ
// in the group, fall in different banks) and a pair-row to an odd length S (consecutive pair-rows
// in different banks).
#pragma once

#include "fft_radix.cuh"

namespace mem {
namespace fft {

// cos and sin of 2 pi j / R, j < R, in double at compile time (Taylor series after reduction to
// an eighth of a turn)
MEM_HD constexpr double taylor_cos(double x) {
    double t = 1.0, s = 1.0;
    for (int i = 1; i < 14; ++i) {
        t *= -x * x / ((2 * i - 1) * (2 * i));
        s += t;
    }
    return s;
}
MEM_HD constexpr double taylor_sin(double x) {
    double t = x, s = x;
    for (int i = 1; i < 14; ++i) {
        t *= -x * x / ((2 * i) * (2 * i + 1));
        s += t;
    }
    return s;
}
MEM_HD constexpr double cos_turn(int j, int R) {
    j %= R;
    if (2 * j > R) j = R - j;                      // [0, 1/2]
    const double tau = 6.283185307179586476925;
    if (8 * j <= R) return taylor_cos(tau * j / R);
    if (8 * j <= 3 * R) return taylor_sin(tau * (R - 4 * j) / (4.0 * R));
    return -taylor_cos(tau * (R - 2 * j) / (2.0 * R));
}
MEM_HD constexpr double sin_turn(int j, int R) {   // cos of a quarter turn less
    return cos_turn(4 * (j % R) + 3 * R, 4 * R);
}
template <int R>
struct Trig {
    float c[R], s[R];
    MEM_HD constexpr Trig() : c(), s() {
        for (int j = 0; j < R; ++j) {
            c[j] = (float)cos_turn(j, R);
            s[j] = (float)sin_turn(j, R);
        }
    }
};

MEM_HD float2 cfma(float2 a, float s, float2 acc) {          // a s + acc
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 1000
    return __ffma2_rn(a, make_float2(s, s), acc);
#else
    return make_float2(a.x * s + acc.x, a.y * s + acc.y);
#endif
}

template <int P, int DIR>
MEM_HD void dft_odd_prime(float2* v) {
    constexpr int H = (P - 1) / 2;
    constexpr Trig<P> T;
    float2 s[H], d[H];
#pragma unroll
    for (int j = 0; j < H; ++j) {
        s[j] = cadd(v[1 + j], v[P - 1 - j]);
        d[j] = csub(v[1 + j], v[P - 1 - j]);
    }
    const float2 x0 = v[0];
#pragma unroll
    for (int k = 1; k <= H; ++k) {
        float2 a = x0, b = make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 0; j < H; ++j) {
            a = cfma(s[j], T.c[((j + 1) * k) % P], a);
            b = cfma(d[j], T.s[((j + 1) * k) % P], b);
        }
        const float2 r = rot90<DIR>(b);            // -DIR i b
        v[k] = cadd(a, r);
        v[P - k] = csub(a, r);
    }
    float2 t = x0;
#pragma unroll
    for (int j = 0; j < H; ++j) t = cadd(t, s[j]);
    v[0] = t;
}

MEM_HD constexpr int first_factor(int R) {                // the pass-1 length of a composite R
    return R % 8 == 0 && R > 8 && R != 16 ? 8
           : R % 4 == 0 && R > 4 ? 4
           : R % 2 == 0 && R > 2 ? 2
           : R % 3 == 0 && R > 3 ? 3
           : R % 5 == 0 && R > 5 ? 5
           : R;
}

template <int R, int DIR>
MEM_HD void dft_any(float2* v) {
    if constexpr (R == 2) {
        const float2 a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    } else if constexpr (R == 4 || R == 8 || R == 16) {
        dft<R, DIR>(v);
    } else if constexpr (first_factor(R) == R) {
        dft_odd_prime<R, DIR>(v);
    } else {
        constexpr int P = first_factor(R), Q = R / P;
        constexpr Trig<R> T;
#pragma unroll
        for (int b = 0; b < Q; ++b) {
            float2 u[P];
#pragma unroll
            for (int a = 0; a < P; ++a) u[a] = v[Q * a + b];
            dft_any<P, DIR>(u);
#pragma unroll
            for (int k = 0; k < P; ++k)
                v[Q * k + b] = b * k ? cmul(u[k], make_float2(T.c[b * k], -DIR * T.s[b * k])) : u[k];
        }
        float2 y[R];
#pragma unroll
        for (int k = 0; k < P; ++k) {
            float2 u[Q];
#pragma unroll
            for (int b = 0; b < Q; ++b) u[b] = v[Q * k + b];
            dft_any<Q, DIR>(u);
#pragma unroll
            for (int j = 0; j < Q; ++j) y[k + P * j] = u[j];
        }
#pragma unroll
        for (int k = 0; k < R; ++k) v[k] = y[k];
    }
}

// Buf: an object with float2& at(int p, int i), place i of pair-row p (0 <= p < H); W: the N
// twiddles exp(-2 pi i k / N).
template <int N_, int R1_, int R2_>
struct MixShape {
    static constexpr int N = N_, R1 = R1_, R2 = R2_;
    static constexpr int H = N / 2, HS = H + 1, LP = R2 + 1, S = (R1 * LP) | 1;
    static constexpr int HR = R2 / 2;
    static constexpr bool DUAL = R1 <= 16;
    static_assert(R1 * R2 == N && R2 % 2 == 0, "N = R1 R2 with an even R2");

    static MEM_HD int pos(int k) { return (k % R1) * LP + k / R1; }     // place of frequency k
    static MEM_HD int nat(int b) { return (b / R2) * LP + b % R2; }     // place of element b
    static MEM_HD int odd_col(int c) { return c == 0 ? H : N - c; }

    // rows, pass 1, from registers: v[m] = element t + R2 m
    template <class Buf>
    static MEM_HD void rows_fwd1_store(const Buf& b, const float2* W, int p, int t, float2* v) {
        dft_any<R1, 1>(v);
#pragma unroll
        for (int k = 0; k < R1; ++k) b.at(p, k * LP + t) = k ? cmul(v[k], W[t * k]) : v[k];
    }
    template <bool NORM, class Buf>
    static MEM_HD void rows_fwd1(const Buf& b, const float2* W, int p, int t, float mean, float inv) {
        float2 v[R1];
#pragma unroll
        for (int m = 0; m < R1; ++m) {
            const float2 z = b.at(p, m * LP + t);
            v[m] = NORM ? make_float2((z.x - mean) * inv, (z.y - mean) * inv) : z;
        }
        rows_fwd1_store(b, W, p, t, v);
    }
    template <class Buf>
    static MEM_HD void rows_fwd2(const Buf& b, int p, int k1) {
        float2 v[R2];
#pragma unroll
        for (int i = 0; i < R2; ++i) v[i] = b.at(p, k1 * LP + i);
        dft_any<R2, 1>(v);
#pragma unroll
        for (int i = 0; i < R2; ++i) b.at(p, k1 * LP + i) = v[i];
    }
    // z = Z_p[c], y = Z_p[N - c] -> (row 2p, row 2p+1) of column c, and back
    static MEM_HD void split(bool packed, float2 z, float2 y, float2* e, float2* o) {
        if (packed) {
            *e = make_float2(z.x, y.x);
            *o = make_float2(z.y, y.y);
        } else {
            *e = make_float2(0.5f * (z.x + y.x), 0.5f * (z.y - y.y));
            *o = make_float2(0.5f * (z.y + y.y), 0.5f * (y.x - z.x));
        }
    }
    static MEM_HD void merge(bool packed, float2 e, float2 o, float2* z, float2* y) {
        if (packed) {
            *z = make_float2(e.x, o.x);
            *y = make_float2(e.y, o.y);
        } else {
            *z = make_float2(e.x - o.y, e.y + o.x);
            *y = make_float2(e.x + o.y, o.x - e.y);
        }
    }
    template <class Buf>
    static MEM_HD void cols_split(const Buf& b, int p, int c) {               // R1 > 16 only
        float2 &z = b.at(p, pos(c)), &y = b.at(p, pos(odd_col(c)));
        float2 e, o;
        split(c == 0, z, y, &e, &o);
        z = e;
        y = o;
    }
    template <class Buf>
    static MEM_HD void cols_merge(const Buf& b, int p, int c) {
        float2 &e = b.at(p, pos(c)), &o = b.at(p, pos(odd_col(c)));
        float2 z, y;
        merge(c == 0, e, o, &z, &y);
        e = z;
        o = y;
    }
    // columns, pass 1: DUAL: u = t / 2 < HR, both parities; else u = t < R2 of split columns
    template <class Buf>
    static MEM_HD void cols_fwd1(const Buf& b, const float2* W, int c, int u) {
        const int q0 = pos(c), q1 = pos(odd_col(c));
        if constexpr (DUAL) {
            float2 e[R1], o[R1];
#pragma unroll
            for (int m = 0; m < R1; ++m)
                split(c == 0, b.at(u + HR * m, q0), b.at(u + HR * m, q1), &e[m], &o[m]);
            dft_any<R1, 1>(e);
            dft_any<R1, 1>(o);
#pragma unroll
            for (int k = 0; k < R1; ++k) {
                b.at(u + HR * k, q0) = k ? cmul(e[k], W[2 * u * k]) : e[k];
                b.at(u + HR * k, q1) = k ? cmul(o[k], W[(2 * u + 1) * k]) : o[k];
            }
        } else {
            const int q = (u & 1) ? q1 : q0;
            float2 v[R1];
#pragma unroll
            for (int m = 0; m < R1; ++m) v[m] = b.at(u / 2 + HR * m, q);
            dft_any<R1, 1>(v);
#pragma unroll
            for (int k = 0; k < R1; ++k) b.at(u / 2 + HR * k, q) = k ? cmul(v[k], W[u * k]) : v[k];
        }
    }
    static constexpr int kColTasks = DUAL ? HR : R2;                    // pass-1 tasks per column
    // columns, pass 2: v[k2] = Y[k1 + R1 k2] of column c
    template <class Buf>
    static MEM_HD void cols_fwd2(const Buf& b, int c, int k1, float2* v) {
        const int q0 = pos(c), q1 = pos(odd_col(c));
#pragma unroll
        for (int t = 0; t < R2; ++t) v[t] = b.at(HR * k1 + t / 2, (t & 1) ? q1 : q0);
        dft_any<R2, 1>(v);
    }
    // the spectrum Y[k1 + R1 k2] = v[k2] as it is, in the places that pass 2 reads
    template <class Buf>
    static MEM_HD void cols_put(const Buf& b, int c, int k1, const float2* v) {
        const int q0 = pos(c), q1 = pos(odd_col(c));
#pragma unroll
        for (int t = 0; t < R2; ++t) b.at(HR * k1 + t / 2, (t & 1) ? q1 : q0) = v[t];
    }
    template <class Buf>
    static MEM_HD void cols_get(const Buf& b, int c, int k1, float2* v) {
        const int q0 = pos(c), q1 = pos(odd_col(c));
#pragma unroll
        for (int t = 0; t < R2; ++t) v[t] = b.at(HR * k1 + t / 2, (t & 1) ? q1 : q0);
    }
    template <class Buf>
    static MEM_HD float2& col_at(const Buf& b, int c, int j) {                // Y[j] as cols_put left it
        const int k1 = j % R1, k2 = j / R1;
        return b.at(HR * k1 + k2 / 2, (k2 & 1) ? pos(odd_col(c)) : pos(c));
    }
    template <class Buf>
    static MEM_HD void cols_inv1(const Buf& b, const float2* W, int c, int k1, float2* v) {
        const int q0 = pos(c), q1 = pos(odd_col(c));
        dft_any<R2, -1>(v);
#pragma unroll
        for (int t = 0; t < R2; ++t)
            b.at(HR * k1 + t / 2, (t & 1) ? q1 : q0) = t ? cmulc(v[t], W[t * k1]) : v[t];
    }
    template <class Buf>
    static MEM_HD void cols_inv2(const Buf& b, int c, int u) {
        const int q0 = pos(c), q1 = pos(odd_col(c));
        if constexpr (DUAL) {
            float2 e[R1], o[R1];
#pragma unroll
            for (int k = 0; k < R1; ++k) {
                e[k] = b.at(u + HR * k, q0);
                o[k] = b.at(u + HR * k, q1);
            }
            dft_any<R1, -1>(e);
            dft_any<R1, -1>(o);
#pragma unroll
            for (int m = 0; m < R1; ++m)
                merge(c == 0, e[m], o[m], &b.at(u + HR * m, q0), &b.at(u + HR * m, q1));
        } else {
            const int q = (u & 1) ? q1 : q0;
            float2 v[R1];
#pragma unroll
            for (int k = 0; k < R1; ++k) v[k] = b.at(u / 2 + HR * k, q);
            dft_any<R1, -1>(v);
#pragma unroll
            for (int m = 0; m < R1; ++m) b.at(u / 2 + HR * m, q) = v[m];
        }
    }
    template <class Buf>
    static MEM_HD void rows_inv1(const Buf& b, const float2* W, int p, int k1) {
        float2 v[R2];
#pragma unroll
        for (int i = 0; i < R2; ++i) v[i] = b.at(p, k1 * LP + i);
        dft_any<R2, -1>(v);
#pragma unroll
        for (int i = 0; i < R2; ++i) b.at(p, k1 * LP + i) = i ? cmulc(v[i], W[i * k1]) : v[i];
    }
    // v[m] = (row 2p, row 2p+1) at element t + R2 m
    template <class Buf>
    static MEM_HD void rows_inv2(const Buf& b, int p, int t, float2* v) {
#pragma unroll
        for (int k = 0; k < R1; ++k) v[k] = b.at(p, k * LP + t);
        dft_any<R1, -1>(v);
    }
    // the packed column's low-pass for the pair (j, N - j): Y' = Y gp + conj Y[-j] gm and the same
    // for -j, with g0 = G(j, 0), gh = G(j, N/2), gp = (g0 + gh) / 2, gm = (g0 - gh) / 2
    template <class Buf>
    static MEM_HD void packed_filter(const Buf& b, int j, float g0, float gh) {
        const int jm = j == 0 ? 0 : N - j;
        float2 &a = col_at(b, 0, j), &m = col_at(b, 0, jm);
        const float gp = 0.5f * (g0 + gh), gm = 0.5f * (g0 - gh);
        const float2 x = a, y = m;
        a = make_float2(x.x * gp + y.x * gm, x.y * gp - y.y * gm);
        if (jm != j) m = make_float2(y.x * gp + x.x * gm, y.y * gp - x.y * gm);
    }
    // columns 0 and N/2 at row j from the packed column
    template <class Buf>
    static MEM_HD void packed_split(const Buf& b, int j, float2* y0, float2* yh) {
        const float2 x = col_at(b, 0, j), m = col_at(b, 0, j == 0 ? 0 : N - j);
        *y0 = make_float2(0.5f * (x.x + m.x), 0.5f * (x.y - m.y));
        *yh = make_float2(0.5f * (x.y + m.y), 0.5f * (m.x - x.x));
    }
};

}  // namespace fft
}  // namespace mem
