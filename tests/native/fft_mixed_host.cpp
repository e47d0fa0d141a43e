// Host build of the mixed-radix image transforms (manifoldem_python_gb300/csrc/fft_mixed.cuh): for
// each shape the spectrum of an image, the low-passed image and the inverse of the spectrum, as
// binary floats on standard output.  The passes run task by task in the order of the kernels'
// barriers.
#include <cmath>
#include <cstdio>
#include <vector>

#include "fft_mixed.cuh"

using namespace mem::fft;

template <class Sh>
struct HostBuf {
    mutable std::vector<float2> s;
    HostBuf() : s(Sh::H * Sh::S) {}
    float2& at(int p, int i) const { return s.at(p * Sh::S + i); }
};

template <class Sh>
static void run() {
    constexpr int N = Sh::N, H = Sh::H, R1 = Sh::R1, R2 = Sh::R2;
    std::vector<float2> W(N);
    for (int k = 0; k < N; ++k)
        W[k] = make_float2((float)std::cos(-2 * M_PI * k / N), (float)std::sin(-2 * M_PI * k / N));
    auto pixel = [&](int r, int c) {
        return (float)(std::sin(0.37 * r + 0.011 * c * c) + 0.3 * std::cos(0.9 * c - 0.2 * r * c));
    };
    auto gain = [&](int j, int c) {
        const int f = j < N - j ? j : N - j;
        return 1.0f / (1.0f + 0.01f * f * f + 0.02f * c * c);
    };
    HostBuf<Sh> b;
    auto forward = [&]() {
        for (int p = 0; p < H; ++p)
            for (int c = 0; c < N; ++c)
                b.at(p, Sh::nat(c)) = make_float2(pixel(2 * p, c), pixel(2 * p + 1, c));
        for (int p = 0; p < H; ++p)
            for (int t = 0; t < R2; ++t)
                Sh::template rows_fwd1<true>(b, W.data(), p, t, 0.25f, 2.0f);
        for (int p = 0; p < H; ++p)
            for (int k = 0; k < R1; ++k) Sh::rows_fwd2(b, p, k);
        if (!Sh::DUAL)
            for (int p = 0; p < H; ++p)
                for (int c = 0; c < H; ++c) Sh::cols_split(b, p, c);
        for (int c = 0; c < H; ++c)
            for (int u = 0; u < Sh::kColTasks; ++u) Sh::cols_fwd1(b, W.data(), c, u);
    };
    auto inverse = [&](std::vector<float>& out) {
        for (int c = 0; c < H; ++c)
            for (int u = 0; u < Sh::kColTasks; ++u) Sh::cols_inv2(b, c, u);
        if (!Sh::DUAL)
            for (int p = 0; p < H; ++p)
                for (int c = 0; c < H; ++c) Sh::cols_merge(b, p, c);
        for (int p = 0; p < H; ++p)
            for (int k = 0; k < R1; ++k) Sh::rows_inv1(b, W.data(), p, k);
        for (int p = 0; p < H; ++p)
            for (int t = 0; t < R2; ++t) {
                float2 v[R1];
                Sh::rows_inv2(b, p, t, v);
                for (int m = 0; m < R1; ++m) {
                    out[(2 * p) * N + t + R2 * m] = v[m].x;
                    out[(2 * p + 1) * N + t + R2 * m] = v[m].y;
                }
            }
    };
    // spectrum
    std::vector<float2> spec(N * Sh::HS);
    forward();
    for (int c = 0; c < H; ++c)
        for (int k = 0; k < R1; ++k) {
            float2 v[R2];
            Sh::cols_fwd2(b, c, k, v);
            if (c == 0) Sh::cols_put(b, c, k, v);
            for (int i = 0; i < R2; ++i) spec[(k + R1 * i) * Sh::HS + c] = v[i];
        }
    for (int j = 0; j < N; ++j)
        Sh::packed_split(b, j, &spec[j * Sh::HS], &spec[j * Sh::HS + H]);
    // low-pass
    std::vector<float> low(N * N), back(N * N);
    forward();
    for (int c = 0; c < H; ++c)
        for (int k = 0; k < R1; ++k) {
            float2 v[R2];
            Sh::cols_fwd2(b, c, k, v);
            if (c == 0) {
                Sh::cols_put(b, c, k, v);
                continue;
            }
            for (int i = 0; i < R2; ++i) {
                const float g = gain(k + R1 * i, c);
                v[i] = make_float2(v[i].x * g, v[i].y * g);
            }
            Sh::cols_inv1(b, W.data(), c, k, v);
        }
    for (int j = 0; j <= N / 2; ++j) Sh::packed_filter(b, j, gain(j, 0), gain(j, H));
    for (int k = 0; k < R1; ++k) {
        float2 v[R2];
        Sh::cols_get(b, 0, k, v);
        Sh::cols_inv1(b, W.data(), 0, k, v);
    }
    inverse(low);
    // inverse of the spectrum
    for (int c = 0; c < H; ++c)
        for (int k = 0; k < R1; ++k) {
            float2 v[R2];
            for (int i = 0; i < R2; ++i) {
                const int j = k + R1 * i;
                v[i] = spec[j * Sh::HS + c];
                if (c == 0) {
                    const float2 h = spec[j * Sh::HS + H];
                    v[i] = make_float2(v[i].x - h.y, v[i].y + h.x);
                }
            }
            Sh::cols_inv1(b, W.data(), c, k, v);
        }
    inverse(back);
    const int dims[2] = {N, R1};
    std::fwrite(dims, sizeof(int), 2, stdout);
    std::fwrite(spec.data(), sizeof(float2), spec.size(), stdout);
    std::fwrite(low.data(), sizeof(float), low.size(), stdout);
    std::fwrite(back.data(), sizeof(float), back.size(), stdout);
}

int main() {
    run<MixShape<20, 5, 4>>();
    run<MixShape<48, 6, 8>>();
    run<MixShape<70, 7, 10>>();
    run<MixShape<54, 9, 6>>();
    run<MixShape<66, 11, 6>>();
    run<MixShape<52, 13, 4>>();
    run<MixShape<180, 15, 12>>();
    run<MixShape<192, 12, 16>>();
    run<MixShape<196, 14, 14>>();
    run<MixShape<250, 25, 10>>();
    run<MixShape<256, 16, 16>>();
    run<MixShape<300, 15, 20>>();
    run<MixShape<144, 8, 18>>();
    run<MixShape<360, 20, 18>>();
    return 0;
}
