// Host build of the pair sums (manifoldem_python_gb300/csrc/float_sums.cuh): per kind of input, how
// many values were compared, how many the pair did not decide, how many decided ones differ from
// the FP64 sum's float and how many an undecided pair would have got wrong; one line each.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "float_sums.cuh"

using namespace mem;

static bool same(float a, float b) {
    return std::memcmp(&a, &b, sizeof a) == 0 || (std::isnan(a) && std::isnan(b));
}

struct Count {
    long values = 0, undecided = 0, wrong = 0, caught = 0;
    void add(bool decided, float got, float plain, float ref) {
        ++values;
        if (decided) {
            wrong += !same(got, ref);
        } else {
            ++undecided;
            caught += !same(plain, ref);
        }
    }
    void print(const char* name) const {
        std::printf("%s %ld %ld %ld %ld\n", name, values, undecided, wrong, caught);
    }
};

// chains of up to 64 values as a thread of the Wiener kernel walks them
template <class Draw>
static void wiener(const char* name, int chains, int c, Draw draw) {
    Count n;
    std::vector<float> x(c + 65);
    for (int q = 0; q < chains; ++q) {
        draw(x);
        SlidingSquares p;
        SlidingSquares64 r;
        for (int t = c; t > 0; --t) {
            p.start(x[t]);
            r.start(x[t]);
        }
        p.started();
        for (int i = 0; i < 64; ++i) {
            float v;
            const bool ok = p.plus_fifth(c, i, &v);
            Pair d = p.w;
            d.add(0.2f);
            d.lo += (float)(0.2 - (double)0.2f);
            n.add(ok, v, d.hi + d.lo, r.plus_fifth());
            p.step(x[i + 1 + c], x[i + 1]);
            r.step(x[i + 1 + c], x[i + 1]);
        }
    }
    n.print(name);
}

template <class Draw>
static void parts(const char* name, int sums, int terms, Draw draw) {
    Count n;
    for (int q = 0; q < sums; ++q) {
        PartSum p;
        double r = 0.0;
        for (int s = 0; s < terms; ++s) {
            const float x = draw(s);
            p.add(x);
            if (s % PartSum::kRun == PartSum::kRun - 1) p.s.settle();
            r += x;
        }
        float v;
        const bool ok = p.value(terms, &v);
        n.add(ok, v, p.s.hi + p.s.lo, (float)r);
    }
    n.print(name);
}

int main() {
    std::mt19937_64 g(7);
    std::normal_distribution<double> normal;
    std::uniform_real_distribution<double> uni(0.0, 1.0);
    auto ctf = [&](std::vector<float>& x) {
        const double k2 = uni(g) * 0.5;
        for (float& v : x) v = (float)std::sin(-M_PI * (20 + 40 * uni(g)) * k2 * 20 - 0.1);
    };
    wiener("ctf_c20", 15000, 20, ctf);
    wiener("ctf_c1", 8000, 1, ctf);
    wiener("ctf_c200", 1500, 200, ctf);
    wiener("normal", 8000, 20, [&](std::vector<float>& x) {
        for (float& v : x) v = (float)normal(g);
    });
    wiener("six_decades", 8000, 20, [&](std::vector<float>& x) {
        for (float& v : x) v = (float)(normal(g) * std::pow(10.0, 6 * uni(g) - 4));
    });
    wiener("large_leaves", 4000, 5, [&](std::vector<float>& x) {
        for (float& v : x) v = (float)(uni(g) < 0.03 ? 1e4 * normal(g) : normal(g));
    });
    wiener("range_ends", 2000, 4, [&](std::vector<float>& x) {
        for (float& v : x) v = (float)(normal(g) * std::pow(10.0, 80 * uni(g) - 42));
    });
    wiener("zeros", 100, 3, [&](std::vector<float>& x) {
        for (float& v : x) v = 0.f;
    });
    wiener("not_finite", 200, 3, [&](std::vector<float>& x) {
        for (float& v : x) v = uni(g) < 0.02 ? (uni(g) < 0.5 ? INFINITY : NAN) : (float)normal(g);
    });
    for (int terms : {1, 2, 3, 15, 64}) {
        char name[40];
        std::snprintf(name, sizeof name, "normal_%d", terms);
        parts(name, 60000, terms, [&](int) { return (float)normal(g); });
        std::snprintf(name, sizeof name, "decades_%d", terms);
        parts(name, 60000, terms,
              [&](int) { return (float)(normal(g) * std::pow(10.0, 16 * uni(g) - 8)); });
        std::snprintf(name, sizeof name, "short_%d", terms);         // few bits: ties
        parts(name, 60000, terms, [&](int) {
            return (float)std::ldexp((double)(int)(g() % 4096) - 2048, (int)(g() % 26));
        });
        std::snprintf(name, sizeof name, "sparse_%d", terms);
        parts(name, 60000, terms, [&](int) { return uni(g) < 0.7 ? -0.f : (float)normal(g); });
        std::snprintf(name, sizeof name, "cancel_%d", terms);
        float kept = 0.f;
        parts(name, 60000, terms, [&](int s) {
            if (s % 2) return -kept;
            kept = (float)(normal(g) * std::pow(10.0, 12 * uni(g)));
            return s == 0 && uni(g) < 0.5 ? (float)(kept * 1.00001) : kept;
        });
        std::snprintf(name, sizeof name, "range_ends_%d", terms);
        parts(name, 60000, terms,
              [&](int) { return (float)(normal(g) * std::pow(10.0, 84 * uni(g) - 46)); });
        std::snprintf(name, sizeof name, "not_finite_%d", terms);
        parts(name, 20000, terms, [&](int) {
            return uni(g) < 0.1 ? (uni(g) < 0.5 ? INFINITY : -INFINITY) : (float)normal(g);
        });
    }
    return 0;
}
