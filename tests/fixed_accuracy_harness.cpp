// Host build of the fixed-point quadrature (mpgb_fixed.cuh) for
// tests/test_fixed_accuracy.py: tight tolerances and
// signed errors.
#include <cmath>
#include <vector>

#include "../mpart_gb300/csrc/mpgb_fixed.cuh"

using namespace mpgb;
typedef long double LD;

namespace {
constexpr int kNB = 6;

fx::Rule rule(double rel) {
    const LD w0 = 1.0L / 30, wM = 0.4L, w1 = 4.0L / 15, r = std::sqrt(0.5L);
    auto frac = [](LD w) { return (uint64_t)std::ldexp(w, 64); };
    fx::Rule R{};
    R.ok = 1;
    R.rho = frac(r);
    R.c0 = frac(1.0L / 6);
    R.cM = frac(2.0L / 3);
    R.w0 = frac(w0);
    R.wM = frac(wM);
    R.w1 = frac(w1);
    R.rel = frac(rel);
    for (int j = 0; j < fx::kMoments; ++j) {
        R.mLo[j] = (uint64_t)(std::ldexp(w1 * std::pow((1 - r) / 2, (LD)j), 64) + 0.5L);
        R.mHi[j] = (uint64_t)(std::ldexp(w1 * std::pow((1 + r) / 2, (LD)j), 64) + 0.5L);
    }
    return R;
}


template <bool EXPR>
void rect(LD v, LD& g, LD& gp) {
    if (EXPR) {
        g = gp = std::exp(v);
    } else {
        const LD x = std::exp(-std::fabs(v));
        g = std::log1p(x) + (v > 0 ? v : 0);
        gp = v > 0 ? 1 / (1 + x) : x / (1 + x);
    }
}

// int g' t^j exp(-(x t)^2 / 2) of the integrand a + exp(-(x t)^2 / 2) sum_j b_j t^j,
// fixed point minus long double, relative to the latter (which subdivides alike).
template <bool EXPR>
void moments(const double* b, double a, double x, double tol, double* err) {
    const fx::Rule R = rule(tol);
    fx::Poly<kNB, true> p;
    bool bad = false;
    for (int j = 0; j < kNB; ++j) p.c[j] = (uint64_t)fx::toFixed58(b[j], bad) + (1ull << 63);
    p.a = (uint64_t)fx::toFixed58(a, bad) + (1ull << 63);
    bad |= !fx::setEnvelope(p, x);
    const int ms = fx::momentShift(x);
    fx::Sums<kNB> S;
    fx::Threshold thr;
    bad |= !fx::threshold<EXPR>(tol / std::fabs(x), tol, thr);
    fx::integrate<EXPR, kNB, true, kNB>(p, R, 30, 0, 1 << 16, thr, ms, S);
    struct Iv { LD lo, hi; };
    std::vector<Iv> st{{0, 1}};
    LD M[kNB] = {};
    const LD r = std::sqrt(0.5L), w[5] = {1.0L / 30, 4.0L / 15, 0.4L, 4.0L / 15, 1.0L / 30};
    while (!st.empty()) {
        const Iv v = st.back();
        st.pop_back();
        const LD m = (v.lo + v.hi) / 2, h = v.hi - v.lo, t[5] = {v.lo, m - h / 2 * r, m, m + h / 2 * r, v.hi};
        LD g[5], e[5], ih = 0;
        for (int i = 0; i < 5; ++i) {
            LD q = 0, gp;
            for (int j = kNB - 1; j >= 0; --j) q = q * t[i] + b[j];
            e[i] = std::exp(-(LD)x * x * t[i] * t[i] / 2);
            rect<EXPR>(a + e[i] * q, g[i], gp);
            e[i] *= gp;
            ih += h * w[i] * g[i];
        }
        const LD ic = h * ((g[0] + g[4]) / 6 + 2 * g[2] / 3), ax = std::fabs((LD)x);
        if (std::fabs(ih - ic) * ax < std::fmax(tol * ic * ax, (LD)tol)) {
            for (int i = 0; i < 5; ++i) {
                LD tp = h * w[i] * e[i];
                for (int j = 0; j < kNB; ++j, tp *= t[i]) M[j] += tp;
            }
        } else {
            st.push_back({m, v.hi});
            st.push_back({v.lo, m});
        }
    }
    const LD unit = EXPR ? std::ldexp(1.0L, S.E - 62) : 0x1p-62L;
    for (int j = 0; j < kNB; ++j) {
        const LD f = (LD)S.m[j] * unit * std::ldexp(1.0L, -ms * (EXPR ? j : j + 1));
        err[j] = bad ? NAN : (double)(f / M[j] - 1);
    }
}
template <bool EXPR>
void tight(const double* b, double x, double absTol, double* out) {
    const fx::Rule R = rule(0.0);
    fx::Poly<kNB, false> p;
    bool bad = false;
    for (int j = 0; j < kNB; ++j) p.c[j] = (uint64_t)fx::toFixed58(b[j], bad) + (1ull << 63);
    p.a = p.Z = 0;
    p.wideZ = false;
    fx::Sums<0> S;
    fx::Threshold thr;
    out[0] = out[1] = 0;
    if (!fx::threshold<EXPR>(absTol / std::fabs(x), 0.0, thr)) return;
    fx::integrate<EXPR, kNB, false, 0>(p, R, 30, 0, 1 << 16, thr, 0, S);
    out[0] = S.over ? -1.0 : S.nInt;
    // the integral, by 4,096 five-point intervals
    LD G = 0;
    const LD r = std::sqrt(0.5L), w[5] = {1.0L / 30, 4.0L / 15, 0.4L, 4.0L / 15, 1.0L / 30};
    for (int q = 0; q < 4096; ++q) {
        const LD h = 1.0L / 4096, m = (q + 0.5L) * h, t[5] = {q * h, m - h / 2 * r, m, m + h / 2 * r, (q + 1) * h};
        for (int i = 0; i < 5; ++i) {
            LD v = 0;
            for (int j = kNB - 1; j >= 0; --j) v = v * t[i] + b[j];
            G += h * w[i] * (EXPR ? std::exp(v) : std::log1p(std::exp(-std::fabs(v))) + (v > 0 ? v : 0));
        }
    }
    out[1] = (double)(std::fabs((EXPR ? std::ldexp((LD)S.g, S.E - 62) : S.g * 0x1p-57L) - G) / (EXPR ? G : 1.0L));
}
}  // namespace

// out: intervals (0: left to FP64, -1: more than 2^16), error of int g (Exp: relative).
extern "C" void fa_tight(int expr, const double* b, double x, double absTol, double* out) {
    if (expr) tight<true>(b, x, absTol, out);
    else tight<false>(b, x, absTol, out);
}

// n points: coefficients b (n x 6), a, x -> the mean of err over them (6).
extern "C" void fa_moment_bias(int expr, const double* b, const double* a, const double* x, long n, double tol,
                               double* mean) {
    LD s[kNB] = {};
    for (long i = 0; i < n; ++i) {
        double e[kNB];
        if (expr) moments<true>(b + i * kNB, a[i], x[i], tol, e);
        else moments<false>(b + i * kNB, a[i], x[i], tol, e);
        for (int j = 0; j < kNB; ++j) s[j] += e[j];
    }
    for (int j = 0; j < kNB; ++j) mean[j] = (double)(s[j] / n);
}

// Intervals reported when the budget runs out (the field is set to -7 before).
extern "C" int fa_over(int budget) {
    const fx::Rule R = rule(0.0);
    fx::Poly<kNB, false> p;
    bool bad = false;
    for (int j = 0; j < kNB; ++j) p.c[j] = (uint64_t)fx::toFixed58(0.5 - 0.3 * j, bad) + (1ull << 63);
    p.a = p.Z = 0;
    p.wideZ = false;
    fx::Sums<0> S;
    S.nInt = -7;
    fx::integrate<false, kNB, false, 0>(p, R, 30, 0, budget, fx::Threshold{1, 0}, 0, S);
    return S.over ? S.nInt : -1;
}
