// Host build of the fixed-point quadrature (mpgb_fixed.cuh) for
// tests/test_fixed_accuracy.py: tight tolerances.
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
