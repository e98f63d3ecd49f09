// Host build of the fixed-point quadrature (mpgb_fixed.cuh) for
// tests/test_fixed.py, with the same traversal in long double beside it.
#include <cmath>
#include <utility>
#include <vector>

#include "../mpart_gb300/csrc/mpgb_fixed.cuh"

using namespace mpgb;

extern "C" void fx_softplus(const double* x, double* g, double* gp, long n) {
    for (long i = 0; i < n; ++i) {
        bool bad = false;
        uint64_t d = 0;
        const uint64_t v = fx::softPlus<true>((uint64_t)fx::toFixed58(x[i], bad) + (1ull << 63), d);
        // (value as hi + lo, so that the fraction's last bits reach the test)
        g[2 * i] = std::ldexp((double)(v >> 32), -25);
        g[2 * i + 1] = std::ldexp((double)(v & 0xffffffffull), -57);
        gp[2 * i] = std::ldexp((double)(d >> 32), -31);
        gp[2 * i + 1] = std::ldexp((double)(d & 0xffffffffull), -63);
        if (bad) g[2 * i] = NAN;
    }
}

extern "C" void fx_exp(const double* x, double* m, int* E, long n) {
    for (long i = 0; i < n; ++i) {
        bool bad = false;
        const uint64_t v = fx::expMant((uint64_t)fx::toFixed58(x[i], bad) + (1ull << 63), E[i]);
        m[2 * i] = std::ldexp((double)(v >> 32), -30);
        m[2 * i + 1] = std::ldexp((double)(v & 0xffffffffull), -62);
        if (bad) m[2 * i] = NAN;
    }
}

namespace {
constexpr int kNB = 6, kNM = 8;

template <bool EXPR, bool ENV>
void node(const double* b, double a, double Z, long double t, long double& g, long double& gp, long double& ge) {
    long double v = 0, e = 1;
    for (int j = kNB - 1; j >= 0; --j) v = v * t + b[j];
    if (ENV) {
        e = std::exp2(-(long double)Z * t * t);
        v = a + e * v;
    }
    if (EXPR) {
        g = gp = std::exp(v);
    } else {
        const long double x = std::exp(-std::fabs(v));
        g = std::log1p(x) + (v > 0 ? v : 0);
        gp = v > 0 ? 1 / (1 + x) : x / (1 + x);
    }
    ge = gp * e;
}

// Worst differences (of int g, of the moments; Exp: relative to int g) and
// the interval counts of both.
template <bool EXPR, bool ENV>
void one(const double* b, double a, double Z, double xd, double tol, bool simpson, int minSub, double* out) {
    const double rho = simpson ? 0.5 : std::sqrt(0.5);
    const double cw[2] = {1.0 / 3, 4.0 / 3};
    double fw[3] = {1.0 / 15, 4.0 / 5, 8.0 / 15};  // ends, middle, +- rho
    if (simpson) {
        fw[0] = 1.0 / 6;
        fw[1] = 1.0 / 3;
        fw[2] = 2.0 / 3;
    }
    auto frac = [](double w) { return (uint64_t)std::ldexp(w, 64); };
    fx::Rule R{};
    R.rho = frac(rho);
    R.c0 = frac(0.5 * cw[0]);
    R.cM = frac(0.5 * cw[1]);
    R.w0 = frac(0.5 * fw[0]);
    R.wM = frac(0.5 * fw[1]);
    R.w1 = frac(0.5 * fw[2]);
    R.rel = frac(tol);
    auto mul = [](uint64_t x, uint64_t y) {
        return (uint64_t)(((unsigned __int128)x * y + ((unsigned __int128)1 << 63)) >> 64);
    };
    R.mLo[0] = R.mHi[0] = R.w1;
    for (int j = 1; j < fx::kMoments; ++j) {
        R.mLo[j] = mul(R.mLo[j - 1], (1ull << 63) - (R.rho >> 1));
        R.mHi[j] = mul(R.mHi[j - 1], (1ull << 63) + (R.rho >> 1));
    }
    fx::Poly<kNB, ENV> p;
    bool bad = false;
    for (int j = 0; j < kNB; ++j) p.c[j] = (uint64_t)fx::toFixed58(b[j], bad) + (1ull << 63);
    p.a = (uint64_t)fx::toFixed58(a, bad) + (1ull << 63);
    p.wideZ = Z >= 126;
    p.Z = (uint64_t)(Z * (p.wideZ ? 0x1p53 : 0x1p57));
    const double th = tol / xd;
    fx::Threshold thr{(uint64_t)(th * 0x1p57), 0};
    if (EXPR) {
        uint64_t u;
        __builtin_memcpy(&u, &th, 8);
        thr.m = ((u & 0x000fffffffffffffull) | (1ull << 52)) << 10;
        thr.E = (int)(u >> 52) - 1023;
    }
    fx::Sums<kNM> S;
    // (the envelope 2^(-Z t^2) is that of x = sqrt(2 Z ln 2))
    const int ms = ENV ? fx::momentShift(std::sqrt(2.0 * Z * std::log(2.0))) : 0;
    fx::integrate<EXPR, kNB, ENV, kNM>(p, R, 30, minSub, 1 << 16, thr, ms, S);
    long double G = 0, M0 = 0, M[kNM] = {};
    struct Iv { long double lo, hi; int level; };
    std::vector<Iv> st{{0, 1, 0}};
    int n = 0;
    while (!st.empty() && n < 100000) {
        const Iv iv = st.back();
        st.pop_back();
        ++n;
        const long double m = (iv.lo + iv.hi) / 2, h = (iv.hi - iv.lo) / 2;
        const long double t[5] = {iv.lo, m - h * rho, m, m + h * rho, iv.hi};
        const double w[5] = {fw[0], fw[2], fw[1], fw[2], fw[0]};
        long double g[5], gp[5], ge[5], ih = 0;
        for (int i = 0; i < 5; ++i) {
            node<EXPR, ENV>(b, a, Z, t[i], g[i], gp[i], ge[i]);
            ih += h * w[i] * g[i];
        }
        const long double ic = h * (cw[0] * (g[0] + g[4]) + cw[1] * g[2]);
        if ((std::fabs(ih - ic) * xd < std::fmax(tol * ic * xd, (long double)tol) || iv.level == 29) &&
            iv.level >= minSub) {
            G += ih;
            for (int i = 0; i < 5; ++i) {
                M0 += h * w[i] * gp[i];
                long double tp = h * w[i] * ge[i];
                for (int j = 0; j < kNM; ++j, tp *= t[i]) M[j] += tp;
            }
        } else {
            st.push_back({m, iv.hi, iv.level + 1});
            st.push_back({iv.lo, m, iv.level + 1});
        }
    }
    const long double gs = EXPR ? std::ldexp(1.0L, S.E - 62) : 0x1p-57L, ws = EXPR ? gs : 0x1p-62L;
    const long double unit = EXPR ? G : 1.0L;
    out[0] = (double)(std::fabs(S.g * gs - G) / unit);
    out[1] = ENV ? (double)(std::fabs(S.m0 * ws - M0) / unit) : 0.0;
    for (int j = 0; j < kNM; ++j) {
        const long double f = std::ldexp(1.0L, ENV ? -ms * (EXPR ? j : j + 1) : 0);
        out[1] = std::fmax(out[1], (double)(std::fabs(S.m[j] * ws * f - M[j]) / unit));
    }
    out[2] = S.over ? -1 : S.nInt;
    out[3] = n;
}
}  // namespace

extern "C" void fx_integrate(int expr, int env, const double* b, double a, double Z, double xd, double tol,
                             int simpson, int minSub, double* out) {
    if (expr && env) one<true, true>(b, a, Z, xd, tol, simpson, minSub, out);
    else if (expr) one<true, false>(b, a, Z, xd, tol, simpson, minSub, out);
    else if (env) one<false, true>(b, a, Z, xd, tol, simpson, minSub, out);
    else one<false, false>(b, a, Z, xd, tol, simpson, minSub, out);
}
