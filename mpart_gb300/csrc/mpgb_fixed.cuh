// 64-bit fixed-point arithmetic for the quadrature of the rectified integrand.
//
// Why.  A GB300 SM issues FP64 at 2 lanes a clock (measured: 1.6, DFMA or
// DADD) but 32 x 32 + 64-bit integer multiply-adds (IMAD.WIDE) at 55 and
// integer additions at 115.  A quadrature node of the adaptive rule is an
// exponential, a logarithm, a reciprocal and a short polynomial on arguments
// of known range, so it can be carried in 64-bit fixed point: a product's high
// word is three IMAD.WIDE, a twentieth of a DFMA's time.  The fraction has 57
// to 63 bits, so every step rounds at 2^-57 or below where a double near 1
// rounds at 2^-53: the integrand, its weighted sums and the error estimate
// that drives the subdivision are closer to the exact ones than in FP64 where
// they are of ordinary size.  Values far below it have fewer digits than a
// double: such quadratures, and arguments outside the range (|d_D f| possibly
// above 31, non-finite values, other rules), keep the FP64 path (integrateFixed
// in mpgb_kernels.cuh lists them).
//
// The functions are plain C++ on uint64_t, the same on the host (tests) and
// the device.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define MPGB_FX_TABLE __device__ const
#else
#define MPGB_FX_TABLE static const
#endif

#include "mpgb_fixed_tables.h"

#ifdef __CUDACC__
#define MPGB_HD __device__ __forceinline__
#else
#define MPGB_HD inline
#endif

namespace mpgb {
namespace fx {

MPGB_HD uint32_t hi32(uint64_t x) { return (uint32_t)(x >> 32); }
MPGB_HD uint32_t lo32(uint64_t x) { return (uint32_t)x; }
// a b + c of 32-bit factors and a 64-bit addend: one IMAD.WIDE each.
#ifdef __CUDA_ARCH__
MPGB_HD uint64_t mulWide(uint32_t a, uint32_t b) {
    uint64_t r;
    asm("mul.wide.u32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
    return r;
}
MPGB_HD uint64_t madWide(uint32_t a, uint32_t b, uint64_t c) {
    uint64_t r;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}
MPGB_HD int64_t madWideS(int32_t a, int32_t b, int64_t c) {
    int64_t r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}
#else
MPGB_HD uint64_t mulWide(uint32_t a, uint32_t b) { return (uint64_t)a * b; }
MPGB_HD uint64_t madWide(uint32_t a, uint32_t b, uint64_t c) { return (uint64_t)a * b + c; }
MPGB_HD int64_t madWideS(int32_t a, int32_t b, int64_t c) { return (int64_t)a * b + c; }
#endif

// a b / 2^64 rounded, for a + b <= 2^64; the product of the low words is left
// out and its mean added with the rounding (zero stays zero).
MPGB_HD uint64_t mulhi(uint64_t a, uint64_t b) {
    const uint64_t mid = madWide(hi32(a), lo32(b), madWide(lo32(a), hi32(b), 0xC0000000ull));
    return madWide(hi32(a), hi32(b), hi32(mid));
}

// The same for any a, b: two middle products, each with its rounding and half
// the mean of the low one.
MPGB_HD uint64_t mulhiAny(uint64_t a, uint64_t b) {
    const uint64_t m1 = madWide(lo32(a), hi32(b), 0xA0000000ull), m2 = madWide(hi32(a), lo32(b), 0xA0000000ull);
    return madWide(hi32(a), hi32(b), hi32(m1)) + hi32(m2);
}

// floor(a b / 2^32).
MPGB_HD uint64_t mul32(uint64_t a, uint32_t b) { return madWide(hi32(a), b, hi32(mulWide(lo32(a), b))); }

// a b / 2^32, rounded; ties up, or down with down = 1.
MPGB_HD uint64_t mul32Round(uint64_t a, uint32_t b, uint32_t down = 0) {
    return madWide(hi32(a), b, hi32(madWide(lo32(a), b, (uint64_t)(0x80000000u - down))));
}

// a b / 2^32 of two 32-bit numbers, rounded.
MPGB_HD uint32_t hi(uint32_t a, uint32_t b) { return hi32(madWide(a, b, 0x80000000ull)); }

MPGB_HD uint64_t shr(uint64_t x, int n) { return n < 64 ? x >> n : 0; }
// x / 2^n rounded to nearest (n < 0: x 2^-n).
MPGB_HD uint64_t scaleRound(uint64_t x, int n) {
    return n < 0 ? x << -n : (n < 64 ? (x + ((1ull << n) >> 1)) >> n : 0);
}
// The same with ties to even.
MPGB_HD uint64_t scaleEven(uint64_t x, int n) {
    return n <= 0 ? x << -n : (n < 64 ? (x + ((1ull << (n - 1)) - 1) + ((x >> n) & 1)) >> n : 0);
}
// x / 2^n rounded to nearest, n >= 0.
MPGB_HD uint64_t shrRound(uint64_t x, int n) { return n < 64 ? (x + ((1ull << n) >> 1)) >> n : 0; }

#ifdef __CUDA_ARCH__
MPGB_HD uint64_t expTab(uint32_t j) { return __ldg((const unsigned long long*)kExpTab + j); }
MPGB_HD void logTab(uint32_t j, uint64_t& lg, uint32_t& inv) {
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(kLogTab) + j);
    lg = ((uint64_t)v.y << 32) | v.x;
    inv = v.z;
}
#else
MPGB_HD uint64_t expTab(uint32_t j) { return kExpTab[j]; }
MPGB_HD void logTab(uint32_t j, uint64_t& lg, uint32_t& inv) {
    lg = kLogTab[j].lg;
    inv = kLogTab[j].inv;
}
#endif

// 2^-W for W with 57 fraction bits: the mantissa 2^-frac(W) in (1/2, 1), 63
// fraction bits, and the integer part n (2^-W = mantissa 2^-n).
MPGB_HD uint64_t exp2neg(uint64_t W, int& n) {
    n = (int)(hi32(W) >> 25);
    const uint64_t T = expTab((hi32(W) >> 20) & 31);
    const uint64_t s = (W << 12) >> 1;  // 16 r, r = the fraction below the table's step
    const uint32_t R = hi32(s);
    uint32_t q = kE6 - hi(R, kE7);
    q = kE5 - hi(R, q);
    q = kE4 - hi(R, q);
    const uint64_t q3 = kE3 - ((uint64_t)hi(R, q) << 11);
    const uint64_t q2 = kE2 - mulhi(s, q3);
    const uint64_t q1 = kE1 - mulhi(s, q2);
    return T - mulhi(T, mulhi(s, q1));
}

// exp(-u), u with 58 fraction bits, u < 32: 63 fraction bits, below 1.
MPGB_HD uint64_t expNeg(uint64_t u) {
    int n;
    const uint64_t m = exp2neg(mulhiAny(u, kLog2e63), n);
    return m >> n;
}

// log(1 + e) (63 fraction bits) for e in [0, 1) with 63, and with RECIP
// 1 / (1 + e) (63 fraction bits).  1 + e times a tabulated reciprocal is
// 1 + r, r < 1/32: log1p(r) by its series; the reciprocal from its series to
// 30 bits and one Newton step.
template <bool RECIP>
MPGB_HD uint64_t log1p(uint64_t e, uint64_t& recip) {
    uint64_t lg;
    uint32_t inv;
    logTab(hi32(e) >> 26, lg, inv);
    const uint64_t v = e | 0x8000000000000000ull;  // 1 + e
    const uint64_t s = (mul32(v, inv) << 7) >> 1;  // 16 r (62 fraction bits of 1 + r)
    const uint32_t R = hi32(s);
    uint32_t q = kL9 - hi(R, kL10);
    q = kL8 - hi(R, q);
    q = kL7 - hi(R, q);
    q = kL6 - hi(R, q);
    q = kL5 - hi(R, q);
    const uint64_t q4 = kL4 - ((uint64_t)hi(R, q) << 11);
    const uint64_t q3 = kL3 - mulhi(s, q4);
    const uint64_t q2 = kL2 - mulhi(s, q3);
    const uint64_t q1 = kL1 - mulhi(s, q2);
    if constexpr (RECIP) {
        uint32_t z = (1u << 12) - hi(R, 1u << 8);
        z = (1u << 16) - hi(R, z);
        z = (1u << 20) - hi(R, z);
        z = (1u << 24) - hi(R, z);
        z = hi(R, (1u << 28) - hi(R, z));     // 1 - 1 / (1 + r), 32 fraction bits
        const uint32_t y = inv - hi(inv, z);  // 31 fraction bits
        const int64_t eps = (int64_t)(0x4000000000000000ull - mul32(v, y));  // 1 - v y, 62 fraction bits
        const int64_t c = (int64_t)(int32_t)(y >> 1) * (int32_t)(eps >> 3);  // y eps, 89 fraction bits
        recip = ((uint64_t)y << 32) + (uint64_t)(c >> 26);
    }
    return lg + (mulhi(s, q1) >> 1);
}

// SoftPlus at d = D / 2^58 - 32, |d| < 32: g = log(1 + e^-|d|) + max(d, 0)
// with 57 fraction bits and, with DERIV, g' = 1 / (1 + e^-d) with 63.
template <bool DERIV>
MPGB_HD uint64_t softPlus(uint64_t D, uint64_t& gp) {
    const bool pos = (D >> 63) != 0;
    const uint64_t x = D ^ 0x8000000000000000ull;
    const uint64_t u = pos ? x : 0 - x;
    uint64_t r = 0;
    const uint64_t l = log1p<DERIV>(expNeg(u), r);
    if constexpr (DERIV) gp = pos ? r : 0x8000000000000000ull - r;
    return ((l + 32) >> 6) + (pos ? u >> 1 : 0);
}

// e^d at d = D / 2^58 - 32, |d| < 32: m 2^E with m in [1/2, 1), 62 fraction bits.
MPGB_HD uint64_t expMant(uint64_t D, int& E) {
    // 64 - d log2(e) = (64 + 32 log2(e)) - (d + 32) log2(e), 57 fraction bits
    constexpr uint64_t kBias = (64ull << 57) + (kLog2e63 >> 1);
    int n;
    const uint64_t m = exp2neg(kBias - mulhiAny(D, kLog2e63), n);
    E = 64 - n;
    return m >> 1;
}

// x with 58 fraction bits; bad is set for |x| >= 32 and non-finite x.
MPGB_HD int64_t toFixed58(double x, bool& bad) {
#ifdef __CUDA_ARCH__
    const uint64_t b = (uint64_t)__double_as_longlong(x);
#else
    uint64_t b;
    __builtin_memcpy(&b, &x, 8);
#endif
    const int e = (int)((b >> 52) & 0x7ff);
    if (e > 1027) bad = true;
    const uint64_t m = ((b & 0x000fffffffffffffull) | 0x0010000000000000ull) << 10;
    const int sh = 1027 - e;  // (subnormal x: shifted out)
    const int64_t v = sh <= 0 ? (int64_t)m : (sh < 64 ? (int64_t)(((m >> (sh - 1)) + 1) >> 1) : 0);
    return (b >> 63) ? -v : v;
}

// x 2^sc rounded to an integer, for |x| 2^sc < 2^62; finite x.
MPGB_HD int64_t toFixed(double x, int sc) {
#ifdef __CUDA_ARCH__
    const uint64_t b = (uint64_t)__double_as_longlong(x);
#else
    uint64_t b;
    __builtin_memcpy(&b, &x, 8);
#endif
    const int e = (int)((b >> 52) & 0x7ff);
    const int sh = 1084 - e - sc;  // (62 - the product's exponent) - 1
    if (e == 0 || sh > 62) return 0;  // below half a unit (subnormals too)
    const uint64_t m = ((b & 0x000fffffffffffffull) | 0x0010000000000000ull) << 10;
    const int64_t v = sh < 0 ? (int64_t)m : (int64_t)(((m >> sh) + 1) >> 1);
    return (b >> 63) ? -v : v;
}

// The exponent bound of a double: |x| < 2^expBound(x) (finite x; a very small
// number for 0); 1025 for infinities and NaN.
MPGB_HD int expBound(double x) {
#ifdef __CUDA_ARCH__
    const uint32_t h = (uint32_t)__double2hiint(x);
#else
    uint64_t b;
    __builtin_memcpy(&b, &x, 8);
    const uint32_t h = (uint32_t)(b >> 32);
#endif
    return (int)((h >> 20) & 0x7ff) - 1022;
}

// The significand of a double with its top bit at 2^63: |x| = this times
// 2^(expBound(x) - 64) (not for subnormals).
MPGB_HD uint64_t mantissa64(double x) {
#ifdef __CUDA_ARCH__
    const uint64_t b = (uint64_t)__double_as_longlong(x);
#else
    uint64_t b;
    __builtin_memcpy(&b, &x, 8);
#endif
    return ((b & 0x000fffffffffffffull) | 0x0010000000000000ull) << 11;
}

// Products of leading-basis values in fixed point: phi = (h 2^27 + l) 2^-57,
// 0 <= l < 2^27, |phi| <= 1, times a basis value (bh 2^31 + bl) 2^-58, |B| < 16.
// The constant is the mean of what the shift and the left-out product of the
// low words drop.
struct Limbs {
    int32_t h, l;
};
MPGB_HD Limbs limbMul(Limbs p, int32_t bh, int32_t bl) {
    const int64_t m = madWideS(p.l << 4, bh, madWideS(p.h, bl, 3ll << 29));
    const int64_t v = madWideS(p.h, bh, m >> 31);
    return {(int32_t)(v >> 27), (int32_t)v & 0x07ffffff};
}

// The adaptive rule in fixed point: three coarse and five fine nodes (-1, 0, 1
// and -rho, rho) with weights scaled to sum to 1, 64 fraction bits; mLo, mHi:
// the weights of -rho and rho times their position in [0, 1] to the power j.
constexpr int kMoments = 12;
struct Rule {
    int ok;
    uint64_t rho, c0, cM, w0, wM, w1, rel;
    uint64_t mLo[kMoments], mHi[kMoments];
};


// d_D f along one quadrature, t in [0, 1]: sum_j c_j t^j (ENV false) or
// a + exp2(-Z t^2) sum_j c_j t^j (the envelope of the Hermite functions).
// c_0 and a carry the bias 32 (2^63) that keeps every partial sum positive.
template <int NB, bool ENV>
struct Poly {
    uint64_t c[NB];  // 58 fraction bits; every entry biased
    uint64_t a;      // 58 fraction bits, biased
    uint64_t Z;      // 57 fraction bits, or 53 where it is 126 or more (wideZ)
    bool wideZ;
};

// The envelope 2^(-Z t^2) for t2 = t^2, t2 = 1 by its flag: m 2^-n, m with 63
// fraction bits.
struct Envelope {
    uint64_t m;
    int n;
};
template <int NB>
MPGB_HD Envelope envelope(const Poly<NB, true>& p, uint64_t t2, bool one) {
    Envelope e{0, 127};
    uint64_t W = one ? p.Z : mulhiAny(t2, p.Z);
    if (p.wideZ) {
        if (W >> 60) return e;
        W <<= 4;
    }
    e.m = exp2neg(W, e.n);
    return e;
}

// Z and its format for |x_D| < 52.6 (false beyond), from 64-bit products: in
// FP64 the constant's own rounding would be common to all points.
template <int NB>
MPGB_HD bool setEnvelope(Poly<NB, true>& p, double x) {
    constexpr uint64_t kHalfLog2e = 0xb8aa3b295c17f0bcull;  // 1 / (2 ln 2), 64 fraction bits
    const int e = expBound(x);
    const uint64_t X = mantissa64(x);
    const uint64_t z = mulhiAny(mulhiAny(X, X), kHalfLog2e);  // x^2 / (2 ln 2) = z 2^(2 e - 64)
    const bool ok = e < 6 || (e == 6 && z < (2000ull << 52));
    p.wideZ = e > 4 || (e == 4 && z >= (126ull << 56));
    p.Z = ok ? scaleRound(z, (p.wideZ ? 11 : 7) - 2 * e) : 0;
    return ok;
}

// sum_j c_j t^j, biased; t with 64 fraction bits.  acc' = acc + 2^63 steps as
// c_j' + t acc' - t 2^63.
template <int NB, bool ENV>
MPGB_HD uint64_t horner(const Poly<NB, ENV>& p, uint64_t t) {
    uint64_t acc = p.c[NB - 1];
    const uint64_t th = t >> 1;
#pragma unroll
    for (int j = NB - 2; j >= 0; --j) acc = (p.c[j] - th) + mulhiAny(acc, t);
    return acc;
}

// A node: g (SoftPlus: 57 fraction bits; Exp: mantissa with 62 and exponent
// E), f = g' (62 fraction bits; Exp: g itself), fe = g' times the envelope's
// mantissa and n its exponent (fe 2^-n).
struct Node {
    uint64_t g, f, fe;
    int E, n;
};

template <bool EXPR, bool DERIV>
MPGB_HD void rect(uint64_t D, Node& o, uint64_t& gp63) {
    o.E = 0;
    o.f = o.fe = 0;
    o.n = 0;
    gp63 = 0;
    if constexpr (EXPR) {
        o.g = expMant(D, o.E);
        if constexpr (DERIV) {
            o.f = o.g;
            gp63 = o.g << 1;
        }
    } else {
        o.g = softPlus<DERIV>(D, gp63);
        if constexpr (DERIV) o.f = gp63 >> 1;
    }
}

template <bool EXPR, bool DERIV, int NB, bool ENV>
MPGB_HD Node nodeAt(const Poly<NB, ENV>& p, uint64_t t) {
    Node o;
    uint64_t gp;
    if constexpr (ENV) {
        const Envelope v = envelope(p, mulhiAny(t, t), false);
        const uint64_t e = shrRound(v.m, v.n);
        rect<EXPR, DERIV>(p.a + mulhiAny(horner(p, t), e << 1) - e, o, gp);
        if constexpr (DERIV) {
            o.fe = mulhi(gp, v.m);
            o.n = v.n;
        }
    } else {
        rect<EXPR, DERIV>(horner(p, t), o, gp);
    }
    return o;
}

// t = 0 and t = 1.
template <bool EXPR, bool DERIV, int NB, bool ENV>
MPGB_HD Node nodeEnd(const Poly<NB, ENV>& p, bool one) {
    uint64_t q = p.c[0];
    if (one) {
#pragma unroll
        for (int j = 1; j < NB; ++j) q += p.c[j] - 0x8000000000000000ull;
    }
    Node o;
    uint64_t gp;
    if constexpr (ENV) {
        const Envelope v = one ? envelope(p, 0, true) : Envelope{0x7fffffffffffffffull, 0};
        const uint64_t e = shrRound(v.m, v.n);
        rect<EXPR, DERIV>(p.a + mulhiAny(q, e << 1) - e, o, gp);
        if constexpr (DERIV) {
            o.fe = mulhi(gp, v.m);
            o.n = v.n;
        }
    } else {
        rect<EXPR, DERIV>(q, o, gp);
    }
    return o;
}

// Integrals over [0, 1]: g (SoftPlus: 57 fraction bits; Exp: 62, times 2^E),
// with NM > 0 m0 = int g' (ENV; 62 fraction bits) and m[j] = int g' t^j (times
// the envelope with ENV); Exp: all times 2^E.  ENV: the moments are those of
// (2^ms t)^j, SoftPlus times 2^ms (see momentShift).
template <int NM>
struct Sums {
    uint64_t g, m0, m[NM > 0 ? NM : 1];
    int E, nInt;
    bool over;
};

// ms for an envelope exp(-(x t)^2 / 2): 2^ms about |x| / 2.  The moments feed
// polynomials in y = x t whose coefficients grow as x^j, while the envelope
// confines t to a few 1 / |x|: unscaled, their fixed fraction would lose
// x^j of its size (1.7e-14 in an order-5 gradient at |x| = 10).  With
// 2^ms <= |x| / 1.41 the weights (2^ms t)^j exp(-(x t)^2 / 2) stay below 2.5.
MPGB_HD int momentShift(double x) {
    const int e = expBound(x * 0.70710678118654752) - 1;  // floor(log2(|x| / 1.41))
    return e < 0 ? 0 : (e > 5 ? 5 : e);
}

// absTol / |x_D| against sums of g scaled by 2^-level: SoftPlus as an integer
// with 57 fraction bits, Exp as m 2^(E - 62).
struct Threshold {
    uint64_t m;
    int E;
};
// The threshold of a quadrature.  False (the point keeps FP64) where neither
// tolerance stands 2^6 units above the sums' last bit: the integers would cut
// a smaller one to zero, or test rounding against it, and an accept test that
// never holds runs to the interval budget (relTol 0, absTol 5e-18, x_D = 1:
// 255 intervals in FP64).
constexpr double kMinRelTol = 0x1p-44;
template <bool EXPR>
MPGB_HD bool threshold(double ta, double relTol, Threshold& thr) {
    const int e = expBound(ta);
    const uint64_t M = mantissa64(ta);
    if constexpr (EXPR) {
        thr.m = M >> 1;
        thr.E = e - 1;
    } else {
        thr.m = e > 5 ? 1ull << 62 : shr(M, 7 - e);  // (x_D = 0: infinite)
        thr.E = 0;
    }
    return relTol >= kMinRelTol || e > -50;  // (ta >= 2^-50)
}

// One interval of the rule from its five nodes (ends A, B, middle M, inner V,
// W): the nodes' g on one exponent E (Exp), the fine sum ih (per unit width) and
// whether |ih - ic| < max(relTol ic, (absTol / |x_D|) 2^level).  (Exp's threshold is
// rounded up: a difference of zero passes however large g is, as in FP64.)
struct Interval {
    uint64_t a, b, m, v, w, ih;
    int E;
    bool small;
};
template <bool EXPR>
MPGB_HD Interval intervalSums(const Node& A, const Node& B, const Node& V, const Node& M, const Node& W,
                              const Rule& Q, Threshold thr, int level) {
    Interval o;
    o.a = A.g;
    o.b = B.g;
    o.m = M.g;
    o.v = V.g;
    o.w = W.g;
    o.E = 0;
    if constexpr (EXPR) {
        int E = A.E > B.E ? A.E : B.E;
        E = M.E > E ? M.E : E;
        E = V.E > E ? V.E : E;
        E = W.E > E ? W.E : E;
        o.E = E;
        o.a = shr(o.a, E - A.E);
        o.b = shr(o.b, E - B.E);
        o.m = shr(o.m, E - M.E);
        o.v = shr(o.v, E - V.E);
        o.w = shr(o.w, E - W.E);
    }
    const uint64_t ab = o.a + o.b, vw = o.v + o.w;
    const uint64_t ic = mulhi(ab, Q.c0) + mulhi(o.m, Q.cM);
    o.ih = mulhi(ab, Q.w0) + mulhi(o.m, Q.wM) + mulhi(vw, Q.w1);
    const uint64_t err = o.ih > ic ? o.ih - ic : ic - o.ih;
    uint64_t tol = mulhi(ic, Q.rel), ta;
    if constexpr (EXPR) {
        const int sh = o.E - thr.E - level;
        ta = sh < 0 ? ~0ull : shr(thr.m - 1, sh) + 1;
    } else {
        ta = (thr.m >> (63 - level)) ? ~0ull : thr.m << level;
    }
    tol = ta > tol ? ta : tol;
    o.small = err < tol;
    return o;
}

// Adds an accepted interval's fine sum to the value g 2^E (SoftPlus: E unused).
// Exp: the exponent follows the largest contribution (the interval's exponent
// less its level), so a narrow peak keeps its bits.
template <bool EXPR>
MPGB_HD void addValue(uint64_t ih, int E, int level, uint64_t& g, int& gE) {
    int dn = level;
    if constexpr (EXPR) {
        const int e = E - level;
        if (e > gE) {
            g = shr(g, e - gE);
            gE = e;
        }
        dn = gE - e;
    }
    g += shrRound(ih, dn);
    if constexpr (EXPR) {
        if (g >> 62) {
            g >>= 1;
            ++gE;
        }
    }
}

// The adaptive traversal of `integrate` (depth first, left first; the same
// rule, accept test and order of accepted sums) on [0, 1].  An interval is
// (lo, level), lo with 32 fraction bits and width 2^-level; the pending right
// halves have distinct levels (a bit mask), and a stack indexed by level holds
// the node at their right end.  An accepted interval's moments are formed
// about its left end and shifted to t = 0 by repeated multiply-adds with lo.
template <bool EXPR, int NB, bool ENV, int NM>
MPGB_HD void integrate(const Poly<NB, ENV>& p, const Rule& Q, int maxSub, int minSub, int maxIntervals,
                       Threshold thr, int ms, Sums<NM>& R) {
    constexpr bool D = NM > 0;
    uint64_t stG[32], stF[D && !EXPR ? 32 : 1], stFe[D && ENV ? 32 : 1];
    int stE[EXPR ? 32 : 1], stN[D && ENV ? 32 : 1];
    R.g = R.m0 = 0;
    R.E = -200;
    R.over = false;
#pragma unroll
    for (int j = 0; j < (NM > 0 ? NM : 1); ++j) R.m[j] = 0;
    Node A = nodeEnd<EXPR, D>(p, false), B = nodeEnd<EXPR, D>(p, true);
    uint32_t lo = 0, pend = 0;
    int level = 0;
    int count = 0;
    while (true) {
        const uint64_t mid = ((uint64_t)lo << 32) + (0x8000000000000000ull >> level);
        const uint64_t dr = Q.rho >> (level + 1);
        const Node V = nodeAt<EXPR, D>(p, mid - dr), M = nodeAt<EXPR, D>(p, mid), W = nodeAt<EXPR, D>(p, mid + dr);
        const Interval q = intervalSums<EXPR>(A, B, V, M, W, Q, thr, level);
        const uint64_t a = q.a, b = q.b, m = q.m, v = q.v, w = q.w, ih = q.ih;
        const int E = q.E;
        const bool accept = (q.small || level == maxSub - 1) && level >= minSub;
        ++count;
        if (accept) {
            int dn = level;  // (exponents as in addValue)
            if constexpr (EXPR) {
                const int e = E - level;
                if (e > R.E) {
                    const int up = e - R.E;
                    R.g = shr(R.g, up);
                    R.m0 = shr(R.m0, up);
#pragma unroll
                    for (int j = 0; j < (NM > 0 ? NM : 1); ++j) R.m[j] = shr(R.m[j], up);
                    R.E = e;
                }
                dn = R.E - e;
            }
            R.g += shrRound(ih, dn);
            if constexpr (D) {
                uint64_t fa, fb, fm, fv, fw;
                int tail = 0;  // the moments' units below: 2^(-62 - tail)
                if constexpr (ENV) {
                    // The shift to t = 0 multiplies an interval's moments, and
                    // their rounding, by up to 2^(ms j): intervals under a small
                    // envelope (largest at the left end) carry more bits, as many
                    // as the shifted moments leave room for.  (Without them an
                    // order-5 J_k was 2e-15 of its integral off at |x_D| = 10.)
                    tail = A.n - ms * NM - 1;
                    tail = tail > 0 ? tail : 0;
                    const int da = EXPR ? E - tail : -tail;
                    fa = shrRound(A.fe, da + A.n - A.E); fb = shrRound(B.fe, da + B.n - B.E);
                    fm = shrRound(M.fe, da + M.n - M.E); fv = shrRound(V.fe, da + V.n - V.E);
                    fw = shrRound(W.fe, da + W.n - W.E);
                    if constexpr (EXPR) {
                        R.m0 = R.g;
                    } else {
                        R.m0 += shrRound(mulhi(A.f + B.f, Q.w0) + mulhi(M.f, Q.wM) + mulhi(V.f + W.f, Q.w1), level);
                    }
                } else if constexpr (EXPR) {
                    fa = a; fb = b; fm = m; fv = v; fw = w;
                } else {
                    fa = A.f; fb = B.f; fm = M.f; fv = V.f; fw = W.f;
                }
                uint64_t mu[NM];
                // (The shift to t = 0 multiplies units by up to 2^(5 ms): its
                // ties are rounded either way.  Halves up, without the tail's
                // bits, were 6e-17 of the fifth moment of every point, 1e-15
                // of an order-5 gradient.)
                fb = mulhi(fb, Q.w0);
                fm = mulhi(fm, Q.wM);
                mu[0] = mulhi(fa, Q.w0) + fb + fm + mulhi(fv + fw, Q.w1);
#pragma unroll
                for (int j = 1; j < NM; ++j) mu[j] = fb + ((fm + ((1ull << j) >> 1)) >> j) + mulhi(fv, Q.mLo[j]) + mulhi(fw, Q.mHi[j]);
#pragma unroll
                for (int j = 0; j < NM; ++j) {
                    if constexpr (ENV) mu[j] = scaleEven(mu[j], level * j + dn - ms * (EXPR ? j : j + 1));
                    else mu[j] = shrRound(mu[j], level * j + dn);
                }
#pragma unroll
                for (int i = 0; i + 1 < NM; ++i) {
#pragma unroll
                    for (int j = NM - 1; j > i; --j) {
                        if constexpr (ENV) mu[j] += mul32Round(mu[j - 1], lo, (uint32_t)mu[j] & 1) << ms;
                        else mu[j] += mul32Round(mu[j - 1], lo);
                    }
                }
                if (ENV && tail) {
#pragma unroll
                    for (int j = 0; j < NM; ++j) mu[j] = scaleEven(mu[j], tail);
                }
#pragma unroll
                for (int j = 0; j < NM; ++j) R.m[j] += mu[j];
            }
            if constexpr (EXPR) {
                if (R.g >> 62) {
                    R.g >>= 1;
                    R.m0 >>= 1;
#pragma unroll
                    for (int j = 0; j < (NM > 0 ? NM : 1); ++j) R.m[j] >>= 1;
                    ++R.E;
                }
            }
            if (pend == 0) break;
#ifdef __CUDA_ARCH__
            const int L = 31 - __clz((int)pend);
#else
            const int L = 31 - __builtin_clz(pend);
#endif
            pend ^= 1u << L;
            lo += 1u << (32 - level);
            level = L;
            A = B;
            B.g = stG[L];
            if constexpr (EXPR) B.E = stE[L];
            if constexpr (D) {
                if constexpr (EXPR) B.f = B.g;
                else B.f = stF[L];
                if constexpr (ENV) {
                    B.fe = stFe[L];
                    B.n = stN[L];
                }
            }
        } else {
            ++level;
            pend |= 1u << level;
            stG[level] = B.g;
            if constexpr (EXPR) stE[level] = B.E;
            if constexpr (D && !EXPR) stF[level] = B.f;
            if constexpr (D && ENV) {
                stFe[level] = B.fe;
                stN[level] = B.n;
            }
            B = M;
        }
        if (count >= maxIntervals) {
            R.over = true;
            break;
        }
    }
    R.nInt = count;
}

}  // namespace fx
}  // namespace mpgb
