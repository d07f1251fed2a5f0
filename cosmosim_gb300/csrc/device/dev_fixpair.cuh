// dev_fixpair.cuh — softened pair terms on the integer pipes.
//
// GB300 runs 2 FP64 operations per clock and SM, 1/64 of its FP32 rate; its
// 32 x 32 -> 64-bit integer multiply-adds run far faster. A softened pair term
// m d / (d^2 + eps^2)^(3/2) costs 9 FP64 operations even with the last step of m/r^3
// by integers; here r^2 and m/r^3 (or 1/r) take none, and the FP64 pipe keeps what
// needs FP64's range: three differences and three sums (192 + 192 cycles a warp
// and scheduler, beside about 160 instructions on the other pipes).
//
// 1/r and m/r^3 for FP64 differences dx, dy, dz and eps^2, with no FP64 operation:
// r^2 is summed from the differences' significands, shifted right to the largest
// one's exponent (or eps's), its top bit then at 62, and kept to 2^-58 relative; 1/r
// from an FP32 rsqrt seed y0 and a series in e = 1 - r^2 y0^2 (one high-word
// product, |e| < 2^-20: y0 (1 + e/2 + 3/8 e^2), y0^3 (1 + 3/2 e + 15/8 e^2), the next
// term below 2^-59), every product keeping its high 64 bits; the result is rounded
// once and packed. So a term is within 1.02 x 2^-53 (1.016 in 180,000 modelled pairs) of the exact function of its
// differences, where FP64 operations round r^2 three times more. Differences and
// sums stay FP64: a fixed-point grid for the positions or the sums would lose the
// bits of bodies much closer to the origin, or much lighter, than the system's
// largest.
#pragma once

#include <math.h>
#include <string.h>

#include "dev_internal.cuh"

__device__ __forceinline__ unsigned long long mulw(unsigned a, unsigned b)
{
    return (unsigned long long)a * b;
}
__device__ __forceinline__ unsigned hi32(unsigned long long v) { return (unsigned)(v >> 32); }
__device__ __forceinline__ unsigned long long shr_clamp(unsigned long long v, unsigned n)
{
    unsigned long long r; // PTX clamps the shift: n >= 64 gives 0
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(n));
    return r;
}

__device__ __forceinline__ unsigned long long shl_clamp(unsigned long long v, unsigned n)
{
    unsigned long long r; // n >= 64 gives 0
    asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(n));
    return r;
}
__device__ __forceinline__ long long mulws(int a, int b) { return (long long)a * b; }

// eps^2 as the pair terms take it.
struct PairEps {
    unsigned long long e2n; // significand, top bit at 61 (0 for eps = 0)
    int e2s;                // biased exponent + 1022: r2 gets e2n >> (2 er - e2s)
    unsigned eh;            // high word of |eps|
    double eps2;
};

// eps^2 zero while eps is not, subnormal or infinite: an exponent of 2047 takes
// every pair to the plain expression.
__host__ __device__ inline PairEps pair_eps(double eps)
{
    PairEps p;
    p.eps2 = eps * eps;
    unsigned long long b, c;
    const double a = fabs(eps);
    memcpy(&b, &p.eps2, sizeof(b));
    memcpy(&c, &a, sizeof(c));
    const int eb = (int)(b >> 52);
    p.eh = (unsigned)(c >> 32);
    p.e2n = 0ull;
    p.e2s = 0;
    if (eb > 0 && eb < 2047) {
        p.e2n = ((b & 0xfffffffffffffull) | (1ull << 52)) << 9;
        p.e2s = eb + 1022;
    } else if (!(eps == 0.0)) {
        p.eh = 0x7ff00000u;
    }
    return p;
}

// r^2 = r2 2^(2 (er - 1023) - 60), r2 in [2^60, 2^64), and its seed.
struct PairR {
    unsigned long long S; // Y^2
    long long e60;        // (1 - r^2 y0^2) 2^60
    unsigned Y;           // y0 = Y 2^(ey - 158), seed of (r2 2^-32)^(-1/2)
    int ey, er;           // er: the largest difference's (or eps's) biased exponent
};

__device__ __forceinline__ unsigned long long pair_word(double d, int er)
{
    const unsigned h = (unsigned)__double2hiint(d), l = (unsigned)__double2loint(d);
    const unsigned top = (h & 0xfffffu) | 0x100000u; // a subnormal's shifts out
    const unsigned long long v = ((unsigned long long)__funnelshift_l(l, top, 10) << 32) | (l << 10);
    return shr_clamp(v, (unsigned)(er - (int)(h >> 20 & 0x7ffu)));
}

__device__ __forceinline__ PairR pair_r(const PairEps &p, double dx, double dy, double dz)
{
    PairR r;
    const unsigned M = 0x7fffffffu;
    r.er = (int)(max(max((unsigned)__double2hiint(dx) & M, (unsigned)__double2hiint(dy) & M),
                     max((unsigned)__double2hiint(dz) & M, p.eh)) >> 20);
    const unsigned long long x = pair_word(dx, r.er), y = pair_word(dy, r.er),
                             z = pair_word(dz, r.er);
    // the words are below 2^63; the dropped low products and the cut shifts are 2.5
    // on average
    const unsigned long long hh = mulw(hi32(x), hi32(x)) + mulw(hi32(y), hi32(y)) +
                                  mulw(hi32(z), hi32(z));
    const unsigned long long xy = mulw(hi32(x), (unsigned)x) + mulw(hi32(y), (unsigned)y),
                             zz = mulw(hi32(z), (unsigned)z);
    const unsigned long long r2 = hh + (xy >> 31) + (zz >> 31) +
                                  shr_clamp(p.e2n, (unsigned)(2 * r.er - p.e2s)) + 2ull;
    float s;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(__uint2float_rz(hi32(r2))));
    const unsigned sb = __float_as_uint(s);
    r.ey = (int)(sb >> 23); // 110..113
    r.Y = (sb << 8) | 0x80000000u;
    r.S = mulw(r.Y, r.Y);
    // r2 S 2^-64 = (1 - e) 2^(284 - 2 ey); |e| < 2^-20, so a power of 2^64 may wrap
    const int k = 284 - 2 * r.ey; // 58..64
    const long long D = (long long)(shl_clamp(1ull, (unsigned)k) - __umul64hi(r2, r.S));
    r.e60 = (D << 2) >> (k - 58);
    return r;
}

// F 2^(E - 1086) to nearest, for F >= 2^32; E comes back as the result's biased
// exponent (out of 1 .. 2045: no number).
__device__ __forceinline__ double pair_pack(unsigned long long F, int &E)
{
    const int lz = __clz((int)hi32(F));
    const unsigned hi = __funnelshift_l((unsigned)F, hi32(F), lz), lo = (unsigned)F << lz;
    E -= lz;
    const unsigned long long v =
        ((unsigned long long)(((unsigned)(E - 1) << 20) + (hi >> 11)) << 32) |
        __funnelshift_r(lo, hi, 11);
    return __longlong_as_double((long long)(v + (lo >> 10 & 1u)));
}

// num / 8 e^2 2^60, the series' second term.
__device__ __forceinline__ int pair_e2(long long e60, unsigned num)
{
    const int eh = (int)(e60 >> 9);
    return (int)((((unsigned)(mulws(eh, eh) >> 32) >> 4) * num) >> 9);
}

static __device__ __noinline__ double pair_plain_1(double dx, double dy, double dz, double eps2)
{
    return 1.0 / sqrt(fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2))));
}

// (dx^2 + dy^2 + dz^2 + eps^2)^(-1/2); the plain expression where an exponent
// would leave FP64's normal range.
__device__ __forceinline__ double pair_inv_r(const PairEps &p, double dx, double dy, double dz)
{
    const PairR r = pair_r(p, dx, dy, dz);
    const long long c60 = (r.e60 >> 1) + pair_e2(r.e60, 3u);
    const unsigned long long C = (1ull << 63) + (unsigned long long)(c60 << 3); // (1 + c) 2^63
    const unsigned long long V = mulw(r.Y, hi32(C)) + hi32(mulw(r.Y, (unsigned)C));
    int E = r.ey - r.er + 1934; // V = Y (1 + c) 2^31, 1/r = V 2^(ey - er + 848)
    const double v = pair_pack(V, E);
    // er is 0 where all are zero, 2047 for infinities and NaN; above 64 a
    // subnormal difference does not count
    return (unsigned)(r.er - 65) < 1980u && (unsigned)(E - 1) < 2045u
               ? v
               : pair_plain_1(dx, dy, dz, p.eps2);
}

static __device__ __noinline__ double pair_plain_3(double dx, double dy, double dz, double eps2,
                                                   double m)
{
    const double r2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2)));
    return m / (r2 * sqrt(r2));
}

// m (dx^2 + dy^2 + dz^2 + eps^2)^(-3/2), 0 for m = +0; the plain expression for a mass
// that is not positive and normal and where an exponent would leave the normal range.
__device__ __forceinline__ double pair_m_r3(const PairEps &p, double dx, double dy, double dz,
                                            double m)
{
    const PairR r = pair_r(p, dx, dy, dz);
    const long long c60 = r.e60 + (r.e60 >> 1) + pair_e2(r.e60, 15u);
    const unsigned long long C = (1ull << 63) + (unsigned long long)(c60 << 3); // (1 + c) 2^63
    const unsigned long long W = mulw(r.Y, hi32(r.S)) + hi32(mulw(r.Y, (unsigned)r.S));
    const unsigned mh = (unsigned)__double2hiint(m), ml = (unsigned)__double2loint(m);
    const int em = (int)(mh >> 20); // with the sign: 2048 and more for a negative mass
    const unsigned long long Mm =
        ((unsigned long long)__funnelshift_l(ml, (mh & 0xfffffu) | 0x100000u, 11) << 32) | (ml << 11);
    const unsigned long long F = __umul64hi(__umul64hi(W, C), Mm);
    // F = Y^3 (1 + c) Mm 2^-97, m/r^3 = F 2^(3 (ey - er) + em + 1648)
    int E = 3 * (r.ey - r.er) + em + 2734;
    const double v = pair_pack(F, E);
    if ((unsigned)(r.er - 65) < 1980u && (unsigned)(E - 1) < 2045u && (unsigned)(em - 1) < 2046u)
        return v;
    return (mh | ml) == 0u ? 0.0 : pair_plain_3(dx, dy, dz, p.eps2, m);
}
