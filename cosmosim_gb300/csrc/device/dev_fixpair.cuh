// dev_fixpair.cuh — softened pair terms on the integer pipes.
//
// GB300 runs 2 FP64 operations per clock and SM, 1/64 of its FP32 rate; its
// 32 x 32 -> 64-bit integer multiply-adds run far faster. A softened pair
// m d / (d^2 + eps^2)^(3/2) costs 9 FP64 operations even with m/r^3 formed by
// integers (576 issue cycles per warp and scheduler); formed by integers from
// end to end it takes about 240 instructions (m/r: 150) on two pipes, 330
// cycles (210), and no FP64 operation.
//
// Positions are 64-bit fixed point on one grid per system: X = x 2^g, rounded,
// |X| < 2^61, so differences are exact in 64 bits. r^2 = dx^2 + dy^2 + dz^2 +
// eps^2 is summed from the differences shifted up together (the largest, or
// eps, then has its top bit at 61) and kept to 2^-57 relative. 1/r comes from
// an FP32 rsqrt seed y0: e = 1 - r^2 y0^2 by one high-word product, then the
// binomial series y0 (1 - e)^(-1/2) or y0^3 (1 - e)^(-3/2) to second order
// (|e| < 2^-20: the next term is below 2^-59), every product keeping its high
// 64 bits. Terms are added to a 128-bit fixed-point sum (the walk's, of
// fewer terms and a tighter bound, to 96 bits), so a sum does not depend on its
// order. (64-bit sums whose unit followed the largest term took
// about 60 instructions less a pair but were 4-15 times less exact than FP64.)
//
// What rounds: the positions (half a grid unit), the truncated products (about
// 2^-55 of a term in all) and the last bit of the 128-bit sum. The grid is
// 2^-61 of the largest coordinate; FIX_EPS_BITS keeps eps above 2^48 units, so a
// pair at the softening length, the closest that matters, still has its
// difference to 2^-48, and every longer one better. The walk also takes wider
// systems (a few bodies thrown far out): their grid keeps eps above 2^50 units,
// cells beyond 2^61 units lie on a coarser grid of 2^far units and meet bodies
// within 2^60 units only, so a difference is at least 2^(60 - far) >= 2^50
// coarse units, as exact as the others; tasks with a body further out keep
// FP64. Measured on a quasar with bodies out to 2^15 to 2^21 softening lengths,
// every pair summed (theta 0), against extended precision: rms error 3.5e-16
// to 1.7e-15 of the acceleration, in FP64 3.5e-15 to 4.1e-15. Systems that do
// not fit (no softening, a span above 2^13 softening lengths, for the walk
// 2^21; non-finite or extreme values) keep the FP64 kernels.
#pragma once

#include <math.h>
#include <string.h>

#include "dev_internal.cuh"

constexpr int FIX_POS_BITS = 61; // |X| < 2^61
constexpr int FIX_EPS_BITS = 48; // eps 2^g >= 2^48
constexpr int FIX_WIDE_EPS_BITS = 50; // the same for a grid with far cells
constexpr int FIX_FAR_MAX = 10;

// The grid's exponent for coordinates below 2^ex and eps in [2^(ee - 1), 2^ee),
// and its far cells' exponent.
__device__ inline int fix_scale(int ex, int ee, int &far)
{
    const int g = FIX_POS_BITS - max(ex, ee);
    far = 0;
    if (g + ee - 1 >= FIX_EPS_BITS)
        return g;
    const int wide = FIX_WIDE_EPS_BITS - (ee - 1);
    far = wide - g;
    return wide;
}

// The grid of n bodies whose largest |coordinate| is xmax and largest mass
// mmax (n mmax bounds the sums), with the given eps and eps^2.
__device__ inline FixGrid fix_grid(double xmax, double mmax, double n, double eps, double eps2,
                                   int far_max = 0)
{
    FixGrid f;
    f.ok = 0;
    f.far = f.g = f.U3 = f.U1 = f.e2s = 0;
    f.eh = 0u;
    f.e2n = 0ull;
    eps = fabs(eps);
    // exponents far inside FP64's, so that every power of two below is normal
    if (!(xmax <= 0x1p200 && mmax > 0x1p-200 && mmax <= 0x1p200 && eps >= 0x1p-200 &&
          eps <= 0x1p200))
        return f;
    // the larger of the coordinates and eps fits 61 bits
    f.g = fix_scale(xmax > 0.0 ? ilogb(xmax) + 1 : -1000, ilogb(eps) + 1, f.far);
    if (f.far > far_max)
        return f;
    const long long E = (long long)ldexp(eps, f.g);
    f.eh = (unsigned)(E >> 32);
    // eps^2 = S 2^k, S the 53-bit significand; r2's unit is 2^(64 - 2 s - 2 g)
    const long long b = __double_as_longlong(eps2);
    const int k = (int)((b >> 52) & 0x7ff) - 1075;
    f.e2n = (((unsigned long long)b & 0xfffffffffffffull) | (1ull << 52)) << 9;
    f.e2s = 64 + 9 - k - 2 * f.g;
    // |sum of a| <= n mmax max(r / (r^2 + eps^2)^1.5) <= n mmax 0.385 / eps^2
    f.U3 = ilogb(n * mmax * 0.385 / eps2) + 1 - 119;
    f.U1 = ilogb(n * mmax / eps) + 1 - 119;
    f.ok = 1;
    return f;
}

// 2^e as a double, -1000 <= e <= 1000.
__device__ __forceinline__ double fix_pow2(int e)
{
    return __longlong_as_double((long long)(e + 1023) << 52);
}

__device__ __forceinline__ long long fix_pos(double x, double scale) // scale = 2^g
{
    return __double2ll_rn(x * scale);
}

// A mass as its significand with the top bit at 63 and the biased exponent in
// the 11 free low bits; 0 for a massless (or subnormal) body.
__device__ __forceinline__ unsigned long long fix_mass(double m)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(m);
    const unsigned e = (unsigned)(b >> 52) & 0x7ffu;
    return (m > 0.0 && e > 0u) ? ((((b & 0xfffffffffffffull) | (1ull << 52)) << 11) | e) : 0ull;
}

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

// High 64 bits of a b from the three upper partial products, each taken from
// its high word: 0 to 3 below, 1.25 on average.
__device__ __forceinline__ unsigned long long mulhi(unsigned long long a, unsigned long long b)
{
    return mulw(hi32(a), hi32(b)) + hi32(mulw(hi32(a), (unsigned)b)) +
           hi32(mulw((unsigned)a, hi32(b)));
}
__device__ __forceinline__ long long mulws(int a, int b) { return (long long)a * b; }

__device__ __forceinline__ unsigned long long sar_clamp(unsigned long long v, unsigned n)
{
    long long r; // PTX clamps the shift: n >= 64 gives the sign
    asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"((long long)v), "r"(n));
    return (unsigned long long)r;
}

// r^2 of a pair and its rsqrt seed.
struct FixR {
    long long x, y, z;    // differences (in grid units) 2^s, |.| < 2^62
    int nx, ny, nz;       // their signs (0 or -1)
    unsigned long long S; // Y^2
    long long e57;        // (1 - r^2 y0^2) 2^57
    unsigned Y;           // y0 = Y 2^(ey - 158)
    int ey, s;
};

// up: the differences are in 2^up grid units
__device__ __forceinline__ FixR fix_pair(const FixGrid &f, long long dx, long long dy, long long dz,
                                         int up = 0)
{
    FixR p;
    const int xh0 = (int)(dx >> 32), yh0 = (int)(dy >> 32), zh0 = (int)(dz >> 32);
    p.nx = xh0 >> 31;
    p.ny = yh0 >> 31;
    p.nz = zh0 >> 31;
    p.s = __clz((xh0 ^ p.nx) | (yh0 ^ p.ny) | (zh0 ^ p.nz) | (int)f.eh) - 2; // 0..15
    p.x = (long long)((unsigned long long)dx << p.s);
    p.y = (long long)((unsigned long long)dy << p.s);
    p.z = (long long)((unsigned long long)dz << p.s);
    p.s -= up;
    const int xh = (int)(p.x >> 32), yh = (int)(p.y >> 32), zh = (int)(p.z >> 32);
    const long long hh = mulws(xh, xh) + mulws(yh, yh) + mulws(zh, zh);
    const long long hl = mulws(xh, (int)((unsigned)p.x >> 2)) + mulws(yh, (int)((unsigned)p.y >> 2)) +
                         mulws(zh, (int)((unsigned)p.z >> 2));
    // r^2 = r2 2^(64 - 2 s - 2 g), r2 in [2^58, 2^62]; the dropped low
    // products are 1 on average
    const unsigned long long r2 = (unsigned long long)(hh + (hl >> 29)) +
                                  shr_clamp(f.e2n, (unsigned)(f.e2s - 2 * p.s)) + 1ull;
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint2float_rz(hi32(r2))));
    const unsigned yb = __float_as_uint(y);
    p.ey = (int)(yb >> 23); // 111..114
    p.Y = (yb << 8) | 0x80000000u;
    p.S = mulw(p.Y, p.Y);
    // r2 S 2^-63 = (1 - e) 2^(285 - 2 ey)
    const unsigned long long T = mulhi(r2 << 1, p.S);
    const int k = 285 - 2 * p.ey; // 57..63
    p.e57 = (long long)((1ull << k) - T) >> (k - 57);
    return p;
}

// e^2 2^70 from e 2^57, for the series' second term.
__device__ __forceinline__ unsigned fix_e2(long long e57)
{
    const int eh = (int)(e57 >> 6);
    return (unsigned)(mulws(eh, eh) >> 32);
}

// ---- terms from FP64 differences ------------------------------------------
//
// 1/r and m/r^3 for FP64 differences dx, dy, dz and eps^2, with no FP64 operation:
// r^2 is summed from the differences' significands, shifted right to the largest
// one's exponent (or eps's), its top bit then at 61, and kept to 2^-56 relative; 1/r
// from an FP32 rsqrt seed y0 and a series in e = 1 - r^2 y0^2 (one high-word
// product, |e| < 2^-20: y0 (1 + e/2 + 3/8 e^2), y0^3 (1 + 3/2 e + 15/8 e^2), the next
// term below 2^-59), every product keeping its high 64 bits; the result is rounded
// once and packed. So a term is within 1.1 x 2^-53 of the exact function of its
// differences, where FP64 operations round r^2 three times more. Differences and
// sums stay FP64: a fixed-point grid for the positions or the sums would lose the
// bits of bodies much closer to the origin, or much lighter, than the system's
// largest.

// eps^2 as the pair terms take it.
struct PairEps {
    unsigned long long e2n; // significand, top bit at 61 (0 for eps = 0)
    int e2s;                // biased exponent + 1020: r2 gets e2n >> (2 er - e2s)
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
        p.e2s = eb + 1020;
    } else if (!(eps == 0.0)) {
        p.eh = 0x7ff00000u;
    }
    return p;
}

// r^2 = r2 2^(2 (er - 1023) - 58), r2 in [2^58, 2^62], and its seed.
struct PairR {
    unsigned long long S; // Y^2
    long long e57;        // (1 - r^2 y0^2) 2^57
    unsigned Y;           // y0 = Y 2^(ey - 158), seed of (r2 2^-32)^(-1/2)
    int ey, er;           // er: the largest difference's (or eps's) biased exponent
};

__device__ __forceinline__ unsigned long long pair_word(double d, int er)
{
    const unsigned h = (unsigned)__double2hiint(d), l = (unsigned)__double2loint(d);
    const unsigned top = (h & 0xfffffu) | 0x100000u; // a subnormal's shifts out
    const unsigned long long v = ((unsigned long long)__funnelshift_l(l, top, 9) << 32) | (l << 9);
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
    // the words are below 2^62; the dropped low products are 1 on average
    const unsigned long long hh = mulw(hi32(x), hi32(x)) + mulw(hi32(y), hi32(y)) +
                                  mulw(hi32(z), hi32(z));
    const unsigned long long hl = mulw(hi32(x), (unsigned)x) + mulw(hi32(y), (unsigned)y) +
                                  mulw(hi32(z), (unsigned)z);
    const unsigned long long r2 =
        hh + (hl >> 31) + shr_clamp(p.e2n, (unsigned)(2 * r.er - p.e2s)) + 1ull;
    float s;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(__uint2float_rz(hi32(r2))));
    const unsigned sb = __float_as_uint(s);
    r.ey = (int)(sb >> 23); // 111..114
    r.Y = (sb << 8) | 0x80000000u;
    r.S = mulw(r.Y, r.Y);
    // r2 S 2^-63 = (1 - e) 2^(285 - 2 ey)
    const unsigned long long T = mulhi(r2 << 1, r.S);
    const int k = 285 - 2 * r.ey; // 57..63
    r.e57 = (long long)((1ull << k) - T) >> (k - 57);
    return r;
}

// F 2^(E - 1086) rounded to nearest, for F > 0; E is then the result's biased
// exponent plus the leading zeros of F. Returned as bits, the exponent in E.
__device__ __forceinline__ double pair_pack(unsigned long long F, int &E)
{
    const int lz = __clz((int)hi32(F)); // the callers' F are above 2^58
    const unsigned hi = __funnelshift_l((unsigned)F, hi32(F), lz), lo = (unsigned)F << lz;
    E -= lz;
    const unsigned long long v =
        ((unsigned long long)(((unsigned)(E - 1) << 20) + (hi >> 11)) << 32) |
        __funnelshift_r(lo, hi, 11);
    return __longlong_as_double((long long)(v + (lo >> 10 & 1u)));
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
    const int q = (int)(((fix_e2(r.e57) >> 4) * 3u) >> 12); // 3/8 e^2 2^57
    const long long c57 = (r.e57 >> 1) + q;
    const unsigned long long C = (1ull << 63) + (unsigned long long)(c57 << 6); // (1 + c) 2^63
    const unsigned long long V = mulw(r.Y, hi32(C)) + hi32(mulw(r.Y, (unsigned)C));
    int E = r.ey - r.er + 1933; // V = Y (1 + c) 2^31, 1/r = V 2^(ey - er + 847)
    const double v = pair_pack(V, E);
    // er is 0 where all are zero, 2047 for infinities and NaN; above 64 a
    // subnormal difference does not count
    return (unsigned)(r.er - 65) < 1980u && (unsigned)(E - 1) < 2045u
               ? v
               : pair_plain_1(dx, dy, dz, p.eps2);
}

// 128-bit sum, words from the lowest.
struct Fix128 {
    unsigned w0, w1, w2, w3;

    __device__ __forceinline__ void clear() { w0 = w1 = w2 = w3 = 0u; }
    // adds (v 2^64) >> sh, sh >= 0; neg (0 or ~0): subtracts it, and one unit
    __device__ __forceinline__ void add(unsigned long long v, unsigned sh, unsigned neg)
    {
        const unsigned hi = hi32(v) ^ neg, lo = (unsigned)v ^ neg;
        const unsigned t2 = (unsigned)((int)hi >> (sh & 31u)); // v < 2^63: hi's top bit is the sign
        const unsigned t1 = __funnelshift_r(lo, hi, sh), t0 = __funnelshift_r(neg, lo, sh);
        const unsigned w = sh >> 5;
        const unsigned o3 = w == 0u ? t2 : neg;
        const unsigned o2 = w == 0u ? t1 : w == 1u ? t2 : neg;
        const unsigned o1 = w == 0u ? t0 : w == 1u ? t1 : w == 2u ? t2 : neg;
        const unsigned o0 = w == 1u ? t0 : w == 2u ? t1 : w == 3u ? t2 : neg;
        sum(o0, o1, o2, o3);
    }
    // adds another sum
    __device__ __forceinline__ void sum(unsigned o0, unsigned o1, unsigned o2, unsigned o3)
    {
        asm("add.cc.u32 %0, %0, %4;\n\taddc.cc.u32 %1, %1, %5;\n\t"
            "addc.cc.u32 %2, %2, %6;\n\taddc.u32 %3, %3, %7;"
            : "+r"(w0), "+r"(w1), "+r"(w2), "+r"(w3)
            : "r"(o0), "r"(o1), "r"(o2), "r"(o3));
    }
    // the sum (two's complement) times 2^U
    __device__ __forceinline__ double value(int U) const
    {
        const bool n = (int)w3 < 0;
        unsigned long long hi = ((unsigned long long)w3 << 32) | w2,
                           lo = ((unsigned long long)w1 << 32) | w0;
        if (n) {
            lo = 0ull - lo;
            hi = ~hi + (lo == 0ull);
        }
        const double v = ldexp(fma((double)hi, 0x1p64, (double)lo), U);
        return n ? -v : v;
    }
};

// 96-bit sum without the 128-bit sum's lowest word. Terms are cut downwards,
// half a unit on average: value() puts back half of their count (a sum of
// nothing, or of terms that are all zero, stays zero).
struct Fix96 {
    unsigned w0, w1, w2;

    __device__ __forceinline__ void clear() { w0 = w1 = w2 = 0u; }
    __device__ __forceinline__ void add(unsigned long long v, unsigned sh, unsigned neg)
    {
        const unsigned hi = hi32(v) ^ neg, lo = (unsigned)v ^ neg;
        const unsigned long long x = ((unsigned long long)hi << 32) | lo; // top bit: the sign
        const unsigned long long top = sar_clamp(x, sh);
        const unsigned low = sh < 32u ? lo << ((32u - sh) & 31u) : (unsigned)sar_clamp(x, sh - 32u);
        sum(low, (unsigned)top, hi32(top));
    }
    __device__ __forceinline__ void sum(unsigned o0, unsigned o1, unsigned o2)
    {
        asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
            : "+r"(w0), "+r"(w1), "+r"(w2)
            : "r"(o0), "r"(o1), "r"(o2));
    }
    __device__ __forceinline__ double value(int U, int cnt) const
    {
        const long long hi = (long long)(((unsigned long long)w2 << 32) | w1);
        if ((hi == 0 && w0 == 0u) || (hi == -1 && (unsigned)cnt >= 0u - w0))
            return 0.0;
        return ldexp(fma((double)hi, 0x1p32, (double)w0 + 0.5 * (double)cnt), U + 32);
    }
};

// Adds one term m d / r^3 to three sums.
template <class Acc>
__device__ __forceinline__ void fix_add3(const FixGrid &f, long long dx, long long dy, long long dz,
                                         unsigned long long mass, Acc &x, Acc &y, Acc &z,
                                         int up = 0)
{
    const FixR p = fix_pair(f, dx, dy, dz, up);
    const int q = (int)(((fix_e2(p.e57) >> 4) * 15u) >> 12); // 15/8 e^2 2^57
    const long long c57 = p.e57 + (p.e57 >> 1) + q;
    const unsigned long long C = (1ull << 63) + (unsigned long long)(c57 << 6); // (1 + c) 2^63
    const unsigned long long W = mulw(p.Y, hi32(p.S)) + hi32(mulw(p.Y, (unsigned)p.S));
    const unsigned long long F = mulhi(mulhi(W, C), mass & ~0x7ffull);
    // F d 2^s = term 2^(64 - X)
    const int X = 3 * p.ey + (int)((unsigned)mass & 0x7ffu) + 2 * p.s + 2 * f.g - 1543;
    const unsigned sh = (unsigned)max(f.U3 - X + 64, 1);
    const int any = (int)hi32(mass) >> 31; // a massless term is zero, of either sign
    x.add(mulhi(F, (unsigned long long)(p.x < 0 ? -p.x : p.x)), sh, (unsigned)(p.nx & any));
    y.add(mulhi(F, (unsigned long long)(p.y < 0 ? -p.y : p.y)), sh, (unsigned)(p.ny & any));
    z.add(mulhi(F, (unsigned long long)(p.z < 0 ? -p.z : p.z)), sh, (unsigned)(p.nz & any));
}

// Sum of m / r terms.
struct FixSum1 {
    Fix128 a;

    __device__ __forceinline__ void add(const FixGrid &f, long long dx, long long dy, long long dz,
                                        unsigned long long mass)
    {
        const FixR p = fix_pair(f, dx, dy, dz);
        const int q = (int)(((fix_e2(p.e57) >> 4) * 3u) >> 12); // 3/8 e^2 2^57
        const long long c57 = (p.e57 >> 1) + q;
        const unsigned long long C = (1ull << 63) + (unsigned long long)(c57 << 6);
        const unsigned long long V = mulw(p.Y, hi32(C)) + hi32(mulw(p.Y, (unsigned)C));
        const unsigned long long F = mulhi(V, mass & ~0x7ffull);
        // m / r = F 2^X
        const int X = p.ey + (int)((unsigned)mass & 0x7ffu) + p.s + f.g - 1259;
        a.add(F, (unsigned)max(f.U1 - X + 64, 0), 0u);
    }
};
