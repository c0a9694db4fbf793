// Exact FP64 building blocks that cost fewer FP64 instructions than the literal
// expressions they replace.  GB300 issues two FP64 instructions per clock per SM against
// 128 integer/FP32 lanes, so moving exact work off the FP64 pipe pays directly.
//
// 1. Comparisons against zero or a non-negative threshold t on the IEEE bit pattern.
//    For finite (non-NaN) x and t >= +0:  x > t  <=>  int64(bits(x)) > int64(bits(t)),
//    since non-negative doubles order like their bit patterns and every negative double
//    (or -0) has a negative int64 pattern.  |x| and -x are exact bit operations.
//
// 2. Division by a constant y from a precomputed double-word reciprocal zh + zl
//    (zh = RN(1/y), zl = RN(1/y - zh)):
//        q0 = RN(a*zh + RN(a*zl))            within 2^-52 ulp of a/y before its last rounding
//    q0 is RN(a/y) unless a/y lies that close to a rounding boundary.  With integer significands
//    X, Y in [2^52, 2^53) that needs |2^s X - (2m+1) Y| < 4 (s = 53 where X >= Y, 54 below), which
//    at most a few X solve, found once from the residues of X modulo Y (multiplication by an
//    arbitrary-precision constant: N. Brisebarre, J.-M. Muller, IEEE Trans. Comput. 57(2),
//    2008); the significands that do round wrongly are kept (none where Y ends in two zero
//    bits) and take the IEEE division, as do zeros, |a| outside [2^-959, 2^977) and those whose
//    quotient is outside [2^-960, 2^1020): below, a*zl loses bits as a subnormal number (of a
//    significand next to a boundary and y near 2^27 the quotient came out wrong for |a| < 2^-940);
//    above, the two products can be infinities of opposite sign.
//    Cost: 1 DMUL + 1 DFMA.
//    By 6 there are none: with a = A 2^e the quotient is A/3 2^(e-1), and a third of an integer
//    is never closer than 1/6 ulp to a rounding boundary.
//    By a value known on the device only (recip_v, div_v) the quotient is corrected:
//        r  = RN(a - q0*y)                   exact (FMA; the remainder is representable)
//        q  = RN(q0 + r*zh)                  = RN(a/y)
//    The last step is Markstein's theorem (P. Markstein, IBM J. Res. Dev. 34(1), 1990;
//    see also N. Brisebarre, J.-M. Muller, S. K. Raina, IEEE Trans. Comput. 53(8),
//    2004): with zh the correctly rounded reciprocal and q0 faithful, the corrected
//    quotient is the correctly rounded one.  Cost: 1 DMUL + 3 DFMA.
//
// |x| and -x as plain expressions on the bit pattern are recognised by the compiler and
// turned back into FP64 instructions (DADD 0 + |x|): k_dsvl ran 6 DADD per cell for its 3
// differences.  dmag and dflip split the double into its two words with a mov, so that the
// sign is handled on the integer pipe (64 instructions issue there for one FP64 instruction).
#pragma once
#include <cstdint>

namespace madv {

constexpr long long SIGN_BIT = (long long)0x8000000000000000ULL;
constexpr long long ABS_MASK = 0x7fffffffffffffffLL;

__device__ __forceinline__ long long dbits(double x) { return __double_as_longlong(x); }
// the two words of x, and back
__device__ __forceinline__ void dsplit(double x, int& hi, int& lo) {
    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(x));
}
__device__ __forceinline__ double djoin(int hi, int lo) {
    double r;
    asm("mov.b64 %0, {%1, %2};" : "=d"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ int dhigh(double x) {
    int hi, lo;
    dsplit(x, hi, lo);
    return hi;
}
// bits of |x|
__device__ __forceinline__ long long dmag(double x) {
    int hi, lo;
    dsplit(x, hi, lo);
    long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi & 0x7fffffff));
    return r;
}
// -x, and -x where f
__device__ __forceinline__ double dflip(double x, bool f = true) {
    int hi, lo;
    dsplit(x, hi, lo);
    return djoin(f ? hi ^ (int)0x80000000 : hi, lo);
}
__device__ __forceinline__ double dabs(double x) {
    int hi, lo;
    dsplit(x, hi, lo);
    return djoin(hi & 0x7fffffff, lo);
}
// copysign(m, x) for m >= 0
__device__ __forceinline__ double dsigned(double m, double x) {
    int hi, lo;
    dsplit(m, hi, lo);
    return djoin(hi | (dhigh(x) & (int)0x80000000), lo);
}
// An integer that orders like x (both zeros 0; x not NaN): the magnitude, negated below 0.
__device__ __forceinline__ long long dkey(double x) {
    const long long s = (long long)(dhigh(x) >> 31);
    return (dmag(x) ^ s) - s;
}
__host__ inline long long dbits_host(double x) {
    long long b;
    __builtin_memcpy(&b, &x, sizeof(b));
    return b;
}

// x > 0.0
__device__ __forceinline__ bool gt0(double x) { return dbits(x) > 0; }
// x < 0.0 (-0 is not below 0): the pattern of -x is positive
__device__ __forceinline__ bool lt0(double x) { return dbits(dflip(x)) > 0; }
// x is NaN (a quiet one, as every FP64 instruction returns)
__device__ __forceinline__ bool is_nan(double x) { return (dhigh(x) & 0x7fffffff) > 0x7ff00000; }
// |x| > 0.0
__device__ __forceinline__ bool nz(double x) { return dmag(x) != 0; }
// x > t, with tb = bits(t), t >= +0
__device__ __forceinline__ bool gt_t(double x, long long tb) { return dbits(x) > tb; }
// x < -t, with tb = bits(t), t >= +0
__device__ __forceinline__ bool lt_negt(double x, long long tb) { return dbits(dflip(x)) > tb; }
// |x| > t, with tb = bits(t), t >= +0
__device__ __forceinline__ bool abs_gt_t(double x, long long tb) { return dmag(x) > tb; }


// 3. Scaling by 2 and by 1/2 on the bit pattern, equal to the FP multiply (round to nearest
//    even) for every input: a normal result is an exponent step; a zero or subnormal x has
//    |x| = a * 2^-1074 with a its magnitude bits (exponent field 1 included), so 2x is the
//    pattern 2a and x/2 the pattern RN(a/2); 2x past the largest finite double is infinity.
//    Infinities and NaNs pass through.  No FP64 instruction is issued.
__device__ __forceinline__ double twice(double x) {
    int hi, lo;
    dsplit(x, hi, lo);
    const unsigned m = (unsigned)hi & 0x7fffffffu;
    if (m - 0x00100000u < 0x7fd00000u) return djoin(hi + 0x00100000, lo);  // normal, and normal result
    const long long b = dbits(x), a = dmag(x), sg = b & SIGN_BIT;
    long long r;
    if (a < (1LL << 52)) r = sg | (a << 1);                  // zero or subnormal
    else if (a < (0x7ffLL << 52)) r = sg | (0x7ffLL << 52);  // overflow
    else r = b;                                              // infinity, NaN
    return __longlong_as_double(r);
}
__device__ __forceinline__ double half(double x) {
    int hi, lo;
    dsplit(x, hi, lo);
    const unsigned m = (unsigned)hi & 0x7fffffffu;
    if (m - 0x00200000u < 0x7fd00000u) return djoin(hi - 0x00100000, lo);  // normal result
    const long long b = dbits(x), a = dmag(x), sg = b & SIGN_BIT;
    long long r;
    if (a >= (0x7ffLL << 52)) r = b;                  // infinity, NaN
    else r = sg | ((a >> 1) + (a & (a >> 1) & 1));    // subnormal result, ties to even
    return __longlong_as_double(r);
}

// Riemann upwinding of the reference:  v = (u > 0) ? l : r;  v = (|u| > t) ? v : (l+r)/2
// (0.5 * x as half(x): the same bits, no FP64 multiply)
__device__ __forceinline__ double upwind(double u, double l, double r, long long tb) {
    if (dmag(u) > tb) return dhigh(u) >= 0 ? l : r;
    return half(l + r);
}

// 4. The sign of a product, x*y > 0, without the multiply: the operands are non-zero with
//    equal signs and the product does not round to zero.  With M the 53-bit significand (the
//    magnitude bits of a subnormal, exponent field taken as 1) and E the exponent field,
//    |x*y| = Mx*My * 2^(Ex+Ey-2150), which rounds to zero exactly when it is <= 2^-1075,
//    i.e. Mx*My <= 2^(1075-Ex-Ey).  Normal operands with Ex+Ey >= 972 never do (the common
//    case, decided by the signs alone); the rest compare the 106-bit significand product.
//    Operands are not NaN.
__device__ __forceinline__ bool prod_gt0(double x, double y) {
    const int hx = dhigh(x), hy = dhigh(y);
    if ((hx ^ hy) < 0) return false;
    const int ex = (int)(((unsigned)hx >> 20) & 0x7ff), ey = (int)(((unsigned)hy >> 20) & 0x7ff);
    if (ex >= 1 && ey >= 1 && ex + ey >= 972) return true;
    const long long ax = dmag(x), ay = dmag(y);
    if (ax == 0 || ay == 0) return false;
    if (ex == 0x7ff || ey == 0x7ff) return true;  // an infinity times a non-zero
    const unsigned long long mx = ex ? (unsigned long long)((ax & 0x000fffffffffffffLL) | (1LL << 52)) : ax;
    const unsigned long long my = ey ? (unsigned long long)((ay & 0x000fffffffffffffLL) | (1LL << 52)) : ay;
    const int k = 1075 - (ex ? ex : 1) - (ey ? ey : 1);
    if (k < 0) return true;
    if (k >= 106) return false;
    const unsigned long long lo = mx * my, hi = __umul64hi(mx, my);
    if (k >= 64) {
        const unsigned long long t = 1ULL << (k - 64);
        return hi > t || (hi == t && lo != 0);
    }
    return hi != 0 || lo > (1ULL << k);
}

struct RecipC {
    double y, zh, zl;
    unsigned bad[4];  // low words of the significands that the two-step quotient misrounds
    int nbad;         // -1: more than 4, the quotient is corrected
    unsigned exlo, exn;  // exponent fields of a that are divided so: exn from exlo (0: y not normal)
};

// The integer significands X in [2^52, 2^53) whose quotient by Y (the same range) comes within
// 2^-52 ulp of a rounding boundary: at most 16 (out holds them).
__host__ inline int hard_significands(unsigned long long Y, unsigned long long out[16]) {
    const unsigned long long lo = 1ULL << 52, hi = 1ULL << 53;
    const int v = (Y & 1) ? 0 : (Y & 2) ? 1 : 2;
    if (v == 2) return 0;  // 2^v divides 2^s X - (2m+1) Y, which is not 0: at least 4
    const unsigned long long Y0 = Y >> v, inv2 = (Y0 + 1) / 2;
    int n = 0;
    for (int s = 53; s <= 54; ++s) {
        unsigned long long inv = 1 % Y0;  // of 2^(s-v) modulo Y0
        for (int q = 0; q < s - v; ++q) inv = (unsigned long long)((unsigned __int128)inv * inv2 % Y0);
        for (int N = -3; N <= 3; ++N) {  // the difference over 2^v
            if (N % 2 == 0 || (v == 1 && (N == 3 || N == -3))) continue;
            const unsigned long long r = N > 0 ? (unsigned long long)N % Y0 : (Y0 - (unsigned long long)(-N) % Y0) % Y0;
            for (unsigned long long X = (unsigned long long)((unsigned __int128)r * inv % Y0); X < hi; X += Y0)
                if (X >= lo && (X >= Y) == (s == 53) && n < 16) out[n++] = X;
        }
    }
    return n;
}

__host__ inline RecipC make_recip(double y) {
    RecipC r;
    r.y = y;
    r.zh = 1.0 / y;
    // 1/y - zh = (1 - zh*y)/y; the residual 1 - zh*y is exact with an FMA
    const double e = __builtin_fma(-r.zh, y, 1.0);
    r.zl = e / y;
    r.nbad = 0;
    r.exlo = r.exn = 0;
    for (unsigned& q : r.bad) q = 0;
    const long long b = dbits_host(y);
    const int ex = (int)(b >> 52) & 0x7ff;
    if (ex < 64 || ex > 1983) return r;  // the reciprocal's words could under- or overflow
    const int lo = ex > 1024 ? ex - 960 : 64, hi = ex < 980 ? ex + 1020 : 2000;
    r.exlo = (unsigned)lo;
    r.exn = (unsigned)(hi - lo);
    unsigned long long X[16];
    const int n = hard_significands((unsigned long long)(b & 0x000fffffffffffffLL) | (1ULL << 52), X);
    for (int q = 0; q < n; ++q) {
        const double a = (double)X[q];
        if (__builtin_fma(a, r.zh, a * r.zl) == a / y) continue;
        if (r.nbad == 4) {
            r.nbad = -1;
            return r;
        }
        r.bad[r.nbad++] = (unsigned)X[q];
    }
    for (int q = r.nbad; q < 4; ++q) r.bad[q] = r.nbad ? r.bad[0] : 0;
    return r;
}

__device__ __forceinline__ double div_corrected(double a, const RecipC& r) {
    const double q0 = __fma_rn(a, r.zh, a * r.zl);
    const double rem = __fma_rn(-q0, r.y, a);
    return __fma_rn(rem, r.zh, q0);
}
__device__ __forceinline__ double div_c(double a, const RecipC& r) {
    int hi, lo;
    dsplit(a, hi, lo);
    const unsigned ex = ((unsigned)hi >> 20) & 0x7ff;
    if (ex - r.exlo >= r.exn) {
        // Zeros are common (still fluid, equal neighbours) and cost no division: one lane's took its
        // warp's 20 FP64 instructions, 21 instead of 5 for a tracing coefficient.
        if ((((unsigned)hi << 1) | (unsigned)lo) == 0 && dhigh(r.y) > 0) return a;
        return a / r.y;
    }
    if (r.nbad != 0) {
        if (r.nbad < 0) return div_corrected(a, r);
        const unsigned l = (unsigned)lo;
        if (l == r.bad[0] || l == r.bad[1] || l == r.bad[2] || l == r.bad[3]) return a / r.y;
    }
    return __fma_rn(a, r.zh, a * r.zl);
}

// Division by a value y that several numerators share, formed on the device: the same
// sequence with zh = RN(1/y) by the division and zl = RN(e zh), e = 1 - zh y exact (FMA), which
// is 1/y - zh to a relative 2^-52.  ok: y is in a range where nothing under- or overflows.
struct RecipV {
    RecipC r;
    bool ok;
};
__device__ __forceinline__ RecipV recip_v(double y) {
    RecipV v;
    const unsigned ex = ((unsigned)dhigh(y) >> 20) & 0x7ff;
    v.ok = ex >= 823 && ex < 1223;  // 2^-200 .. 2^200
    v.r.y = y;
    v.r.zh = 1.0 / y;
    v.r.zl = __fma_rn(-v.r.zh, y, 1.0) * v.r.zh;
    return v;
}
__device__ __forceinline__ double div_v(double a, const RecipV& v) {
    const unsigned ex = ((unsigned)dhigh(a) >> 20) & 0x7ff;
    if (!v.ok || ex < 323 || ex >= 1723) {  // |a| outside 2^-700 .. 2^700
        if (v.ok && !nz(a)) return dflip(a, dhigh(v.r.y) < 0);  // a species the cell has none of
        return a / v.r.y;
    }
    return div_corrected(a, v.r);
}

// a / 6 with r6 = make_recip(6): exact for zeros too (zl > 0 keeps their sign)
__device__ __forceinline__ double div_6(double a, const RecipC& r6) {
    const unsigned ex = ((unsigned)dhigh(a) >> 20) & 0x7ff;
    if ((ex < 64 && nz(a)) || ex >= 2000) return a / 6.0;
    return __fma_rn(a, r6.zh, a * r6.zl);
}

// std::min(std::max(v, std::min(a, b)), std::max(a, b)) of the PPM interface clamp, the four
// comparisons on integer keys: 3 keys and 4 comparisons cost about 35 integer instructions,
// 4 FP64 comparisons the issue slots of 256.  v is an FP64 result of a and b: NaN if either
// is, and passed on then.
__device__ __forceinline__ double clamp_between(double v, double a, double b) {
    if ((dhigh(v) & 0x7fffffff) > 0x7ff00000) return v;
    const long long ka = dkey(a), kb = dkey(b), kv = dkey(v);
    const bool ba = kb < ka, ab = ka < kb;
    const double lo = ba ? b : a, hi = ab ? b : a;
    const long long klo = ba ? kb : ka, khi = ab ? kb : ka;
    return kv < klo ? lo : (khi < kv ? hi : v);
}

}  // namespace madv
