// gb_ozconv.h -- exact integer -> FP64 conversions of the error-free digit
// splitting (host and device code, no intrinsics beyond count-leading-zeros and
// a bit cast, so that the same functions compile into a CPU check).
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define OZ_HD __host__ __device__ __forceinline__
#else
#define OZ_HD inline
#endif

OZ_HD int oz_clz64(unsigned long long x)
{
#ifdef __CUDA_ARCH__
    return __clzll((long long)x);
#else
    return x ? __builtin_clzll(x) : 64;
#endif
}

OZ_HD double oz_bits_to_double(unsigned long long u)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double d;
    memcpy(&d, &u, sizeof d);
    return d;
#endif
}

// (hi 2^SH + lo) 2^(s - 16 - SH) rounded once to nearest-even, s = e + f -
// OZ_SCALE_OFFSET: hi holds levels 0-2 in units of 2^-16, lo the lower levels in
// units of 2^-(16 + SH) (SH = 32 for levels 3-6, 40 for levels 3-7). General
// 128-bit form (any hi, lo).
template <int SH>
OZ_HD double oz_to_double(long long hi, long long lo, int s)
{
    __int128 z = ((__int128)hi << SH) + (__int128)lo;
    if (z == 0) return 0.0;
    unsigned long long sign = 0;
    if (z < 0) {
        sign = 1ull << 63;
        z = -z;
    }
    const unsigned __int128 u = (unsigned __int128)z;
    const unsigned long long zh = (unsigned long long)(u >> 64), zl = (unsigned long long)u;
    const int nb = zh ? 128 - oz_clz64(zh) : 64 - oz_clz64(zl);
    int E = nb - 1 + s - 16 - SH;
    unsigned long long m;
    if (nb <= 53) {
        m = zl << (53 - nb);
    } else {
        const int sh = nb - 53;
        const unsigned __int128 q = u >> sh;
        const unsigned __int128 rem = u - (q << sh);
        const unsigned __int128 half = (unsigned __int128)1 << (sh - 1);
        m = (unsigned long long)q;
        if (rem > half || (rem == half && (m & 1))) ++m;
        if (m >> 53) {
            m >>= 1;
            ++E;
        }
    }
    if (E < -1022 || E > 1023)                     // outside the normal range: scale in FP64
        return ldexp((double)hi, s - 16) + ldexp((double)lo, s - 16 - SH);
    return oz_bits_to_double(sign | ((unsigned long long)(E + 1023) << 52) | (m & ((1ull << 52) - 1)));
}

// z 2^e0 rounded once to nearest-even, z any 128-bit integer (the exact sum of a
// Gram entry's split partials, hi 2^40 + lo summed over the splits)
OZ_HD double oz_i128_to_double(__int128 z, int e0)
{
    if (z == 0) return 0.0;
    unsigned long long sign = 0;
    if (z < 0) {
        sign = 1ull << 63;
        z = -z;
    }
    const unsigned __int128 u = (unsigned __int128)z;
    const unsigned long long zh = (unsigned long long)(u >> 64), zl = (unsigned long long)u;
    const int nb = zh ? 128 - oz_clz64(zh) : 64 - oz_clz64(zl);
    int E = nb - 1 + e0;
    unsigned long long m;
    if (nb <= 53) {
        m = zl << (53 - nb);
    } else {
        const int sh = nb - 53;
        const unsigned __int128 q = u >> sh;
        const unsigned __int128 rem = u - (q << sh);
        const unsigned __int128 half = (unsigned __int128)1 << (sh - 1);
        m = (unsigned long long)q;
        if (rem > half || (rem == half && (m & 1))) ++m;
        if (m >> 53) {
            m >>= 1;
            ++E;
        }
    }
    if (E < -1022 || E > 1023) {                   // outside the normal range: scale in FP64
        const double mag = ldexp((double)zh, e0 + 64) + ldexp((double)zl, e0);
        return sign ? -mag : mag;
    }
    return oz_bits_to_double(sign | ((unsigned long long)(E + 1023) << 52) | (m & ((1ull << 52) - 1)));
}

// The same value for SH = 40 in 64-bit arithmetic, for |hi| < 2^41 and |lo| < 2^62
// (eight levels of at most 2^24 each). z = hi 2^40 + lo = T 2^18 + R with T =
// floor(z / 2^18) (|T| < 2^63) and 0 <= R < 2^18; |z| is carried as U 2^e where
// U is exact (|z| < 2^63) or U keeps at least 55 bits and the discarded bits are
// folded into its lowest bit (round to odd), so that rounding U once to 53 bits
// (nearest-even) gives the correctly rounded |z| -- the result of the general
// form bit for bit.
OZ_HD double oz_to_double40(long long hi, long long lo, int s)
{
    const long long T = hi * (1LL << 22) + (lo >> 18);
    const unsigned long long R = (unsigned long long)(lo & 0x3ffffLL);
    if (T == 0 && R == 0) return 0.0;
    unsigned long long sign = 0, Tm = (unsigned long long)T, Rm = R;
    if (T < 0) {
        sign = 1ull << 63;
        Tm = R ? (unsigned long long)(-(T + 1)) : (unsigned long long)(-T);
        Rm = R ? (1ull << 18) - R : 0;
    }
    unsigned long long U;
    int e;
    if (Tm < (1ull << 45)) {
        U = (Tm << 18) | Rm;
        e = 0;
    } else if (Tm < (1ull << 55)) {
        U = (Tm << 9) | (Rm >> 9) | (unsigned long long)((Rm & 0x1ffull) != 0);
        e = 9;
    } else {
        U = Tm | (unsigned long long)(Rm != 0);
        e = 18;
    }
    const int nb = 64 - oz_clz64(U);
    int E = nb - 1 + e + s - 56;
    unsigned long long m;
    if (nb <= 53) {
        m = U << (53 - nb);
    } else {
        const int sh = nb - 53;
        m = U >> sh;
        const unsigned long long rem = U & ((1ull << sh) - 1), half = 1ull << (sh - 1);
        if (rem > half || (rem == half && (m & 1))) ++m;
        if (m >> 53) {
            m >>= 1;
            ++E;
        }
    }
    if (E < -1022 || E > 1023)
        return ldexp((double)hi, s - 16) + ldexp((double)lo, s - 56);
    return oz_bits_to_double(sign | ((unsigned long long)(E + 1023) << 52) | (m & ((1ull << 52) - 1)));
}

// ---------------------------------------------------------------- 32-bit forms
// The kernels that split and round are bound by the instructions they issue, and the
// 64-bit shifts and comparisons above are several each. These work in 32-bit
// words: clamped shifts (amounts past 31 give zero), funnel shifts and carries.

// x >> s, 0 for s > 31
OZ_HD uint32_t oz_shr(uint32_t x, uint32_t s)
{
#ifdef __CUDA_ARCH__
    uint32_t r;
    asm("shr.b32 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(s));
    return r;
#else
    return s > 31 ? 0 : x >> s;
#endif
}
// low word of (hi:lo) >> s, s clamped to 32
OZ_HD uint32_t oz_fsr(uint32_t lo, uint32_t hi, uint32_t s)
{
#ifdef __CUDA_ARCH__
    return __funnelshift_rc(lo, hi, s);
#else
    if (s > 32) s = 32;
    return (uint32_t)((((unsigned long long)hi << 32) | lo) >> s);
#endif
}
// high word of (hi:lo) << s, s < 32
OZ_HD uint32_t oz_fsl(uint32_t lo, uint32_t hi, uint32_t s)
{
#ifdef __CUDA_ARCH__
    return __funnelshift_l(lo, hi, s);
#else
    return s ? (hi << s) | (lo >> (32 - s)) : hi;
#endif
}
OZ_HD int oz_clz32(uint32_t x)
{
#ifdef __CUDA_ARCH__
    return __clz((int)x);
#else
    return x ? __builtin_clz(x) : 32;
#endif
}

#define OZ_SHIFT0 1025              // scale e of an entry's row or column + this = its shift base
#define OZ_SHIFT_NONE 20000         // shift base that leaves nothing of an entry

// The biased digits of the double (hi, lo) against scale e, sb = e + OZ_SHIFT0: the integer
// U = T + 0x80808080808080 of gb_tc05.h in bytes 1..7 of the result (byte 0 is left
// over). The significand, left-justified in 64 bits, goes right by r + 3, r = e +
// 1022 - exponent, so that it ends seven bits below T's rounding bit: s' = 2 s + f
// with s = 2^7 floor(2 T'), T' = mant 2^-r. Rounding half up and the sign are then
// one exclusive-or and one addition, U 2^8 = floor((s' ^ m) + (2 B + 1) 2^7), m all
// ones for a negative entry: for it ~s' = -s' - 1, and the bits below the rounding
// bit cannot reach a carry in either sign. 18 instructions, no branch; the kernels
// that split are bound by the integer pipe (half rate), and the plain 64-bit form
// takes about 45.
OZ_HD unsigned long long oz_digits(uint32_t hi, uint32_t lo, int sb)
{
    const int ex = (int)((hi >> 20) & 0x7ff);
    const int sh = ex ? sb - ex : 255;                     // 0 and subnormals: nothing
    const uint32_t mh = oz_fsl(lo, hi, 11) | 0x80000000u, ml = lo << 11;
    const int over = sh - 32 > 0 ? sh - 32 : 0;
    const uint32_t sl = oz_shr(oz_fsr(ml, mh, (uint32_t)sh), (uint32_t)over);
    const unsigned long long sp = (unsigned long long)oz_shr(mh, (uint32_t)sh) << 32 | sl;
    const long long m = (long long)((int)hi >> 31);
    return (sp ^ (unsigned long long)m) + 0x8080808080808080ull;
}

// The eight level sums v (exact integers, |v| <= 2^24, weights 2^(8 (7 - L))) as
// sum v 2^(s - 56), rounded once to nearest-even: what oz_to_double40 gives for
// their (hi, lo). The sum, below 2^82, in three words; the leading 64 bits by
// funnel shifts, the rest into a sticky bit.
OZ_HD double oz_levels_to_double(const int v[8], int s)
{
    const long long lo = (((long long)v[6] * 256 + v[7]) + (long long)v[5] * 65536) + (long long)v[4] * 16777216 +
                         ((long long)v[3] << 32);
    const long long hi = ((long long)v[1] * 256 + v[2]) + (long long)v[0] * 65536;
    // z = hi 2^40 + lo
    uint32_t w0 = (uint32_t)lo;
    unsigned long long up = (unsigned long long)(lo >> 32) + ((unsigned long long)hi << 8);
    const uint32_t sign = (uint32_t)(up >> 63) ? 0xffffffffu : 0u;
    // |z|
    w0 = (w0 ^ sign) - sign;
    up = (up ^ ((unsigned long long)sign << 32 | sign)) + (unsigned long long)(sign && w0 == 0);
    uint32_t w1 = (uint32_t)up, w2 = (uint32_t)(up >> 32);
    int nb = 96;
    if (w2 == 0) {
        w2 = w1;
        w1 = w0;
        w0 = 0;
        nb = 64;
        if (w2 == 0) {
            w2 = w1;
            w1 = 0;
            nb = 32;
            if (w2 == 0) return 0.0;
        }
    }
    const int lz = oz_clz32(w2);
    nb -= lz;
    const uint32_t th = oz_fsl(w1, w2, lz), tl = oz_fsl(w0, w1, lz);
    const uint32_t rest = w0 << lz;
    const int E = nb - 1 + s - 56;
    if (E < -1022 || E > 1022) return oz_to_double40(hi, lo, s);
    const uint32_t sticky = (tl & 0x3ffu) | rest;
    const uint32_t mh = th >> 11, ml = oz_fsl(tl, th, 21);
    const uint32_t inc = (tl >> 10) & 1u & (uint32_t)(sticky != 0 || (ml & 1u));
    unsigned long long b = (((unsigned long long)mh << 32) | ml) + inc;
    b += (unsigned long long)(uint32_t)((E + 1022) << 20) << 32;
    return oz_bits_to_double(b | (unsigned long long)(sign & 0x80000000u) << 32);
}
