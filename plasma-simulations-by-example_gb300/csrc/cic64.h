/*
 * cic64.h -- pieces of the float64 cloud-in-cell kernels that keep work off
 * the float64 pipe.  GB300 issues a float64 instruction of a warp in 16
 * clocks of its SM, in which the four schedulers issue 64 others, so a test,
 * a truncation or a quotient done on the integer pipes is nearly free beside
 * one done in float64.  Every function returns the bits of the plain
 * expression it stands for (units that use them are built with -fmad=false).
 */
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace espic {

/* x == +-0 on the 32-bit halves of its bits: a 64-bit test of the bits
 * compiles to a float64 compare */
__device__ __forceinline__ bool zero_bits(double x) {
    return (((unsigned int)__double2hiint(x) << 1) | (unsigned int)__double2loint(x)) == 0u;
}

/* isfinite without a float64 compare */
__device__ __forceinline__ bool finite_bits(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }

/* a / b correctly rounded, given y = RN(1/b) for b > 0: q = a y, the exact
 * remainder r = a - b q (one FMA), then q + r y rounded -- Markstein's
 * correction (P. Markstein, IBM J. Res. Develop. 34(1), 1990), which yields
 * the correctly rounded quotient for normal operands, so results equal the
 * division's bit for bit; a = +-0 returns a y, the zero of the right sign. */
__device__ __forceinline__ double div_rcp(double a, double b, double y) {
    const double q = a * y;
    const double r = __fma_rn(-q, b, a);
    const double q2 = __fma_rn(r, y, q);
    return zero_bits(a) ? q : q2;
}

/* integers in the order of the doubles (-0 and +0 equal); the order of NaN is
 * that of a value beyond infinity of its sign */
__device__ __forceinline__ long long order_key(double x) {
    const long long b = __double_as_longlong(x);
    const long long m = b & 0x7fffffffffffffffll;
    return b < 0 ? -m : m;
}

/* F 2^-64 as a double, F of at most 53 significant bits; F = 0 gives `zero` */
__device__ __forceinline__ double fixed64(unsigned long long F, double zero) {
    const int n = __clzll((long long)F) & 63;
    const unsigned long long m = F << n; /* the leading bit on top */
    const double x = __longlong_as_double(((long long)(1022 - n) << 52) + (long long)((m << 1) >> 12));
    return F ? x : zero;
}

/* lc, a logical coordinate along an axis of n nodes, as its cell, the offset
 * off = lc - cell and rest = 1 - off, with the bits of the float64
 * expressions and integer operations alone: from 1 on, lc's fraction is a
 * 64-bit fixed point number that both differences take exactly; below 1, off
 * is lc, and rest counts units of 2^-53, the spacing of doubles from 1/2 to 1,
 * by which lc is rounded with ties to even (an lc above 1/2 is a whole number
 * of them).  False, with nothing set, for lc outside [0, n - 1) or not
 * finite: the caller then takes its general path. */
__device__ __forceinline__ bool cell_of(double lc, int n, int &cell, double &off, double &rest) {
    const int hi = __double2hiint(lc);
    if ((unsigned)hi >= 0x41300000u) return false; /* negative, 2^20 or more, not finite */
    const int e = (hi >> 20) - 1023;               /* lc >= 1: e in 0..19 */
    const unsigned long long b = (unsigned long long)__double_as_longlong(lc);
    if (e < 0) {
        cell = 0;
        off = lc;
        const unsigned long long m = (b & 0xfffffffffffffull) | 0x10000000000000ull; /* lc = m 2^(e-52) */
        const int t = e < -63 ? 62 : -1 - e;
        const unsigned long long D = t ? (m + ((1ull << (t - 1)) - 1ull) + ((m >> t) & 1ull)) >> t : m;
        rest = fixed64((0x20000000000000ull - D) << 11, 1.0);
        return true;
    }
    const int c = ((hi & 0xfffff) | 0x100000) >> (20 - e);
    if (c > n - 2) return false;
    const unsigned long long F = (b << 12) << e;
    cell = c;
    off = fixed64(F, 0.0);
    rest = fixed64(0ull - F, 1.0);
    return true;
}

/* the 24 leading bits of x as a float (0 below 2^-126; false above the float
 * range), within 2^-23 |x| of x */
__device__ __forceinline__ bool cut_float(double x, float &xf) {
    const int hi = __double2hiint(x);
    const unsigned lo = (unsigned)__double2loint(x);
    const int fe = ((hi >> 20) & 0x7ff) - 896; /* float exponent field */
    xf = 0.0f;
    if (fe >= 1) xf = __int_as_float((hi & (int)0x80000000) | (fe << 23) | ((hi & 0xfffff) << 3) | (int)(lo >> 29));
    return fe <= 254;
}

/* A double's magnitude for round_product: its 53-bit mantissa 10 bits up, and
 * its exponent field (numbers below 2^-1022 count as 0). */
struct Mantissa {
    unsigned long long m;
    int f;
};

__device__ __forceinline__ Mantissa mantissa_of(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int f = (int)(b >> 52) & 0x7ff;
    return {f ? ((b & 0xfffffffffffffull) | 0x10000000000000ull) << 10 : 0ull, f};
}

/* The magnitude of the exact product of two such numbers, rounded to the
 * nearest integer (ties to even), for products below 2^51: the 128-bit
 * product of the mantissas (one shifted 11 bits instead of 10, which makes
 * 21), its lower half folded into a sticky bit.  About 30 integer
 * operations, half the time of the one float64 FMA that does the same
 * (RN(a b + 1.5 2^52)). */
__device__ __forceinline__ unsigned long long round_product(Mantissa a, Mantissa b) {
    const unsigned long long bm = b.m << 1;
    unsigned long long h = __umul64hi(a.m, bm);
    h |= (a.m * bm) != 0ull;
    const int t = 2107 - (a.f + b.f);
    if (t > 63) return 0ull;
    return (h + ((1ull << (t - 1)) - 1ull) + ((h >> t) & 1ull)) >> t;
}

/* The magnitude of RN(a b) rounded to the nearest integer (both to even), for
 * products below 2^51: what a float64 multiplication and a conversion give.
 * As round_product, with the product rounded to 53 bits first.  About 45
 * integer operations in place of the multiplication and the 18 that a rounding
 * of its bits takes. */
__device__ __forceinline__ unsigned long long round_twice(Mantissa a, Mantissa b) {
    const unsigned long long bm = b.m << 1;
    unsigned long long h = __umul64hi(a.m, bm); /* 62 or 63 bits, or 0 */
    h |= (a.m * bm) != 0ull;
    const int d = 9 + (int)(h >> 62);
    const unsigned long long r = (h + ((1ull << (d - 1)) - 1ull) + ((h >> d) & 1ull)) >> d;
    const int s = 2107 - (a.f + b.f) - d, t = s > 62 ? 62 : s; /* a b = r 2^-s, s >= 1; 0 from 55 on */
    return (r + ((1ull << (t - 1)) - 1ull) + ((r >> t) & 1ull)) >> t;
}

/* (double)c, rounded to nearest even, by integer operations */
__device__ __forceinline__ double count_to_double(long long c) {
    const unsigned long long a = c < 0 ? 0ull - (unsigned long long)c : (unsigned long long)c;
    const int n = __clzll((long long)a) & 63;
    const unsigned long long m = a << n, h = m >> 11; /* 53 bits, the leading one on top */
    const unsigned tail = (unsigned)m & 0x7ffu;
    const unsigned long long up = tail > 0x400u - (unsigned)(h & 1ull); /* half and odd, or more than half */
    const unsigned long long b = ((unsigned long long)(1085 - n) << 52) + h + up;
    const double x = __longlong_as_double((long long)(b | ((unsigned long long)c & 0x8000000000000000ull)));
    return a ? x : 0.0;
}

/* The warp's Field_::scatter of `value` at cell offsets d with e = 1 - d, each
 * corner weight value*(1-di)*(1-dj)*(1-dk) (the reference's operand order)
 * rounded once to an integer count of 1/fx and added to acc.  fx is a power
 * of two, so it multiplies the value once instead of eight weights.
 * unit_cell: d lies in [0, 1), so that no weight exceeds the value; where the
 * value's count is below 2^51, the last product of each weight and its
 * rounding are integer operations, so that the float64 pipe and the others
 * carry like loads (6M particles on 97x89x117 nodes: 497 us with float64
 * products and differences 1 - d, 401 us now; 20,000 particles take 13 us
 * either way).  Two neighbouring lanes add to the two x corners of one
 * particle, which mostly lie in one 32-byte sector.  Every
 * lane of the warp calls it; n0: the cell's first node; a particle that is
 * not live adds nothing. */
__device__ __forceinline__ void scatter8(unsigned long long *acc, uint32_t n0, int64_t sy, int64_t sz,
                                         const double d[3], const double e[3], double value, double fx,
                                         bool unit_cell, bool live) {
    const unsigned FULL = 0xffffffffu;
    const bool odd = threadIdx.x & 1;
    const double v = value * fx;
    const double a0 = v * e[0], a1 = v * d[0];
    /* (j, k) rows of low and high x corners */
    const double lo[2] = {a0 * e[1], a0 * d[1]}, hi[2] = {a1 * e[1], a1 * d[1]};
    const int64_t row[4] = {0, sy, sz, sy + sz};
    /* decided for the warp, so that the float64 products and conversions sit
     * behind a branch */
    const bool small = __all_sync(FULL, !live || (unit_cell && (__double2hiint(v) & 0x7fffffff) < 0x43200000));
    const uint32_t mate = __shfl_xor_sync(FULL, n0, 1);
    unsigned long long *even = acc + (odd ? mate : n0) + odd, *other = acc + (odd ? n0 : mate) + odd;
    const Mantissa me = mantissa_of(e[2]), md = mantissa_of(d[2]);
#pragma unroll
    for (int r = 0; r < 4; r++) {
        long long ql, qh;
        if (small) {
            const long long sign = (long long)(__double2hiint(v) >> 31); /* -1 or 0 */
            ql = (long long)round_twice(mantissa_of(lo[r & 1]), r < 2 ? me : md);
            qh = (long long)round_twice(mantissa_of(hi[r & 1]), r < 2 ? me : md);
            ql = (ql ^ sign) - sign;
            qh = (qh ^ sign) - sign;
        } else {
            ql = __double2ll_rn(lo[r & 1] * (r < 2 ? e[2] : d[2]));
            qh = __double2ll_rn(hi[r & 1] * (r < 2 ? e[2] : d[2]));
        }
        if (!live) ql = qh = 0;
        const long long got = __shfl_xor_sync(FULL, odd ? ql : qh, 1);
        const long long ce = odd ? got : ql, co = odd ? qh : got;
        if (ce) atomicAdd(even + row[r], (unsigned long long)ce);
        if (co) atomicAdd(other + row[r], (unsigned long long)co);
    }
}

}  // namespace espic
