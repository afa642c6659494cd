/* cic64_host.cpp -- TEST INFRASTRUCTURE: the integer formulas of csrc/cic64.h
 * compiled as host code, against the float64 expressions they stand for.  The
 * device intrinsics they use are restated here.  Built by
 * tests/test_cic64_host.py with g++ into a temporary folder that also holds an
 * empty cuda_runtime.h. */
#include <cmath>
#include <cstdint>
#include <cstring>
#include <random>

#define __device__
#define __forceinline__ inline

static inline int64_t bits(double x) {
    int64_t b;
    memcpy(&b, &x, 8);
    return b;
}
static inline int __double2hiint(double x) { return (int)(bits(x) >> 32); }
static inline int __double2loint(double x) { return (int)bits(x); }
static inline long long __double_as_longlong(double x) { return bits(x); }
static inline double __longlong_as_double(long long b) {
    double x;
    memcpy(&x, &b, 8);
    return x;
}
static inline float __int_as_float(int b) {
    float x;
    memcpy(&x, &b, 4);
    return x;
}
static inline int __clzll(long long x) { return x ? __builtin_clzll(x) : 64; }
static inline unsigned long long __umul64hi(unsigned long long a, unsigned long long b) {
    return (unsigned long long)(((unsigned __int128)a * b) >> 64);
}
static inline double __fma_rn(double a, double b, double c) { return fma(a, b, c); }
static inline long long __double2ll_rn(double x) { return llrint(x); }
/* named by scatter8, which this file does not call */
static const struct { int x; } threadIdx = {0};
static inline bool __all_sync(unsigned, bool p) { return p; }
template <class T>
static inline T __shfl_xor_sync(unsigned, T v, int) {
    return v;
}
static inline void atomicAdd(unsigned long long *, unsigned long long) {}

#include "cic64.h"

using namespace espic;

static std::mt19937_64 rng(64);
static double unit() { return (double)(rng() >> 11) * 0x1p-53; }
static bool same(double a, double b) { return bits(a) == bits(b); }

/* logical coordinates: uniform, near whole numbers, tiny, with few bits */
static double coordinate(int kind, int n) {
    switch (kind) {
        case 0: return unit() * (n - 1);
        case 1: return unit();
        case 2: return ldexp(unit(), -(int)(rng() % 1074));
        case 3: return (double)(rng() % (n - 1)) + ldexp((double)(rng() % 3), -(int)(1 + rng() % 60));
        case 4: return ldexp((double)(rng() % (1 << 20)) + 0.5, -(int)(rng() % 70));
        case 5: return nextafter((double)(1 + rng() % (n - 1)), rng() & 1 ? 0.0 : 1e9);
        default: return rng() % 2 ? 0.0 : (double)(rng() % n);
    }
}

extern "C" long long cic_cells(long long count, int n) {
    long long bad = 0;
    for (long long i = 0; i < count; i++) {
        const double lc = coordinate((int)(i % 7), n);
        int c;
        double off, rest;
        const bool ok = cell_of(lc, n, c, off, rest), in = lc >= 0 && lc < n - 1;
        if (ok != in) {
            bad++;
        } else if (ok) {
            const double want = lc - (double)(int)lc;
            bad += c != (int)lc || !same(off, want) || !same(rest, 1 - want);
        }
    }
    const double out[] = {-1.0, -0.0, -1e-300, 1048576.0, 1e300, INFINITY, -INFINITY, NAN, -NAN, (double)(n - 1)};
    for (double lc : out) {
        int c;
        double off, rest;
        bad += cell_of(lc, n, c, off, rest);
    }
    return bad;
}

/* products below 2^51 of two factors, and their rounded counts */
extern "C" long long cic_products(long long count) {
    long long bad = 0;
    for (long long i = 0; i < count; i++) {
        double a = ldexp(unit(), (int)(rng() % 120) - 68), b = unit();
        if (i % 3 == 0) a = ldexp((double)(1 + rng() % 4096), (int)(rng() % 40) - 30); /* ties */
        if (i % 5 == 0) b = ldexp((double)(rng() % 2049), -11);
        if (i % 64 == 1) a = i % 128 == 1 ? 0.0 : 4e-320;
        if (!(a * b < 0x1p51)) continue;
        bad += (long long)round_twice(mantissa_of(a), mantissa_of(b)) != llrint(a * b);
        /* the exact product rounded once: RN(a b + 1.5 2^52) by one FMA */
        const double shifted = fma(a, b, 0x1.8p52);
        bad += (long long)round_product(mantissa_of(a), mantissa_of(b)) != (long long)(shifted - 0x1.8p52);
    }
    return bad;
}

extern "C" long long cic_counts(long long count) {
    long long bad = 0;
    for (long long i = 0; i < count; i++) {
        long long c = (long long)(rng() >> (rng() % 64));
        if (i % 4 == 0) c = (long long)(((rng() >> 11) << (rng() % 11)) + (1ull << (rng() % 12))); /* ties and carries */
        if (i % 2) c = -c;
        bad += !same(count_to_double(c), (double)c);
    }
    const long long edge[] = {0, 1, -1, (1ll << 53) - 1, 1ll << 53, (1ll << 53) + 1, (1ll << 54) + 2, (1ll << 54) + 6,
                              INT64_MAX, INT64_MIN, INT64_MAX - 511, INT64_MAX - 512, -(1ll << 62) - 256};
    for (long long c : edge) bad += !same(count_to_double(c), (double)c);
    return bad;
}

extern "C" long long cic_quotients(long long count) {
    long long bad = 0;
    for (long long i = 0; i < count; i++) {
        double a = (unit() + (i & 1)) * (rng() & 1 ? 1 : -1), b = 1 + unit();
        if (i % 4 == 0) b = 2 - ldexp((double)(1 + rng() % 1000), -52); /* reciprocals farthest from exact */
        a = ldexp(a, (int)(rng() % 400) - 200);
        b = ldexp(b, (int)(rng() % 400) - 200);
        if (i % 64 == 3) a = i & 64 ? 0.0 : -0.0;
        bad += !same(div_rcp(a, b, 1.0 / b), a / b);
    }
    return bad;
}

/* integer order and tests against float64's */
extern "C" long long cic_keys(long long count) {
    long long bad = 0;
    for (long long i = 0; i < count; i++) {
        double v[2];
        for (double &x : v) {
            const uint64_t r = rng();
            memcpy(&x, &r, 8);
            if (i % 8 == 0) x = rng() & 1 ? 0.0 : -0.0;
            if (i % 8 == 1) x = rng() & 1 ? INFINITY : -INFINITY;
        }
        bad += zero_bits(v[0]) != (v[0] == 0) || finite_bits(v[0]) != (bool)std::isfinite(v[0]);
        if (std::isnan(v[0]) || std::isnan(v[1])) continue;
        bad += (order_key(v[0]) < order_key(v[1])) != (v[0] < v[1]);
        float f;
        if (cut_float(v[0], f))
            bad += !(std::fabs((double)f - v[0]) <= std::fmax(std::ldexp(std::fabs(v[0]), -23), 0x1p-126));
        else
            bad += std::fabs(v[0]) < 0x1p127;
    }
    return bad;
}
