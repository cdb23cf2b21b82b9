// ysg_tables.cuh -- sine, cosine and exponential to half a unit in the last
// place, for tables that are formed once and used for every sample.
//
// The time stage's twiddles, taper and e^{eps t} (k_time_tables of k_ifft.cu)
// are formed on the device.  Its library's functions are within 1.36 (sincos)
// and 0.85 (exp) units on those arguments, the host's within 0.51 and 0.50,
// so the device tables are formed in sums of two doubles (Dekker 1971, Knuth
// TAOCP 4.2.2) from the Taylor series of a reduced argument: the leading terms
// in two doubles, the tail in one.
#pragma once
#include <math.h>

#include <cuda_runtime.h>

namespace ysg {

// h + l, |l| at most half a unit of h
struct Two {
    double h, l;
};

__device__ __forceinline__ Two two_sum(double a, double b)
{
    const double s = __dadd_rn(a, b), t = __dsub_rn(s, a);
    return Two{s, __dadd_rn(__dsub_rn(a, __dsub_rn(s, t)), __dsub_rn(b, t))};
}
__device__ __forceinline__ Two two_fast(double a, double b)      // |a| >= |b|
{
    const double s = __dadd_rn(a, b);
    return Two{s, __dsub_rn(b, __dsub_rn(s, a))};
}
__device__ __forceinline__ Two two_mul(double a, double b)
{
    const double p = __dmul_rn(a, b);
    return Two{p, fma(a, b, -p)};
}
__device__ __forceinline__ Two two_mul(Two a, Two b)
{
    const Two p = two_mul(a.h, b.h);
    return two_fast(p.h, __dadd_rn(p.l, fma(a.h, b.l, __dmul_rn(a.l, b.h))));
}
__device__ __forceinline__ Two two_add(Two a, Two b)
{
    const Two s = two_sum(a.h, b.h), t = two_sum(a.l, b.l);
    const Two u = two_fast(s.h, __dadd_rn(s.l, t.h));
    return two_fast(u.h, __dadd_rn(u.l, t.l));
}
__device__ __forceinline__ Two two_add(Two a, double b)
{
    const Two s = two_sum(a.h, b);
    return two_fast(s.h, __dadd_rn(s.l, a.l));
}
__device__ __forceinline__ Two two_scale(double s, Two a) { return Two{s * a.h, s * a.l}; }    // s a power of two

// sin a and cos a, |a| <= 4: a = q pi/2 + r, series of r / 4, then twice
// (sin, 1 - cos)(2x) = (2 sin (1 - (1 - cos)), 2 sin^2).
__device__ __forceinline__ void table_sincos(double a, double* sn, double* cs)
{
    const double q = rint(a * 0.6366197723675814);
    const Two half_pi{-1.5707963267948966, -6.123233995736766e-17};
    const Two x = two_scale(0.25, two_add(two_mul(Two{q, 0.0}, half_pi), a));
    const Two z = two_mul(x, x), z2 = two_mul(z, z);
    const double y = z.h, y3 = y * y * y;
    // 1 - cos x = z/2 - z^2/24 + z^3/6! - ..
    const double tv = y3 * fma(y, fma(y, fma(y, fma(y, 1.0 / 87178291200.0, -1.0 / 479001600.0), 1.0 / 3628800.0),
                                      -1.0 / 40320.0), 1.0 / 720.0);
    const Two c24{-1.0 / 24.0, -2.3129646346357427e-18};
    Two v = two_add(two_add(two_scale(0.5, z), two_mul(z2, c24)), tv);
    // sin x = x (1 - z/6 + z^2/120 - z^3/7! + ..)
    const double ts = y3 * fma(y, fma(y, fma(y, -1.0 / 6227020800.0, 1.0 / 39916800.0), -1.0 / 362880.0), 1.0 / 5040.0);
    const Two c6{-1.0 / 6.0, -9.25185853854297e-18}, c120{1.0 / 120.0, 1.1564823173178714e-19};
    Two s = two_add(two_mul(x, two_add(two_add(two_mul(z, c6), two_mul(z2, c120)), -ts)), x);
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const Two sv = two_mul(s, v), ss = two_mul(s, s);
        s = two_add(two_scale(2.0, s), two_scale(-2.0, sv));
        v = two_scale(2.0, ss);
    }
    const double si = s.h, co = two_add(Two{-v.h, -v.l}, 1.0).h;
    const int k = (int)q;
    *sn = k & 1 ? co : si;
    *cs = k & 1 ? si : co;
    if (k & 2) *sn = -*sn;
    if ((k + 1) & 2) *cs = -*cs;
}

// e^a: a = k ln 2 + r, series of r / 16 for e^y - 1, then four times
// E(2y) = 2 E + E^2.
__device__ __forceinline__ double table_exp(double a)
{
    if (!(fabs(a) < 700.0)) return exp(a);
    const double k = rint(a * 1.4426950408889634);
    const Two ln2{-0.6931471805599453, -2.3190468138462996e-17};
    const Two r = two_add(two_mul(Two{k, 0.0}, ln2), a);
    const Two y = two_scale(0.0625, r), y2 = two_mul(y, y);
    const double t = y.h, t2 = t * t;
    const double tail = t2 * t2 * fma(t, fma(t, fma(t, fma(t, fma(t, 1.0 / 362880.0, 1.0 / 40320.0), 1.0 / 5040.0),
                                                    1.0 / 720.0), 1.0 / 120.0), 1.0 / 24.0);
    const Two c6{1.0 / 6.0, 9.25185853854297e-18};
    Two e = two_add(two_add(two_add(two_mul(two_mul(y2, y), c6), tail), two_scale(0.5, y2)), y);
#pragma unroll 1
    for (int q = 0; q < 4; q++) e = two_add(two_scale(2.0, e), two_mul(e, e));
    return scalbn(two_add(e, 1.0).h, (int)k);
}

}  // namespace ysg
