// crmath.cuh -- x^y rounded to nearest from a double-double evaluation.
//
// The reference's adaptive step controllers call pow(r, -0.2)
// (PropagationCK.cpp:116, :123, PropagationBP.cpp:104, :111) and DiffusionSDE
// calls pow(|rigidity|/4e9, alpha) (DiffusionSDE.cpp:263).  glibc's pow is
// within 0.52 ulp, so it returns the correctly rounded result except in rare
// near-midpoint cases; CUDA's pow has a 2-ulp bound and differs from glibc in
// the last place on a few per cent of inputs, which changes accept/reject
// decisions of the step controller.  cr_pow evaluates log and exp in
// double-double arithmetic (about 100 bits) with the classic reductions:
//   log: x = 2^k m, m in [sqrt(1/2), sqrt(2)), log m = 2 atanh((m-1)/(m+1))
//        by its odd power series;
//   exp: t = j ln2 + u, u / 2^8 by its Taylor series, squared 8 times.
// and rounds hi + lo once.  Valid for finite x > 0 and finite y with
// |y log x| < 700; other inputs fall back to pow().  Host and device, as the
// quotients, roots and reciprocals without divisions at the end.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define CRP_HD __host__ __device__ __forceinline__
#else
#define CRP_HD inline
#endif

namespace crp {

struct dd {
    double hi, lo;
};

CRP_HD dd dd_two_sum(double a, double b) {
    double s = a + b;
    double bb = s - a;
    double e = (a - (s - bb)) + (b - bb);
    return {s, e};
}

CRP_HD dd dd_fast_two_sum(double a, double b) {
    double s = a + b;
    return {s, b - (s - a)};
}

CRP_HD dd dd_two_prod(double a, double b) {
    double p = a * b;
    return {p, fma(a, b, -p)};
}

CRP_HD dd dd_add(dd a, dd b) {
    dd s = dd_two_sum(a.hi, b.hi);
    dd t = dd_two_sum(a.lo, b.lo);
    s.lo += t.hi;
    s = dd_fast_two_sum(s.hi, s.lo);
    s.lo += t.lo;
    return dd_fast_two_sum(s.hi, s.lo);
}

CRP_HD dd dd_mul(dd a, dd b) {
    dd p = dd_two_prod(a.hi, b.hi);
    p.lo += a.hi * b.lo + a.lo * b.hi;
    return dd_fast_two_sum(p.hi, p.lo);
}

CRP_HD dd dd_mul_d(dd a, double b) {
    dd p = dd_two_prod(a.hi, b);
    p.lo += a.lo * b;
    return dd_fast_two_sum(p.hi, p.lo);
}

CRP_HD dd dd_div(dd a, dd b) {
    double q1 = a.hi / b.hi;
    dd r = dd_add(a, dd_mul_d(b, -q1));
    double q2 = r.hi / b.hi;
    r = dd_add(r, dd_mul_d(b, -q2));
    double q3 = r.hi / b.hi;
    dd q = dd_fast_two_sum(q1, q2);
    return dd_add(q, dd{q3, 0.0});
}

// ln 2 and its tail
#define CRP_LN2_HI 6.93147180559945286227e-01
#define CRP_LN2_LO 2.31904681384629955842e-17

// natural log of x > 0 (finite, normal) in double-double
CRP_HD dd dd_log(double x) {
    int k;
    double m = frexp(x, &k);  // x = m 2^k, m in [0.5, 1)
    if (m < 0.70710678118654752440) {
        m *= 2.0;
        k -= 1;
    }
    // s = (m - 1) / (m + 1); m - 1 is exact (Sterbenz)
    dd num = {m - 1.0, 0.0};
    dd den = dd_two_sum(m, 1.0);
    dd s = dd_div(num, den);
    dd z = dd_mul(s, s);
    // atanh(s)/s = sum_{i>=0} z^i / (2i+1), |z| <= 0.0295; 20 terms reach 2^-100
    dd acc = {1.0 / 41.0, 0.0};
    for (int i = 19; i >= 0; --i) {
        double c = 1.0 / (2 * i + 1);
        dd cdd = {c, fma(-c, (double)(2 * i + 1), 1.0) / (double)(2 * i + 1)};
        acc = dd_add(dd_mul(acc, z), cdd);
    }
    dd lm = dd_mul(dd_mul_d(s, 2.0), acc);
    dd kl = dd_add(dd_two_prod((double)k, CRP_LN2_HI), dd_two_prod((double)k, CRP_LN2_LO));
    return dd_add(kl, lm);
}

// exp of a double-double t with |t| < 700, in double-double
CRP_HD dd dd_exp(dd t) {
    double j = rint(t.hi / CRP_LN2_HI);
    dd u = dd_add(t, dd_add(dd_two_prod(-j, CRP_LN2_HI), dd_two_prod(-j, CRP_LN2_LO)));
    // u / 256, Taylor to degree 10, then square 8 times
    u.hi = ldexp(u.hi, -8);
    u.lo = ldexp(u.lo, -8);
    dd acc = {1.0 / 3628800.0, 0.0};  // 1/10!
    for (int i = 9; i >= 1; --i) {
        double f = 1.0;
        for (int q = 2; q <= i; ++q) f *= q;  // i! exact for i <= 9
        dd c = {1.0 / f, fma(-1.0 / f, f, 1.0) / f};
        acc = dd_add(dd_mul(acc, u), c);
    }
    // acc = sum_{i=1..10} u^(i-1)/i! ; e^u - 1 = u * acc
    dd em1 = dd_mul(u, acc);
    // (1 + em1)^256 via e^(2v) - 1 = (e^v - 1)(e^v + 1)
    for (int i = 0; i < 8; ++i) em1 = dd_mul(em1, dd_add(em1, dd{2.0, 0.0}));
    dd r = dd_add(em1, dd{1.0, 0.0});
    int ji = (int)j;
    r.hi = ldexp(r.hi, ji);
    r.lo = ldexp(r.lo, ji);
    return r;
}

// x^y for normal x, |y| <= 1, to a relative error below 2^-63 and rounded, if that
// error cannot change the rounding (true for all but 0.6 % of inputs).  The
// same reductions as below, with the leading terms of each series in
// double-double and their tails, at most 2^-12.5 of the sum, in double:
//   log: s = (m-1)/(m+1), z = s^2 <= 0.0295: 2 s (1 + z/3 + z^2 P(z)); error of the
//        tail 3 ulp of 2^-12.5 times |2 s| <= 0.35: below 2^-64.5;
//   exp: v = u / 8, |v| <= 0.0434: v + v^2/2 + v^3 Q(v); error of the tail 3 ulp of
//        2^-16: 2^-67.5, three doublings of the argument: below 2^-64.
// A tenth of the full evaluation's operations.
CRP_HD bool pow_quick(double x, double y, double &result) {
    int k;
    double m = frexp(x, &k);
    if (m < 0.70710678118654752440) {
        m *= 2.0;
        k -= 1;
    }
    const double num = m - 1.0;
    const dd den = dd_fast_two_sum(m > 1.0 ? m : 1.0, m > 1.0 ? 1.0 : m);
    const double inv = 1.0 / den.hi;
    const double q1 = num * inv;
    const double q2 = fma(-q1, den.lo, fma(-q1, den.hi, num)) * inv;
    const double zh = q1 * q1, zl = fma(q1, q1, -zh) + 2.0 * q1 * q2;
    double P = 1.0 / 27.0;
    P = fma(P, zh, 1.0 / 25.0); P = fma(P, zh, 1.0 / 23.0); P = fma(P, zh, 1.0 / 21.0);
    P = fma(P, zh, 1.0 / 19.0); P = fma(P, zh, 1.0 / 17.0); P = fma(P, zh, 1.0 / 15.0);
    P = fma(P, zh, 1.0 / 13.0); P = fma(P, zh, 1.0 / 11.0); P = fma(P, zh, 1.0 / 9.0);
    P = fma(P, zh, 1.0 / 7.0); P = fma(P, zh, 1.0 / 5.0);
    const double third = 1.0 / 3.0, third_lo = 1.0 / 54043195528445952.0;  // 1/3 - RN(1/3) = 2^-54 / 3
    const double p = zh * third, pe = fma(zh, third, -p) + zh * third_lo + zl * third;
    const dd B = dd_fast_two_sum(p, zh * zh * P);
    const double Bl = B.lo + pe;
    const double w = q1 * B.hi, we = fma(q1, B.hi, -w) + q1 * Bl + q2 * B.hi + q2;
    const dd l = dd_fast_two_sum(q1, w);
    const double a = k * CRP_LN2_HI, ae = fma((double)k, CRP_LN2_HI, -a) + k * CRP_LN2_LO;
    const dd L = dd_two_sum(a, 2.0 * l.hi);
    const double Ll = L.lo + (2.0 * (l.lo + we) + ae);
    const double th = y * L.hi, tl = fma(y, L.hi, -th) + y * Ll;
    if (!(fabs(th) < 699.0)) return false;
    const double j = rint(th * (1.0 / CRP_LN2_HI));
    const double b = j * CRP_LN2_HI;
    const dd u = dd_fast_two_sum(th - b, (tl - fma(j, CRP_LN2_HI, -b)) - j * CRP_LN2_LO);
    const double vh = 0.125 * u.hi, vl = 0.125 * u.lo;
    const double ah = vh * vh, al = fma(vh, vh, -ah) + 2.0 * vh * vl;
    double Q = 1.0 / 3628800.0;
    Q = fma(Q, vh, 1.0 / 362880.0); Q = fma(Q, vh, 1.0 / 40320.0); Q = fma(Q, vh, 1.0 / 5040.0);
    Q = fma(Q, vh, 1.0 / 720.0); Q = fma(Q, vh, 1.0 / 120.0); Q = fma(Q, vh, 1.0 / 24.0);
    Q = fma(Q, vh, 1.0 / 6.0);
    const dd e0 = dd_fast_two_sum(vh, 0.5 * ah);
    const dd e1 = dd_fast_two_sum(e0.hi, vh * ah * Q);
    double eh = e1.hi, el = e1.lo + e0.lo + vl + 0.5 * al;
#pragma unroll
    for (int i = 0; i < 3; i++) {  // (1 + e)^2 - 1 = 2 e + e^2
        const double sq = eh * eh, sl = fma(eh, eh, -sq) + 2.0 * eh * el;
        const dd t = dd_fast_two_sum(2.0 * eh, sq);
        eh = t.hi;
        el = t.lo + 2.0 * el + sl;
    }
    const dd r = dd_fast_two_sum(1.0, eh);
    const double lo = r.lo + el, eps = 4.336808689942018e-19;  // 2^-61 (r.hi in [0.7, 1.42])
    const double below = r.hi + (lo - eps), above = r.hi + (lo + eps);
    result = ldexp(below, (int)j);
    return below == above;
}

CRP_HD double cr_pow(double x, double y) {
    if (!(x > 0.0) || !(x < INFINITY) || !(fabs(y) < INFINITY) || x < 2.2250738585072014e-308)
        return pow(x, y);
    if (y == 0.0 || x == 1.0) return 1.0;
    double quick;
    if (fabs(y) <= 1.0 && pow_quick(x, y, quick)) return quick;
    dd l = dd_log(x);
    dd t = dd_mul_d(l, y);
    if (!(fabs(t.hi) < 700.0)) return pow(x, y);
    dd r = dd_exp(t);
    return r.hi + r.lo;
}

// a / b, rounded to nearest, for rb = 1 / b rounded to nearest (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor",
// 1990): the first correction leaves a quotient within one ulp, whose remainder
// is exact, and the second rounds it correctly.  a and a / b nonzero and far
// from the ends of the exponent range.
CRP_HD double quotient(double a, double b, double rb) {
    double q = a * rb;
    q = fma(fma(-q, b, a), rb, q);
    return fma(fma(-q, b, a), rb, q);
}

// sqrt(n2), rounded to nearest, for |n2 - 1| < 2^-27.  With n2 = 1 + e the square root
// is 1 + e/2 - e^2/8, and e/2 is a multiple of half the spacing of doubles there:
// the small last term only decides the ties, downwards, so rounding 1 + e/2 down
// gives the correctly rounded root.  (On the host the directed rounding is made
// from the exact remainder of the nearest one.)
CRP_HD double root_near_1(double n2) {
#ifdef __CUDA_ARCH__
    return __fma_rd(0.5, n2, 0.5);
#else
    const double r = fma(0.5, n2, 0.5);
    return fma(0.5, n2, 0.5 - r) < 0 ? nextafter(r, 0.0) : r;
#endif
}

// 1 / r, rounded to nearest, for |r - 1| < 2^-27: 1/r = 1 - d + d^2 for r = 1 + d is
// 2 - r with its ties rounded up.
CRP_HD double reciprocal_near_1(double r) {
#ifdef __CUDA_ARCH__
    return __dsub_ru(2.0, r);
#else
    const double v = 2.0 - r;
    return (2.0 - v) - r > 0 ? nextafter(v, 2.0) : v;
#endif
}

}  // namespace crp
