// FP64 elementary functions and edge ends with few FP64 instructions, for the
// drop-in form's flux kernels and their reverse, and for the outer points'
// state update in both forms.
//
// GB300 executes one FP64 instruction per warp and SM in 16 cycles, against
// four FP32 or integer ones per cycle, so the flux kernels are bound by the
// number of FP64 instructions alone.  What can be done beside the FP64 pipe
// without touching the FP64 result is done there: comparisons on the bit
// patterns, argument reductions and seeds in FP32, and the high-order terms
// of an expansion, small enough that FP32's relative error of 2^-24 stays
// below 2^-52 of the result (but for exp(-S^2) at |S| > 2, where the error of
// S^2 itself is larger).
//
// Errors against long double (tests/test_fast64_math.py): quotients and
// reciprocal roots 0.503 ulp, exp32 1.02 (rms 0.34), erf 1.01 2^-53, and
// exp(-S^2) 1.1 ulp below |S| = 1, then up to 1.6, 3.8, 8.8, 22 and 30 ulp (rms
// 0.35, 0.47, 0.86, 1.8, 3.1) in each unit of |S| up to 6, where the expression
// exp(-S * S) that it replaces has an rms error of 0.74, 2.1, 3.4, 6.8 and 9.6.
// Arguments outside the ranges below (which a physical state does not reach, and
// every Inf / NaN) take CUDA's functions.
//
// FP64 instructions per call: gauss_erf 10 (exp and erf: about 50), exp32 5
// (about 16), rsqrt_rcp 7 for both, ratio64 3.
#pragma once
#include "qlskum_math.cuh"

namespace qlskum {
namespace fast64 {

__device__ __forceinline__ unsigned abs_hi(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }

__device__ __forceinline__ double flip(double x, unsigned sign)
{
    return __hiloint2double((int)((unsigned)__double2hiint(x) ^ sign), __double2loint(x));
}

// |x| <= 1e-5 (the limiter's cut, limiters_mod.h:70) on the bit pattern; false for NaN.
__device__ __forceinline__ bool within_cut(double x)
{
    return (__double_as_longlong(x) & 0x7fffffffffffffffLL) <= __double_as_longlong(10e-6);
}

// Not so small that its low parts, 2^-46 of it, leave FP32's normal range.
__device__ __forceinline__ bool large_enough(float x) { return fabsf(x) > 1e-24f; }

// a / b; a zero numerator, which the limiter has at every extremum where eps^2 = 0, off the FP64 pipe.
static __device__ __noinline__ double div_slow(double a, double b)
{
    if ((__double_as_longlong(a) << 1) == 0 && abs_hi(b) - 0x00100000u < 0x7fe00000u)  // b normal
        return flip(a, (unsigned)__double2hiint(b) & 0x80000000u);
    return a / b;
}
static __device__ __noinline__ double rsqrt_slow(double x) { return rsqrt(x); }
static __device__ __noinline__ double exp32_slow(double x) { return 32.0 * exp(x); }
static __device__ __noinline__ double2 gauss_erf_slow(double s) { return make_double2(1.1283791670955126 * exp(-s * s), erf(s)); }

// The 29 low mantissa bits of x that d2f(x) cuts off, as a float (d2f(x)
// normal; a rest below FP32's normal range may flush to zero).
__device__ __forceinline__ float d2f_rest(double x)
{
    const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x) & 0x1fffffffu;
    // 2^-52 first: the product with 2^e, the float of x's exponent, is then exact wherever it is normal
    return copysignf((float)l, __uint_as_float(h)) * 2.220446049250313e-16f * __uint_as_float((((h >> 20) & 0x7ffu) - 896u) << 23);
}

// num / den for finite num, den > 0: the quotient to 2^-44 from FP32 (hi and
// rest of both), corrected once by its FP64 remainder.  A numerator (the
// limiter's is eps^2 alone at an extremum), denominator or quotient whose rests
// FP32 cannot hold takes the division; so do zero, overflow, Inf and NaN.
__device__ __forceinline__ double ratio64(double num, double den)
{
    const float dh = d2f(den), nh = d2f(num);
    const float r = __fdividef(1.0f, dh);
    const float q = nh * r;
    if (!(fabsf(r) > 1e-37f && fabsf(r) < 1e24f && large_enough(nh) && large_enough(q) && fabsf(q) < 1e37f))
        return div_slow(num, den);
    const float res = fmaf(-dh, q, nh) + fmaf(-d2f_rest(den), q, d2f_rest(num));
    const double v = f2d(q) + f2d(res * r);
    return fma(fma(-den, v, num), f2d(r), v);
}

// The same as a call, for places that are no inner loop: inlined three times
// into an outer point's update it made the mixed flux kernel with 72 registers
// spill (4 to 5 us of the 1,357 us per iteration at 1.02 M points).
static __device__ __noinline__ double ratio64_call(double num, double den) { return ratio64(num, den); }

// r = 1 / sqrt(x) and h = 1 / x from the FP32 seed y of r, whose square is
// exact in FP64: with e = 1 - x y^2, r = y (1 + e/2 + 3 e^2 / 8) and
// h = y^2 (1 + e + e^2), the next terms below 2^-60.
__device__ __forceinline__ void rsqrt_rcp(double x, double &r, double &h)
{
    const float s = rsqrtf(d2f(x));
    if (!(s > 1e-18f && s < 1e18f)) {  // x, whose root this is, is a normal float
        r = rsqrt_slow(x);
        h = div_slow(1.0, x);
        return;
    }
    const double y = f2d(s);
    const double y2 = y * y;
    const double e = fma(-x, y2, 1.0);
    r = fma(__dmul_rn(y, e), fma(0.375, e, 0.5), y);
    h = fma(y2, fma(e, e, e), y2);
}

// 32 exp(x) from tab[i] = 32 2^(i/512): x = k ln2/512 + r, |r| <= 2^-10.5,
// exp(r) - 1 = r (1 + r (1/2 + r/6 + r^2/24)), the last two terms in FP32.
__device__ __forceinline__ double exp32(double x, const double *__restrict__ tab)
{
    if (abs_hi(x) >= 0x40800000u) return exp32_slow(x);  // |x| >= 512 or NaN
    const float kf = rintf(d2f(x) * 738.65986f);
    const double kd = f2d(kf);
    const int k = (int)kf;
    const double r = fma(-kd, 0.0013538030870311431, x);
    const float rf = d2f(r);
    const double h = 0.5 + f2d(rf * fmaf(rf, 0.041666667f, 0.16666667f));
    // the reduction's low part, below 2^-50, added to exp(r) - 1
    const double p = fma(r, fma(r, h, 1.0), f2d(kf * -4.5293883e-20f));
    const double t = __ldg(tab + (k & 511));
    const double ts = __hiloint2double(__double2hiint(t) + ((k >> 9) << 20), __double2loint(t));
    return fma(ts, p, ts);
}

// e = 2 exp(-s^2) / sqrt(pi) and E = erf(s) together, from
// tab[j] = {2 exp(-x^2) / sqrt(pi), erf(x)} at the nearest x = j / 1024 to |s|,
// d = |s| - x (exact, |d| <= 2^-11):
//   exp(-s^2) = exp(-x^2) exp(-u), u = d (2 x + d), by its series, u^3 on in FP32;
//   erf(s) = erf(x) + 2/sqrt(pi) d [(f0 + f1) / 2 + d (f0' - f1') / 12],
// the corrected trapezoid over f = exp(-t^2) (error d^5 f'''' / 720 < 2^-60),
// its correction, below 2^-24, in FP32.
__device__ __forceinline__ void gauss_erf(double s, const double2 *__restrict__ tab, double &e, double &E)
{
    const unsigned ah = abs_hi(s);
    if (ah >= 0x40180000u) {  // |s| >= 6 or NaN
        const double2 v = gauss_erf_slow(s);
        e = v.x;
        E = v.y;
        return;
    }
    const double a = __hiloint2double((int)ah, __double2loint(s));
    const float jf = rintf(d2f(a) * 1024.0f);
    const double2 t = __ldg(tab + (int)jf);
    const float xf = jf * 0.0009765625f;
    const double x = f2d(xf);
    const double d = a - x;
    const double u = d * fma(2.0, x, d);
    const float uf = d2f(u), df = d2f(d);
    const double h = 0.5 - f2d(uf * fmaf(uf, fmaf(uf, 0.0083333333f, -0.041666667f), 0.16666667f));
    const double p = u * fma(u, h, -1.0);
    e = fma(t.x, p, t.x);
    // d/6 (s e - x e0)
    const float pf = d2f(p);
    const float w = 0.16666667f * df * d2f(t.x) * fmaf(df, 1.0f + pf, xf * pf);
    const double z = fma(0.5, t.x + e, f2d(w));
    E = flip(fma(d, z, t.y), (unsigned)__double2hiint(s) & 0x80000000u);
}

// One component of the limited reconstruction (interior_fluxes_mod.h:72-83,
// limiters_mod.h:64-104): q + phi dn with dn = -(delx dqx + dely dqy) / 2
// given; dp = qmax - q (dn > 0) or qmin - q.  The common factor dn of the
// limiter's numerator and denominator cancels.
__device__ __forceinline__ double limited(double q, double dn, double dp, double eps2)
{
    double phi = 1.0;
    if (!within_cut(dn)) {
        const double base = fma(dp, dp, eps2);
        const double t = ratio64(fma(dn, dp + dp, base), fma(dn, fma(2.0, dn, dp), base));
        // min(t, 1), 1 for NaN: t is non-negative, so its bits order like its value
        if ((unsigned long long)__double_as_longlong(t) < 0x3ff0000000000000ULL) phi = t;
    }
    return fma(phi, dn, q);
}

// One edge end: q~ -> prim (q_variables_mod.h:230-253) and the half-range
// moments (split_fluxes_mod.h:14-26) from q~ turned into the owner's (t, n)
// frame (interior points' frame is (x, y)).  With b = -2 q~4 = 4 beta,
// r = 1 / sqrt(b) and h = 1 / b: p / rho = 2 h, u = 2 h q~, S = u sqrt(beta) = r q~,
// beta |u|^2 = S1^2 + S2^2, rho = exp(q~1 + S1^2 + S2^2) 32 h^2 r, and the
// moments B = exp(-S^2) / (2 sqrt(pi beta)) = r e / 2.  h has its own expansion
// (r^2 would carry r's rounding twice, and rho takes it to the power 2.5).
struct End {
    double rho, ut, un, pbr, usq, E1, E2;
    double r, e1, e2;  // e = 2 exp(-S^2) / sqrt(pi)
};

__device__ __forceinline__ void end(const DevCloud &c, int f, double nx, double ny, const double t[4], End &s)
{
    double qs = t[1], qn = t[2];
    if (f != kInterior) {
        qs = fma(t[1], ny, -__dmul_rn(t[2], nx));
        qn = fma(t[1], nx, __dmul_rn(t[2], ny));
    }
    double h;
    rsqrt_rcp(-2.0 * t[3], s.r, h);
    const double S1 = qs * s.r, S2 = qn * s.r;
    s.pbr = h + h;
    s.ut = qs * s.pbr;
    s.un = qn * s.pbr;
    s.usq = fma(s.ut, s.ut, __dmul_rn(s.un, s.un));
    s.rho = exp32(fma(S1, S1, fma(S2, S2, t[0])), c.exp_tab) * (h * h * s.r);
    gauss_erf(S1, c.gauss_tab, s.e1, s.E1);
    gauss_erf(S2, c.gauss_tab, s.e2, s.E2);
}

// What the reverse reads back instead of evaluating it again, as planes of ns
// doubles: rho, r, exp(-S1^2) and exp(-S2^2) over sqrt(pi), erf(S1), erf(S2).
__device__ __forceinline__ void keep_end(double *__restrict__ o, long long ns, const End &s)
{
    o[0] = s.rho;
    o[ns] = s.r;
    o[2 * ns] = 0.5 * s.e1;
    o[3 * ns] = 0.5 * s.e2;
    o[4 * ns] = s.E1;
    o[5 * ns] = s.E2;
}

// Adds one end's weighted split-flux pair 2 (wx Gx(s1) + wy Gy(s2)) to v (wx,
// wy half the weights).  With al = wx rho (1 + s1 E1), ga = wy rho (1 + s2 E2)
// and be = 2 (wx rho s1 B1 + wy rho s2 B2), the pair (split_fluxes_mod.h:14-84
// and :86-164) is
//   v0 = al ut + ga un + be,  v1 = ut v0 + al p/rho,  v2 = un v0 + ga p/rho,
//   v3 = (usq v0 + p/rho (7 v0 - be)) / 2;  twice v3 is added.
// sx, sy: the sign bits of s1, s2 (0 for +1).  Every product is in an explicit
// fma or alone, here and below, so that no kernel contracts it differently.
__device__ __forceinline__ void split_pair(const End &k, unsigned sx, unsigned sy, double wx, double wy, double v[4])
{
    const double wr = wx * k.rho, yr = wy * k.rho;
    const double al = fma(wr, flip(k.E1, sx), wr), ga = fma(yr, flip(k.E2, sy), yr);
    const double be = k.r * fma(flip(wr, sx), k.e1, __dmul_rn(flip(yr, sy), k.e2));
    const double v0 = fma(al, k.ut, fma(ga, k.un, be));
    v[0] += v0;
    v[1] = fma(k.ut, v0, fma(al, k.pbr, v[1]));
    v[2] = fma(k.un, v0, fma(ga, k.pbr, v[2]));
    v[3] = fma(k.pbr, fma(7.0, v0, -be), fma(k.usq, v0, v[3]));
}

// Adds 2 w times a boundary end's quadrant flux (quadrant_fluxes_mod.h:6-211),
// the t half range of sign bit sx times the n half range of sign bit sn:
//   f = ut A1 + s1 B1,  m = un A2 + s2 B2,
//   G0 = rho A2 f,  G1 = rho A2 (ut f + p/rho A1),  G2 = rho f m,
//   G3 = rho (A2 (usq f + p/rho (7 f - s1 B1)) + s2 un B2 f) / 2; twice G3 is added.
__device__ __forceinline__ void quad_x(const End &k, unsigned sx, unsigned sn, double w, double v[4])
{
    const double A1 = fma(0.5, flip(k.E1, sx), 0.5), A2 = fma(0.5, flip(k.E2, sn), 0.5);
    const double hr = 0.5 * k.r;
    const double B1 = hr * flip(k.e1, sx), B2 = hr * flip(k.e2, sn);
    const double wr = 2.0 * w * k.rho, wa = wr * A2;
    const double f = fma(k.ut, A1, B1);
    const double wf = wr * f;
    v[0] = fma(wa, f, v[0]);
    v[1] = fma(wa, fma(k.ut, f, __dmul_rn(k.pbr, A1)), v[1]);
    v[2] = fma(wf, fma(k.un, A2, B2), v[2]);
    v[3] = fma(wa, fma(k.usq, f, __dmul_rn(k.pbr, fma(7.0, f, -B1))), fma(wf, __dmul_rn(k.un, B2), v[3]));
}

// a b - c d with one rounding of the difference (Kahan): the second product's
// rounding error is added back.
__device__ __forceinline__ double diff_of_products(double a, double b, double c, double d)
{
    const double w = c * d;
    const double e = fma(-c, d, w);
    return fma(a, b, -w) + e;
}

// The weight of half-range d's flux difference over an edge with rotated
// vector sn in point i's residual: the row of the directional 2x2 solve
// (interior_fluxes_mod.h:140-145 and its likes) times the edge's least-squares
// weights; twice on the wall (flux_residual_mod.h:29), 0 for a half-range the
// class does not use.
__device__ __forceinline__ double flux_weight(const DevCloud &c, int i, int f, int d, double2 sn)
{
    if ((f == kWall && d == 2) || (f == kOuter && d == 3)) return 0.0;
    const double4_32a m = c.fgeo[4 * (size_t)i + d];  // sxx, syy, sxy, 1/det
    const double w = m.w * (d < 2 ? diff_of_products(m.y, sn.x, m.z, sn.y) : diff_of_products(m.x, sn.y, m.z, sn.x));
    return f == kWall ? 2.0 * w : w;
}

// Doubles in the order of signed integers (for max / min off the FP64 pipe);
// its own inverse.
__device__ __forceinline__ long long order_key(long long b) { return b ^ ((b >> 63) & 0x7fffffffffffffffLL); }

// dist / speed * cfl of one edge (state_update_mod.h:483-488)
__device__ __forceinline__ double edge_dt(double dist, double speed, double cfl)
{
    return cfl * ratio64(dist, speed);
}

// ------------------------------------------------------------ points
// The point formulas of qlskum_math.cuh with every multiply-add explicit, so
// that the module, fused and recording kernels, whatever the compiler inlines
// around them, give the same bits.

__device__ __forceinline__ double beta_of(const double P[4]) { return ratio64(0.5 * P[0], P[3]); }

// q_variables_mod.h:19-33, with log(rho) and log(beta) given
__device__ __forceinline__ void q_of(const double P[4], double log_rho, double log_beta, double Q[4])
{
    const double beta = beta_of(P);
    const double usq = fma(P[1], P[1], __dmul_rn(P[2], P[2]));
    Q[0] = fma(-beta, usq, fma(2.5, log_beta, log_rho));
    const double b2 = 2.0 * beta;
    Q[1] = b2 * P[1];
    Q[2] = b2 * P[2];
    Q[3] = -b2;
}

__device__ __forceinline__ void q_of(const double P[4], double Q[4]) { q_of(P, log(P[0]), log(beta_of(P)), Q); }

// |u| + 3 sqrt(p / rho) of state_update_mod.h:483-485
__device__ __forceinline__ double wave_speed(const double P[4])
{
    const double u = __dsqrt_rn(fma(P[1], P[1], __dmul_rn(P[2], P[2])));
    return fma(3.0, __dsqrt_rn(ratio64(P[3], P[0])), u);
}

// One half range of conserved_vector_Ubar (state_update_mod.h:35-90) at an
// outer point: the state's outflowing one (s = 1) or the free stream's
// inflowing one (s = -1).  With r = 1 / sqrt(2 p / rho) = sqrt(beta), S = un r,
// A = (1 + s erf(S)) / 2 and rho B = rho s exp(-S^2) / (2 sqrt(pi beta)) = s e p r / 2.
__device__ __forceinline__ void half_range(double s, double gm1, double rho, double u1, double u2, double p,
                                           double nx, double ny, const double2 *__restrict__ tab, double U[4])
{
    const double ut = fma(u1, ny, -__dmul_rn(u2, nx)), un = fma(u1, nx, __dmul_rn(u2, ny));
    const double x = ratio64_call(p + p, rho);
    double r, h, e, E;
    rsqrt_rcp(x, r, h);
    gauss_erf(un * r, tab, e, E);
    const double A = fma(0.5 * s, E, 0.5), m = __dmul_rn(rho, A);
    const double mB = __dmul_rn(0.5 * s * p, __dmul_rn(e, r));
    U[0] = m;
    U[1] = __dmul_rn(m, ut);
    U[2] = fma(m, un, mB);
    U[3] = fma(ratio64_call(p, gm1), A, 0.5 * fma(m, fma(ut, ut, __dmul_rn(un, un)), __dmul_rn(un, mB)));
}

// primitive_to_conserved (state_update_mod.h:18-33); for an outer point
// conserved_vector_Ubar, the free stream's half given in Uinf.
__device__ __forceinline__ void conserved(int f, double gm1, double nx, double ny, const double P[4],
                                          const double Uinf[4], const double2 *__restrict__ tab, double U[4])
{
    if (f != kOuter) {
        const double t1 = P[0] * P[1], t2 = P[0] * P[2];
        U[0] = P[0];
        U[3] = fma(2.5, P[3], 0.5 * fma(t1, P[1], __dmul_rn(t2, P[2])));
        U[1] = fma(t1, ny, -__dmul_rn(t2, nx));
        U[2] = fma(t1, nx, __dmul_rn(t2, ny));
        return;
    }
    half_range(1.0, gm1, P[0], P[1], P[2], P[3], nx, ny, tab, U);
#pragma unroll
    for (int r = 0; r < 4; r++) U[r] += Uinf[r];
}

// One SSPRK stage of one point (state_update_mod.h:111-282): P is updated in
// place; returns the point's res_sqr (0 on outer points).  An outer point's two
// or three half ranges are one thread's serial chain, which a small cloud's
// kernel waits for: with CUDA's exp, erf, sqrt and division (and the free
// stream's half evaluated again for prim_old) it set the mixed flux kernel's
// time below 100,000 points (9,600 points: 22.5 us, now 15.1).
__device__ __forceinline__ double stage(const CaseConst &K, const double2 *__restrict__ tab, int f, double nx,
                                        double ny, double P[4], const double4_32a *__restrict__ prim_old_i,
                                        const double F[4], int rk)
{
    double U[4], Uinf[4] = {0.0, 0.0, 0.0, 0.0};
    if (f == kOuter) half_range(-1.0, K.gamma - 1.0, K.rho_inf, K.u1_inf, K.u2_inf, K.pr_inf, nx, ny, tab, Uinf);
    conserved(f, K.gamma - 1.0, nx, ny, P, Uinf, tab, U);
    const double rho = U[0];
    if (rk != 3) {
#pragma unroll
        for (int j = 0; j < 4; j++) U[j] = fma(-0.5, F[j], U[j]);
    } else {
        double Po[4], Uo[4];
        ld4(*prim_old_i, Po);
        conserved(f, K.gamma - 1.0, nx, ny, Po, Uinf, tab, Uo);
#pragma unroll
        for (int j = 0; j < 4; j++) U[j] = fma(2.0 / 3.0, Uo[j], __dmul_rn(1.0 / 3.0, fma(-0.5, F[j], U[j])));
    }
    if (f == kWall) U[2] = 0.0;
    const double m1 = fma(U[1], ny, __dmul_rn(U[2], nx)), m2 = fma(U[2], ny, -__dmul_rn(U[1], nx));
    const double d = U[0] - rho;
    const double inv = __drcp_rn(U[0]);
    P[0] = U[0];
    P[1] = m1 * inv;
    P[2] = m2 * inv;
    P[3] = fma(0.4, U[3], -__dmul_rn(0.2 * inv, fma(m1, m1, __dmul_rn(m2, m2))));
    return f == kOuter ? 0.0 : __dmul_rn(d, d);
}

}  // namespace fast64
}  // namespace qlskum
