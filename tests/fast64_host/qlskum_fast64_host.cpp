// Host entry points to the FP64 form's fast functions (qlskum_fast64.cuh) and to
// the reverse of its flux (qlskum_reverse64.cuh), for checking them on a machine
// without a GPU (tests/test_fast64_math.py, test_reverse64_math.py).  Same source as the device code, with the CUDA
// intrinsics it uses defined here; those that approximate on the device
// (__fdividef, rsqrtf: 2 ulp) are moved off the correctly rounded value by
// `seed_shift` ulps.
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include <cuda_runtime.h>

namespace {

float seed_shift = 0.0f;

template <typename To, typename From> inline To bits(From x)
{
    static_assert(sizeof(To) == sizeof(From), "");
    To y;
    std::memcpy(&y, &x, sizeof y);
    return y;
}

inline int __double2hiint(double x) { return (int)(bits<uint64_t>(x) >> 32); }
inline int __double2loint(double x) { return (int)(uint32_t)bits<uint64_t>(x); }
inline double __hiloint2double(int hi, int lo) { return bits<double>((uint64_t)(uint32_t)hi << 32 | (uint32_t)lo); }
inline long long __double_as_longlong(double x) { return bits<long long>(x); }
inline double __longlong_as_double(long long x) { return bits<double>(x); }
inline unsigned __float_as_uint(float x) { return bits<unsigned>(x); }
inline float __uint_as_float(unsigned x) { return bits<float>(x); }
inline float shifted(float x) { return x * (1.0f + seed_shift * 1.1920929e-7f); }
inline float __fdividef(float a, float b) { return shifted(a / b); }
inline float rsqrtf(float x) { return shifted((float)(1.0 / std::sqrt((double)x))); }
inline float __frcp_rn(float x) { return 1.0f / x; }
inline double rsqrt(double x) { return 1.0 / std::sqrt(x); }
inline double __dmul_rn(double a, double b) { return a * b; }
inline double __dsqrt_rn(double x) { return std::sqrt(x); }
inline double __drcp_rn(double x) { return 1.0 / x; }
template <typename T> inline T __ldg(const T *p) { return *p; }

}  // namespace

#define __noinline__
#define QLSKUM_HOST_INTRINSICS
#include "qlskum_fast64.cuh"
#include "qlskum_reverse64.cuh"

using namespace qlskum;

namespace {

// The tables as qlskum_host.cpp lays them out.
struct Tables {
    std::vector<double2> gauss;
    std::vector<double> exp;
    Tables() : gauss(kGaussTab), exp(kExpTab)
    {
        const long double rpi = 1.128379167095512573896158903121545172L;
        for (int j = 0; j < kGaussTab; j++) {
            const long double x = j / 1024.0L;
            gauss[j] = make_double2((double)(rpi * expl(-x * x)), (double)erfl(x));
        }
        for (int i = 0; i < kExpTab; i++) exp[i] = (double)exp2l(5.0L + i / 512.0L);
    }
} tables;

double ulps(double got, long double want)
{
    const double w = (double)want;
    if (got == w || (std::isnan(got) && std::isnan(w))) return 0.0;
    const long double ulp = std::fabs(std::nextafter(w, INFINITY) - w);
    return (double)(std::fabs((long double)got - want) / ulp);
}

}  // namespace

extern "C" {

// Ulps of rounding (2^-53 relative or thereabouts) that the approximate seeds are off by.
void qlskum_f64_seed_shift(double ulps_of_float) { seed_shift = (float)ulps_of_float; }

// out[i]: the function's distance from the value in long double, in ulps of that value.
void qlskum_f64_ratio(int n, const double *num, const double *den, double *out)
{
    for (int i = 0; i < n; i++) out[i] = ulps(fast64::ratio64(num[i], den[i]), (long double)num[i] / den[i]);
}

void qlskum_f64_rsqrt_rcp(int n, const double *x, double *out_r, double *out_h)
{
    for (int i = 0; i < n; i++) {
        double r, h;
        fast64::rsqrt_rcp(x[i], r, h);
        out_r[i] = ulps(r, 1.0L / sqrtl((long double)x[i]));
        out_h[i] = ulps(h, 1.0L / x[i]);
    }
}

void qlskum_f64_exp32(int n, const double *x, double *out)
{
    for (int i = 0; i < n; i++) out[i] = ulps(fast64::exp32(x[i], tables.exp.data()), 32.0L * expl((long double)x[i]));
}

// e: ulps of its value, and those of the expression exp(-s s); E: units of 2^-53.
void qlskum_f64_gauss_erf(int n, const double *s, double *out_e, double *out_plain, double *out_E)
{
    const long double rpi = 1.128379167095512573896158903121545172L;
    for (int i = 0; i < n; i++) {
        double e, E;
        fast64::gauss_erf(s[i], tables.gauss.data(), e, E);
        const long double g = expl(-(long double)s[i] * s[i]);
        out_e[i] = ulps(e, rpi * g);
        out_plain[i] = ulps(std::exp(-s[i] * s[i]), g);
        out_E[i] = (double)(std::fabs(E - erfl((long double)s[i])) * 9007199254740992.0L);
    }
}

// The limited reconstruction q + phi dn of one component, and the factor phi itself.
void qlskum_f64_limited(int n, const double *q, const double *dn, const double *dp, const double *eps2, double *out,
                        double *phi)
{
    for (int i = 0; i < n; i++) {
        out[i] = fast64::limited(q[i], dn[i], dp[i], eps2[i]);
        phi[i] = fast64::limited(0.0, dn[i], dp[i], eps2[i]) / dn[i];
    }
}

// One end of an edge of a class-f point with half ranges `dir` and their
// weights w = {x, y, second x, second y}, as the flux kernels evaluate it.
// in: [q4 dx4 dy4 mx4 mn4] (20) -> v (4), kept (6).
void qlskum_f64_end(int f, int dir, const double *in, double e2, double delx, double dely, double nx, double ny,
                    const double *w, double *v, double *kept)
{
    DevCloud c;
    c.gauss_tab = tables.gauss.data();
    c.exp_tab = tables.exp.data();
    const double hx = -0.5 * delx, hy = -0.5 * dely;
    double t[4];
    for (int r = 0; r < 4; r++) {
        const double dn = std::fma(hx, in[4 + r], hy * in[8 + r]);
        t[r] = fast64::limited(in[r], dn, (dn >= 0.0 ? in[12 + r] : in[16 + r]) - in[r], e2);
    }
    fast64::End s;
    fast64::end(c, f, nx, ny, t, s);
    fast64::keep_end(kept, 1, s);
    const unsigned neg = 0x80000000u;
    const unsigned sx = (dir & kXpos) ? 0u : neg, sy = (dir & kYpos) ? 0u : neg, s2 = f == kOuter ? 0u : neg;
    const bool inner = f == kInterior;
    for (int r = 0; r < 4; r++) v[r] = 0.0;
    fast64::split_pair(s, sx, sy, inner ? 0.5 * w[0] : 0.0, 0.5 * w[1], v);
    if (!inner) fast64::quad_x(s, sx, s2, 0.5 * w[0], v);
    if ((dir & (kXpos | kXneg)) == (kXpos | kXneg)) {
        if (inner) fast64::split_pair(s, neg, 0u, 0.5 * w[2], 0.0, v);
        else fast64::quad_x(s, neg, s2, 0.5 * w[2], v);
    }
    if ((dir & (kYpos | kYneg)) == (kYpos | kYneg)) fast64::split_pair(s, 0u, neg, 0.0, 0.5 * w[3], v);
    v[3] *= 0.5;
}

// Its reverse for the bar b of v.  out: bars of the 20 inputs, then bdelx,
// bdely, bnx, bny, as adjk::k_flux distributes them.
void qlskum_f64_end_vjp(int f, int dir, const double *in, double e2, double delx, double dely, double nx, double ny,
                        const double *w, const double *kept, const double *b, double *out)
{
    const double hx = -0.5 * delx, hy = -0.5 * dely;
    adjk::RevEnd s;
    adjk::EndBar o;
    double bt[4];
    adjk::rev_end(f, nx, ny, hx, hy, in, in + 4, in + 8, in + 12, in + 16, e2, kept, 1, s);
    adjk::flux_bars(f, dir, s.k, w[0], w[1], w[2], w[3], b, o);
    adjk::end_vjp(s, o, bt);
    for (int r = 0; r < 24; r++) out[r] = 0.0;
    out[22] = s.t[1] * bt[2] - s.t[2] * bt[1];
    out[23] = s.t[1] * bt[1] + s.t[2] * bt[2];
    if (f != kInterior) {
        const double bs = bt[1], bn = bt[2];
        bt[1] = bs * ny + bn * nx;
        bt[2] = bn * ny - bs * nx;
    }
    for (int r = 0; r < 4; r++) {
        double bdn, bdp;
        adjk::limited_vjp(s.l[r], bt[r], bdn, bdp);
        out[r] = bt[r] - bdp;
        out[4 + r] = hx * bdn;
        out[8 + r] = hy * bdn;
        out[(s.l[r].dn >= 0.0 ? 12 : 16) + r] = bdp;
        out[20] -= 0.5 * bdn * in[4 + r];
        out[21] -= 0.5 * bdn * in[8 + r];
    }
}

}
