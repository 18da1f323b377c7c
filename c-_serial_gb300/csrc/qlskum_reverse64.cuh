// Reverse of one edge end of the FP64 flux residual, the unit of adjk::k_flux
// (qlskum_adjoint.cu), in the forms of qlskum_fast64.cuh; checked on the CPU
// against adj::end64_vjp (tests/test_reverse64_math.py).
#pragma once
#include "qlskum_adjoint.cuh"
#include "qlskum_fast64.cuh"

namespace qlskum {
namespace adjk {

using adj::KinBar;

// The reverse of fp64::edge_flux: F = delta sum_e v_e, v_e the folded-weight
// sum of an edge's half-range flux differences, so the bar of v_e is
// delta F-bar at every edge and the bar of a flux at the neighbour's end that
// times the edge's weight, at the owner's end its negative.

// The limiter at one component, kept for its reverse: t = num / den and
// 1 / den where it is active, else t = 1 and 0.
struct Limiter {
    double dn, dp, t, rden;
};

__device__ __forceinline__ double limited(double q, double dn, double dp, double eps2, Limiter &l)
{
    l.dn = dn;
    l.dp = dp;
    l.t = 1.0;
    l.rden = 0.0;
    if (!fast64::within_cut(dn)) {
        const double base = fma(dp, dp, eps2);
        const double rd = rcp64(fma(dn, fma(2.0, dn, dp), base));
        const double t = fma(dn, dp + dp, base) * rd;
        if ((unsigned long long)__double_as_longlong(t) < 0x3ff0000000000000ULL) {
            l.t = t;
            l.rden = rd;
        }
    }
    return fma(l.t, dn, q);
}

// The bars of q~ -> those of dn and dp (dp's enters q and qmax or qmin).
// q~ = q + t dn, t = (base + 2 dn dp) / (base + dn dp + 2 dn^2), base = dp^2 + eps2.
__device__ __forceinline__ void limited_vjp(const Limiter &l, double bt, double &bdn, double &bdp)
{
    const double g = l.dn * bt * l.rden;
    const double dp2 = l.dp + l.dp;
    bdn = fma(l.t, bt, g * fma(-l.t, fma(4.0, l.dn, l.dp), dp2));
    bdp = g * fma(-l.t, dp2 + l.dn, fma(2.0, l.dn, dp2));
}

// Bars of one end's log(rho), u_t, u_n, p / rho, erf(S1), erf(S2) and of the
// moments B1, B2.
struct EndBar {
    double ell, ut, un, p, E1, E2, B1, B2;
};

// Reverse of fast64::split_pair for the bar b of v.
__device__ __forceinline__ void split_pair_vjp(const Kin<double> &k, unsigned sx, unsigned sy, double wx, double wy,
                                               const double b[4], EndBar &o)
{
    const double wr = wx * k.rho, yr = wy * k.rho, ws = fast64::flip(wr, sx), ys = fast64::flip(yr, sy);
    const double al = wr * fma(0.5, fast64::flip(k.E1, sx), 0.5), ga = yr * fma(0.5, fast64::flip(k.E2, sy), 0.5);
    const double be = fma(ws, k.B1, ys * k.B2);
    const double v0 = fma(al, k.ut, fma(ga, k.un, be));
    const double h3 = 0.5 * b[3];
    // the bar of v0 without and with the 3.5 p / rho v0 of v3
    const double bs = fma(k.ut, b[1], fma(k.un, b[2], fma(k.usq, h3, b[0])));
    const double bv = fma(7.0 * k.pbr, h3, bs);
    const double bbe = fma(-k.pbr, h3, bv);
    const double bp = fma(al, b[1], fma(ga, b[2], h3 * fma(7.0, v0, -be)));
    o.p += bp;
    o.ell += fma(v0, bs, k.pbr * bp);
    o.ut += fma(v0, fma(k.ut, b[3], b[1]), al * bv);
    o.un += fma(v0, fma(k.un, b[3], b[2]), ga * bv);
    o.E1 = fma(0.5 * ws, fma(k.pbr, b[1], bv * k.ut), o.E1);
    o.E2 = fma(0.5 * ys, fma(k.pbr, b[2], bv * k.un), o.E2);
    o.B1 = fma(ws, bbe, o.B1);
    o.B2 = fma(ys, bbe, o.B2);
}

// Reverse of a boundary end's quadrant flux of weight w.
__device__ __forceinline__ void quad_x_vjp(const Kin<double> &k, double s1, double s2, double w, const double b[4],
                                           EndBar &o)
{
    KinBar kb;
    const double bG[4] = {w * b[0], w * b[1], w * b[2], w * b[3]};
    adj::flux_quad_vjp(k, s1, s2, bG, kb);
    o.ell = fma(k.rho, kb.rho, o.ell);
    o.ut += fma(2.0 * k.ut, kb.usq, kb.ut);
    o.un += fma(2.0 * k.un, kb.usq, kb.un);
    o.p += kb.pbr;
    o.E1 += kb.E1;
    o.E2 += kb.E2;
    o.B1 += kb.B1;
    o.B2 += kb.B2;
}

// One end of an edge: its limited reconstruction and the moments from the
// forward's kept values.
struct RevEnd {
    Limiter l[4];
    double t[4];        // q~
    double qs, qn, r, e1, e2;
    Kin<double> k;
};

__device__ __forceinline__ void rev_end(int f, double nx, double ny, double hx, double hy, const double q[4],
                                        const double dx[4], const double dy[4], const double mx[4],
                                        const double mn[4], double e2, const double *__restrict__ kept, long long ns,
                                        RevEnd &s)
{
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const double dn = fma(hx, dx[c], hy * dy[c]);
        s.t[c] = limited(q[c], dn, (__double2hiint(dn) >= 0 ? mx[c] : mn[c]) - q[c], e2, s.l[c]);
    }
    s.k.rho = kept[0];
    s.r = kept[ns];
    s.e1 = kept[2 * ns];
    s.e2 = kept[3 * ns];
    s.k.E1 = kept[4 * ns];
    s.k.E2 = kept[5 * ns];
    s.qs = s.t[1];
    s.qn = s.t[2];
    if (f != kInterior) {
        s.qs = fma(s.t[1], ny, -(s.t[2] * nx));
        s.qn = fma(s.t[1], nx, s.t[2] * ny);
    }
    s.k.pbr = 2.0 * s.r * s.r;
    s.k.ut = s.qs * s.k.pbr;
    s.k.un = s.qn * s.k.pbr;
    s.k.usq = fma(s.k.ut, s.k.ut, s.k.un * s.k.un);
    s.k.B1 = s.r * s.e1;
    s.k.B2 = s.r * s.e2;
}

// Reverse of fast64::end: the bars of the end's moments -> those of q~ in the
// point's (t, n) frame: bt[1], bt[2] are the bars of qs, qn.
//   S = r q, r = b^-1/2, p / rho = 2 / b, u = q p / rho,
//   log(rho) = q~1 + S1^2 + S2^2 - 2.5 log b, b = -2 q~4, erf' = 2 e, B = r e.
__device__ __forceinline__ void end_vjp(const RevEnd &s, const EndBar &o, double bt[4])
{
    const double S1 = s.r * s.qs, S2 = s.r * s.qn;
    const double bS1 = 2.0 * fma(s.e1, o.E1, S1 * fma(-s.k.B1, o.B1, o.ell));
    const double bS2 = 2.0 * fma(s.e2, o.E2, S2 * fma(-s.k.B2, o.B2, o.ell));
    const double br = fma(s.e1, o.B1, fma(s.e2, o.B2, fma(s.qs, bS1, s.qn * bS2)));
    const double bp = fma(s.qs, o.ut, fma(s.qn, o.un, o.p));
    bt[0] = o.ell;
    bt[1] = fma(s.k.pbr, o.ut, s.r * bS1);
    bt[2] = fma(s.k.pbr, o.un, s.r * bS2);
    bt[3] = 0.5 * s.k.pbr * fma(s.r, br, fma(2.0 * s.k.pbr, bp, 5.0 * o.ell));
}

// The bars of an end's moments for the weights (wx, wy) of the edge, w2x / w2y
// those of the second half range of an edge on both sides of an axis.
__device__ __forceinline__ void flux_bars(int f, unsigned dir, const Kin<double> &k, double wx, double wy, double w2x,
                                          double w2y, const double b[4], EndBar &o)
{
    const unsigned neg = 0x80000000u;
    const unsigned sx = (dir & kXpos) ? 0u : neg, sy = (dir & kYpos) ? 0u : neg;
    const bool inner = f == kInterior;
    const double s2 = f == kOuter ? 1.0 : -1.0;
    o = EndBar{0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    split_pair_vjp(k, sx, sy, inner ? wx : 0.0, wy, b, o);
    if (!inner) quad_x_vjp(k, sx ? -1.0 : 1.0, s2, wx, b, o);
    if (w2x != 0.0) {
        if (inner) split_pair_vjp(k, neg, 0u, w2x, 0.0, b, o);
        else quad_x_vjp(k, -1.0, s2, w2x, b, o);
    }
    if (w2y != 0.0) split_pair_vjp(k, 0u, neg, 0.0, w2y, b, o);
}

}  // namespace adjk
}  // namespace qlskum
