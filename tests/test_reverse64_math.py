"""One edge end of the FP64 flux residual and its reverse as the GPU kernels evaluate
them (qlskum_fast64.cuh, qlskum_reverse64.cuh), compiled for the host: the flux
against the solver's plain formulas, the bars against their own reverse."""
import ctypes as C

import numpy as np
import pytest

dp = C.POINTER(C.c_double)
XPOS, XNEG, YPOS, YNEG = 1, 2, 4, 8
D = C.c_double

# class (0 wall, 1 interior, 2 outer) and the half ranges of an edge, both-sides edges
# among them; a wall point has no ypos half range, an outer one no yneg
CASES = [(1, x | y) for x in (XPOS, XNEG, XPOS | XNEG) for y in (YPOS, YNEG, YPOS | YNEG)]
CASES += [(0, x | YNEG) for x in (XPOS, XNEG, XPOS | XNEG)]
CASES += [(2, x | YPOS) for x in (XPOS, XNEG, XPOS | XNEG)]


@pytest.fixture(scope="module")
def libs():
    from qlskum import build
    a, b = C.CDLL(build.build_fast64_host()), C.CDLL(build.build_vjp_host())
    i = C.c_int
    a.qlskum_f64_end.argtypes = [i, i, dp, D, D, D, D, D, dp, dp, dp]
    a.qlskum_f64_end_vjp.argtypes = [i, i, dp, D, D, D, D, D, dp, dp, dp, dp]
    b.qlskum_dbg_prim_to_q.argtypes = [dp, dp]
    b.qlskum_dbg_end_flux.argtypes = [i, i, dp, D, D, D, D, D, dp]
    b.qlskum_dbg_end64_flux_vjp.argtypes = [i, i, dp, D, D, D, D, D, dp, dp]
    b.qlskum_dbg_venkat.argtypes, b.qlskum_dbg_venkat.restype = [D] * 5, D
    return a, b


def P(a):
    return a.ctypes.data_as(dp)


@pytest.mark.parametrize("f, dir", CASES)
@pytest.mark.parametrize("e2", [1e-7, 1e-41, 0.0])
def test_edge_end_and_its_reverse(libs, f, dir, e2):
    """Both sides take the same 100 to 400 operations in other orders, the reverse
    with S^2 <= 2 in its cancellations: 1e-12 of the largest part (4,500 ulps).  The
    plain formulas form dn as (q + dn) - q, off by an ulp of q; the limiter's bars
    are functions of dp / dn and change by up to 4 times the relative error of dn."""
    A, B = libs
    rng = np.random.default_rng(100 * f + dir)
    limited = extrema = 0
    for trial in range(24):
        prim = np.array([rng.uniform(0.7, 1.3), rng.uniform(-0.9, 0.9), rng.uniform(-0.5, 0.5), rng.uniform(0.5, 0.9)])
        q = np.zeros(4)
        B.qlskum_dbg_prim_to_q(P(prim), P(q))
        scale = np.abs(q) + 0.1
        th = rng.uniform(0, 2 * np.pi)
        nx, ny = (0.0, 1.0) if f == 1 else (np.cos(th), np.sin(th))
        delx, dely = rng.uniform(-0.01, 0.01, 2)
        up, down = rng.uniform(1e-4, 0.02, 4) * scale, rng.uniform(1e-4, 0.02, 4) * scale
        up[rng.random(4) < 0.2] = 0.0    # a local extremum
        down[rng.random(4) < 0.2] = 0.0
        x = np.concatenate([q, rng.uniform(-2, 2, 8) * np.tile(scale, 2), q + up, q - down])
        g = delx * x[4:8] + dely * x[8:12]
        phi = np.array([B.qlskum_dbg_venkat(q[r] - 0.5 * g[r], q[r], x[12 + r], x[16 + r], e2) for r in range(4)])
        limited += int((phi < 1.0).sum())
        extrema += int((phi < 1e-3).sum())
        w = rng.standard_normal(4)
        if (dir & 3) != 3:
            w[2] = 0.0
        if (dir & 12) != 12:
            w[3] = 0.0
        b = rng.standard_normal(4)
        # half range -> weight: the first of each axis, then the second of a both-sides edge
        parts = [(0 if dir & XPOS else 1, w[0]), (2 if dir & YPOS else 3, w[1])]
        parts += [(1, w[2])] if (dir & 3) == 3 else []
        parts += [(3, w[3])] if (dir & 12) == 12 else []
        v, kept, want, G = np.zeros(4), np.zeros(6), np.zeros(4), np.zeros(4)
        A.qlskum_f64_end(f, dir, P(x), e2, delx, dely, nx, ny, P(w), P(v), P(kept))
        bars, big = np.zeros(24), np.zeros(24)
        size = np.zeros(4)
        for d, wd in parts:
            B.qlskum_dbg_end_flux(f, d, P(x), e2, delx, dely, nx, ny, P(G))
            want += wd * G
            size += np.abs(wd * G)
            one, bG = np.zeros(24), wd * b
            B.qlskum_dbg_end64_flux_vjp(f, d, P(x), e2, delx, dely, nx, ny, P(bG), P(one))
            bars += one
            big += np.abs(one)
        assert (np.abs(v - want) <= 1e-13 * size.max()).all(), (v, want)
        out = np.zeros(24)
        A.qlskum_f64_end_vjp(f, dir, P(x), e2, delx, dely, nx, ny, P(w), P(kept), P(b), P(out))
        # every bar is that of q~ times factors of up to 4 that may cancel (phi == 0 at an
        # extremum): its own size for q, max and min, times the half edge for the gradient,
        # times the gradient for the edge
        bt = big[:4].max() + big[12:20].max()
        dn = np.abs(0.5 * g)
        tol = 1e-12 + 4 * 2.0 ** -52 * np.abs(q).max() / dn[dn > 0.9e-5].min(initial=1.0)
        for k, part in ((slice(0, 4), 1.0), (slice(4, 12), 0.5 * max(abs(delx), abs(dely))), (slice(12, 20), 1.0),
                        (slice(20, 22), 0.5 * np.abs(x[4:12]).max())):
            assert (np.abs(out[k] - bars[k]) <= tol * bt * part).all(), (k, out[k], bars[k])
        if f != 1:
            # a unit normal only turns (the two take |u|^2 before and after the rotation, which
            # differ in a change of its length)
            t = np.array([-ny, nx])
            assert abs((out[22:] - bars[22:]) @ t) <= tol * max(bt, big[22:].max())
    assert limited >= 20 and (extrema >= 5 or e2 > 1e-10)
