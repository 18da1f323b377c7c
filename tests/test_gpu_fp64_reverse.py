"""The FP64 reverse kernels at each of their launch shapes: residual VJP against
central differences of the residual, in random directions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one cloud per launch shape of the flux reverse, each with a remainder; without
# jitter a cloud has edges on both sides of an axis (dels or deln == 0)
@pytest.mark.parametrize("wall, layers, jitter", [(49, 21, 0.1), (48, 21, 0.0), (113, 111, 0.1), (257, 259, 0.1)])
def test_residual_vjp_launch_shapes(wall, layers, jitter):
    """The map is piecewise smooth (limiter branches, max / min, the time step's
    minimum): 1% noise keeps the switches apart and a step of 1e-8 crosses few.
    Bound: 1e-8 of the Cauchy-Schwarz product, the rounding of the difference
    quotient (a residual correct to 3e-13 of its norm, over 1e-8, is 3e-5 of
    |R|, and |J| |v| exceeds |R| by the cells' inverse size times the noise)
    and of the few crossings; a missing term is ~1e-2."""
    import qlskum
    from qlskum import cloudgen
    c = cloudgen.make_cloud(n_wall=wall, n_layers=layers, first_spacing=5e-3, radius=5.0 if wall < 50 else 20.0,
                            seed=4, jitter=jitter)
    s = qlskum.Solver(c, mach=0.63, aoa=2.0, cfl=0.2, vl_const=50.0, inner_iterations=1)
    s.q_lskum(5)
    rng = np.random.default_rng(8)
    p = s.prim * (1.0 + 1e-2 * rng.standard_normal((c.n, 4)))
    h = 1e-8
    for _ in range(2):
        v = rng.standard_normal((c.n, 4)) * np.array([1.0, 0.5, 0.5, 0.7])
        w = rng.standard_normal((c.n, 4))
        fd = float(np.sum(w * (s.residual(p + h * v) - s.residual(p - h * v))) / (2 * h))
        g = s.residual_vjp(p, w)
        assert abs(fd - float(np.sum(g * v))) <= 1e-8 * np.linalg.norm(g) * np.linalg.norm(v)


def test_repeated_residual_and_vjp():
    """The second and later calls replay a captured graph: the values of a first
    call on another handle (the forward's bits; the VJP's neighbour bars are
    added in no fixed order: 1e-13 of their norm), also after the wall gradient
    has replaced the reverse's buffers."""
    import qlskum
    from qlskum import cloudgen
    c = cloudgen.make_cloud(n_wall=49, n_layers=21, first_spacing=5e-3, radius=5.0, seed=4)
    kw = dict(mach=0.63, aoa=2.0, cfl=0.2, vl_const=50.0, inner_iterations=1)
    rng = np.random.default_rng(3)
    s = qlskum.Solver(c, **kw)
    for k in range(5):
        P = np.tile([1.0, 0.6, 0.02, 1 / 1.4], (c.n, 1)) * (1.0 + 1e-2 * rng.standard_normal((c.n, 4)))
        w = rng.standard_normal((c.n, 4))
        if k == 3:
            s.residual_vjp(P, w, wall=True)
        o = qlskum.Solver(c, **kw)
        assert np.array_equal(s.residual(P), o.residual(P))
        a, b = s.residual_vjp(P, w), o.residual_vjp(P, w)
        assert np.linalg.norm(a - b) <= 1e-13 * np.linalg.norm(b)
