"""The FP64 form at limiter constants whose eps^2 = (vl_const min_dist)^6 lies in, at the
edge of and below FP32's range (min_dist is about 5e-3 here: 1e-14 to 1e-57, and
zero): at a local extremum eps^2 alone is the limiter's numerator."""
import numpy as np
import pytest

import qlskum_oracle
from test_gpu_fp64_kernels import disturbed, flux_bound, stage

pytestmark = pytest.mark.gpu

VL = [50.0, 1.0, 1e-2, 1e-3, 1e-4, 3e-5, 1e-5, 1e-7, 0.0]


def cloud():
    from qlskum import cloudgen
    return cloudgen.make_cloud(n_wall=48, n_layers=21, first_spacing=5e-3, radius=5.0, seed=3)


@pytest.mark.parametrize("vl_const", VL)
def test_flux_residual(vl_const):
    """phi dn changes with dn and dp by at most a few times their own errors, also
    where eps^2 is nothing: the flux kernels' bound."""
    import qlskum
    c = cloud()
    kw = dict(mach=0.63, aoa=2.0, cfl=0.2, vl_const=vl_const, inner_iterations=1)
    P = disturbed(c, 0.63)
    s, o = qlskum.Solver(c, **kw), qlskum_oracle.Oracle(c, **kw)
    stage(s, P, 1)
    o.set_prim(P)
    o.func_delta()
    o.eval_q_variables()
    o.eval_q_derivatives()
    o.eval_q_inner_loop()
    o.eval_update_innerloop()
    o.cal_flux_residual()
    assert (o.q == o.qm[:, 0]).any() and (o.q == o.qm[:, 1]).any()  # local extrema
    err = np.abs(s.field(qlskum.FIELD_FLUX_RES) - o.flux_res).max(0)
    assert (err <= flux_bound(c, P, o.delta)).all(), (err, flux_bound(c, P, o.delta))


@pytest.mark.parametrize("vl_const", VL)
def test_residual_vjp(vl_const):
    """The reverse takes the forward's limiter: central differences of the
    residual in random directions, within 1e-8 of the Cauchy-Schwarz product (the
    rounding of the quotient, few crossed switches)."""
    import qlskum
    c = cloud()
    s = qlskum.Solver(c, mach=0.63, aoa=2.0, cfl=0.2, vl_const=vl_const, inner_iterations=1)
    rng = np.random.default_rng(8)
    p = disturbed(c, 0.63)
    h = 1e-8
    for _ in range(2):
        v = rng.standard_normal((c.n, 4)) * np.array([1.0, 0.5, 0.5, 0.7])
        w = rng.standard_normal((c.n, 4))
        fd = float(np.sum(w * (s.residual(p + h * v) - s.residual(p - h * v))) / (2 * h))
        g = s.residual_vjp(p, w)
        assert abs(fd - float(np.sum(g * v))) <= 1e-8 * np.linalg.norm(g) * np.linalg.norm(v)
