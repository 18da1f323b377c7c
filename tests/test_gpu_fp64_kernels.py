"""The FP64 flux kernels' fast functions and launch forms against the oracle.

Bound of the flux residual: delta sum_e c_e (G_k - G_i) over a point's edges,
each flux G correct to about 10 ulps of its scale and 8 S^2 more for the
density, exp of a sum whose terms are S^2 large (S^2 = beta |u|^2); the
weights c_e of a half range sum to at most 2.5 / min_dist (the cloud
generator's bound); four half ranges, two ends: 20 (10 + 8 S^2) ulps of
(delta / min_dist) max |G|.  The disturbances are small against the speed of
sound, so that an edge end's state stays near the points' at every Mach number.
"""
import numpy as np
import pytest

import qlskum_oracle

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def disturbed(cloud, mach, seed=5):
    rng = np.random.default_rng(seed)
    P = np.empty((cloud.n, 4))
    P[:, 0] = 1.0 + 0.05 * rng.uniform(-1, 1, cloud.n)
    P[:, 1] = 0.97 * mach + 0.02 * rng.uniform(-1, 1, cloud.n)
    P[:, 2] = 0.15 * mach + 0.02 * rng.uniform(-1, 1, cloud.n)
    P[:, 3] = (1.0 + 0.05 * rng.uniform(-1, 1, cloud.n)) / 1.4
    return P


def flux_bound(cloud, P, delta):
    """Per component: the module's bound with |u| + 3 sqrt(p / rho) as the speed of the largest flux."""
    U = float((np.hypot(P[:, 1], P[:, 2]) + 3 * np.sqrt(P[:, 3] / P[:, 0])).max())
    G = P[:, 0].max() * U * np.array([1.0, U, U, U * U])
    S2 = float((0.5 * P[:, 0] / P[:, 3] * (P[:, 1] ** 2 + P[:, 2] ** 2)).max())
    return 20 * (10 + 8 * S2) * EPS * float((delta / cloud.min_dist).max()) * G


def stage(s, P, inner):
    s.set_prim(P)
    s.func_delta()
    s.eval_q_variables()
    s.eval_q_derivatives()
    for _ in range(inner):
        s.eval_q_inner_loop()
        s.eval_update_innerloop()
    s.cal_flux_residual()


# 9: |S| beyond the tables (the library's exp and erf); 0.01: |S| next to 0.
# Without jitter the cloud has edges on both sides of an axis (dels or deln == 0).
@pytest.mark.parametrize("mach", [0.01, 0.85, 3.0, 9.0])
@pytest.mark.parametrize("power", [0.0, -2.0])
def test_flux_residual_over_the_mach_range(mach, power):
    import qlskum
    from qlskum import cloudgen
    c = cloudgen.make_cloud(n_wall=48, n_layers=21, first_spacing=5e-3, radius=5.0, seed=3, jitter=0.0)
    kw = dict(mach=mach, aoa=2.0, cfl=0.2, vl_const=50.0, power=power, inner_iterations=1)
    P = disturbed(c, mach)
    s, o = qlskum.Solver(c, **kw), qlskum_oracle.Oracle(c, **kw)
    o.set_prim(P)
    o.func_delta()
    o.eval_q_variables()
    o.eval_q_derivatives()
    o.eval_q_inner_loop()
    o.eval_update_innerloop()
    o.cal_flux_residual()
    counts, _ = s.connectivity()
    interior = c.flag_1 == 1
    assert (counts[interior].sum(1) > 2 * c.nbhs[interior]).any()  # both-sides edges
    stage(s, P, 1)
    err = np.abs(s.field(qlskum.FIELD_FLUX_RES) - o.flux_res).max(0)
    assert (err <= flux_bound(c, P, o.delta)).all(), (err, flux_bound(c, P, o.delta))


def test_nonfinite_state_is_reported():
    """A NaN in the state goes through the fast functions' library paths and is reported."""
    import qlskum
    from conftest import golden_cloud
    c = golden_cloud("cloud_small")
    s = qlskum.Solver(c, mach=0.63, aoa=2.0, cfl=0.2, vl_const=50.0, inner_iterations=0)
    P = disturbed(c, 0.63)
    P[c.n // 2, 3] = np.nan
    s.set_prim(P)
    with pytest.raises(qlskum.QlskumError) as e:
        s.q_lskum(1)
    assert e.value.status == 3
    s.set_prim(disturbed(c, 0.63))
    s.q_lskum(1)
    assert np.isfinite(s.prim).all()


# the flux kernels' three launch shapes, each with a remainder
@pytest.mark.parametrize("wall, layers", [(49, 21), (113, 111), (257, 259)])
def test_flux_launch_shapes(wall, layers):
    """Fused and module path agree bit for bit, and both with the oracle."""
    import qlskum
    from qlskum import cloudgen
    c = cloudgen.make_cloud(n_wall=wall, n_layers=layers, first_spacing=5e-3, radius=5.0 if wall < 50 else 20.0, seed=4)
    kw = dict(mach=0.63, aoa=2.0, cfl=0.2, vl_const=50.0, inner_iterations=1)
    P = disturbed(c, 0.63)
    o = qlskum_oracle.Oracle(c, threads=16, **kw)
    o.set_prim(P)
    s = qlskum.Solver(c, **kw)
    stage(s, P, 1)
    flux = s.field(qlskum.FIELD_FLUX_RES)
    s.snapshot_prim_old()
    for rk in (1, 2, 3, 4):
        if rk > 1:
            s.eval_q_variables()
            s.eval_q_derivatives()
            s.eval_q_inner_loop()
            s.eval_update_innerloop()
            s.cal_flux_residual()
        s.state_update(rk)
    f = qlskum.Solver(c, **kw)
    f.set_prim(P)
    f.q_lskum(1)
    assert np.array_equal(f.prim, s.prim)
    o.func_delta()
    o.eval_q_variables()
    o.eval_q_derivatives()
    o.eval_q_inner_loop()
    o.eval_update_innerloop()
    o.cal_flux_residual()
    assert (np.abs(flux - o.flux_res).max(0) <= flux_bound(c, P, o.delta)).all()
    o.set_prim(P)
    res, _, top = o.fpi_solver()
    h = f.residual_history()[-1]
    assert np.allclose([h[0], h[2]], [res, top], rtol=1e-10, atol=0)
    # four stages, each within the bound of its flux residual
    assert (np.abs(f.prim - o.prim).max(0) <= 4 * flux_bound(c, P, o.delta) + 8 * EPS * np.abs(P).max(0)).all()


# 1008, 1029 and 1071 points: the last warp of the four-lanes-per-point kernels full or partly empty
@pytest.mark.parametrize("wall", [48, 49, 51])
@pytest.mark.parametrize("power", [0.0, -2.0])
def test_inner_step_on_its_own(wall, power):
    """An inner step whose gradient is not that of the current q, as a caller
    of the modules may order it.  Bound: the weights sum to at most 2.5 /
    min_dist; q (8 ulps) and the old gradient times an edge (8 ulps) meet them."""
    import qlskum
    from qlskum import cloudgen
    c = cloudgen.make_cloud(n_wall=wall, n_layers=21, first_spacing=5e-3, radius=5.0, seed=4)
    kw = dict(mach=0.63, aoa=2.0, cfl=0.2, vl_const=50.0, power=power, inner_iterations=1)
    s, o = qlskum.Solver(c, **kw), qlskum_oracle.Oracle(c, **kw)
    for x in (s, o):
        x.set_prim(disturbed(c, 0.63, 1))
        x.eval_q_variables()
        x.eval_q_derivatives()
        x.set_prim(disturbed(c, 0.63, 2))
        x.eval_q_variables()
        x.eval_q_inner_loop()
        x.eval_update_innerloop()
    d = s.field(qlskum.FIELD_DQ)
    md = c.min_dist[:, None, None]
    reach = 2.5 * 3.0 * np.abs(o.dq).max()  # gradient times an edge of up to 3 min_dist, over min_dist
    assert (np.abs(d - o.dq) <= EPS * (8 * 2.5 * 2 * np.abs(o.q).max() / md + 8 * reach)).all()


@pytest.mark.parametrize("mach", [0.01, 0.85, 3.0, 9.0])
@pytest.mark.parametrize("rk", [1, 3])
def test_stage_over_the_mach_range(mach, rk):
    """The SSPRK stage, with the outer points' half ranges (|S| past the table at
    Mach 9).  A half range is at most 10 roundings and an S to 4 ulps, whose
    dA / dS and S^2 exp(-S^2) are below 0.6: 20 ulps of rho (1, U, U, U^2); half
    the residual's own bound comes with F.  u = m / rho and p = 0.4 (E - m^2 / (2 rho))
    take an error dU to at most 4 times its size over rho (U for u, U^2 for p)."""
    import qlskum
    from qlskum import cloudgen
    c = cloudgen.make_cloud(n_wall=48, n_layers=21, first_spacing=5e-3, radius=5.0, seed=3)
    kw = dict(mach=mach, aoa=2.0, cfl=0.02, vl_const=50.0, inner_iterations=0)
    P = disturbed(c, mach)
    s, o = qlskum.Solver(c, **kw), qlskum_oracle.Oracle(c, **kw)
    for h in (s, o):
        h.set_prim(P)
        h.snapshot_prim_old()
        h.func_delta()
        h.eval_q_variables()
        h.eval_q_derivatives()
        h.cal_flux_residual()
        h.state_update(rk)
    U = float((np.hypot(P[:, 1], P[:, 2]) + 3 * np.sqrt(P[:, 3] / P[:, 0])).max())
    G = P[:, 0].max() * np.array([1.0, U, U, U * U])
    # flux_bound()'s scale is U G
    b = float((0.5 * flux_bound(c, P, o.delta) / G + 20 * EPS).max())
    tol = 4 * b * np.array([1.0, U, U, U * U]) * P[:, 0].max() / o.prim[:, 0].min()
    assert (np.abs(s.prim - o.prim).max(axis=0) <= tol).all()
    outer = c.flag_1 == 2
    assert outer.any() and np.abs(s.prim - P)[outer].max() > 1e-4
