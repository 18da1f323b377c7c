"""A bulk copy that does not arrive is told by every call that hands out results,
also where the state is not finite, until a new state is set.  A test-only kernel
waits on barriers that nothing completes: the wait returns after its bound (a
second per chunk) and the context stays usable."""
import ctypes as C
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ERR_CUDA = 4


@pytest.fixture(scope="module")
def lib():
    """qlskum on the library whose host layer is built beside the test kernel."""
    import qlskum
    from qlskum import build
    path = build.build_lost_copy()
    saved, make = qlskum._lib, build.build
    qlskum._lib, build.build = None, lambda *a, **k: path
    try:
        L = qlskum.load()
    finally:
        build.build = make
    for f in (L.qlskum_test_lost_copy, L.qlskum_test_lost_copy_batch, L.qlskum_test_lost_copy_partition):
        f.argtypes, f.restype = [C.c_void_p], C.c_int
    yield L
    qlskum._lib = saved


def lose(fn, h):
    t = time.monotonic()
    assert fn(h) == 2
    assert time.monotonic() - t < 10.0


def refused(call, *a, **k):
    import qlskum
    with pytest.raises(qlskum.QlskumError) as e:
        call(*a, **k)
    assert e.value.status == ERR_CUDA and "bulk copy" in str(e.value)


def cloud():
    from conftest import golden_cloud
    return golden_cloud("cloud_small")


def test_solver(lib, tmp_path):
    import qlskum
    s = qlskum.Solver(cloud(), mach=0.63, aoa=2.0, cfl=0.2, vl_const=50.0, inner_iterations=1, precision=qlskum.MIXED)
    P = s.prim
    out = np.empty((s.n, 4))
    ptr = out.ctypes.data_as(C.POINTER(C.c_double))
    s.q_lskum(2)
    lose(lib.qlskum_test_lost_copy, s._h)
    s.fpi_solver(3)  # waits for nothing
    calls = [lambda: s.prim, lambda: s._ck(lib.qlskum_get_prim(s._h, ptr)), s.residual_history, s.objective, s.synchronize,
             lambda: s.field(qlskum.FIELD_DQ), lambda: s.q_lskum(1), lambda: s.adjoint_fixed_point("cl", 2),
             lambda: s.adjoint_gradient("cl", 2), lambda: s.write_restart(str(tmp_path / "r"))]
    for call in calls:
        refused(call)
    s.set_prim(P)
    s.q_lskum(1)
    assert np.isfinite(s.prim).all()
    # with a state that is not finite as well
    P[s.n // 2, 3] = np.nan
    s.set_prim(P)
    s.fpi_solver(1)
    lose(lib.qlskum_test_lost_copy, s._h)
    refused(s.q_lskum, 1)
    P[s.n // 2, 3] = 1 / 1.4
    g = s.adjoint_gradient("cl", 2, prim0=P)  # sets a state too
    assert np.isfinite(g["dmach"])


def test_during_the_adjoint_sweep(lib):
    """The sweep's own recomputations come after its check of the primal: the
    read of the gradient tells."""
    import qlskum
    s = qlskum.Solver(cloud(), mach=0.63, aoa=2.0, cfl=0.2, vl_const=50.0, inner_iterations=1, precision=qlskum.MIXED)
    s.q_lskum(5)
    s.adjoint_fixed_point("cl", 2)
    lose(lib.qlskum_test_lost_copy, s._h)
    refused(s.adjoint_fixed_point, "cl", 2)


def test_batch(lib):
    import qlskum
    b = qlskum.Batch([cloud()], [(0, 0.63, 2.0), (0, 0.7, 1.0)], cfl=0.2, vl_const=50.0, inner_iterations=1)
    b.run(1)
    lose(lib.qlskum_test_lost_copy_batch, b._h)
    for call in (lambda: b.run(1), b.objective, lambda: b.prim(1), b.residual_history):
        refused(call)


def test_partition(lib):
    import qlskum
    p = qlskum.Partition(cloud(), 2, mach=0.63, aoa=2.0, cfl=0.2, vl_const=50.0, inner_iterations=1,
                         precision=qlskum.MIXED)
    P = p.prim
    p.q_lskum(1)
    lose(lib.qlskum_test_lost_copy_partition, p._h)
    for call in (lambda: p.prim, p.residual_history, p.objective, lambda: p.q_lskum(1)):
        refused(call)
    p.set_prim(P)
    p.q_lskum(1)
    assert np.isfinite(p.prim).all()
