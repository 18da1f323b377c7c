"""The mixed gradient kernel whose edge list comes by bulk copies: the same bits
at every block size, and the four-lanes form's values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(c, block, lanes, power, inner=2):
    import qlskum
    s = qlskum.Solver(c, mach=0.63, aoa=2.0, cfl=0.2, vl_const=50.0, power=power, inner_iterations=inner,
                      precision=qlskum.MIXED)
    s.set_launch_config(10, block, 0, lanes)
    rng = np.random.default_rng(2)
    s.set_prim(s.prim * (1.0 + 1e-2 * rng.standard_normal((c.n, 4))))
    s.q_lskum(1)
    return s.prim, s.field(qlskum.FIELD_DQ), s.field(qlskum.FIELD_QM)


# few slices, a remainder of a slice, more slices than resident warps
# (152 x 24); lists of up to 20 edges (several chunks)
@pytest.mark.parametrize("wall, layers", [(40, 12), (49, 21), (397, 331)])
@pytest.mark.parametrize("power", [0.0, -2.0])
def test_block_sizes_and_lanes(wall, layers, power):
    """The gradients are sums of at most 20 products in FP32: split over four
    lanes they move by at most 20 ulps of the terms' sum, whose weights sum to at
    most 2.5 / min_dist (x and y half range: twice); two inner steps repeat that.
    The extrema are the same."""
    from conftest import small_cloud
    from qlskum import cloudgen
    c = small_cloud(wall, layers) if wall < 60 else cloudgen.make_cloud(n_wall=wall, n_layers=layers, seed=3,
                                                                       te_spread=0.064)
    ref = run(c, 128, 1, power)
    for block in (64, 256, 512):
        for a, b in zip(ref, run(c, block, 1, power)):
            assert np.array_equal(a, b)
    p4, dq4, qm4 = run(c, 128, 4, power)
    scale = 2 * 2.5 * np.abs(ref[2]).max() / c.min_dist[:, None, None]
    assert (np.abs(dq4 - ref[1]) <= 3 * 20 * 2.0 ** -24 * scale).all()
    assert np.allclose(qm4, ref[2], rtol=0, atol=1e-5 * np.abs(ref[2]).max())
    assert np.allclose(p4, ref[0], rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("lanes", [1, 2, 4])
@pytest.mark.parametrize("power", [0.0, -2.0])
def test_edge_lists_past_l2(lanes, power):
    """Three cases of one cloud are past the size at which the edge lists are
    read evict-first (26 or 37 MB each, 64 MB), one case is not: how they are read
    changes no bit."""
    import qlskum
    from qlskum import cloudgen
    c = cloudgen.make_cloud(n_wall=397, n_layers=331, seed=3, te_spread=0.064)
    out = []
    for cases in (1, 3):
        b = qlskum.Batch([c], [(0, 0.63, 2.0)] * cases, cfl=0.2, vl_const=50.0, power=power, inner_iterations=2)
        b.set_launch_config(128, lanes, 10)
        b.run(3)
        out += [b.prim(k) for k in range(cases)]
    for p in out[1:]:
        assert np.array_equal(out[0], p)


@pytest.mark.parametrize("wall, layers", [(40, 12), (49, 21), (64, 40), (257, 259)])
def test_residual_of_few_and_many_partials(wall, layers):
    """2 to 1,041 block partials (64, 128 and 256 points per block) of the same
    state: the sum in FP64 moves by at most 1,041 roundings of 2^-53 and the maximum not at all."""
    import qlskum
    from conftest import small_cloud
    from qlskum import cloudgen
    c = small_cloud(wall, layers) if wall < 60 else cloudgen.make_cloud(n_wall=wall, n_layers=layers, seed=3)
    out = []
    for variant in (2, 0, 3):
        s = qlskum.Solver(c, mach=0.63, aoa=2.0, cfl=0.2, vl_const=50.0, inner_iterations=0, precision=qlskum.MIXED)
        s.set_launch_config(variant, 128, 0)
        rng = np.random.default_rng(2)
        s.set_prim(s.prim * (1.0 + 1e-2 * rng.standard_normal((c.n, 4))))
        s.q_lskum(1)
        out.append((s.prim, s.residual_history()[0]))
    for prim, h in out[1:]:
        assert np.array_equal(prim, out[0][0])
        assert abs(h[0] / out[0][1][0] - 1.0) <= 1041 * 2.0 ** -53 and h[2] == out[0][1][2]
