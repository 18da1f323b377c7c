"""params.block_size over the range that qlskum_create accepts, above the 512
threads of the largest block the mixed gradient kernel takes: the launch shape
changes no bit of the result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def start(c, seed=2):
    rng = np.random.default_rng(seed)
    return np.tile([1.0, 0.63, 0.02, 1 / 1.4], (c.n, 1)) * (1.0 + 1e-2 * rng.standard_normal((c.n, 4)))


# 33 slices of 32 points (the second block's warps partly idle) and 392
@pytest.mark.parametrize("wall, layers", [(49, 21), (113, 111)])
@pytest.mark.parametrize("form", ["fp64", "mixed"])
def test_block_sizes_of_a_solver(wall, layers, form):
    import qlskum
    from qlskum import cloudgen
    c = cloudgen.make_cloud(n_wall=wall, n_layers=layers, first_spacing=5e-3, radius=5.0 if wall < 50 else 20.0, seed=4)
    out = []
    for block in (128, 32, 96, 512, 544, 768, 1024):
        s = qlskum.Solver(c, mach=0.63, aoa=2.0, cfl=0.2, vl_const=50.0, inner_iterations=2, block_size=block,
                          precision=qlskum.MIXED if form == "mixed" else qlskum.FP64)
        assert s.launch_config()["point_block"] == block
        s.set_prim(start(c))
        s.q_lskum(3)
        out.append((s.prim, s.field(qlskum.FIELD_DQ), s.field(qlskum.FIELD_QM)))
    for o in out[1:]:
        for a, b in zip(out[0], o):
            assert np.array_equal(a, b)


def test_block_sizes_of_a_partition():
    import qlskum
    from qlskum import cloudgen
    c = cloudgen.make_cloud(n_wall=113, n_layers=111, first_spacing=5e-3, radius=20.0, seed=4)
    out = []
    for block in (128, 544, 1024):
        p = qlskum.Partition(c, 2, mach=0.63, aoa=2.0, cfl=0.2, vl_const=50.0, inner_iterations=2, block_size=block,
                             precision=qlskum.MIXED)
        p.set_prim(start(c))
        p.q_lskum(3)
        out.append(p.prim)
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
