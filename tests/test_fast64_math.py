"""The FP64 form's fast functions (csrc/qlskum_fast64.cuh) compiled for the host,
against long double; the approximate FP32 seeds moved by up to their 2 ulps."""
import ctypes as C

import numpy as np
import pytest

dp = C.POINTER(C.c_double)
N = 200_000


@pytest.fixture(scope="module")
def L():
    from qlskum import build
    lib = C.CDLL(build.build_fast64_host())
    lib.qlskum_f64_seed_shift.argtypes = [C.c_double]
    lib.qlskum_f64_seed_shift.restype = None
    return lib


def run(fn, *arrays, out=1):
    """fn(n, arrays..., outputs...) -> the outputs."""
    a = [np.ascontiguousarray(x, np.float64) for x in arrays]
    o = [np.empty(a[0].size) for _ in range(out)]
    fn.restype = None
    fn(C.c_int(a[0].size), *[x.ctypes.data_as(dp) for x in a + o])
    return o if out > 1 else o[0]


def spread(rng, decades, n=N):
    return 10.0 ** rng.uniform(-decades, decades, n)


@pytest.mark.parametrize("shift", [-2.0, 0.0, 2.0])
@pytest.mark.parametrize("decades", [2, 45, 150])
def test_quotient_and_roots(L, shift, decades):
    """Half an ulp from the last rounding; before it the quotient is off by its
    seed's error to the third power (2^-21.5, so 2^-64) and the series are cut at
    2^-61: below 0.01 ulp.  Where the seed is out of FP32's range rsqrt(x) is the
    host's 1 / sqrt(x), two roundings and their binades."""
    L.qlskum_f64_seed_shift(shift)
    rng = np.random.default_rng(decades)
    num, den = spread(rng, decades) * rng.choice([-1.0, 1.0], N), spread(rng, decades)
    assert run(L.qlskum_f64_ratio, num, den).max() <= 0.51
    r, h = run(L.qlskum_f64_rsqrt_rcp, den, out=2)
    assert r.max() <= (0.51 if decades == 2 else 1.51) and h.max() <= 0.51


def test_quotient_of_special_values(L):
    """Zero, infinity and NaN, and the ends of FP32's range: the division's value."""
    L.qlskum_f64_seed_shift(0.0)
    v = np.array([0.0, 5e-324, 1e-310, 1.1754943508222875e-38, 1e-38, 1e-37, 1e-30, 1e-24, 1.0, 1e24, 1e30, 1e37,
                  3.5e38, 1e300, np.inf, np.nan])
    num, den = (x.ravel() for x in np.meshgrid(np.concatenate([v, -v]), v))
    assert run(L.qlskum_f64_ratio, num, den).max() <= 0.51


@pytest.mark.parametrize("eps2", [0.0, 1e-300, 6.4e-41, 1.2e-38, 1.6e-38, 1e-30, 1e-24, 1e-20, 1e-6])
def test_limiter_at_an_extremum(L, eps2):
    """dp == 0: phi = eps^2 / (eps^2 + 2 dn^2), whatever the size of eps^2; two
    FMAs' roundings, the quotient and phi dn / dn: 4 ulps."""
    L.qlskum_f64_seed_shift(0.0)
    rng = np.random.default_rng(3)
    dn = spread(rng, 1, 1000) * 1e-3 * rng.choice([-1.0, 1.0], 1000)
    z = np.zeros_like(dn)
    q = rng.uniform(0.5, 2.0, dn.size)
    got, phi = run(L.qlskum_f64_limited, q, dn, z, z + eps2, out=2)
    want = eps2 / (eps2 + 2.0 * dn * dn)
    assert np.allclose(phi, want, rtol=4 * 2.0 ** -52, atol=1e-320)
    assert np.allclose(got, q + want * dn, rtol=2.0 ** -52, atol=0)


def test_exp(L):
    """The table's rounding and the last one: half an ulp each, the table's doubled
    where the result lies in the binade below; 0.1 for the polynomial."""
    rng = np.random.default_rng(5)
    assert run(L.qlskum_f64_exp32, rng.uniform(-30, 30, N)).max() <= 1.6
    assert run(L.qlskum_f64_exp32, np.array([-600.0, -512.0, -511.99, 0.0, 511.99, 512.0, 600.0])).max() <= 1.6


def test_gauss_and_erf(L):
    """erf: the table's rounding and the last one, 2^-53.  2 exp(-s^2) / sqrt(pi): the
    same as exp's (1.6 ulps), the roundings of u <= 2 |s| 2^-11 (8 u ulps with the
    binade below) and u^3 / 6 from FP32, off by 4 2^-23 of it: u^3 2^29 ulps.  From
    |s| = 1 on smaller than the error of the expression exp(-s s)."""
    rng = np.random.default_rng(6)
    s = rng.uniform(0, 6.5, N) * rng.choice([-1.0, 1.0], N)
    e, plain, E = run(L.qlskum_f64_gauss_erf, s, out=3)
    a = np.abs(s)
    assert E.max() <= 1.05
    inside = a < 6.0
    u = a / 1024.0
    assert (e <= 1.6 + 8 * u + u ** 3 * 2.0 ** 29)[inside].all()
    for lo in (1, 2, 3, 4, 5):
        b = (a >= lo) & (a < lo + 1)
        assert np.sqrt((e[b] ** 2).mean()) <= np.sqrt((plain[b] ** 2).mean())
