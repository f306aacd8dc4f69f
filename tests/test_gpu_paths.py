"""
Derivative paths of orbits whose lengths end at, just before and just after the
parts the sequential build works in (256 points, runs of 8), and of orbits that
leave its common step -- real ones, points in the Xrange side table, growth and
decay beyond the lazy normalisation's bounds: the oracle's values, bit for bit.
"""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from fractalshades_gb300 import _native as nat
    c = nat.Context(0)
    yield c
    c.close()


def _orbit(kind, n):
    r = np.random.default_rng(n)
    z = r.uniform(-1., 1., n) + 1j * r.uniform(-1., 1., n)
    if kind == "real":
        z = z.real + 0j
    elif kind == "growing":
        z *= 4.
    elif kind == "shrinking":
        z *= 1e-3
    elif kind == "mixed":
        z *= 10. ** r.uniform(-30, 3, n)
    z[0] = 0.
    return z


@pytest.mark.parametrize("scale_e", [-2000, -30, 0])
@pytest.mark.parametrize("kind", ["plain", "real", "growing", "shrinking", "mixed", "side"])
@pytest.mark.parametrize("n", [2, 3, 8, 9, 10, 17, 256, 257, 258, 264, 265, 513, 700])
def test_paths_vs_oracle(ctx, n, kind, scale_e):
    from fractalshades_gb300 import _native as nat
    Zn = _orbit(kind, n)
    side = dict(xr_idx=None, xr_m=None, xr_e=None)
    if kind == "side" and n > 8:
        idx = np.arange(5, n, 7, dtype=np.int32)
        Zn[idx] = 0.
        side = dict(xr_idx=idx, xr_m=np.full(idx.size, 1.25 - 1.5j), xr_e=np.full(idx.size, -1500, dtype=np.int32))
    div_iter, scale_m = 10 ** 6, 1.375
    for order in (n, 10 ** 9):
        if order > n:
            div_iter = max(n - 1, 1)
        for xr in (False, True):
            if not xr and (scale_e < -1000 or kind == "side"):
                continue
            ref = nat.Reference(ctx, Zn, div_iter=div_iter, order=order, xr_paths=xr, calc_dzndc=True,
                                calc_dzndz=True, scale_m=scale_m, scale_e=scale_e, bla=False,
                                **(side if xr else {}))
            args = (side["xr_idx"], side["xr_m"], side["xr_e"]) if xr else ()
            want_c = orc.dzndc_path_m2(Zn, div_iter, order, xr, scale_m, scale_e, *args)
            want_z = orc.dzndz_path_m2(Zn, div_iter, xr, *args)
            for got, want in ((ref.download("dzndc"), want_c), (ref.download("dzndz"), want_z)):
                if not xr:
                    assert np.array_equal(got.view(np.float64), want.view(np.float64), equal_nan=True)
                    continue
                # mantissa and exponent, as the reference leaves them
                assert np.array_equal(got[0].view(np.float64), np.asarray(want[0]).view(np.float64),
                                      equal_nan=True)
                assert np.array_equal(got[1], want[1])
            ref.free()
