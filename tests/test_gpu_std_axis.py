"""
The standard loops where the integer products do not hold: a row of pixels on
the axis has zero factors at every step, and chaotic pixels overflow their
derivatives long before max_iter.  Bit for bit against the oracle, at the sizes
that take the loops' different forms, and at a cost near an ordinary image's.
"""
import numpy as np
import pytest

from test_gpu_std_sizes import LIN, check

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from fractalshades_gb300 import _native as nat
    c = nat.Context(0)
    yield c
    c.close()


MODELS = [dict(), dict(d2=True, backshift=3), dict(nexp=2), dict(nexp=2, d2=True, backshift=3), dict(nexp=4),
          dict(nexp=3, d2=True)] + [dict(flavor=f) for f in (1, 2, 3, 4, 5)] + [
          dict(flavor=f, backshift=3) for f in (1, 2, 3, 4, 5)]


# odd ny: a row on the real axis; 1100 iterations: derivatives overflow
@pytest.mark.parametrize("nx,ny", [(1, 1), (49, 51), (98, 101), (201, 203)])
@pytest.mark.parametrize("kw", MODELS, ids=lambda kw: "-".join(f"{k}{v}" for k, v in kw.items()) or "m2")
def test_axis_row(ctx, kw, nx, ny):
    wide = dict(center=-0.4 + 0j, dx=4.) if kw.get("flavor") else dict(center=-0.5 + 0j, dx=3.)
    check(ctx, nx, ny, max_iter=1100, **wide, **kw)


# a column at x = 0, and both at the origin
@pytest.mark.parametrize("flavor", [1, 2, 3, 4, 5])
def test_axis_column(ctx, flavor):
    check(ctx, 49, 51, flavor=flavor, center=0j, dx=3., max_iter=1100)


@pytest.mark.parametrize("kw", [dict(flavor=1), dict(flavor=2), dict(flavor=3), dict(flavor=4), dict(options=True)],
                         ids=lambda kw: "-".join(f"{k}{v}" for k, v in kw.items()))
def test_axis_row_costs_about_an_ordinary_image(ctx, kw):
    """Both images have pixels that run to max_iter.  On the axis each of
    their steps is an attempt by the integer products (an ordinary step) and
    a step by the multiplies, which holds up a lone pixel no longer than the
    attempt does: twice an ordinary image, 2.6 times with what the launch and
    its first steps add."""
    from fractalshades_gb300 import _native as nat
    flavor, options = kw.get("flavor", 0), kw.get("options", False)

    def best(ny):
        xs, ys = np.linspace(-0.5, 0.5, 49), np.linspace(-0.5, 0.5, ny)
        n = 49 * ny
        Z = np.zeros((6, n)) if flavor else np.zeros((5, n), dtype=np.complex128)
        sr, si = -np.ones((1, n), dtype=np.int8), np.zeros((1, n), dtype=np.int32)
        tile = nat.make_tile(xs=xs, ys=ys, lin_mat=LIN, Z=Z, stop_reason=sr, stop_iter=si, center=-0.5 + 0j,
                             dx=4. if flavor else 3., i_znorbit=4 if options else 0)
        calc = nat.make_calc(max_iter=1000, M_divergence=1000., epsilon_stationnary=0.01, flavor=flavor,
                             calc_d2zndc2=options, backshift=3 if options else 0)
        ms = []
        for _ in range(8):
            ctx.std_tiles(calc, [tile])
            ms.append(ctx.stats()["kernel_ms"])
        return min(ms)

    assert best(51) <= 2.6 * best(50)
