"""
Tables of a reference: built beside its derivative path on a second stream,
built alone on one (no path asked for, or derived for another view size) -- the
same BLA tree and the same image, from orbits too short for a tree up to
several blocks of it.
"""
import numpy as np
import pytest

from fractalshades_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu
LIN = np.array([[1., -0.], [0., 1.]])


@pytest.fixture(scope="module")
def ctx():
    from fractalshades_gb300 import _native as nat
    c = nat.Context(0)
    yield c
    c.close()


def _orbit(n, seed):
    r = np.random.default_rng(seed)
    z = 0.4 * np.exp(2j * np.pi * r.uniform(size=n)) * r.uniform(0.5, 2., n)
    z[0] = 0.
    return z


def _image(ctx, ref, flavor, mode, drift):
    from fractalshades_gb300 import _native as nat
    xs, ys = syn.image_axes(33, 21)
    n = xs.size * ys.size
    Z = np.zeros((2, n), dtype=np.complex128) if flavor == 0 else np.zeros((6, n))
    sr, si = -np.ones((1, n), dtype=np.int8), np.zeros((1, n), dtype=np.int32)
    kw = dict(drift_m=drift, drift_e=-40, i_dzndc=1) if flavor == 0 else \
        dict(drift_m=drift.real, drift_e=-40, drifty_m=drift.imag, drifty_e=-40)
    tile = nat.make_tile(xs=xs, ys=ys, lin_mat=LIN, Z=Z, stop_reason=sr, stop_iter=si, ref=ref,
                         dx_m=1.25, dx_e=-40, **kw)
    ctx.perturb_tiles(nat.make_calc(max_iter=700, M_divergence=1000., flavor=flavor, calc_dzndc=True,
                                    bla=True, mode=mode), [tile])
    return Z, sr, si


@pytest.mark.parametrize("mode", ["fe32", "fp64"])
@pytest.mark.parametrize("flavor", [0, 1])
@pytest.mark.parametrize("n", [2, 7, 8, 9, 16, 17, 63, 64, 65, 1023, 2056, 2474, 9000])
def test_tables_beside_a_path_and_alone(ctx, n, flavor, mode):
    from fractalshades_gb300 import _native as nat
    Zn = _orbit(n, n)
    kc = float(np.ldexp(1.25, -40))
    kw = dict(div_iter=10 ** 6, order=n, flavor=flavor, scale_m=1.25, scale_e=-40, bla=True)
    both = nat.Reference(ctx, Zn, calc_dzndc=True, kc=kc, **kw)
    alone = nat.Reference(ctx, Zn, calc_dzndc=False, kc=kc, **kw)
    derived = nat.Reference(ctx, Zn, calc_dzndc=True, kc=1e-3, **kw).derive_bla(kc)
    if n >= 8:
        M, r = both.download("bla")
        for other in (alone, derived):
            Mo, ro = other.download("bla")
            assert np.array_equal(M.view(np.float64), Mo.view(np.float64), equal_nan=True)
            assert np.array_equal(r, ro, equal_nan=True)
    a = _image(ctx, both, flavor, mode, 0.25 + 0.125j)
    b = _image(ctx, derived, flavor, mode, 0.25 + 0.125j)
    for x, y in zip(a, b):
        assert np.array_equal(x.view(np.uint8), y.view(np.uint8))


@pytest.mark.parametrize("flavor", [0, 1])
def test_tables_of_many_live_references(ctx, flavor):
    """Tables that share blocks of a context's pool do not touch: every
    reference of a set built, partly freed and built again holds the tables it
    holds alone."""
    from fractalshades_gb300 import _native as nat
    lens = [3, 9, 17, 100, 257, 1000, 4095, 4096, 4097, 20000]
    names = ("dzndc", "bla") if flavor == 0 else ("bs_paths", "bla")

    def build(c, n):
        return nat.Reference(c, _orbit(n, n), div_iter=10 ** 6, order=n, flavor=flavor, scale_m=1.25,
                             scale_e=-40, calc_dzndc=True, bla=True, kc=float(np.ldexp(1.25, -40)))

    def tables(ref, n):
        out = []
        for k in names:
            if k == "bla" and n < 8:
                continue
            t = ref.download(k)
            out += list(t) if isinstance(t, tuple) else [t]
        return [np.ascontiguousarray(x).view(np.uint8) for x in out if x is not None]

    live = {n: build(ctx, n) for n in lens}
    for n in lens[::2]:
        live[n].free()
        live[n] = build(ctx, n)
    other = nat.Context(0)
    for n in lens:
        alone = build(other, n)
        for a, b in zip(tables(live[n], n), tables(alone, n)):
            assert np.array_equal(a, b)
        alone.free()
    other.close()
    for r in live.values():
        r.free()
