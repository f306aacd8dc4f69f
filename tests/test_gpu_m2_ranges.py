"""
The FP64 and Xrange power-2 loops where their products and sums leave the
fast forms (values below 2^-480 in FP64, zero parts, orbits on the real axis,
the critical point, derivatives that underflow), against the oracle; and the
claim order of rectangles (8 x 4 blocks with remainders) against an explicit
list of the same positions.
"""
import functools

import mpmath
import numpy as np
import pytest

from fractalshades_gb300 import synthetic as syn
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
LIN = np.array([[1., -0.], [0., 1.]])


@pytest.fixture(scope="module")
def ctx():
    from fractalshades_gb300 import _native as nat
    c = nat.Context(0)
    yield c
    c.close()


@functools.lru_cache(maxsize=None)
def _axis_nucleus(p, c0):
    """Nucleus of period p on the real axis, by Newton from c0."""
    with mpmath.workdps(800):
        c = mpmath.mpf(c0)
        for _ in range(40):
            a, d = mpmath.mpf(0), mpmath.mpf(0)
            for _ in range(p):
                d = 2 * a * d + 1
                a = a * a + c
            c -= a / d
        return mpmath.mpc(c, 0)


def _view(where, dx, xr, nx=24, ny=18, max_iter=4000, offset=(0.07, -0.03)):
    if where == "axis":
        return syn.prepare_m2(p=16, dps=800, dx=dx, nx=nx, ny=ny, max_iter=max_iter, offset=offset,
                              center=_axis_nucleus(16, "-1.62541"), xr_mode=xr)
    return syn.prepare_m2(p=361, dps=1100, dx=dx, nx=nx, ny=ny, max_iter=max_iter, offset=offset,
                          xr_mode=xr)


def _reference(ctx, w, interior):
    from fractalshades_gb300 import _native as nat
    return nat.Reference(ctx, w.Zn, div_iter=w.div_iter, order=w.order, xr_idx=w.xr_idx, xr_m=w.xr_m,
                         xr_e=w.xr_e, xr_paths=w.xr_mode, calc_dzndc=True, calc_dzndz=interior,
                         scale_m=w.dx_m, scale_e=w.dx_e, bla=True, kc=w.kc, bla_eps=1e-6)


def _run(ctx, w, ref, mode, interior=False, explicit=False, calc_dzndc=True):
    from fractalshades_gb300 import _native as nat
    n = w.nx * w.ny
    Z = np.full((1 + interior + calc_dzndc, n), np.nan, dtype=np.complex128)
    sr, si = np.full((1, n), -5, dtype=np.int8), np.full((1, n), -7, dtype=np.int32)
    pos = dict(pix=(w.xs[None, :] + 1j * w.ys[:, None]).ravel()) if explicit else dict(xs=w.xs, ys=w.ys)
    t = nat.make_tile(lin_mat=LIN, Z=Z, stop_reason=sr, stop_iter=si, ref=ref, dx_m=w.dx_m, dx_e=w.dx_e,
                      drift_m=w.drift_m, drift_e=w.drift_e, i_dzndz=1 if interior else -1,
                      i_dzndc=1 + interior if calc_dzndc else -1, **pos)
    ctx.perturb_tiles(nat.make_calc(max_iter=w.max_iter, M_divergence=w.M, epsilon_stationnary=1e-3,
                                    mode=mode, calc_dzndc=calc_dzndc, interior=interior, bla=True,
                                    xr_semantics=w.xr_mode), [t])
    return Z, si, sr


@pytest.mark.parametrize("interior", [False, True])
@pytest.mark.parametrize("where", ["axis", "bulb"])
@pytest.mark.parametrize("dx,xr", [("1e-3", False), ("1e-7", False), ("1e-30", False), ("1e-150", False),
                                   ("1e-200", False), ("1e-290", False), ("1e-5", True),
                                   ("1e-305", True), ("1e-340", True), ("1e-700", True)])
def test_m2_ranges_vs_oracle(ctx, where, dx, xr, interior):
    w = _view(where, dx, xr)
    Mb, rb, _, st = orc.make_bla_m2(w.Zn, w.kc, 1e-6)
    side = (w.xr_idx, w.xr_m, w.xr_e)
    kw = dict(Zn=w.Zn, ref_div_iter=w.div_iter, ref_order=w.order, lin_mat=LIN, dx_m=w.dx_m, dx_e=w.dx_e,
              drift_m=w.drift_m, drift_e=w.drift_e, max_iter=w.max_iter, M=w.M, eps_stat=1e-3, xr_mode=xr,
              bla=(Mb, rb, st), interior=interior, xr_idx=w.xr_idx, xr_m=w.xr_m, xr_e=w.xr_e,
              dZndc=orc.dzndc_path_m2(w.Zn, w.div_iter, w.order, xr, w.dx_m, w.dx_e, *side))
    if interior:
        kw["dZndz"] = orc.dzndz_path_m2(w.Zn, w.div_iter, xr, *side)
    Zo, _, sro, sio = orc.perturb_m2((w.xs[None, :] + 1j * w.ys[:, None]).ravel(), **kw)
    Z, si, sr = _run(ctx, w, _reference(ctx, w, interior), "xr64" if xr else "fp64", interior)
    # a BLA radius may differ from the oracle's by an ulp of hypot, which can
    # change the steps of a pixel on it: none of these few hundred
    assert np.array_equal(si, sio) and np.array_equal(sr, sro)
    for k in range(Z.shape[0]):
        if interior and k == 1 and xr:
            continue                     # the Xrange branch does not write dzndz
        np.testing.assert_allclose(Z[k], Zo[k], rtol=1e-13, atol=0)


@pytest.mark.parametrize("interior", [False, True])
@pytest.mark.parametrize("mode,dx", [("fp64", "1e-12"), ("xr64", "1e-305")])
def test_m2_without_dzndc(ctx, mode, dx, interior):
    """A derivative that is not asked for has no table on the device."""
    from fractalshades_gb300 import _native as nat
    w = _view("axis", dx, mode == "xr64")
    full = _run(ctx, w, _reference(ctx, w, interior), mode, interior)
    ref = nat.Reference(ctx, w.Zn, div_iter=w.div_iter, order=w.order, xr_idx=w.xr_idx, xr_m=w.xr_m,
                        xr_e=w.xr_e, xr_paths=w.xr_mode, calc_dzndc=False, calc_dzndz=interior,
                        scale_m=w.dx_m, scale_e=w.dx_e, bla=True, kc=w.kc, bla_eps=1e-6)
    Z, si, sr = _run(ctx, w, ref, mode, interior, calc_dzndc=False)
    assert np.array_equal(si, full[1]) and np.array_equal(sr, full[2])
    assert np.array_equal(Z[0], full[0][0])


@pytest.mark.parametrize("mode", ["fp64", "xr64", "fe32"])
@pytest.mark.parametrize("nx,ny", [(1, 1), (7, 3), (8, 4), (9, 5), (31, 4), (33, 2), (5, 41), (64, 64), (65, 67)])
def test_claim_order_of_rectangles(ctx, mode, nx, ny):
    w = _view("bulb", "1e-9", mode == "xr64", nx=max(nx, 2), ny=max(ny, 2), max_iter=1500)
    w.nx, w.ny, w.xs, w.ys = nx, ny, w.xs[:nx], w.ys[:ny]
    ref = _reference(ctx, w, False)
    a, b = _run(ctx, w, ref, mode), _run(ctx, w, ref, mode, explicit=True)
    assert (a[1] > 0).all()
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("M", [4., 30., 1e3, 1e8, 1e17])
def test_fe32_escape_radius(ctx, M):
    """The FP32 loop leaves the escape test out where the orbit's exponent
    rules an escape out; from the values at a radius of 2.5, plain iteration
    tells at which step a larger one is passed."""
    w = syn.seahorse_workload(nx=40, max_iter=6000)
    ref = _reference(ctx, w, False)
    w.M = 2.5
    Z0, si0, sr0 = _run(ctx, w, ref, "fe32")
    w.M = M
    Z, si, sr = _run(ctx, w, ref, "fe32")
    assert (sr0 == 1).all() and (sr == 1).all()
    dx = float(np.ldexp(w.dx_m, w.dx_e))
    c = complex(w.center) + dx * (w.xs[None, :] + 1j * w.ys[:, None]).ravel()
    z, more = Z0[0].copy(), np.zeros(Z0.shape[1], dtype=np.int64)
    for _ in range(12):
        go = np.abs(z) <= M
        z = np.where(go, z * z + c, z)
        more += go
    # the FP32 values are good to about 1e-4 of |z| here and double that at each
    # further step; a pixel that lands on the radius to within that may take one
    # step more or less, which a few steps of squaring make rare
    off = si[0] - si0[0] != more
    assert off.sum() <= 0.01 * off.size and np.abs(si[0] - si0[0] - more).max() <= 1


@pytest.mark.parametrize("nx,ny", [(283, 275), (331, 353), (411, 397)])
def test_xr64_images_above_two_ctas_an_sm(ctx, nx, ny):
    """Images that two CTAs an SM do not hold at once run in the Xrange loop's
    three-CTA kernel: the pixels of a smaller launch, and its statistics."""
    w = _view("bulb", "1e-305", True, nx=nx, ny=ny, max_iter=1200)
    ref = _reference(ctx, w, False)
    a = _run(ctx, w, ref, "xr64")
    big = ctx.stats()
    xs, ys = w.xs, w.ys
    cut = 100
    w.nx, w.ny, w.xs, w.ys = cut, cut, xs[:cut], ys[:cut]
    b = _run(ctx, w, ref, "xr64")
    for x, y in zip(a, b):
        assert np.array_equal(x.reshape(x.shape[0], ny, nx)[:, :cut, :cut], y.reshape(y.shape[0], cut, cut))
    assert big["pixels"] == nx * ny and big["pixel_iters"] == a[1].sum()
    assert 0 < big["full_steps"] <= big["pixel_iters"]
