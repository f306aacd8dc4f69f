"""
The standard loops over the sizes at which their launch changes form (eight
lanes per pixel up to 64 pixels per SM, 64-thread CTAs up to 256, 256-thread
CTAs above; warps of 32 and groups of 16 pixels with remainders), and over
limits that move the tests read from exponents: bit for bit against the oracle.
"""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu
LIN = np.array([[1., -0.], [0., 1.]])


@pytest.fixture(scope="module")
def ctx():
    from fractalshades_gb300 import _native as nat
    c = nat.Context(0)
    yield c
    c.close()


def check(ctx, nx, ny, *, flavor=0, nexp=0, center=-0.5 + 0j, dx=3., max_iter=150, M=1000., eps=0.01,
          d2=False, backshift=0, block=0):
    from fractalshades_gb300 import _native as nat
    xs = np.linspace(-0.5, 0.5, nx) if nx > 1 else np.array([0.21])
    ys = np.linspace(-0.4, 0.4, ny) if ny > 1 else np.array([0.13])
    pix = (xs[None, :] + 1j * ys[:, None]).ravel()
    if flavor:
        Zo, sio, sro = orc.std_bs(pix, center, LIN, dx, flavor, max_iter, M, backshift=backshift)
    elif nexp:
        Zo, sio, sro = orc.std_mn(pix, center, LIN, dx, max_iter, M, eps, nexp, d2, backshift)
    else:
        Zo, sio, sro = orc.std_m2(pix, center, LIN, dx, max_iter, M, eps, d2, backshift)
    Z = np.zeros_like(Zo)
    sr = -np.ones((1, pix.size), dtype=np.int8)
    si = np.zeros((1, pix.size), dtype=np.int32)
    t = nat.make_tile(xs=xs, ys=ys, lin_mat=LIN, Z=Z, stop_reason=sr, stop_iter=si, center=center,
                      dx=dx, i_znorbit=(6 if flavor else 3 + d2) if backshift else 0)
    ctx.std_tiles(nat.make_calc(max_iter=max_iter, M_divergence=M, epsilon_stationnary=eps,
                                flavor=flavor, nexp=nexp, calc_d2zndc2=d2, backshift=backshift,
                                block=block), [t])
    assert np.array_equal(si, sio) and np.array_equal(sr, sro)
    # (bits; a NaN's sign and payload are not compared)
    a, b = Z.view(np.float64), Zo.view(np.float64)
    assert np.array_equal(np.isnan(a), np.isnan(b))
    k = ~np.isnan(a)
    assert np.array_equal(a[k].view(np.uint64), b[k].view(np.uint64))
    assert ctx.stats()["pixel_iters"] == int(sio.sum())


# odd ny: a row on the real axis, where factors are 0
@pytest.mark.parametrize("nx,ny", [(1, 1), (1, 17), (5, 3), (31, 1), (33, 47), (96, 101), (98, 101),
                                   (197, 197), (199, 201), (401, 303)])
def test_std_m2_sizes(ctx, nx, ny):
    check(ctx, nx, ny)


@pytest.mark.parametrize("flavor", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("nx,ny", [(33, 47), (99, 101), (401, 303)])
def test_std_bs_sizes(ctx, flavor, nx, ny):
    check(ctx, nx, ny, flavor=flavor, center=-0.4 + 0j, dx=4.)


@pytest.mark.parametrize("kw", [
    dict(nexp=2), dict(nexp=3), dict(nexp=4), dict(nexp=7), dict(nexp=3, d2=True),
    dict(nexp=2, d2=True, backshift=2), dict(nexp=5, d2=True, backshift=4), dict(d2=True),
    dict(d2=True, backshift=3), dict(flavor=1, backshift=3), dict(flavor=5, backshift=2)],
    ids=lambda kw: "-".join(f"{k}{v}" for k, v in kw.items()))
def test_std_models_and_options(ctx, kw):
    check(ctx, 121, 83, center=-0.3 + 0j, **kw)


@pytest.mark.parametrize("block", [0, 32, 256])
@pytest.mark.parametrize("kw", [
    dict(max_iter=1), dict(max_iter=2), dict(max_iter=3), dict(max_iter=4), dict(max_iter=17),
    dict(eps=0.), dict(eps=1.5), dict(eps=1e-160), dict(M=2.), dict(M=0.1), dict(M=1e160),
    dict(M=1e140, max_iter=60), dict(flavor=2, M=1e160), dict(flavor=1, max_iter=1), dict(flavor=3, max_iter=2),
    dict(dx=1e-200, center=0j), dict(dx=1e200), dict(flavor=1, dx=1e200), dict(center=0j, dx=1e-3)],
    ids=lambda kw: "-".join(f"{k}{v}" for k, v in kw.items()))
def test_std_limits(ctx, kw, block):
    check(ctx, 41, 57, block=block, **kw)
