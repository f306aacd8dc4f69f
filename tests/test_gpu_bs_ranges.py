"""
The double form of the Burning Ship perturbation loop over the cases its step
tells apart -- references on the real axis and off it, deltas from the size of
the view down to products below the double range, with and without the
Jacobian, every flavor -- against the oracle.
"""
import numpy as np
import pytest

from fractalshades_gb300 import synthetic as syn
from fractalshades_gb300.numpy_utils import xrange as fsx
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
LIN = np.array([[1., -0.], [0., 1.]])


@pytest.fixture(scope="module")
def ctx():
    from fractalshades_gb300 import _native as nat
    c = nat.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("hess", [True, False])
@pytest.mark.parametrize("width", ["1e-2", "1e-6", "1e-30", "1e-140", "1e-170", "1e-250"])
@pytest.mark.parametrize("flavor,seed", [(1, 4), (1, 5), (1, 77), (2, 4), (3, 4), (4, 4), (5, 4)])
def test_bs_fp64_ranges_vs_oracle(ctx, flavor, seed, width, hess):
    import mpmath
    from fractalshades_gb300 import _native as nat
    # seeds 4, 77: nuclei on the real axis; 5: off it
    t = syn.config4_workload(seed=seed, n_tiles=1, max_iter=600, kind=flavor)[0]
    dx = fsx.mpf_to_Xrange(mpmath.mpf(width))
    kc = float(np.ldexp(dx.m, dx.e))
    xs, ys = syn.image_axes(19, 13)                      # odd: a row and a column at 0
    pix = (xs[None, :] + 1j * ys[:, None]).ravel()
    n = pix.size
    Zn, div, order = t.Zn, t.div_iter, t.ref_order
    Mb, rb, _, st = orc.make_bla_bs(Zn, flavor, kc, 1e-6)
    paths = orc.dzndc_path_bs(Zn, div, order, flavor, float(np.ldexp(dx.m, dx.e))) if hess else None
    drift = dict(driftx_m=0.01 * dx.m, driftx_e=dx.e, drifty_m=0., drifty_e=0)
    Zo, _, sro, sio = orc.perturb_bs(pix, Zn=Zn, ref_div_iter=div, ref_order=order, lin_mat=LIN,
                                     dx_m=dx.m, dx_e=dx.e, max_iter=600, M=1000., flavor=flavor,
                                     calc_hessian=hess, bla=(Mb, rb, st), dpaths=paths, **drift)
    ref = nat.Reference(ctx, Zn, div_iter=div, order=order, flavor=flavor, calc_dzndc=hess,
                        scale_m=dx.m, scale_e=dx.e, bla=True, kc=kc, bla_eps=1e-6)
    Z = np.zeros((6 if hess else 2, n))
    sr, si = -np.ones((1, n), dtype=np.int8), np.zeros((1, n), dtype=np.int32)
    tile = nat.make_tile(xs=xs, ys=ys, lin_mat=LIN, Z=Z, stop_reason=sr, stop_iter=si, ref=ref,
                         dx_m=dx.m, dx_e=dx.e, drift_m=drift["driftx_m"], drift_e=dx.e,
                         drifty_m=0., drifty_e=0)
    ctx.perturb_tiles(nat.make_calc(max_iter=600, M_divergence=1000., flavor=flavor, calc_dzndc=hess,
                                    bla=True, mode="fp64"), [tile])
    assert np.array_equal(si, sio) and np.array_equal(sr, sro)
    k = ~np.isnan(Zo[:Z.shape[0]])
    assert np.array_equal(k, ~np.isnan(Z))
    # bit for bit, but for the sign of a zero
    assert np.array_equal(Z[k], Zo[:Z.shape[0]][k])


@pytest.mark.parametrize("hess", [True, False])
@pytest.mark.parametrize("width", ["1e-5", "1e-30", "1e-200", "1e-320"])
@pytest.mark.parametrize("mode", ["fe32", "fp64"])
def test_bs_real_reference_alone_and_in_a_mixed_launch(ctx, mode, width, hess):
    """A launch whose references are all real takes the kernel of the real
    axis; in one launch with a reference off it, the general one: the same
    pixels bit for bit."""
    import mpmath
    from fractalshades_gb300 import _native as nat
    if mode == "fp64" and width == "1e-320":
        pytest.skip("below the double form's range")
    dx = fsx.mpf_to_Xrange(mpmath.mpf(width))
    kc = float(np.ldexp(dx.m, dx.e))
    xs, ys = syn.image_axes(37, 29)
    n = xs.size * ys.size
    refs = []
    for seed in (4, 5):                                  # on the real axis, off it
        t = syn.config4_workload(seed=seed, n_tiles=1, max_iter=600, kind=1)[0]
        refs.append(nat.Reference(ctx, t.Zn, div_iter=t.div_iter, order=t.ref_order, flavor=1,
                                  calc_dzndc=hess, scale_m=dx.m, scale_e=dx.e, bla=True, kc=kc,
                                  bla_eps=1e-6))

    def run(which):
        out, tiles = [], []
        for k in which:
            o = (np.zeros((6 if hess else 2, n)), -np.ones((1, n), dtype=np.int8),
                 np.zeros((1, n), dtype=np.int32))
            out.append(o)
            tiles.append(nat.make_tile(xs=xs, ys=ys, lin_mat=LIN, Z=o[0], stop_reason=o[1],
                                       stop_iter=o[2], ref=refs[k], dx_m=dx.m, dx_e=dx.e,
                                       drift_m=0.01 * dx.m, drift_e=dx.e, drifty_m=0., drifty_e=0))
        ctx.perturb_tiles(nat.make_calc(max_iter=3000, M_divergence=1000., flavor=1, calc_dzndc=hess,
                                        bla=True, mode=mode), tiles)
        return out

    for a, b in zip(run([0])[0], run([0, 1])[0]):
        assert np.array_equal(a, b, equal_nan=a.dtype == np.float64)


@pytest.mark.parametrize("seed", [4, 5])
@pytest.mark.parametrize("flavor", [1, 2, 3, 4, 5])
def test_bs_fe32_images_above_three_ctas_an_sm(ctx, flavor, seed):
    """Images that three CTAs an SM do not hold at once run in the four-CTA
    kernel: the pixels of a smaller launch."""
    import mpmath
    from fractalshades_gb300 import _native as nat
    t = syn.config4_workload(seed=seed, n_tiles=1, max_iter=300, kind=flavor)[0]
    dx = fsx.mpf_to_Xrange(mpmath.mpf("1e-8"))
    ref = nat.Reference(ctx, t.Zn, div_iter=t.div_iter, order=t.ref_order, flavor=flavor,
                        calc_dzndc=True, scale_m=dx.m, scale_e=dx.e, bla=True,
                        kc=float(np.ldexp(dx.m, dx.e)), bla_eps=1e-6)
    xs, ys = syn.image_axes(353, 347)

    def run(xs, ys):
        n = xs.size * ys.size
        Z, sr = np.zeros((6, n)), -np.ones((1, n), dtype=np.int8)
        si = np.zeros((1, n), dtype=np.int32)
        tile = nat.make_tile(xs=xs, ys=ys, lin_mat=LIN, Z=Z, stop_reason=sr, stop_iter=si, ref=ref,
                             dx_m=dx.m, dx_e=dx.e, drift_m=0.01 * dx.m, drift_e=dx.e,
                             drifty_m=0., drifty_e=0)
        ctx.perturb_tiles(nat.make_calc(max_iter=300, M_divergence=1000., flavor=flavor,
                                        calc_dzndc=True, bla=True, mode="fe32"), [tile])
        return [x.reshape(x.shape[0], ys.size, xs.size) for x in (Z, sr, si)]

    for big, small in zip(run(xs, ys), run(xs[:90], ys[:70])):
        assert np.array_equal(big[:, :70, :90], small, equal_nan=small.dtype == np.float64)
