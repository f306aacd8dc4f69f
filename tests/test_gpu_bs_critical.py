"""
The FP32 Burning Ship form right after a rebase: the step at the critical point
follows at once unless a BLA step could be taken there.  With a tree that admits
no step (a period of 12, its only radius 0) BLA changes neither the pixels nor,
beyond a look at the tree every eighth point, the time.
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


@pytest.mark.parametrize("edge", [True, False])
@pytest.mark.parametrize("side", [64, 200])
def test_bla_that_admits_nothing(ctx, side, edge):
    from fractalshades_gb300 import _native as nat
    t = syn.config4_workload(seed=4, n_tiles=1, max_iter=3000, edge=edge)[0]
    ref = nat.Reference(ctx, t.Zn, div_iter=t.div_iter, order=t.ref_order, flavor=1, calc_dzndc=True,
                        scale_m=t.dx_m, scale_e=t.dx_e, bla=True, kc=t.kc, bla_eps=1e-6)
    xs, ys = syn.image_axes(side, side)
    n = side * side
    outs, times = [], []
    for bla in (False, True):
        Z, sr = np.zeros((6, n)), -np.ones((1, n), dtype=np.int8)
        si = np.zeros((1, n), dtype=np.int32)
        tile = nat.make_tile(xs=xs, ys=ys, lin_mat=LIN, Z=Z, stop_reason=sr, stop_iter=si, ref=ref,
                             dx_m=t.dx_m, dx_e=t.dx_e, drift_m=0.01 * t.dx_m, drift_e=t.dx_e,
                             drifty_m=0., drifty_e=0)
        calc = nat.make_calc(max_iter=3000, M_divergence=1000., flavor=1, calc_dzndc=True, bla=bla,
                             mode="fe32")
        ms = []
        for _ in range(6):
            ctx.perturb_tiles(calc, [tile])
            ms.append(ctx.stats()["kernel_ms"])
        assert ctx.stats()["bla_steps"] == 0
        outs.append((Z, sr, si))
        times.append(min(ms))
    for a, b in zip(*outs):
        assert np.array_equal(a, b, equal_nan=a.dtype == np.float64)
    # one more table read every eighth point, of some 200 instructions a point
    assert times[1] <= 1.05 * times[0]
