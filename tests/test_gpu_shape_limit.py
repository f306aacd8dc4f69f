"""
ctas_per_sm with the launcher's own choice of CTA: at most that many CTAs an SM,
of 256 threads -- the outputs, and within noise the time, of block = 256.
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


def _std(side):
    """xs, ys, the tile's own arguments, whether a perturbation, and the calculation's"""
    xs, ys = syn.image_axes(side, side)
    return xs, ys, dict(center=-0.5 + 0j, dx=3.), 3, False, dict(max_iter=2000, epsilon_stationnary=0.01)


def _m2(ctx, side, mode):
    from fractalshades_gb300 import _native as nat
    w = syn.prepare_m2(p=361, dps=1100, dx="1e-305", nx=side, max_iter=3000) if mode == "xr64" \
        else syn.seahorse_workload(nx=side)
    ref = nat.Reference(ctx, w.Zn, div_iter=w.div_iter, order=w.order, xr_idx=w.xr_idx, xr_m=w.xr_m,
                        xr_e=w.xr_e, xr_paths=w.xr_mode, calc_dzndc=True, scale_m=w.dx_m,
                        scale_e=w.dx_e, bla=True, kc=w.kc, bla_eps=1e-6)
    kw = dict(ref=ref, dx_m=w.dx_m, dx_e=w.dx_e, drift_m=w.drift_m, drift_e=w.drift_e, i_dzndc=1)
    return w.xs, w.ys, kw, 2, True, dict(max_iter=w.max_iter, mode=mode, calc_dzndc=True, bla=True,
                                         xr_semantics=w.xr_mode)


@pytest.mark.parametrize("kind,side", [("std", 40), ("std", 150), ("fp64", 200), ("xr64", 180)])
def test_limit_keeps_the_shape(ctx, kind, side):
    from fractalshades_gb300 import _native as nat
    # (a tile holds addresses: everything it points to lives to the end of the test)
    xs, ys, tile_kw, nZ, perturb, calc_kw = _std(side) if kind == "std" else _m2(ctx, side, kind)
    n = side * side
    run = ctx.perturb_tiles if perturb else ctx.std_tiles
    outs, times = [], []
    for block in (256, 0):
        Z = np.zeros((nZ, n), dtype=np.complex128)
        sr, si = -np.ones((1, n), dtype=np.int8), np.zeros((1, n), dtype=np.int32)
        tile = nat.make_tile(xs=xs, ys=ys, lin_mat=LIN, Z=Z, stop_reason=sr, stop_iter=si, **tile_kw)
        calc = nat.make_calc(M_divergence=1000., block=block, ctas_per_sm=1, **calc_kw)
        ms = []
        for _ in range(6):
            run(calc, [tile])
            ms.append(ctx.stats()["kernel_ms"])
        outs.append((Z, sr, si))
        times.append(min(ms))
    for x, y in zip(*outs):
        assert np.array_equal(x, y)
    # one and the same launch: 10 % is many times the difference of two runs
    assert abs(times[1] / times[0] - 1.) <= 0.1
