"""
The FP64 and Xrange power-2 loops against the oracle bit for bit (but for the sign
of a zero): the oracle takes the tables that the GPU built, so that no radius
differs by an ulp of hypot, and every other operation of the two is the same.
"""
import numpy as np
import pytest

from fractalshades_gb300 import synthetic as syn
from oracle import oracle as orc
from test_gpu_m2_ranges import LIN, _reference, _run, _view, ctx  # noqa: F401

pytestmark = pytest.mark.gpu


def _same(ctx, w, mode, interior):  # noqa: F811
    xr = mode == "xr64"
    ref = _reference(ctx, w, interior)
    Z, si, sr = _run(ctx, w, ref, mode, interior)
    kw = dict(Zn=w.Zn, ref_div_iter=w.div_iter, ref_order=w.order, lin_mat=LIN, dx_m=w.dx_m, dx_e=w.dx_e,
              drift_m=w.drift_m, drift_e=w.drift_e, max_iter=w.max_iter, M=w.M, eps_stat=1e-3, xr_mode=xr,
              bla=ref.download("bla") + (ref.stages,), interior=interior, xr_idx=w.xr_idx, xr_m=w.xr_m,
              xr_e=w.xr_e, dZndc=ref.download("dzndc"))
    if interior:
        kw["dZndz"] = ref.download("dzndz")
    Zo, _, sro, sio = orc.perturb_m2((w.xs[None, :] + 1j * w.ys[:, None]).ravel(), **kw)
    assert np.array_equal(si, sio) and np.array_equal(sr, sro)
    for k in range(Z.shape[0]):
        if interior and k == 1 and xr:
            continue                     # the Xrange branch does not write dzndz
        a, b = Z[k].view(np.float64), np.ascontiguousarray(Zo[k]).view(np.float64)
        assert np.array_equal(np.isnan(a), np.isnan(b))
        ok = ~np.isnan(a)
        assert np.array_equal(a[ok], b[ok])


@pytest.mark.parametrize("interior", [False, True])
@pytest.mark.parametrize("where", ["axis", "bulb"])
@pytest.mark.parametrize("dx,xr", [("1e-3", False), ("1e-7", False), ("1e-30", False), ("1e-150", False),
                                   ("1e-200", False), ("1e-290", False), ("1e-5", True),
                                   ("1e-305", True), ("1e-340", True), ("1e-700", True)])
def test_m2_bits(ctx, where, dx, xr, interior):  # noqa: F811
    _same(ctx, _view(where, dx, xr), "xr64" if xr else "fp64", interior)


# views whose pixels escape after steps near the orbit's size
@pytest.mark.parametrize("mode", ["fp64", "xr64"])
def test_m2_bits_boundary(ctx, mode):  # noqa: F811
    _same(ctx, syn.edge_workload(nx=20, max_iter=20000, xr_mode=mode == "xr64"), mode, False)


def test_m2_bits_seahorse(ctx):  # noqa: F811
    _same(ctx, syn.seahorse_workload(nx=40), "fp64", False)
