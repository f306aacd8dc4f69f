"""
Performance cases: the iteration paths a program of this framework calls, on
device buffers, through the public entry points (``fractalshades_gb300._native``
Context / Reference, the calls the model classes make).

A case names its path with ``kind`` and gives the image size and the options:

  std    standard escape-time loops: ``flavor`` 0 the Mandelbrot family
         (``nexp`` 0 the power-2 model, else the power-n model), 1 .. 5 the
         Burning Ship family; ``options`` adds d2zndc2 and the orbit point
         n - 3 (the inputs of Milnor shading and field lines)
  m2     power-2 Mandelbrot perturbation with a reference orbit, BLA and
         derivatives, in ``mode`` fp64 / xr64 / fe32; ``period`` > 0: around the
         nucleus of that period, 1 to 1.4 times 10^-``depth`` wide; 0: the seahorse valley,
         where every pixel escapes; ``interior``: interior detection
  bs     Burning Ship perturbation around a nucleus found from ``center_seed``,
         ``edge``: four nucleus sizes wide (pixels escape), else 1e-30 .. 1e-200
  view   a new view: the reference tables are built from the orbit, one tile is
         rendered with them, the reference is dropped

Sizes, centres and options are those of this repository's synthetic workloads,
tests and benchmark, with odd sizes beside them.
"""
import math

import mpmath
import numpy as np
import torch

from fractalshades_gb300 import _native as nat
from fractalshades_gb300 import synthetic as syn

DEV = "cuda"
LIN = np.array([[1., -0.], [0., 1.]])
M_DIV = 1000.
BACKSHIFT = 3

# nuclei of the synthetic workloads: period -> decimal digits of the stored centre
PERIODS = {361: 1100, 1071: 1100, 1566: 1100, 1691: 1100, 2002: 1100, 2111: 1100,
           2474: 1100, 2482: 1100, 2562: 400}

# views of the standard loop: centre and width of the whole set
STD_VIEW = {0: (-0.5, 0., 3.), 1: (-0.4, 0.5, 4.), 2: (-0.4, 0., 4.), 3: (-0.4, 0., 4.),
            4: (-0.4, 0., 4.), 5: (-0.4, 0., 4.)}

_ctx = None


def context():
    global _ctx
    if _ctx is None:
        _ctx = nat.Context(0)
    return _ctx


def listed():
    return [
        # a frame of an interactive preview: the smallest call
        dict(name="std_frame_64x48", kind="std", flavor=0, nexp=0, nx=64, ny=48, max_iter=200,
             options=False),
        # the standard-loop configuration of the benchmark
        dict(name="std_m2_800x600", kind="std", flavor=0, nexp=0, nx=800, ny=600, max_iter=1000,
             options=False),
        # a final render of the whole set
        dict(name="std_m2_3001x2251", kind="std", flavor=0, nexp=0, nx=3001, ny=2251,
             max_iter=1000, options=False),
        # a Burning Ship image
        dict(name="std_bs_1001x667", kind="std", flavor=1, nexp=0, nx=1001, ny=667, max_iter=1000,
             options=False),
        # a power-3 image with the optional outputs
        dict(name="std_mn3_options_641x479", kind="std", flavor=0, nexp=3, nx=641, ny=479,
             max_iter=500, options=True),
        # the default form above 1e-300: double deltas, every pixel escapes
        dict(name="m2_fp64_seahorse_511x383", kind="m2", mode="fp64", period=0, depth=9, nx=511,
             ny=383, max_iter=6000, interior=False),
        # the default form below 1e-300: Xrange deltas, an interior view
        dict(name="m2_xr64_nucleus_513x511", kind="m2", mode="xr64", period=2562, depth=305,
             nx=513, ny=511, max_iter=200000, interior=False),
        # the headline view of the benchmark
        dict(name="m2_fe32_nucleus_2048", kind="m2", mode="fe32", period=2562, depth=300, nx=2048,
             ny=2048, max_iter=200000, interior=False),
        # the fast form where every pixel escapes
        dict(name="m2_fe32_seahorse_1024", kind="m2", mode="fe32", period=0, depth=9, nx=1024,
             ny=1024, max_iter=6000, interior=False),
        # Burning Ship, double deltas, a boundary view
        dict(name="bs_fp64_edge_255", kind="bs", mode="fp64", center_seed=4, edge=True, side=255,
             max_iter=20000),
        # Burning Ship, fast form, a deep tile
        dict(name="bs_fe32_deep_640", kind="bs", mode="fe32", center_seed=4, edge=False, side=640,
             max_iter=20000),
        # the first tile of a new centre: table build, then a 256 x 256 tile
        dict(name="view_fe32_256", kind="view", mode="fe32", period=2474, depth=600, nx=256,
             ny=256, max_iter=200000, interior=False),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["std", "std", "m2", "m2", "bs", "view"])
    if kind == "std":
        flavor = rng.choice([0, 0, 0, 1, 2, 3, 4, 5])
        nexp = rng.choice([0, 0, 3, 4]) if flavor == 0 else 0
        top = 2400 if flavor == 0 and nexp == 0 else 1000
        return dict(kind="std", flavor=flavor, nexp=nexp, nx=_log_int(rng, 48, top),
                    ny=_log_int(rng, 48, top), max_iter=_log_int(rng, 100, 1000),
                    options=rng.random() < 0.25)
    if kind == "m2":
        mode = rng.choice(["fp64", "xr64", "fe32", "fe32"])
        top = 1800 if mode == "fe32" else 450
        period = rng.choice([0] + sorted(PERIODS)) if mode != "xr64" else rng.choice(sorted(PERIODS))
        if period == 0:
            depth, max_iter = 9, 6000
        else:
            max_iter = _log_int(rng, 20000, 200000)
            lo, hi = {"fp64": (30, 290), "xr64": (301, 1000), "fe32": (30, 1000)}[mode]
            depth = rng.randint(lo, min(hi, (300 if PERIODS[period] == 400 else 1000) + 5))
        return dict(kind="m2", mode=mode, period=period, depth=depth, nx=_log_int(rng, 64, top),
                    ny=_log_int(rng, 64, top), max_iter=max_iter,
                    interior=period != 0 and rng.random() < 0.5)
    if kind == "bs":
        mode = rng.choice(["fp64", "fe32"])
        return dict(kind="bs", mode=mode, center_seed=rng.randint(1, 1000), edge=rng.random() < 0.5,
                    side=_log_int(rng, 48, 200 if mode == "fp64" else 700),
                    max_iter=_log_int(rng, 2000, 20000))
    period = rng.choice([p for p in sorted(PERIODS) if PERIODS[p] == 1100])
    mode = rng.choice(["fe32", "xr64"])
    return dict(kind="view", mode=mode, period=period, depth=rng.randint(301, 1000),
                nx=_log_int(rng, 32, 256), ny=_log_int(rng, 32, 256), max_iter=200000,
                interior=rng.random() < 0.5)


# ---------------------------------------------------------------------------
# what a program has in hand
# ---------------------------------------------------------------------------
def _offsets(seed):
    r = np.random.default_rng(seed)
    return float(r.uniform(-0.04, 0.04)), float(r.uniform(-0.04, 0.04))


def _std_view(case, seed):
    """Screen axes, centre and width of a standard view (shifted a little by
    the seed)."""
    xs, ys = syn.image_axes(case["nx"], case["ny"], case["nx"] / case["ny"])
    cre, cim, dx = STD_VIEW[case["flavor"]]
    ox, oy = _offsets(seed)
    return xs, ys, complex(cre + ox, cim + oy), dx


def _rows(case):
    """(complex Z, rows of Z)"""
    if case["kind"] == "std":
        if case["flavor"] != 0:
            return False, 6 + (2 if case["options"] else 0)
        return True, 3 + (2 if case["options"] else 0)
    if case["kind"] == "bs":
        return False, 6
    return True, 3 if case["interior"] else 2


def _outputs(case, n):
    cplx, nZ = _rows(case)
    f64 = dict(dtype=torch.float64, device=DEV)
    return dict(Z=torch.zeros((nZ, n, 2) if cplx else (nZ, n), **f64),
                stop_reason=torch.full((n,), -1, dtype=torch.int8, device=DEV),
                stop_iter=torch.zeros(n, dtype=torch.int32, device=DEV),
                potential=torch.zeros(n, **f64), dem=torch.zeros(n, **f64))


def _tile(case, out, xs, ys, **kw):
    return nat.make_tile_ptrs(
        nx=xs.numel(), ny=ys.numel(), xs_ptr=xs.data_ptr(), ys_ptr=ys.data_ptr(), lin_mat=LIN,
        Z_ptr=out["Z"].data_ptr(), nZ=_rows(case)[1], stop_reason_ptr=out["stop_reason"].data_ptr(),
        stop_iter_ptr=out["stop_iter"].data_ptr(), potential_ptr=out["potential"].data_ptr(),
        dem_ptr=out["dem"].data_ptr(), **kw)


def _prepare_std(case, seed):
    xs, ys, center, dx = _std_view(case, seed)
    xs, ys = torch.from_numpy(xs).to(DEV), torch.from_numpy(ys).to(DEV)
    out = _outputs(case, xs.numel() * ys.numel())
    opt = case["options"]
    calc = nat.make_calc(max_iter=case["max_iter"], M_divergence=M_DIV,
                         epsilon_stationnary=0.01, flavor=case["flavor"], nexp=case["nexp"],
                         calc_d2zndc2=opt and case["flavor"] == 0,
                         backshift=BACKSHIFT if opt else 0)
    i_orb = (4 if case["flavor"] == 0 else 6) if opt else 0
    tile = _tile(case, out, xs, ys, center=center, dx=dx, i_znorbit=i_orb)
    return dict(kind="std", calc=calc, tile=tile, out=out, keep=(xs, ys))


def _m2_workload(case, seed):
    off = _offsets(seed)
    if case["period"] == 0:
        with mpmath.workdps(30):
            c = mpmath.mpc("-0.743643887037151", "0.131825904205330")
        return syn.prepare_m2(p=None, dps=30, dx="2.e-9", nx=case["nx"], ny=case["ny"],
                              max_iter=case["max_iter"], M=M_DIV, center=c, offset=off)
    return syn.prepare_m2(p=case["period"], dps=PERIODS[case["period"]],
                          dx="%.9fe-%d" % (1. + 10. * abs(off[0]), case["depth"]),
                          nx=case["nx"], ny=case["ny"],
                          max_iter=case["max_iter"], M=M_DIV, offset=off,
                          xr_mode=False if case["mode"] == "fp64" else True)


def _m2_reference(case, w):
    return nat.Reference(context(), w.Zn, div_iter=w.div_iter, order=w.order, xr_idx=w.xr_idx,
                         xr_m=w.xr_m, xr_e=w.xr_e, xr_paths=w.xr_mode, calc_dzndc=True,
                         calc_dzndz=case["interior"], scale_m=w.dx_m, scale_e=w.dx_e, bla=True,
                         kc=w.kc, bla_eps=1e-6)


def _m2_tile(case, w, ref, out, xs, ys):
    # below the double range the derivative is taken per width, not per unit
    scale_e = -w.dx_e if case["depth"] >= 300 else 0
    return _tile(case, out, xs, ys, ref=ref, dx_m=w.dx_m, dx_e=w.dx_e, drift_m=w.drift_m,
                 drift_e=w.drift_e, i_dzndz=1 if case["interior"] else -1,
                 i_dzndc=2 if case["interior"] else 1, dzndc_scale_e=scale_e)


def _prepare_m2(case, seed):
    w = _m2_workload(case, seed)
    xs, ys = torch.from_numpy(w.xs).to(DEV), torch.from_numpy(w.ys).to(DEV)
    out = _outputs(case, xs.numel() * ys.numel())
    calc = nat.make_calc(max_iter=w.max_iter, M_divergence=w.M, epsilon_stationnary=1e-3,
                         mode=case["mode"], calc_dzndc=True, interior=case["interior"], bla=True,
                         xr_semantics=w.xr_mode)
    s = dict(kind=case["kind"], calc=calc, out=out, keep=(xs, ys))
    if case["kind"] == "view":
        s.update(case=case, w=w, xs=xs, ys=ys)
    else:
        s["ref"] = _m2_reference(case, w)
        s["tile"] = _m2_tile(case, w, s["ref"], out, xs, ys)
    return s


def _prepare_bs(case, seed):
    t = syn.config4_workload(seed=case["center_seed"], n_tiles=1, max_iter=case["max_iter"],
                             M=M_DIV, edge=case["edge"])[0]
    xs, ys = syn.image_axes(case["side"], case["side"])
    xs, ys = torch.from_numpy(xs).to(DEV), torch.from_numpy(ys).to(DEV)
    out = _outputs(case, xs.numel() * ys.numel())
    ref = nat.Reference(context(), t.Zn, div_iter=t.div_iter, order=t.ref_order, flavor=1,
                        calc_dzndc=True, scale_m=t.dx_m, scale_e=t.dx_e, bla=True, kc=t.kc,
                        bla_eps=1e-6)
    ox, oy = _offsets(seed)
    calc = nat.make_calc(max_iter=case["max_iter"], M_divergence=M_DIV, flavor=1, calc_dzndc=True,
                         bla=True, mode=case["mode"])
    tile = _tile(case, out, xs, ys, ref=ref, dx_m=t.dx_m, dx_e=t.dx_e, drift_m=ox * t.dx_m,
                 drift_e=t.dx_e, drifty_m=oy * t.dx_m, drifty_e=t.dx_e)
    return dict(kind="bs", calc=calc, tile=tile, out=out, ref=ref, keep=(xs, ys))


def prepare(case, seed):
    context()
    s = {"std": _prepare_std, "m2": _prepare_m2, "view": _prepare_m2, "bs": _prepare_bs}[
        case["kind"]](case, seed)
    torch.cuda.synchronize()      # the buffers are set before the library's stream uses them
    return s


def run(state):
    ctx = context()
    if state["kind"] == "std":
        ctx.std_tiles(state["calc"], [state["tile"]], nat.DEVICE)
    elif state["kind"] == "view":
        ref = _m2_reference(state["case"], state["w"])
        tile = _m2_tile(state["case"], state["w"], ref, state["out"], state["xs"], state["ys"])
        ctx.perturb_tiles(state["calc"], [tile], nat.DEVICE)
        ref.free()
    else:
        ctx.perturb_tiles(state["calc"], [state["tile"]], nat.DEVICE)
    return state["out"]


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: the axes and, for a new view, the orbit, read once; every output
    written once.  Flops: the mean iterations of a pixel of the path (executed
    steps where BLA skips) times the operations of one step."""
    nx, ny = (case["side"], case["side"]) if case["kind"] == "bs" else (case["nx"], case["ny"])
    n = nx * ny
    cplx, nZ = _rows(case)
    nbytes = 8 * (nx + ny) + n * (nZ * (16 if cplx else 8) + 1 + 4 + 16)
    if case["kind"] == "std":
        steps = min(case["max_iter"], 26)
        per = 26 if case["flavor"] == 0 else 32
    elif case["kind"] == "bs":
        steps, per = case["max_iter"] * (0.6 if case["edge"] else 1.), 60
    elif case["period"] == 0:
        steps, per = 1200, 35
    else:
        # a period of the orbit is a few steps: BLA runs and the steps around
        # the critical point
        steps, per = 12. * case["max_iter"] / case["period"], 30
        if case["interior"]:
            steps = min(steps, 24.)
    if case["kind"] == "view":
        nbytes += 16 * case["period"]
    return {"bytes": float(nbytes), "flops": float(n * steps * per)}


# ---------------------------------------------------------------------------
# the values in 64 bits
# ---------------------------------------------------------------------------
def _epilogue(out, zx, zy, absd, n, degree):
    az = torch.hypot(zx, zy)
    x = torch.log(torch.log(az) / math.log(M_DIV)) / math.log(degree)
    q = torch.floor(x)
    out["potential"] = (n.double() - q) - (x - q)
    out["dem"] = az * torch.log(az) / absd


def _cmul(a, b):
    return a[0] * b[0] - a[1] * b[1], a[0] * b[1] + a[1] * b[0]


def _cpow(a, k):
    """a^k for k = 1 .. 4, squares and products left to right."""
    if k == 1:
        return a
    if k == 2:
        return _cmul(a, a)
    if k == 3:
        return _cmul(a, _cmul(a, a))
    return _cmul(_cmul(a, a), _cmul(a, a))


class _Pixels:
    """The pixels still iterating, and where the stopped ones go."""

    def __init__(self, case, seed):
        xs, ys, center, dx = _std_view(case, seed)
        px, py = np.meshgrid(xs, ys)
        self.n = px.size
        self.a = torch.from_numpy(center.real + dx * px.ravel()).to(DEV)
        self.b = torch.from_numpy(center.imag + dx * py.ravel()).to(DEV)
        self.at = torch.arange(self.n, device=DEV)
        self.out = dict(stop_iter=torch.zeros(self.n, dtype=torch.int32, device=DEV),
                        stop_reason=torch.full((self.n,), -1, dtype=torch.int8, device=DEV))

    def stop(self, mask, rows, values, n, reason):
        """Stores the masked pixels; what is left of the values and of c."""
        at = self.at[mask]
        for r, v in zip(rows, values):
            r[at] = v[mask]
        self.out["stop_iter"][at] = n
        self.out["stop_reason"][at] = reason
        keep = ~mask
        self.at, self.a, self.b = self.at[keep], self.a[keep], self.b[keep]
        return [v[keep] for v in values]


def _exact_mandelbrot(case, seed):
    p = _Pixels(case, seed)
    k = case["nexp"] or 2
    z0 = torch.zeros(p.n, dtype=torch.float64, device=DEV)
    rows = [z0.clone() for _ in range(8)]     # zn, dzndz, dzndc, d2zndc2
    v = [z0.clone() for _ in range(8)]
    for n in range(1, case["max_iter"] + 1):
        if p.at.numel() == 0:
            break
        if n == case["max_iter"]:
            p.stop(torch.ones_like(p.at, dtype=torch.bool), rows, v, n, 0)
            break
        z, dz, dc, d2 = (v[0], v[1]), (v[2], v[3]), (v[4], v[5]), (v[6], v[7])
        if case["options"]:
            if case["nexp"]:
                # the model's recurrence, with dzndz in its second term
                zm2 = _cpow(z, k - 2)
                zm1 = _cmul(zm2, z)
                s, t = _cmul(d2, zm1), _cmul(_cmul(((k - 1.) * dz[0], (k - 1.) * dz[1]), dc), zm2)
            else:
                zm1 = z
                s, t = _cmul(d2, z), _cmul(dc, dc)
            d2 = (float(k) * (s[0] + t[0]), float(k) * (s[1] + t[1]))
        else:
            zm1 = _cpow(z, k - 1)
        w = _cmul((k * dc[0], k * dc[1]), zm1)
        dc = (w[0] + 1., w[1])
        dz = _cmul((k * dz[0], k * dz[1]), zm1)
        if n == 1:
            dz = (torch.ones_like(z[0]), torch.zeros_like(z[0]))
        w = _cmul(zm1, z)
        z = (w[0] + p.a, w[1] + p.b)
        v = [z[0], z[1], dz[0], dz[1], dc[0], dc[1], d2[0], d2[1]]
        v = p.stop(z[0] * z[0] + z[1] * z[1] > M_DIV * M_DIV, rows, v, n, 1)
        still = v[2] * v[2] + v[3] * v[3] < 0.01 * 0.01
        v = p.stop(still, rows, v, n, 2)
    pairs = [torch.stack(rows[2 * i:2 * i + 2], dim=1) for i in range(4)]
    out = p.out
    # with the orbit row in Z there is no whole Z here
    out["Z"] = None if case["options"] else torch.stack(pairs[:3])
    _epilogue(out, rows[0], rows[1], torch.hypot(rows[4], rows[5]), out["stop_iter"], k)
    return out


def _sgn(x):
    return torch.where(x < 0., -1., 1.).double()


def _exact_ship(case, seed):
    p = _Pixels(case, seed)
    z0 = torch.zeros(p.n, dtype=torch.float64, device=DEV)
    rows = [z0.clone() for _ in range(6)]
    v = [z0.clone() for _ in range(6)]
    f = case["flavor"]
    for n in range(1, case["max_iter"] + 1):
        if p.at.numel() == 0:
            break
        if n == case["max_iter"]:
            p.stop(torch.ones_like(p.at, dtype=torch.bool), rows, v, n, 0)
            break
        X, Y, xa, xb, ya, yb = v
        if f in (1, 2):
            nX = X * X - Y * Y + p.a
            nxa = 2. * (X * xa - Y * ya) + 1.
            nxb = 2. * (X * xb - Y * yb)
        elif f == 3:
            nX = X * X - Y * Y.abs() + p.a
            nxa = 2. * (X * xa - Y.abs() * ya) + 1.
            nxb = 2. * (X * xb - Y.abs() * yb)
        else:
            q = X * X - Y * Y
            nX = q.abs() + p.a
            nxa = 2. * _sgn(q) * (X * xa - Y * ya)
            nxb = 2. * _sgn(q) * (X * xb - Y * yb)
        if f in (1, 5):
            nY = 2. * (X * Y).abs() - p.b
            nya = 2. * (X.abs() * _sgn(Y) * ya + _sgn(X) * xa * Y.abs())
            nyb = 2. * (X.abs() * _sgn(Y) * yb + _sgn(X) * xb * Y.abs()) - 1.
        elif f == 2:
            nY = 2. * X * Y.abs() - p.b
            nya = 2. * (X * _sgn(Y) * ya + xa * Y.abs())
            nyb = 2. * (X * _sgn(Y) * yb + xb * Y.abs()) - 1.
        else:
            nY = 2. * X * Y - p.b
            nya = 2. * (xa * Y + X * ya)
            nyb = 2. * (xb * Y + X * yb) - 1.
        v = [nX, nY, nxa, nxb, nya, nyb]
        v = p.stop(nX * nX + nY * nY > M_DIV * M_DIV, rows, v, n, 1)
    out = p.out
    out["Z"] = None if case["options"] else torch.stack(rows)
    xa, xb, ya, yb = rows[2:]
    absd = 0.5 * (torch.hypot(xa + yb, xb - ya) + torch.hypot(xa - yb, xb + ya))
    _epilogue(out, rows[0], rows[1], absd, out["stop_iter"], 2)
    return out


def exact(case, seed):
    """The standard loops in plain 64-bit arithmetic.  The perturbation cases
    have none: their views are below the double range or resolved by skipped
    steps whose truncation a plain loop does not share, and their iteration
    counts amplify it."""
    if case["kind"] != "std":
        return None
    return _exact_mandelbrot(case, seed) if case["flavor"] == 0 else _exact_ship(case, seed)
