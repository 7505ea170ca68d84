"""Measured workloads of the engine, each one pass through a public entry point.

`listed()` names the cases, `draw(rng)` gives further ones of the same ranges;
`prepare` makes what a program holds before the call, `run` is the call,
`work` what a pass cannot do without, and `exact` the same outputs in 64 bits.

Kinds:
  entry   LocVolCalib's entry point (f32 `main` or its f64 twin), one
          calibration per call, prices returned to the host
  mix     the batched form: a plan of uneven calibrations, new market inputs
          uploaded, one run, all prices copied back
  serve   a burst of requests to a running server, every result awaited
  tridag  batched f32 tridiagonal solves on device arrays
  tke     one turbulent-kinetic-energy step of the ocean model on device arrays
  op      OptionPricing on device arrays, one price vector per call
"""
import functools
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("futhark-benchmarks_b200")
wl = importlib.import_module("futhark-benchmarks_b200.workloads")
tke = importlib.import_module("futhark-benchmarks_b200.tke")
op = importlib.import_module("futhark-benchmarks_b200.op")

DEVICE = "cuda"


def listed():
    return [
        # The reference's three datasets: few strikes on a long time line, a
        # wide x grid, a grid that needs a cluster.
        {"name": "entry_small", "kind": "entry", "f64": True, "outer": 16, "numX": 32, "numY": 256, "numT": 256},
        {"name": "entry_medium_f32", "kind": "entry", "f64": False, "outer": 128, "numX": 256, "numY": 32,
         "numT": 64},
        {"name": "entry_large", "kind": "entry", "f64": True, "outer": 256, "numX": 256, "numY": 256, "numT": 64},
        # A grid that is a multiple of nothing.
        {"name": "entry_ragged", "kind": "entry", "f64": True, "outer": 50, "numX": 101, "numY": 75, "numT": 130},
        # A book of calibrations repriced with new market inputs.
        {"name": "mix_512", "kind": "mix", "f64": True, "count": 512, "sizes": 0},
        # Requests that arrive together at the serving runtime, FP32 state.
        {"name": "serve_48_f32state", "kind": "serve", "f64": False, "count": 48, "sizes": 1},
        # The tridiagonal test program: its small dataset's size, its benchmark
        # size, and the columns of a 200 x 200 x 100 ocean.
        {"name": "tridag_seq_small", "kind": "tridag", "form": "seq", "rows": 100, "m": 115},
        {"name": "tridag_seq", "kind": "tridag", "form": "seq", "rows": 57600, "m": 115},
        {"name": "tridag_par_ocean", "kind": "tridag", "form": "par", "rows": 40000, "m": 100},
        # The ocean model's benchmark size.
        {"name": "tke_200x200x100", "kind": "tke", "x": 200, "y": 200, "z": 100},
        # OptionPricing: the small dataset's size in the reduction order of the
        # reference's golden outputs, the large one's in the default order.
        {"name": "op_european_seq", "kind": "op", "contract": 1, "paths": 1 << 23, "models": 1, "sequential": True},
        {"name": "op_daily", "kind": "op", "contract": 3, "paths": 131072, "models": 1, "sequential": False},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["entry", "entry", "mix", "serve", "tridag", "tridag", "tke", "op", "op"])
    if kind == "entry":
        # the workloads' grid sizes, or any size between them
        size = (lambda: rng.choice(wl.GRID_SIZES)) if rng.random() < 0.5 else (lambda: _log_int(rng, 24, 256))
        return {"kind": kind, "f64": rng.random() < 0.7, "outer": _log_int(rng, 4, 256), "numX": size(),
                "numY": size(), "numT": _log_int(rng, 8, 256)}
    if kind in ("mix", "serve"):
        hi = 512 if kind == "mix" else 48
        return {"kind": kind, "f64": rng.random() < 0.5, "count": _log_int(rng, hi // 16, hi),
                "sizes": rng.randrange(1 << 20)}
    if kind == "tridag":
        return {"kind": kind, "form": rng.choice(["seq", "par"]), "rows": _log_int(rng, 32, 57600),
                "m": _log_int(rng, 8, 256)}
    if kind == "tke":
        return {"kind": kind, "x": _log_int(rng, 16, 200), "y": _log_int(rng, 16, 200), "z": _log_int(rng, 10, 100)}
    contract = rng.choice([1, 2, 3])
    lo, hi = {1: (1 << 16, 1 << 23), 2: (1 << 14, 1 << 20), 3: (1 << 11, 131072)}[contract]
    models = rng.choice([1, 1, 2, 4])
    return {"kind": "op", "contract": contract, "paths": _log_int(rng, lo, hi) // models, "models": models,
            "sequential": rng.random() < 0.5}


# --- what a program keeps: one context per library, one server --------------

@functools.cache
def _ctx():
    return pkg.Context("#0")


@functools.cache
def _server(f64):
    return pkg.Server(_ctx(), precision=pkg.F64 if f64 else pkg.F32_STATE)


@functools.cache
def _tke_ctx():
    return tke.TkeContext("#0")


@functools.cache
def _op_ctx(sequential):
    c = op.OpContext("#0")
    if sequential:
        c.set_reduction_order(c.ORDER_SEQUENTIAL_F32)
    return c


# --- inputs -----------------------------------------------------------------

def _market(rng):
    """s0, t, alpha, nu, beta on the ranges of the uneven mix."""
    return tuple(float(rng.uniform(lo, hi)) for lo, hi in ((0.02, 0.05), (1.0, 10.0), (0.1, 0.3), (0.4, 0.8),
                                                           (0.3, 0.7)))


def _calibrations(case, seed):
    """The sizes are the case's, the market inputs the seed's."""
    rng = np.random.default_rng(seed)
    return [wl.Calibration(c.outer, c.numX, c.numY, c.numT, *_market(rng))
            for c in wl.uneven_mix(case["count"], case["sizes"])]


def _tridag_inputs(case, seed):
    """Systems of an implicit diffusion step: diagonally dominant."""
    g = torch.Generator(DEVICE).manual_seed(seed)
    shape = (case["rows"], case["m"])
    lower, upper, y = (torch.rand(shape, generator=g, device=DEVICE) + 0.3 for _ in range(3))
    return -lower, 1.0 + lower + upper, -upper, y


def _tke_inputs(case, seed):
    """An ocean with sea floor at every depth and some land, flow in all
    directions and a state that overshoots below zero here and there."""
    g = torch.Generator(DEVICE).manual_seed(seed)
    X, Y, Z = case["x"], case["y"], case["z"]
    u = lambda lo, *shape: torch.rand(shape, generator=g, device=DEVICE) + lo  # noqa: E731
    v = {k: u(-0.6, X, Y, Z) for k in ("tketau", "tketaup1", "tketaum1", "dtketau", "dtketaup1", "dtketaum1")}
    v.update({k: u(-0.5, X, Y, Z) for k in ("utau", "vtau", "wtau")})
    v.update({k: (u(0.0, X, Y, Z) < 0.85).float() for k in ("maskU", "maskV", "maskW")})
    v.update({k: u(0.5, n) for k, n in (("dxt", X), ("dxu", X), ("dyt", Y), ("dyu", Y), ("dzt", Z), ("dzw", Z),
                                        ("cost", Y), ("cosu", Y))})
    v["kbot"] = torch.randint(-1, Z + 2, (X, Y), generator=g, device=DEVICE, dtype=torch.int32)
    v.update({k: u(0.5, X, Y, Z) for k in ("kappaM", "mxl", "forc")})
    v["forc_tke_surface"] = u(-0.7, X, Y)
    return v


def _bridge(times):
    """Brownian bridge over `times`: the last date first, then the midpoint of
    each interval, left half before right."""
    t = [0.0] + list(times)
    rows = [(len(times), 0, 0, math.sqrt(t[-1]), 0.0, 0.0)]

    def halve(lo, hi):
        mid = (lo + hi) // 2
        if mid > lo:
            span = t[hi] - t[lo]
            rows.append((mid, lo, hi, math.sqrt((t[mid] - t[lo]) * (t[hi] - t[mid]) / span), (t[hi] - t[mid]) / span,
                         (t[mid] - t[lo]) / span))
            halve(lo, mid)
            halve(mid, hi)

    halve(0, len(times))
    cols = np.array(rows, np.float64).T
    return np.ascontiguousarray(cols[:3], np.int32), np.ascontiguousarray(cols[3:], np.float32)


def _op_inputs(case, seed):
    """Index levels, volatilities, drifts and rates around the reference's
    datasets; Sobol direction numbers of 30 bits."""
    rng = np.random.default_rng(seed)
    contract, M = case["contract"], case["models"]
    D, U, n_disc = {1: (1, 1, 1), 2: (5, 3, 5), 3: (367, 3, 2)}[contract]
    near = lambda v, rel: np.asarray(v) * rng.uniform(1 - rel, 1 + rel, np.shape(v))  # noqa: E731
    years = np.arange(1, D + 1) / {1: 1.02, 2: 1.0, 3: 366.0}[contract]
    inds, data = _bridge(near(years[:1], 0.01) if D == 1 else years)
    cs = np.zeros((M, U, U))
    vols, drifts = np.zeros((M, D, U)), np.zeros((M, D, U))
    for m in range(M):
        corr = np.array([[1.0, 0.6, 0.8], [0.6, 1.0, 0.6], [0.8, 0.6, 1.0]])
        off = rng.uniform(-0.05, 0.05, (3, 3))
        corr += np.triu(off, 1) + np.triu(off, 1).T
        cs[m] = np.linalg.cholesky(corr)[:U, :U]
        vols[m] = near([0.19, 0.19, 0.15], 0.1)[:U]
        drifts[m] = rng.uniform(-0.03, 0.02, U) * (1 / 366.0 if contract == 3 else 1.0)
        if contract == 3:  # the first date is today
            vols[m, 0] = drifts[m, 0] = 0.0
    f = lambda v: np.ascontiguousarray(v, np.float32)  # noqa: E731
    sobol = torch.quasirandom.SobolEngine(D * U, scramble=False).sobolstate.numpy()
    return {"dir_vs": np.ascontiguousarray(sobol, np.int32), "md_cs": f(cs), "md_vols": f(vols),
            "md_drifts": f(drifts), "md_sts": f(near(np.tile([3758.05, 11840.0, 1200.0], (M, 1)), 0.02)[:, :U]),
            "md_detvals": f(rng.uniform(0.98, 1.0, (M, 1))),
            "md_discts": f(np.cumprod(rng.uniform(0.96, 0.99, (M, n_disc)), axis=1)),
            "bb_inds": inds, "bb_data": data}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "entry":
        call = _ctx().main_f64 if case["f64"] else _ctx().main
        return {"kind": kind, "call": call,
                "args": (case["outer"], case["numX"], case["numY"], case["numT"],
                         *_market(np.random.default_rng(seed)))}
    if kind == "mix":
        calibs = _calibrations(case, seed)
        return {"kind": kind, "calibs": calibs, "f64": case["f64"],
                "plan": _ctx().plan(calibs, pkg.F64 if case["f64"] else pkg.F32_STATE)}
    if kind == "serve":
        return {"kind": kind, "server": _server(case["f64"]), "f64": case["f64"],
                "calibs": _calibrations(case, seed)}
    if kind == "tridag":
        ins = _tridag_inputs(case, seed)
        return {"kind": kind, "ctx": _ctx(), "case": case, "ins": ins, "out": torch.empty_like(ins[0])}
    if kind == "tke":
        dims = (case["x"], case["y"], case["z"])
        ins = _tke_inputs(case, seed)
        outs = {k: torch.empty(dims[:2] if k == "tke_surf_corr_out" else dims, device=DEVICE)
                for k in tke.STEP_OUTPUTS}
        scratch = torch.empty(_tke_ctx().scratch_bytes(*dims), dtype=torch.uint8, device=DEVICE)
        ptrs = {k: ins[k].data_ptr() for k in tke.STEP_INPUTS}
        ptrs.update({k: v.data_ptr() for k, v in outs.items()}, scratch=scratch.data_ptr())
        return {"kind": kind, "ctx": _tke_ctx(), "dims": dims, "ptrs": ptrs, "outs": outs, "keep": (ins, scratch)}
    host = _op_inputs(case, seed)
    ctx = _op_ctx(case["sequential"])
    dims = op.dims_of((case["contract"], case["paths"], *(host[k] for k in op.ARRAY_NAMES)))
    ins = {k: torch.from_numpy(v).to(DEVICE) for k, v in host.items()}
    out = torch.empty(case["models"], device=DEVICE)
    scratch = torch.empty(ctx.scratch_bytes(case["contract"], case["paths"], dims), dtype=torch.uint8, device=DEVICE)
    return {"kind": "op", "ctx": ctx, "case": case, "dims": dims, "ptrs": {k: v.data_ptr() for k, v in ins.items()},
            "out": out, "scratch": scratch, "keep": ins}


def run(state):
    kind = state["kind"]
    if kind == "entry":
        return state["call"](*state["args"])
    if kind == "mix":
        plan = state["plan"]
        plan.set_params(state["calibs"])
        plan.run()
        prices = plan.prices()
        # the FP32-state variant's prices are single precision
        return prices if state["f64"] else prices.astype(np.float32)
    if kind == "serve":
        server = state["server"]
        tickets = [server.submit(c) for c in state["calibs"]]
        prices = np.concatenate([server.result(t) for t in tickets])
        return prices if state["f64"] else prices.astype(np.float32)
    if kind == "tridag":
        case, out = state["case"], state["out"]
        state["ctx"].tridag_device(case["form"], case["rows"], case["m"], *(t.data_ptr() for t in state["ins"]),
                                   out.data_ptr())
        return out
    if kind == "tke":
        state["ctx"].step(state["dims"], state["ptrs"])
        return state["outs"]
    case = state["case"]
    state["ctx"].price(case["contract"], case["paths"], state["dims"], state["ptrs"], state["out"].data_ptr(),
                       state["scratch"].data_ptr())
    return state["out"]


def work(case):
    kind = case["kind"]
    if kind in ("entry", "mix", "serve"):
        if kind == "entry":
            steps, options, count = (case["outer"] * case["numX"] * case["numY"] * (case["numT"] - 1), case["outer"],
                                     1)
        else:
            calibs = wl.uneven_mix(case["count"], case["sizes"])
            steps, options, count = wl.total_work(calibs), wl.total_options(calibs), case["count"]
        # a cell's step: variance 4, explicit terms and combine 25, the two
        # tridiagonal systems' coefficients 24, their solves 20, combines 4
        return {"bytes": 56 * count + 8 * options, "flops": 77 * steps}
    if kind == "tridag":
        n = case["rows"] * case["m"]
        return {"bytes": 20 * n, "flops": (9 if case["form"] == "seq" else 33) * n}
    if kind == "tke":
        cells = case["x"] * case["y"] * case["z"]
        return {"bytes": 60 * cells + 12 * case["x"] * case["y"], "flops": 165 * cells}
    D, U, _ = {1: (1, 1, 1), 2: (5, 3, 5), 3: (367, 3, 2)}[case["contract"]]
    # an inverse Gaussian about 32, a bridge step 5, a correlated price about
    # 30 with its exponential; once per model from the correlation on
    return {"bytes": 4 * D * (U * (30 + 2 * case["models"]) + 6) + 4 * case["models"] * 20,
            "flops": case["paths"] * D * U * (37 + 30 * case["models"])}


# --- the same in 64 bits ----------------------------------------------------

def _dense(lower, diag, upper):
    """[..., n, n] matrices of tridiagonal systems given by their diagonals."""
    m = torch.diag_embed(diag)
    m.diagonal(-1, -2, -1).copy_(lower[..., 1:])
    m.diagonal(1, -2, -1).copy_(upper[..., :-1])
    return m


def _second_derivative(x):
    """[n, 3] weights, zero at the ends."""
    w = torch.zeros(len(x), 3, dtype=torch.float64, device=DEVICE)
    lo, hi = x[1:-1] - x[:-2], x[2:] - x[1:-1]
    w[1:-1, 0], w[1:-1, 1], w[1:-1, 2] = 2 / lo / (lo + hi), -2 * (1 / lo + 1 / hi) / (lo + hi), 2 / hi / (lo + hi)
    return w


def _exact_entry(case, seed):
    outer, X, Y, T = case["outer"], case["numX"], case["numY"], case["numT"]
    s0, t, alpha, nu, beta = _market(np.random.default_rng(seed))
    if not case["f64"]:  # the f32 entry point's arguments
        s0, t, alpha, nu, beta = (float(np.float32(v)) for v in (s0, t, alpha, nu, beta))
    f = dict(dtype=torch.float64, device=DEVICE)
    dx, dy = 20 * alpha * s0 * math.sqrt(t) / X, 10 * nu * math.sqrt(t) / Y
    at_x, at_y = int(s0 / dx), Y // 2
    x = torch.arange(X, **f) * dx - at_x * dx + s0
    y = torch.arange(Y, **f) * dy - at_y * dy + math.log(alpha)
    Wx, Wy = _second_derivative(x), _second_derivative(y)
    line = t * np.arange(T) / max(T - 1.0, 1.0)
    strikes = 0.001 * torch.arange(outer, **f)
    res = (x[None, None, :] - strikes[:, None, None]).clamp(min=0).expand(outer, Y, X)
    shift = lambda v, by, axis: torch.roll(v, by, axis)  # noqa: E731  (the end weights are zero)
    for k in range(T - 2, -1, -1):
        dt = 1.0 / (line[k + 1] - line[k])
        var = torch.exp(2 * (beta * torch.log(x)[None, :] + y[:, None] - 0.5 * nu * nu * line[k]))  # [Y, X]
        u = 0.5 * var * (Wx[:, 0] * shift(res, 1, 2) + Wx[:, 1] * res + Wx[:, 2] * shift(res, -1, 2))
        gy = 0.5 * nu * nu * Wy
        v = gy[:, 0, None] * shift(res, 1, 1) + gy[:, 1, None] * res + gy[:, 2, None] * shift(res, -1, 1)
        rhs = dt * res + 0.5 * u + v
        h = -0.25 * var[:, :, None] * Wx[None]
        A = _dense(h[..., 0], dt + h[..., 1], h[..., 2])  # a system per y
        u = torch.linalg.solve(A, rhs.permute(1, 2, 0)).permute(2, 0, 1)
        h = -0.5 * gy
        A = _dense(h[:, 0], dt + h[:, 1], h[:, 2])
        rhs = dt * u - 0.5 * v
        res = torch.linalg.solve(A, rhs.permute(1, 0, 2).reshape(Y, -1)).reshape(Y, outer, X).permute(1, 0, 2)
    return res[:, at_y, at_x].cpu().numpy()


def _thomas(a, b, c, y):
    """Tridiagonal solves along the last axis."""
    n = b.shape[-1]
    cp, yp = [c[..., 0] / b[..., 0]], [y[..., 0] / b[..., 0]]
    for i in range(1, n):
        d = b[..., i] - a[..., i] * cp[-1]
        cp.append(c[..., i] / d)
        yp.append((y[..., i] - a[..., i] * yp[-1]) / d)
    out = [yp[-1]]
    for i in range(n - 2, -1, -1):
        out.append(yp[i] - cp[i] * out[-1])
    return torch.stack(out[::-1], -1)


def _flux(velfac, vel, dx, t, mask, axis):
    """Superbee advection flux towards the next cell along `axis`; what lies
    outside the grid is masked."""
    n = t.shape[axis]
    pad = lambda v: torch.cat([torch.zeros_like(v.narrow(axis, 0, 1)), v,  # noqa: E731
                               torch.zeros_like(v.narrow(axis, 0, 1)), torch.zeros_like(v.narrow(axis, 0, 1))], axis)
    t4, m4 = pad(t), pad(mask)
    tm, tc, tp, tpp = (t4.narrow(axis, k, n) for k in range(4))
    mm, mc, mp, mpp = (m4.narrow(axis, k, n) for k in range(4))
    sv = velfac * vel
    cfl = (sv / dx).abs()
    rjp, rj, rjm = (tpp - tp) * mp * mpp, (tp - tc) * mc * mp, (tc - tm) * mm * mc
    div = torch.where(rj.abs() < 1e-20, torch.full_like(rj, 1e-20), rj)
    cr = torch.where(vel > 0, rjm, rjp) / div
    cr = torch.maximum((2 * cr).clamp(max=1), cr.clamp(max=2)).clamp(min=0)
    return sv * (tp + tc) * 0.5 - sv.abs() * ((1 - cr) + cfl * cr) * rj * 0.5


def _exact_tke(case, seed):
    v = {k: (t.double() if t.is_floating_point() else t.long()) for k, t in _tke_inputs(case, seed).items()}
    X, Y, Z = case["x"], case["y"], case["z"]
    tau, dzt, dzw = v["tketau"], v["dzt"], v["dzw"]
    cost, cosu = v["cost"][None, :, None], v["cosu"][None, :, None]
    dxt, dxu = v["dxt"][:, None, None], v["dxu"][:, None, None]
    dyt, dyu = v["dyt"][None, :, None], v["dyu"][None, :, None]
    ix, iy, iz = torch.arange(X, device=DEVICE), torch.arange(Y, device=DEVICE), torch.arange(Z, device=DEVICE)
    inner = ((ix >= 2) & (ix < X - 2))[:, None] & ((iy >= 2) & (iy < Y - 2))[None, :]
    inner3 = inner[:, :, None]
    zero = torch.zeros_like(tau)
    # vertical diffusion and dissipation, implicit
    delta = zero.clone()
    delta[:, :, :-1] = 0.5 * (v["kappaM"][:, :, :-1] + v["kappaM"][:, :, 1:]) / dzt[1:]
    delta = torch.where(inner3, delta, zero)
    below = torch.cat([zero[:, :, :1], delta[:, :, :-1]], 2)
    floor = (v["kbot"] - 1)[:, :, None]
    water = (floor >= 0) & (iz >= floor) & inner3
    edge = (floor >= 0) & (iz == floor) & inner3
    h = torch.where(iz == Z - 1, 0.5 * dzw, dzw)
    a = torch.where(water & ~edge & (iz > 0), -below / h, zero)
    decay = 0.7 * tau.clamp(min=0).sqrt() / v["mxl"]
    b = torch.where(edge, 1 + delta / dzw + decay,
                    torch.where(iz == Z - 1, 1 + below / h + decay, 1 + (delta + below) / dzw + decay))
    b = torch.where(water, b, torch.where(inner3, torch.ones_like(b), zero))
    c = torch.where(water, -delta / dzw, zero)
    d = tau + v["forc"]
    d[:, :, -1] += v["forc_tke_surface"] / (0.5 * dzw[-1])
    d = torch.where(water, d, zero)
    b = torch.where(inner3, b, torch.ones_like(b))  # columns whose solution is not used
    new = torch.where(water, _thomas(a, b, c, d), v["tketaup1"])
    top = new[:, :, -1]
    surf = torch.where(inner & (top < 0), -top * 0.5 * dzw[-1], torch.zeros_like(top))
    new[:, :, -1] = torch.where(inner, top.clamp(min=0), top)
    # lateral diffusion of the top level
    fe, fn = zero[:, :, -1].clone(), zero[:, :, -1].clone()
    t = tau[:, :, -1]
    fe[:-1] = (2000 * (t[1:] - t[:-1]) / (cost * dxu)[:-1, :, 0]) * v["maskU"][:-1, :, -1]
    fn[:, :-1] = 2000 * (t[:, 1:] - t[:, :-1]) / dyu[:, :-1, 0] * v["maskV"][:, :-1, -1] * cosu[:, :-1, 0]
    lat = (fe - torch.roll(fe, 1, 0)) / (cost * dxt)[:, :, 0] + (fn - torch.roll(fn, 1, 1)) / (cost * dyt)[:, :, 0]
    new[:, :, -1] += torch.where(inner, v["maskW"][:, :, -1] * lat, torch.zeros_like(lat))
    # advection
    ok_x, ok_y = (iy >= 2) & (iy < Y - 2), (ix >= 2) & (ix < X - 2)
    east = ((ix >= 1) & (ix < X - 2))[:, None, None] & ok_x[None, :, None]
    north = ((iy >= 1) & (iy < Y - 2))[None, :, None] & ok_y[:, None, None]
    mw = v["maskW"]
    fe = torch.where(east, _flux(1.0, v["utau"], cost * dxt, tau, mw, 0), zero)
    fn = torch.where(north, _flux(cosu, v["vtau"], cost * dyt, tau, mw, 1), zero)
    ft = torch.where(inner3 & (iz < Z - 1), _flux(1.0, v["wtau"], dzw, tau, mw, 2), zero)
    dtk = mw * (-(fe - torch.roll(fe, 1, 0)) / (cost * dxt) - (fn - torch.roll(fn, 1, 1)) / (cost * dyt))
    dtk = torch.where(inner3, dtk, v["dtketau"])
    dtk = dtk - (ft - torch.cat([zero[:, :, :1], ft[:, :, :-1]], 2)) / h
    new = new + 1.6 * dtk - 0.6 * v["dtketaum1"]
    return {"tketaup1_out": new, "dtketau_out": dtk, "tke_surf_corr_out": surf}


def _exact_op(case, seed):
    v = {k: torch.from_numpy(a).to(DEVICE) for k, a in _op_inputs(case, seed).items()}
    contract, N, M = case["contract"], case["paths"], case["models"]
    D, U = v["md_vols"].shape[1:]
    bi, li, ri = (v["bb_inds"][k].tolist() for k in range(3))
    sd, lw, rw = (v["bb_data"][k].double() for k in range(3))
    total = torch.zeros(M, dtype=torch.float64, device=DEVICE)
    part = max(1, (1 << 23) // (D * U))
    for at in range(0, N, part):
        n = torch.arange(at + 1, min(N, at + part) + 1, device=DEVICE)
        gray = n ^ (n >> 1)
        x = torch.zeros(len(n), D * U, dtype=torch.long, device=DEVICE)
        for bit in range(30):
            x ^= ((gray >> bit) & 1)[:, None] * v["dir_vs"][:, bit].long()[None]
        z = torch.special.ndtri(x.double() / 2.0 ** 30).reshape(-1, D, U)
        w = torch.zeros(len(n), D + 1, U, dtype=torch.float64, device=DEVICE)
        w[:, bi[0]] = sd[0] * z[:, 0]
        for i in range(1, D):
            w[:, bi[i]] = rw[i] * w[:, ri[i]] + sd[i] * z[:, i] + lw[i] * w[:, li[i]]
        dw = w[:, 1:] - w[:, :-1]
        for m in range(M):
            noise = dw @ torch.tril(v["md_cs"][m].double()).T
            growth = torch.exp(v["md_drifts"][m].double() + noise * v["md_vols"][m].double())
            price = v["md_sts"][m].double() * torch.cumprod(growth, 1)
            disc = v["md_discts"][m].double()
            if contract == 1:
                pay = ((price[:, 0, 0] - 4000.0) * v["md_detvals"][m, 0].double()).clamp(min=0) * disc[0]
            else:
                levels = torch.tensor([3758.05, 11840.0, 1200.0], dtype=torch.float64, device=DEVICE)
                worst = (price / levels).amin(2)
                if contract == 2:
                    last = worst[:, 4]
                    pay = torch.where(last >= 1, 1750.0, torch.where(last > 0.75, 1000.0, last * 1000.0)) * disc[4]
                    for d in (3, 2, 1, 0):
                        pay = torch.where(worst[:, d] >= 1, (1150.0 + 150.0 * d) * disc[d], pay)
                else:
                    low = torch.tensor([2630.6349999999998, 8288.0, 840.0], dtype=torch.float64, device=DEVICE)
                    hit = (price <= low).any(2).any(1) & (price[:, -1] < levels).any(1)
                    pay = 100.0 * disc[0] + torch.where(hit, 1000.0 * worst[:, -1], 1000.0) * disc[1]
            total[m] += pay.sum()
    return total / N


def exact(case, seed):
    kind = case["kind"]
    if kind == "entry":
        # a dense solve per row and step: under a second a step at the largest grid
        return _exact_entry(case, seed)
    if kind == "tridag":
        return _thomas(*(t.double() for t in _tridag_inputs(case, seed)))
    if kind == "tke":
        return _exact_tke(case, seed)
    if kind == "op":
        return _exact_op(case, seed)
    return None  # every calibration of a mix or a burst takes minutes this way
