"""Performance cases of the dispersion engine: what its users have it do.

    listed()              the named cases
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   inputs and handles a program holds before the call
    run(state)            one pass through the public entry points
    work(case)            bytes and flops that one pass cannot do without
    exact(case, seed)     the outputs in 64 bits from plain torch, where they have such values

A case is a dict: ``call`` names the entry point, ``models`` x ``periods`` the
traces, ``layers_min``..``layers_max`` the finite layers of a model, ``lvz`` and
``water`` the fractions of models with a low-velocity layer and with a water top.
"""
import math

import numpy as np
import torch

from modisp_b200 import api, plugin
from modisp_b200.autograd import DifferentiableSolver, misfit
from modisp_b200.ragged import dispersion_ragged


def _case(name, call, models, periods, nmodes, layers, wave, precision, *, group=True, lvz=0., water=0., tol=1e-10,
          t_min=.5, t_max=50., nc=0):
    case = dict(call=call, models=models, periods=periods, nmodes=nmodes, layers_min=layers[0], layers_max=layers[1],
                wave=wave, precision=precision, group=group, lvz=lvz, water=water, tol=tol, t_min=t_min, t_max=t_max,
                nc=nc)
    return dict(case, name=name) if name else case


def listed():
    return [
        # one site model, the quickstart's size: an interactive call
        _case("one_site", "solver", 1, 30, 2, (1, 1), "rayleigh", "float64", t_min=.1, t_max=10.),
        # one crustal model, phase velocities only: the inner call of an iterative inversion
        _case("one_crust_love", "solver", 1, 60, 5, (20, 20), "love", "mixed", group=False),
        # a sampler's population, some models offshore, at the solver's default tolerance
        _case("population", "solver", 53, 41, 3, (5, 14), "rayleigh", "float64", group=False, water=.3, tol=1e-5,
              t_min=1., t_max=40.),
        # batches of random crustal models in plain FP64, both waves
        _case("crust_rayleigh", "solver", 2500, 60, 5, (8, 20), "rayleigh", "float64"),
        _case("crust_love", "solver", 2477, 60, 5, (8, 20), "love", "float64"),
        # mixed precision with low-velocity layers, tensors in and out on the device
        _case("mixed_rayleigh", "device", 20000, 60, 5, (8, 20), "rayleigh", "mixed", lvz=.3),
        _case("mixed_love", "device", 19999, 60, 5, (8, 20), "love", "mixed", lvz=.3),
        # the largest: modisp's own batch path through the backend plugin, host arrays
        _case("plugin_large", "plugin", 100000, 60, 5, (8, 20), "rayleigh", "mixed", lvz=.3),
        # gradient of a misfit: forward and backward of 12-layer models
        _case("misfit_gradient", "gradient", 4096, 40, 3, (12, 12), "rayleigh", "mixed", t_min=1., t_max=40.),
        # full Jacobians of phase and group velocities at known roots, as for a linearised inversion
        _case("jacobians", "jacobian", 1024, 40, 3, (12, 12), "rayleigh", "mixed", t_min=1., t_max=40.),
        # thin-layered gradient models, each with its own periods and mode count
        _case("ragged_deep", "ragged", 1000, 120, 10, (30, 100), "rayleigh", "mixed", t_min=.2, t_max=100.),
        # the legacy uniform grid
        _case("uniform_grid", "uniform", 2000, 60, 5, (8, 20), "rayleigh", "float64", group=False, tol=1e-6, nc=512),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["solver", "solver", "solver", "device", "device", "plugin", "gradient", "jacobian", "ragged",
                       "uniform"])
    most = dict(solver=3000, device=20000, plugin=60000, gradient=4096, jacobian=1024, ragged=1000, uniform=2000)[call]
    models = _log_int(rng, 1 if call == "solver" else 16, most)
    wave = "rayleigh" if call == "uniform" else rng.choice(["rayleigh", "rayleigh", "love"])
    precision = "float64" if call == "uniform" else rng.choice(["float64", "mixed"])
    if call == "ragged":
        low = rng.randint(10, 60)
        return _case(None, call, models, rng.randint(50, 120), rng.randint(1, 10), (low, rng.randint(low, 100)), wave,
                     "mixed", t_min=.2, t_max=100.)
    low = rng.randint(1, 16)
    high = rng.randint(low, 24)
    lvz = rng.choice([0., .3]) if low >= 3 else 0.
    water = rng.choice([0., 0., .3]) if wave == "rayleigh" and call in ("solver", "device", "plugin") and low >= 2 else 0.
    t_min = rng.uniform(.4, 2.)
    return _case(None, call, models, rng.randint(8, 60), rng.randint(1, 3 if call == "jacobian" else 6), (low, high), wave,
                 precision, group=call != "uniform" and (call != "solver" or rng.random() < .7), lvz=lvz, water=water,
                 tol=1e-6 if call == "uniform" else rng.choice([1e-5, 1e-10]) if call == "solver" else 1e-10,
                 t_min=t_min, t_max=t_min * rng.uniform(8., 60.), nc=rng.randint(256, 640) if call == "uniform" else 0)


# ---- inputs ----------------------------------------------------------------
def _models(case, rng):
    """Padded [B, L] (thickness, vp, vs, rho): random crustal models, or (ragged)
    smooth gradients over 80 km cut into thin layers."""
    B, L = case["models"], case["layers_max"] + 1
    n = rng.integers(case["layers_min"], case["layers_max"] + 1, B)[:, None]
    j = np.arange(L)[None, :]
    if case["call"] == "ragged":
        depth = np.minimum((j + .5) * 80. / n, 80.)
        vs = (.2 + 4.3 * depth / 80.) * rng.uniform(.95, 1.05, (B, L))
        h = np.broadcast_to(80. / n, (B, L)).copy()
    else:
        top, bottom = rng.uniform(.3, 1., (B, 1)), rng.uniform(3.5, 4.7, (B, 1))
        vs = (top + (bottom - top) * np.minimum(j / n, 1.)) * rng.uniform(.9, 1.1, (B, L))
        h = rng.uniform(.2, 3., (B, L))
    fastest = np.where(j < n, vs, 0.).max(axis=1, keepdims=True)
    vs = np.where(j == n, np.maximum(vs, 1.02 * fastest), vs)
    slow = np.flatnonzero((rng.uniform(size=B) < case["lvz"]) & (n[:, 0] >= 3))
    at = 1 + (rng.uniform(size=B) * (n[:, 0] - 1)).astype(np.int64)
    vs[slow, at[slow]] = vs[slow, at[slow] - 1] * (1. - rng.uniform(.2, .4, B)[slow])
    vp = vs * rng.uniform(1.7, 2., (B, L))
    rho = 1.74 * vp ** .25
    wet = rng.uniform(size=B) < case["water"]
    vp[wet, 0], vs[wet, 0], rho[wet, 0] = 1.5, 0., 1.03
    half = np.broadcast_to(n, (B, L))  # rows past the last layer repeat the half-space
    vp, vs, rho = (np.where(j > n, np.take_along_axis(x, half, 1), x) for x in (vp, vs, rho))
    return tuple(np.ascontiguousarray(x) for x in (np.where(j < n, h, 0.), vp, vs, rho))


def _periods(case):
    return np.geomspace(case["t_min"], case["t_max"], case["periods"])


def _ragged_periods(case, rng):
    """Every model's periods and mode count; how many of each is the case's, whatever the seed."""
    shape, B = np.random.default_rng(case["models"]), case["models"]
    sizes, modes = shape.integers(50, case["periods"] + 1, B), shape.integers(1, case["nmodes"] + 1, B)
    ends = np.sort(np.exp(rng.uniform(math.log(case["t_min"]), math.log(case["t_max"]), (B, 2))), axis=1)
    return [np.geomspace(a, max(b, 1.5 * a), int(n)) for (a, b), n in zip(ends, sizes)], modes


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    data = dict(case=case, models=_models(case, rng), periods=_periods(case))
    if case["call"] == "ragged":
        data["periods"], data["modes"] = _ragged_periods(case, rng)
    if case["call"] == "gradient":  # observed curves
        T = np.broadcast_to(np.log(data["periods"]), (case["models"], case["nmodes"], case["periods"]))
        data["observed"] = tuple((a + .4 * T) * rng.uniform(.95, 1.05, T.shape) for a in (1.2, .9))
    return data


def prepare(case, seed):
    s = _inputs(case, seed)
    call, L = case["call"], case["layers_max"] + 1
    if call == "solver":
        s["solver"] = api.Solver(precision=case["precision"], group_velocity=case["group"], c_tol_rel=case["tol"])
    elif call == "uniform":
        s["solver"] = api.Solver(search_strategy="uniform", nc=case["nc"], c_tol_rel=case["tol"])
    elif call == "plugin":
        s["solver"] = plugin.QeSolver(case["models"], L, case["periods"], case["nmodes"], shape=True,
                                      single_precision=case["precision"] == "mixed", group_velocity=case["group"])
        s["bounds"] = np.tile([0., np.inf], (case["models"], 1))
    elif call != "ragged":
        s["tensors"] = [torch.from_numpy(x).cuda() for x in s["models"]]
        s["solver"] = DifferentiableSolver(case["models"], L, s["periods"], case["nmodes"], wave=case["wave"],
                                           precision=case["precision"], c_tol_rel=case["tol"])
        if call == "gradient":
            for x in s["tensors"]:
                x.requires_grad_(True)
            s["observed"] = [torch.from_numpy(x).cuda() for x in s["observed"]]
        if call == "jacobian":  # the roots of the current models, from the forward solve
            s["roots"] = s["solver"].solve(*s["tensors"])
    return s


def run(s):
    case = s["case"]
    call = case["call"]
    if call in ("solver", "uniform"):
        r = s["solver"](*s["models"], s["periods"], nmodes=case["nmodes"], wave=case["wave"])
        return dict(phase=r.phase_velocity, group=r.group_velocity, group_flags=r.group_velocity_flags,
                    flags=r.trace_flags, levels=r.search_level, counts=r.root_count, bounds=r.search_bounds,
                    status=r.status, close=r.close_root_risk)
    if call == "plugin":
        velocity, flags, _, levels, counts, extras = s["solver"].run(
            *s["models"], s["periods"], s["bounds"], c_tol_rel=case["tol"], wave=int(case["wave"] == "love"))
        return dict(phase=velocity, group=extras["group_velocity"], group_flags=extras["group_velocity_flags"],
                    flags=flags, levels=levels, counts=counts)
    if call == "device":
        r = s["solver"].solve(*s["tensors"])
        return dict(phase=r["velocity"], group=r["group_velocity"], group_flags=r["group_velocity_flags"],
                    flags=r["flags"], levels=r["levels"], counts=r["counts"])
    if call == "gradient":
        phase, group = s["solver"](*s["tensors"])
        loss = misfit(phase, group, *s["observed"])
        return dict(phase=phase, group=group, loss=loss, gradients=torch.autograd.grad(loss, s["tensors"]))
    if call == "jacobian":
        phase, group = s["solver"].jacobian(*s["tensors"], s["roots"]["velocity"], s["roots"]["group_velocity"])
        return dict(phase=phase, group=group)
    r = dispersion_ragged(*s["models"], s["periods"], nmodes=s["modes"], wave=case["wave"],
                          precision=case["precision"], c_tol_rel=case["tol"])
    return dict(phase=r.phase_velocity, group=r.group_velocity, group_flags=r.group_velocity_flags,
                flags=r.trace_flags, levels=r.search_level, counts=r.root_count)


def work(case):
    """Bytes: models in, results out.  Flops: for every root the evaluations that
    no search can do without -- a sample on either side and one on it -- with the
    derivatives where they are asked for; the uniform grid's every value."""
    layers = .5 * (case["layers_min"] + case["layers_max"])
    traces = case["models"] * case["periods"]
    if case["call"] == "ragged":
        traces = case["models"] * .5 * (50 + case["periods"])
    modes = case["nmodes"] * (.5 if case["call"] == "ragged" else 1.)
    roots = traces * modes
    step = 170. if case["wave"] == "rayleigh" else 24.  # flops of one layer of the recurrence
    read = 32. * case["models"] * (case["layers_max"] + 1)
    out = 12. * traces + roots * (20. if case["group"] else 8.)
    evaluations = 3. + (3. if case["group"] else 0.)
    if case["call"] == "jacobian":
        out, evaluations = roots * 64. * (case["layers_max"] + 1), 12.
    if case["call"] == "gradient":
        out, evaluations = out + read + 16. * roots, evaluations + 12.
    flops = roots * evaluations * layers * step
    if case["call"] == "uniform":
        flops += traces * case["nc"] * layers * step
    return dict(bytes=read + out, flops=flops)


# ---- the outputs in 64 bits, in plain torch ---------------------------------
def _wave(k, kv, h):
    """cosh(r h), sinh(r h) / r, r sinh(r h) times exp(-s), and s, for r^2 = k^2 - kv^2 (s = 0 where r is imaginary)."""
    d = (k - kv) * (k + kv)
    r = d.abs().clamp_min(1e-280).sqrt()
    x = r * h
    flat = x.detach()
    up, down = torch.exp(x - flat), torch.exp(-x - flat)
    trig = d < 0
    c = torch.where(trig, torch.cos(x), .5 * (up + down))
    s = torch.where(trig, torch.sin(x), .5 * (up - down)) / r
    return c, s, d * s, torch.where(trig, torch.zeros_like(flat), flat)


def _normal(e):
    big = torch.stack([x.detach().abs() for x in e]).amax(0).clamp_min(1e-200)
    return [x / big for x in e]


def _secular(love, m, k, w):
    """Secular values and their share of the vector for samples (k, w) of models m = (h, vp, vs, rho), each [S, L]."""
    h, vp, vs, rho = (x.unbind(1) for x in m)
    last, k2 = len(h) - 1, k * k
    kb = w / vs[last]
    rb = ((k - kb) * (k + kb)).clamp_min(0.).sqrt()
    if love:
        e = [rb * rho[last], 1. / vs[last] ** 2]
    else:
        ka = w / vp[last]
        ra = ((k - ka) * (k + ka)).clamp_min(0.).sqrt()
        g2 = 2. * vs[last] ** 2 / w ** 2
        gm, t = g2 * k2 - 1., rho[last]
        e = [(gm * gm - g2 * g2 * k2 * ra * rb) * t * t, -ra * t, (gm - g2 * ra * rb) * t, rb * t, k2 - ra * rb]
    e = _normal(e)
    for j in range(last - 1, -1, -1):
        solid = (vs[j] > 0) & (h[j] > 0)
        v = torch.where(solid, vs[j], torch.ones_like(vs[j]))
        cq, y, z, sq = _wave(k, w / v, h[j])
        if love:
            mu = rho[j] * v * v
            new = [e[0] * cq + e[1] * z * mu, e[0] * y / mu + e[1] * cq]
        else:
            cp, x, u, sp = _wave(k, w / vp[j], h[j])
            t, one = rho[j], torch.exp(-sp - sq)
            g = 2. * v * v / w ** 2
            gam = g * k2
            gm, gg = gam - 1., gam * g
            cc, cy, cz, wx, ux = cp * cq, cp * y, cp * z, cq * x, cq * u
            uy, uz, xy, xz = u * y, u * z, x * y, x * z
            dc = one - cc
            A = cc - 2. * gam * gm * dc - gg * uz - k2 * gm * gm * xy
            D, C = (k2 * cy - ux) / t, (cz - k2 * wx) / t
            I = -((gam + gm) * dc + g * uz + k2 * gm * xy) / t
            P = -(2. * k2 * dc + uz + k2 * k2 * xy) / t ** 2
            E, F = (gg * cz - gm * gm * wx) * t, (gm * gm * cy - gg * ux) * t
            G, H = g * cz - gm * wx, gm * cy - g * ux
            O = -(2. * gg * gm * gm * dc + gg * gg * uz + gm ** 4 * xy) * t ** 2
            J = -(g * gm * (gam + gm) * dc + gam * g * g * uz + gm ** 3 * xy) * t
            K = one + 2. * (cc - A)
            q = -2. * k2 * e[2]
            new = [A * e[0] + E * e[1] + J * q + F * e[3] + O * e[4], D * e[0] + cc * e[1] + H * q - uy * e[3] + F * e[4],
                   I * e[0] + G * e[1] + K * e[2] + H * e[3] + J * e[4],
                   C * e[0] - xz * e[1] + G * q + cc * e[3] + E * e[4], P * e[0] + C * e[1] + I * q + D * e[3] + A * e[4]]
        e = _normal([torch.where(solid, a, b) for a, b in zip(new, e)])
    value = e[0]
    share = value / torch.stack([x.detach() for x in e]).norm(dim=0)
    wet = vs[0] == 0
    if not love and bool(wet.any()):
        c, s, _, _ = _wave(k, w / vp[0], h[0])
        a, b = c * e[0], s * rho[0] * e[1]
        value = torch.where(wet, a - b, value)
        share = torch.where(wet, (a - b).detach() / (a.detach() ** 2 + b.detach() ** 2).sqrt(), share)
    return value, share


def _sample(love, m, model, c, w, chunk=1 << 20):
    """Secular values and shares at velocities c [S], models by index."""
    got = [_secular(love, [x[model[i:i + chunk]] for x in m], w[i:i + chunk] / c[i:i + chunk], w[i:i + chunk])
           for i in range(0, c.numel(), chunk)]
    return (torch.cat([g[q] for g in got]) for q in (0, 1))


def _lowest_speed(love, m):
    """An eighth of the slowest Rayleigh (Love: shear) speed of a model's layers."""
    h, vp, vs, _ = m
    solid = (vs > 0) & ((h > 0) | (torch.arange(h.shape[1], device=h.device) == h.shape[1] - 1))
    speed = vs
    if not love:
        ratio = (vs / vp) ** 2
        a, b = torch.zeros_like(vs), torch.ones_like(vs)
        for _ in range(60):
            x = .5 * (a + b)
            f = ((x - 8.) * x + 24. - 16. * ratio) * x - 16. * (1. - ratio)
            a, b = torch.where(f < 0, x, a), torch.where(f < 0, b, x)
        speed = vs * (.5 * (a + b)).sqrt()
    return .125 * torch.where(solid, speed, torch.full_like(speed, math.inf)).amin(1)


def _search(love, m, model, period, most, density=32, block=64, knots=1024):
    """The first `most` roots of every trace (model index, period), NaN past the last: [traces, most].

    Samples even in the phase count N(c) / T plus a logarithmic term, sign changes as brackets, and a closer look
    wherever the share of the vector has a minimum of one sign."""
    dev = model.device
    h, vp, vs, _ = m
    lo, hi = _lowest_speed(love, m), vs[:, -1] * (1. - 2. ** -52)
    if not love:
        lo = torch.where(vs[:, 0] == 0, .5 * lo, lo)
    frac = torch.linspace(0., 1., knots, dtype=torch.float64, device=dev)
    table = lo[:, None] * (hi / lo)[:, None] ** frac
    table[:, -1] = hi
    count = torch.zeros_like(table)
    for j in range(h.shape[1] - 1):
        for v in (vs, vp)[:1 if love else 2]:
            ok = v[:, j:j + 1] > 0
            slow = torch.where(ok, 1. / v[:, j:j + 1].clamp_min(1e-9) ** 2, torch.zeros_like(v[:, j:j + 1]))
            count += 2. * h[:, j:j + 1] * (slow - 1. / table ** 2).clamp_min(0.).sqrt()
    roots = torch.full((model.numel(), most), math.nan, dtype=torch.float64, device=dev)
    for first in range(0, model.numel(), 65536):
        md, T = model[first:first + 65536], period[first:first + 65536]
        n, w = md.numel(), 2. * math.pi / T
        u = count[md] / T[:, None] + 8. * frac
        rows = torch.arange(n, device=dev)
        found, lows, highs, dips = [], [], [], []
        left = torch.full((n, 2), math.nan, dtype=torch.float64, device=dev)  # velocity and share of the last two samples
        left_g = left.clone()
        held = torch.zeros(n, dtype=torch.int64, device=dev)
        at = torch.zeros(n, dtype=torch.int64, device=dev)
        while rows.numel():
            block = max(64, min(2048, (1 << 20) // rows.numel()))
            target = u[rows, :1] + (at[rows, None] + torch.arange(block, device=dev)) / density
            i = torch.searchsorted(u[rows], target).clamp(1, knots - 1)
            u0, u1 = u[rows].gather(1, i - 1), u[rows].gather(1, i)
            part = ((target - u0) / (u1 - u0)).clamp(0., 1.)
            t = table[md[rows]]
            c = t.gather(1, i - 1) * (1. - part) + t.gather(1, i) * part
            c = torch.minimum(c, hi[md[rows], None])
            _, g = _sample(love, m, md[rows].repeat_interleave(block), c.reshape(-1), w[rows].repeat_interleave(block))
            c, g = torch.cat([left[rows], c], 1), torch.cat([left_g[rows], g.reshape(c.shape)], 1)
            change = (g[:, 1:-1] * g[:, 2:] <= 0) & (c[:, 1:-1] < c[:, 2:])
            r, q = change.nonzero(as_tuple=True)
            found.append(rows[r]), lows.append(c[r, q + 1]), highs.append(c[r, q + 2])
            held += torch.bincount(rows[r], minlength=n)
            dip = ((g[:, :-2] * g[:, 1:-1] > 0) & (g[:, 1:-1] * g[:, 2:] > 0) & (g[:, 1:-1].abs() < g[:, :-2].abs())
                   & (g[:, 1:-1].abs() < g[:, 2:].abs()))
            r, q = dip.nonzero(as_tuple=True)
            dips.append((rows[r], c[r, q], c[r, q + 2]))
            left[rows], left_g[rows] = c[:, -2:], g[:, -2:]
            at[rows] += block
            rows = rows[(held[rows] < most) & (c[:, -1] < hi[md[rows]])]
        tr, a, b = (torch.cat(x) for x in zip(*dips))
        for _ in range(4):  # a pair hidden in a dip
            if not tr.numel():
                break
            x = a[:, None] + (b - a)[:, None] * torch.linspace(0., 1., 33, dtype=torch.float64, device=dev)
            _, s = _sample(love, m, md[tr].repeat_interleave(33), x.reshape(-1), w[tr].repeat_interleave(33))
            s = s.reshape(x.shape)
            r, q = (s[:, :-1] * s[:, 1:] <= 0).nonzero(as_tuple=True)
            found.append(tr[r]), lows.append(x[r, q]), highs.append(x[r, q + 1])
            low = s.abs()[:, 1:-1].argmin(1, keepdim=True) + 1
            none = ~(s[:, :-1] * s[:, 1:] <= 0).any(1)
            tr, a, b = tr[none], x.gather(1, low - 1)[none, 0], x.gather(1, low + 1)[none, 0]
        tr, a, b = torch.cat(found), torch.cat(lows), torch.cat(highs)
        fa, _ = _sample(love, m, md[tr], a, w[tr])
        for _ in range(60):
            x = .5 * (a + b)
            f, _ = _sample(love, m, md[tr], x, w[tr])
            same = (f < 0) == (fa < 0)
            a, b = torch.where(same, x, a), torch.where(same, b, x)
        x, order = torch.sort(.5 * (a + b))
        tr = tr[order]
        tr, order = torch.sort(tr, stable=True)
        x = x[order]
        rank = torch.arange(tr.numel(), device=dev) - torch.searchsorted(tr, tr)
        keep = rank < most
        roots[first + tr[keep], rank[keep]] = x[keep]
    return roots


def _derivatives(love, m, model, c, period, chunk=65536, full=False):
    """Group velocity at every root, and (full) dc/dm and dU/dm, each [R, 4, L]."""
    got = []
    for i in range(0, c.numel(), chunk):
        rows = [x[model[i:i + chunk]].clone().requires_grad_(full) for x in m]
        w = (2. * math.pi / period[i:i + chunk]).requires_grad_(True)
        cc = c[i:i + chunk]
        k = (w.detach() / cc).requires_grad_(True)
        F, _ = _secular(love, rows, k, w)
        fk, fw = torch.autograd.grad(F.sum(), (k, w), create_graph=full)
        U = -fk / fw
        if not full:
            got.append((U.detach(),))
            continue
        fm = torch.stack(torch.autograd.grad(F.sum(), rows, retain_graph=True, materialize_grads=True), 1)
        um = torch.autograd.grad(U.sum(), rows + [k], materialize_grads=True)
        um, uk = torch.stack(um[:4], 1), um[4]
        km = -fm / fk.detach()[:, None, None]
        got.append((U.detach(), -(cc / k.detach())[:, None, None] * km, um + uk[:, None, None] * km))
    return tuple(torch.cat(x) for x in zip(*got))


def exact(case, seed):
    traces = case["models"] * case["periods"]
    if case["call"] == "uniform" or traces * case["layers_max"] > 4_000_000:
        return None  # roots as far as the uniform grid's bisection takes them; too long
    s = _inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    love = case["wave"] == "love"
    m = [torch.from_numpy(x).to(dev) for x in s["models"]]
    B, K, T, L = case["models"], case["nmodes"], case["periods"], case["layers_max"] + 1
    if case["call"] == "ragged":
        sizes = torch.tensor([p.size for p in s["periods"]], device=dev)
        model = torch.arange(B, device=dev).repeat_interleave(sizes)
        period = torch.from_numpy(np.concatenate(s["periods"])).to(dev)
    else:
        model = torch.arange(B, device=dev).repeat_interleave(T)
        period = torch.from_numpy(np.tile(s["periods"], B)).to(dev)
    guide = ((m[0] > 0) & (m[2] < m[2][:, -1:]) & (m[2] > 0)).any(1)
    c = _search(love, m, model, period, K + 1)
    if love:
        c[~guide[model]] = math.nan
    near = torch.zeros_like(c, dtype=torch.bool)  # roots too close for a group velocity
    near[:, :-1] = c[:, 1:] - c[:, :-1] <= .005 * c[:, 1:]
    near[:, 1:] |= near[:, :-1].clone()
    c, near = c[:, :K], near[:, :K]
    have = torch.isfinite(c) & ~near
    tr, rank = have.nonzero(as_tuple=True)
    full = case["call"] in ("gradient", "jacobian")
    if full:
        tr, rank = torch.isfinite(c).nonzero(as_tuple=True)
    d = [x.cpu() for x in _derivatives(love, m, model[tr], c[tr, rank], period[tr], full=full)]
    c, tr, rank, have = c.cpu(), tr.cpu(), rank.cpu(), have.cpu()
    U = torch.full_like(c, math.nan)
    U[tr, rank] = d[0]
    U[~have] = math.nan
    if case["call"] == "ragged":
        modes, sizes = s["modes"], [p.size for p in s["periods"]]
        flat = [torch.cat([x[:, :int(q)].T.reshape(-1) for x, q in zip(v.split(sizes), modes)]) for v in (c, U)]
        return dict(phase=flat[0], group=flat[1], group_flags=None, flags=None, levels=None, counts=None)
    phase, group = (x.reshape(B, T, K).transpose(1, 2).contiguous() for x in (c, U))
    if full:
        both = []
        for q in (1, 2):
            x = torch.zeros((B, K, T, 4, L), dtype=torch.float64)
            x[tr // T, rank, tr % T] = d[q]
            both.append(x)
        empty, missing = ~torch.isfinite(phase), ~torch.isfinite(group)
        if case["call"] == "jacobian":
            both[0][empty], both[1][missing] = math.nan, math.nan
            return dict(phase=both[0], group=both[1])
        dc, du = phase - torch.from_numpy(s["observed"][0]), group - torch.from_numpy(s["observed"][1])
        dc, du = (torch.where(torch.isfinite(x), x, torch.zeros_like(x)) for x in (dc, du))
        grad = 2. * (torch.einsum("bkt,bktpl->pbl", dc, both[0]) + torch.einsum("bkt,bktpl->pbl", du, both[1]))
        return dict(phase=phase, group=group, loss=(dc ** 2).sum() + (du ** 2).sum(), gradients=tuple(grad))
    out = dict(phase=phase, group=group if case["group"] else None, group_flags=None, flags=None, levels=None, counts=None)
    if case["call"] == "plugin" and case["precision"] == "mixed":
        out["phase"] = phase.float().double()
    if case["call"] == "solver":
        bounds = None
        if not case["water"]:
            bounds = torch.stack([_lowest_speed(love, m), torch.nextafter(m[2][:, -1], torch.zeros_like(m[2][:, -1]))], 1)
        out |= dict(bounds=bounds, status=None, close=None)
    return out
