"""The measured work of the engine: calls a vortex-method program makes, through the public entry points.

A time step of such a program is a velocity sum of its particles on themselves (by direct sum or treecode), with a
body the particle sums on its panels, the influence matrix, its solve and the panel sums on the particles, and the
clearing of the layer next to the body; an inverse problem adds the reverse passes.  Each family below is one of these
calls; the listed cases are the sizes of this repository's configurations and tests, the drawn ones span their ranges.
All arrays live on the GPU and every sum runs on torch's current stream, as a program that holds its state there has it.
"""
import math

import torch

import omega2d_gb300 as og

DEV = "cuda"
CORES = {"rm": og.CORE_RM, "gauss": og.CORE_GAUSSIAN, "v2": og.CORE_V2, "wl": og.CORE_WL, "v3": og.CORE_V3}
ACCUM = {"plain": og.PLAIN_F32, "comp": og.COMPENSATED}
RESULT = {"vel": og.VELONLY, "grad": og.VELANDGRAD, "vort": og.VELANDVORT, "shear": og.VELANDSHEAR}
INV2PI = 0.5 / math.pi
EXACT_PAIRS = 4.0e10   # FP64 pairs that plain torch sums in a few seconds
CLEAR_IPS = 0.01       # particle spacing that sets the width of the cleared layer

_ctx = None


def context():
    """The program's one engine context, on torch's current stream."""
    global _ctx
    if _ctx is None:
        _ctx = og.Context(0)
    _ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    return _ctx


def listed():
    return [
        # the smallest steps: the start of a run or a small demonstration flow, one velocity evaluation
        {"name": "self_1000_v2", "family": "self", "layout": "cloud", "n": 1000, "core": "v2", "radius": 0.03,
         "spread": 0.0, "accum": "comp", "result": "vel"},
        # a run of 20,000 particles over ten Euler steps in a freestream
        {"name": "euler_20k_rm", "family": "advect", "layout": "cloud", "n": 20000, "core": "rm", "radius": 0.01,
         "accum": "comp", "order": 1, "steps": 10, "dt": 0.01},
        # adaptive particle sizes: every radius its own, an odd count, the reference's default core
        {"name": "self_33001_v2_adaptive", "family": "self", "layout": "cloud", "n": 33001, "core": "v2",
         "radius": 0.008, "spread": 0.5, "accum": "comp", "result": "vel"},
        # the reference's default core summed in single precision, as its vectorised build does
        {"name": "self_131k_v2_plain", "family": "self", "layout": "patch", "n": 131072, "core": "v2",
         "radius": 0.005, "spread": 0.0, "accum": "plain", "result": "vel"},
        # velocity and its gradient, for strain and vortex stretching diagnostics
        {"name": "self_131k_gauss_grad", "family": "self", "layout": "patch", "n": 131072, "core": "gauss",
         "radius": 0.005, "spread": 0.0, "accum": "comp", "result": "grad"},
        # the large direct step: the million-particle Gaussian patch
        {"name": "self_1m_gauss", "family": "self", "layout": "patch", "n": 1000000, "core": "gauss",
         "radius": 0.005, "spread": 0.0, "accum": "comp", "result": "vel"},
        # probes in the flow and the gradient of a loss on them: forward and backward
        {"name": "probe_500k_10k", "family": "probe", "ns": 500000, "nt": 10000, "core": "gauss", "radius": 0.01,
         "accum": "comp"},
        # the reverse of a particle step: gradients of the particles' own velocities
        {"name": "vjp_self_131k", "family": "vjp", "layout": "patch", "n": 131072, "core": "gauss", "radius": 0.005,
         "accum": "comp"},
        # the million-particle patch by treecode
        {"name": "tree_1m_gauss", "family": "tree", "layout": "patch", "n": 1000000, "core": "gauss",
         "radius": 0.005},
        # a body in the flow: particles on its panels (the solve's right-hand side), panels on the particles
        {"name": "body_200k_2048", "family": "body", "n": 200000, "npan": 2048, "accum": "comp"},
        # the same body's influence matrix and its solve for the sheet strengths (4096 unknowns)
        {"name": "bem_2048", "family": "bem", "npan": 2048, "nunk": 2},
        # particles cropped out of the layer next to the body, once per step
        {"name": "clear_200k_2048", "family": "clear", "n": 200000, "npan": 2048, "method": 0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["self", "self", "self", "result", "advect", "probe", "vjp", "tree", "body", "bem", "clear"])
    accum = rng.choice(["comp", "comp", "plain"])
    layout = rng.choice(["patch", "cloud"])
    if family == "self":
        core = rng.choice(["gauss", "v2", "rm", "gauss", "v2", "wl", "v3"])
        spread = rng.choice([0.0, 0.0, 0.0, 0.5])
        top = 300000 if spread else 1000000 if core in ("gauss", "rm") else 500000
        n = _log(rng, 300, top)
        return {"family": "self", "layout": layout, "n": n, "core": core,
                "radius": round(rng.uniform(0.5, 5.0) / math.sqrt(n), 6), "spread": spread, "accum": accum,
                "result": "vel"}
    if family == "result":
        n = _log(rng, 1000, 300000)
        return {"family": "self", "layout": layout, "n": n, "core": "gauss",
                "radius": round(rng.uniform(0.5, 5.0) / math.sqrt(n), 6), "spread": 0.0, "accum": accum,
                "result": rng.choice(["grad", "vort", "shear"])}
    if family == "advect":
        n = _log(rng, 500, 60000)
        return {"family": "advect", "layout": layout, "n": n, "core": rng.choice(["rm", "gauss", "v2"]),
                "radius": round(rng.uniform(1.0, 3.0) / math.sqrt(n), 6), "accum": accum,
                "order": rng.choice([1, 2, 3]), "steps": rng.randint(1, 8), "dt": 0.01}
    if family == "probe":
        return {"family": "probe", "ns": _log(rng, 5000, 1000000), "nt": _log(rng, 200, 20000),
                "core": rng.choice(["gauss", "gauss", "v2"]), "radius": round(rng.uniform(0.005, 0.02), 6),
                "accum": accum}
    if family == "vjp":
        n = _log(rng, 2000, 250000)
        return {"family": "vjp", "layout": layout, "n": n, "core": "gauss",
                "radius": round(rng.uniform(0.5, 5.0) / math.sqrt(n), 6), "accum": accum}
    if family == "tree":
        n = _log(rng, 30000, 1000000)
        return {"family": "tree", "layout": layout, "n": n, "core": "gauss",
                "radius": round(rng.uniform(1.0, 5.0) / math.sqrt(n), 6)}
    if family == "body":
        return {"family": "body", "n": _log(rng, 2000, 500000), "npan": _log(rng, 64, 4096), "accum": accum}
    if family == "bem":
        return {"family": "bem", "npan": _log(rng, 64, 3000), "nunk": rng.choice([1, 2, 2])}
    return {"family": "clear", "n": _log(rng, 2000, 500000), "npan": _log(rng, 64, 4096),
            "method": rng.choice([0, 0, 1])}


# ---------------------------------------------------------------- inputs

def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _particles(case, g):
    """x, y, r, s of a Gaussian vortex patch (strengths follow the vorticity, total 1) or of a uniform cloud of
    particles of both signs; `spread` > 0 gives every particle its own radius within that share."""
    n = case["n"]
    if case["layout"] == "patch":
        xy = 0.25 * torch.randn(2, n, generator=g, device=DEV)
        s = torch.exp(-(xy[0] ** 2 + xy[1] ** 2) / 0.125)
        s = s / s.sum()
    else:
        xy = 2.0 * torch.rand(2, n, generator=g, device=DEV) - 1.0
        s = torch.randn(n, generator=g, device=DEV) / math.sqrt(n)
    r = torch.full((n,), case["radius"], device=DEV)
    if case.get("spread"):
        r = r * (1.0 + case["spread"] * (2.0 * torch.rand(n, generator=g, device=DEV) - 1.0))
    return xy[0].contiguous(), xy[1].contiguous(), r, s


def _annulus(n, g, inner, outer):
    rad = torch.sqrt(torch.rand(n, generator=g, device=DEV) * (outer ** 2 - inner ** 2) + inner ** 2)
    th = 2.0 * math.pi * torch.rand(n, generator=g, device=DEV)
    return rad * torch.cos(th), rad * torch.sin(th)


def _circle(npan):
    """Nodes and panel node pairs of a unit-diameter circle, clockwise (the fluid is outside)."""
    th = -2.0 * math.pi * torch.arange(npan, dtype=torch.float64, device=DEV) / npan
    i = torch.arange(npan, dtype=torch.int32, device=DEV)
    idx = torch.stack([i, (i + 1) % npan], 1).reshape(-1).contiguous()
    return (0.5 * torch.cos(th)).float(), (0.5 * torch.sin(th)).float(), idx


def prepare(case, seed):
    g = _generator(seed)
    st = {"case": case, "ctx": context()}
    f = case["family"]
    if f in ("self", "advect", "vjp", "tree"):
        st["x"], st["y"], st["r"], st["s"] = _particles(case, g)
        n = case["n"]
        st["u"], st["v"] = torch.zeros(n, device=DEV), torch.zeros(n, device=DEV)
        if f == "self":
            m = {"vel": 0, "grad": 4}.get(case["result"], 1)
            st["extra"] = [torch.zeros(n, device=DEV) for _ in range(m)]
        if f == "vjp":
            st["lu"], st["lv"] = torch.randn(2, n, generator=g, device=DEV).unbind(0)
            st["grads"] = [torch.zeros(n, device=DEV) for _ in range(3)]
    elif f == "probe":
        ns, nt = case["ns"], case["nt"]
        st["x"], st["y"] = (2.0 * torch.rand(2, ns, generator=g, device=DEV) - 1.0).unbind(0)
        st["s"] = torch.randn(ns, generator=g, device=DEV) / math.sqrt(ns)
        st["r"] = torch.full((ns,), case["radius"], device=DEV)
        st["tx"], st["ty"] = (torch.rand(2, nt, generator=g, device=DEV) - 0.5).unbind(0)
        st["u"], st["v"] = torch.zeros(nt, device=DEV), torch.zeros(nt, device=DEV)
        st["grads"] = [torch.zeros(ns, device=DEV) for _ in range(3)]
    else:
        npan = case["npan"]
        st["nx"], st["ny"], st["idx"] = _circle(npan)
        if f == "body":
            st["x"], st["y"] = _annulus(case["n"], g, 0.55, 3.0)
            st["s"] = 1.0e-2 * torch.randn(case["n"], generator=g, device=DEV)
            st["vs"], st["ss"] = torch.randn(2, npan, generator=g, device=DEV).unbind(0)
            st["pu"], st["pv"] = torch.zeros(npan, device=DEV), torch.zeros(npan, device=DEV)
            st["u"], st["v"] = torch.zeros(case["n"], device=DEV), torch.zeros(case["n"], device=DEV)
        elif f == "bem":
            # velocity at the panel centres of a freestream and some vortices outside the body, as the right-hand side
            vx, vy = _annulus(64, g, 0.8, 3.0)
            gam = 0.3 * torch.randn(64, generator=g, device=DEV)
            x0, y0, x1, y1, tx, ty, _ = _panels(st["nx"], st["ny"], st["idx"])
            dx = 0.5 * (x0 + x1)[:, None] - vx.double()[None, :]
            dy = 0.5 * (y0 + y1)[:, None] - vy.double()[None, :]
            k = gam.double()[None, :] * INV2PI / (dx * dx + dy * dy)
            u, v = 1.0 - (k * dy).sum(1), (k * dx).sum(1)
            m = npan * case["nunk"]
            t, nrm = -(u * tx + v * ty), -(-u * ty + v * tx)
            st["b"] = (torch.stack([t, nrm], 1).reshape(-1) if case["nunk"] == 2 else t).contiguous()
            st["A"] = torch.zeros(m * m, dtype=torch.float64, device=DEV)
            st["sol"] = torch.zeros(m, dtype=torch.float64, device=DEV)
        else:
            # most particles in the flow, some of them (the newest) inside the layer
            st["x"], st["y"] = _annulus(case["n"], g, 0.499, 1.5)
            st["s"] = 1.0e-2 * torch.randn(case["n"], generator=g, device=DEV)
            st["r"] = torch.full((case["n"],), CLEAR_IPS, device=DEV)
    return st


def run(st):
    case, ctx = st["case"], st["ctx"]
    f = case["family"]
    if f == "self":
        out = [st["u"], st["v"]] + st["extra"]
        for t in out:
            t.zero_()
        og.points_affect_points_dev(ctx, CORES[case["core"]], RESULT[case["result"]], ACCUM[case["accum"]], st["x"],
                                    st["y"], st["r"], st["s"], st["x"], st["y"], st["r"], st["u"], st["v"],
                                    extra=st["extra"], finalize=True, fs=(1.0, 0.0))
        return out
    if f == "advect":
        x, y = st["x"].clone(), st["y"].clone()
        og.advect_dev(ctx, CORES[case["core"]], ACCUM[case["accum"]], case["order"], x, y, st["r"], st["s"],
                      (1.0, 0.0), case["dt"], case["steps"])
        return [x, y]
    if f == "vjp":
        for t in st["grads"]:
            t.zero_()
        og.points_affect_points_vjp_self_dev(ctx, CORES[case["core"]], ACCUM[case["accum"]], st["x"], st["y"],
                                             st["r"], st["s"], st["lu"], st["lv"], *st["grads"])
        return list(st["grads"])
    if f == "tree":
        st["u"].zero_()
        st["v"].zero_()
        og.points_affect_points_tree_dev(ctx, CORES[case["core"]], st["x"], st["y"], st["r"], st["s"], st["x"],
                                         st["y"], st["r"], st["u"], st["v"], finalize=True, fs=(1.0, 0.0))
        return [st["u"], st["v"]]
    if f == "probe":
        # velocities at the probes, then the gradient of sum |velocity|^2 with respect to the particles
        core, accum = CORES[case["core"]], ACCUM[case["accum"]]
        st["u"].zero_()
        st["v"].zero_()
        og.points_affect_points_dev(ctx, core, og.VELONLY, accum, st["x"], st["y"], st["r"], st["s"], st["tx"],
                                    st["ty"], None, st["u"], st["v"], finalize=True)
        for t in st["grads"]:
            t.zero_()
        og.points_affect_points_vjp_dev(ctx, core, accum, st["x"], st["y"], st["r"], st["s"], st["tx"], st["ty"],
                                        None, 2.0 * st["u"], 2.0 * st["v"], *st["grads"])
        return [st["u"], st["v"]] + list(st["grads"])
    geo = (st["nx"], st["ny"], st["idx"])
    if f == "body":
        accum = ACCUM[case["accum"]]
        out = [st["pu"], st["pv"], st["u"], st["v"]]
        for t in out:
            t.zero_()
        og.points_affect_panels_dev(ctx, accum, st["x"], st["y"], st["s"], *geo, st["pu"], st["pv"], finalize=True,
                                    fs=(1.0, 0.0))
        og.panels_affect_points_dev(ctx, accum, *geo, st["vs"], st["ss"], st["x"], st["y"], st["u"], st["v"],
                                    finalize=True, fs=(1.0, 0.0))
        return out
    if f == "bem":
        og.panels_on_panels_coeff_dev(ctx, case["nunk"], *geo, None, st["A"])
        st["sol"].zero_()
        og.solve_gmres_f64_dev(ctx, st["A"], st["b"], st["sol"])
        return [st["sol"]]
    x, y = st["x"].clone(), st["y"].clone()
    s = st["s"].clone() if case["method"] == 0 else None
    circ, cnt = og.clear_inner_layer_dev(ctx, case["method"], og.CLEAR_CUTOFF, CLEAR_IPS, *geo, x, y, s,
                                         st["r"] if case["method"] == 0 else None)
    return {"x": x, "y": y, "s": s, "removed": circ, "count": cnt}


def work(case):
    f = case["family"]
    n = case.get("n", 0)
    if f in ("self", "advect", "vjp"):
        per = og.flops_per_pair(CORES[case["core"]], RESULT[case.get("result", "vel")], True)
        extra = {"vel": 0, "grad": 4}.get(case.get("result", "vel"), 1)
        calls = case.get("order", 1) * case.get("steps", 1)
        # the reverse evaluates the core and its derivative and sums three gradients per pair
        per = 2 * per if f == "vjp" else per
        arrays = {"self": 4 + 2 * (2 + extra), "advect": 6 * calls, "vjp": 6 + 6}[f]
        return {"bytes": 4.0 * n * arrays, "flops": float(per) * n * n * calls}
    if f == "tree":
        # per particle and level a few dozen well-separated cells of about 24 complex terms, and about 100 near pairs
        return {"bytes": 4.0 * n * 8, "flops": n * (math.log(max(n, 64) / 32, 4) * 27 * 24 * 8 + 1900.0)}
    if f == "probe":
        per = og.flops_per_pair(CORES[case["core"]], og.VELONLY, False)
        return {"bytes": 4.0 * (2 * 4 * case["ns"] + 3 * case["ns"] + 8 * case["nt"]),
                "flops": 3.0 * per * case["ns"] * case["nt"]}
    npan = case["npan"]
    if f == "body":
        return {"bytes": 4.0 * (3 * n + 2 * n + 4 * n + 4 * npan + 6 * npan), "flops": (39.0 + 47.0) * n * npan}
    if f == "bem":
        m = npan * case["nunk"]
        # the matrix written and read once, and about 35 products with it
        return {"bytes": 2 * 8.0 * m * m, "flops": 90.0 * npan * npan + 35 * 2.0 * m * m}
    return {"bytes": 4.0 * 7 * n, "flops": 20.0 * n * npan}


# ---------------------------------------------------------------- 64-bit results

def _panels(nx, ny, idx):
    i = idx.long().reshape(-1, 2)
    x, y = nx.double(), ny.double()
    x0, y0, x1, y1 = x[i[:, 0]], y[i[:, 0]], x[i[:, 1]], y[i[:, 1]]
    ln = torch.sqrt((x1 - x0) ** 2 + (y1 - y0) ** 2)
    return x0, y0, x1, y1, (x1 - x0) / ln, (y1 - y0) / ln, ln


def _core(core, d2, z, grad):
    """K and B = 2 dK/d(d^2) of the core at squared distance d2; z is the sum of the radii's squares (rm, gauss, wl),
    fourth powers (v2) or sixth powers (v3)."""
    b = None
    if core == "rm":
        k = 1.0 / (d2 + z)
        b = -2.0 * k * k if grad else None
    elif core == "gauss":
        x = d2 / z
        e = torch.exp(-x)
        mid = -torch.expm1(-x) / d2
        k = torch.where(x > 16.0, 1.0 / d2, torch.where(x < 0.001, 1.0 / z, mid))
        if grad:
            # g'(x), g = (1 - e^-x)/x: by its series below x = 0.02
            ser = -0.5 + x * (1.0 / 3 + x * (-1.0 / 8 + x * (1.0 / 30 - x / 144.0)))
            gp = torch.where(x < 0.02, ser, (e * (x + 1.0) - 1.0) / (x * x))
            g = torch.where(x < 0.02, 1.0 - x * (0.5 - x * (1.0 / 6 - x / 24.0)), mid * z)
            b = torch.where(x < 0.001, -2.0 * g / (z * z), 2.0 * gp / (z * z))
    elif core == "v2":
        k = torch.rsqrt(d2 * d2 + z)
        b = -2.0 * k ** 3 * d2 if grad else None
    elif core == "wl":
        dd = d2 + z
        k = (dd + z) / (dd * dd)
    else:
        k = (d2 ** 3 + z) ** (-1.0 / 3.0)
    return k, b


def _term(core, r):
    return r.double() ** {"v2": 4, "v3": 6}.get(core, 2)


def _chunks(nt, ns):
    step = max(1, int(3.0e7 // ns))
    return [(a, min(nt, a + step)) for a in range(0, nt, step)]


def _exact_self(case, x, y, zs, s):
    """Unscaled velocity (and gradient-type result) of the particles on themselves."""
    n, res = x.numel(), case.get("result", "vel")
    cols = {"vel": 2, "grad": 6}.get(res, 3)
    out = [torch.zeros(n, dtype=torch.float64, device=DEV) for _ in range(cols)]
    for a, b in _chunks(n, n):
        dx, dy = x[a:b, None] - x[None, :], y[a:b, None] - y[None, :]
        d2 = dx * dx + dy * dy
        k, bb = _core(case["core"], d2, zs[a:b, None] + zs[None, :], res != "vel")
        gk = k * s[None, :]
        out[0][a:b] = -(gk * dy).sum(1)
        out[1][a:b] = (gk * dx).sum(1)
        if res == "vel":
            continue
        gb = bb * s[None, :]
        if res == "grad":
            out[2][a:b] = -(gb * dx * dy).sum(1)                 # du/dx
            out[3][a:b] = (gb * dx * dx + gk).sum(1)             # dv/dx
            out[4][a:b] = -(gb * dy * dy + gk).sum(1)            # du/dy
            out[5][a:b] = (gb * dx * dy).sum(1)                  # dv/dy
        elif res == "vort":
            out[2][a:b] = (gb * d2 + 2.0 * gk).sum(1)
        else:
            out[2][a:b] = (0.5 * gb.abs() * d2).sum(1)
    return out


def _exact_advect(case, st):
    zs, s = _term(case["core"], st["r"]), st["s"].double()
    dt = case["dt"]

    def vel(x, y):
        u, v = _exact_self(case, x, y, zs, s)
        return 1.0 + u * INV2PI, v * INV2PI

    x, y = st["x"].double(), st["y"].double()
    for _ in range(case["steps"]):
        u1, v1 = vel(x, y)
        if case["order"] == 1:
            x, y = x + dt * u1, y + dt * v1
            continue
        c = 2.0 / 3.0 if case["order"] == 2 else 0.5
        u2, v2 = vel(x + c * dt * u1, y + c * dt * v1)
        if case["order"] == 2:
            x, y = x + dt * (0.25 * u1 + 0.75 * u2), y + dt * (0.25 * v1 + 0.75 * v2)
            continue
        u3, v3 = vel(x + 0.75 * dt * u2, y + 0.75 * dt * v2)
        x = x + dt * (2.0 * u1 + 3.0 * u2 + 4.0 * u3) / 9.0
        y = y + dt * (2.0 * v1 + 3.0 * v2 + 4.0 * v3) / 9.0
    return [x, y]


def _exact_vjp(case, st):
    """Gradients of sum lu u + lv v of the finalized velocities: both roles of every particle."""
    x, y, s = st["x"].double(), st["y"].double(), st["s"].double()
    lu, lv = st["lu"].double() * INV2PI, st["lv"].double() * INV2PI
    zs = _term(case["core"], st["r"])
    n = x.numel()
    gx, gy, gs = (torch.zeros(n, dtype=torch.float64, device=DEV) for _ in range(3))
    for a, b in _chunks(n, 2 * n):
        # rows: the particle whose gradient is formed; columns: the other one, as its target and as its source
        dx, dy = x[None, :] - x[a:b, None], y[None, :] - y[a:b, None]
        k, bb = _core(case["core"], dx * dx + dy * dy, zs[a:b, None] + zs[None, :], True)
        gs[a:b] = (k * (-lu[None, :] * dy + lv[None, :] * dx)).sum(1)
        wu = s[a:b, None] * lu[None, :] - s[None, :] * lu[a:b, None]
        wv = s[a:b, None] * lv[None, :] - s[None, :] * lv[a:b, None]
        q = bb * (-wu * dy + wv * dx)
        gx[a:b] = -(q * dx + k * wv).sum(1)
        gy[a:b] = -(q * dy - k * wu).sum(1)
    return [gx, gy, gs]


def _exact_probe(case, st):
    x, y, s, tx, ty = (st[q].double() for q in ("x", "y", "s", "tx", "ty"))
    zs = _term(case["core"], st["r"])
    ns, nt = x.numel(), tx.numel()
    u, v = torch.zeros(nt, dtype=torch.float64, device=DEV), torch.zeros(nt, dtype=torch.float64, device=DEV)
    for a, b in _chunks(nt, ns):
        dx, dy = tx[a:b, None] - x[None, :], ty[a:b, None] - y[None, :]
        gk = _core(case["core"], dx * dx + dy * dy, zs[None, :], False)[0] * s[None, :]
        u[a:b], v[a:b] = -(gk * dy).sum(1) * INV2PI, (gk * dx).sum(1) * INV2PI
    lu, lv = 2.0 * u * INV2PI, 2.0 * v * INV2PI
    gx, gy, gs = (torch.zeros(ns, dtype=torch.float64, device=DEV) for _ in range(3))
    for a, b in _chunks(ns, nt):
        dx, dy = tx[None, :] - x[a:b, None], ty[None, :] - y[a:b, None]
        k, bb = _core(case["core"], dx * dx + dy * dy, zs[a:b, None], True)
        w = -lu[None, :] * dy + lv[None, :] * dx
        gs[a:b] = (k * w).sum(1)
        q = bb * w
        gx[a:b] = -s[a:b] * (q * dx + k * lv[None, :]).sum(1)
        gy[a:b] = -s[a:b] * (q * dy - k * lu[None, :]).sum(1)
    return [u, v, gx, gy, gs]


def _star(x0, y0, x1, y1, tx, ty):
    """The angle under which a panel is seen and the log of its end points' distance ratio."""
    dx0, dy0, dx1, dy1 = tx - x0, ty - y0, tx - x1, ty - y1
    us = torch.atan2(dx0 * (y1 - y0) - dy0 * (x1 - x0), dx0 * dx1 + dy0 * dy1)
    vs = 0.5 * torch.log((dx0 * dx0 + dy0 * dy0) / (dx1 * dx1 + dy1 * dy1))
    return us, vs


def _exact_body(case, st):
    x0, y0, x1, y1, tx, ty, ln = _panels(st["nx"], st["ny"], st["idx"])
    x, y, s, g, q = (st[w].double() for w in ("x", "y", "s", "vs", "ss"))
    npan, n = x0.numel(), x.numel()
    A, B = g * tx + q * ty, q * tx - g * ty
    su, sv = torch.zeros_like(x0), torch.zeros_like(x0)
    u, v = torch.zeros_like(x), torch.zeros_like(x)
    for a, b in _chunks(n, npan):
        us, vs = _star(x0[None, :], y0[None, :], x1[None, :], y1[None, :], x[a:b, None], y[a:b, None])
        su += (s[a:b, None] * us).sum(0)
        sv += (s[a:b, None] * vs).sum(0)
        u[a:b] = us @ A + vs @ B
        v[a:b] = vs @ A - us @ B
    pu, pv = -(su * tx - sv * ty) / ln, -(su * ty + sv * tx) / ln
    return [1.0 + pu * INV2PI, pv * INV2PI, 1.0 + u * INV2PI, v * INV2PI]


def _exact_bem(case, st):
    x0, y0, x1, y1, tx, ty, ln = _panels(st["nx"], st["ny"], st["idx"])
    xm, ym = 0.5 * (x0 + x1), 0.5 * (y0 + y1)

    def block(tang, us, vs, sx, sy):
        """Components along the target's tangent and normal of a unit vortex or source sheet's velocity."""
        vu, vv = (us * sx - vs * sy, us * sy + vs * sx) if tang else (us * sy + vs * sx, vs * sy - us * sx)
        return vu * tx[:, None] + vv * ty[:, None], -vu * ty[:, None] + vv * tx[:, None]

    us, vs = _star(x0[None, :], y0[None, :], x1[None, :], y1[None, :], xm[:, None], ym[:, None])
    ur, vr = _star(x0[:, None], y0[:, None], x1[:, None], y1[:, None], xm[None, :], ym[None, :])
    fact = ln[None, :] / ln[:, None]
    npan, nunk = case["npan"], case["nunk"]
    M = torch.zeros(npan, nunk, npan, nunk, dtype=torch.float64, device=DEV)
    for q in range(nunk):
        fwd = block(q == 0, us, vs, tx[None, :], ty[None, :])
        rev = block(q == 0, ur, vr, tx[:, None], ty[:, None])
        for p in range(nunk):
            c = 0.5 * (fwd[p] - fact * rev[p])
            c.fill_diagonal_(math.pi if p == q else 0.0)
            M[:, p, :, q] = c * INV2PI
    m = npan * nunk
    return [torch.linalg.solve(M.reshape(m, m), st["b"])]


def exact(case, seed):
    f = case["family"]
    pairs = {"self": 1.0, "advect": float(case.get("order", 1) * case.get("steps", 1)), "vjp": 2.0, "tree": 1.0}
    if f in pairs and pairs[f] * float(case["n"]) ** 2 > EXACT_PAIRS:
        return None
    if f == "clear":
        return None   # which side of the layer a particle lies on, and its cuts, follow single-precision steps
    st = prepare(case, seed)
    if f in ("self", "tree"):
        out = _exact_self(case, st["x"].double(), st["y"].double(), _term(case["core"], st["r"]), st["s"].double())
        return [1.0 + out[0] * INV2PI, out[1] * INV2PI] + [t * INV2PI for t in out[2:]]
    return {"advect": _exact_advect, "vjp": _exact_vjp, "probe": _exact_probe, "body": _exact_body,
            "bem": _exact_bem}[f](case, st)
