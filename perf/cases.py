"""The work that this framework's performance is judged on, as cases.

A case is one call of a public entry point on CUDA tensors, as a program that
has moved its fields to the GPU makes it: a whole time loop of one grid, one
weather-stencil sweep, one CFD run, or one pass of a planned batch.  ``listed``
names a fixed set over the range the entry points are used in (NPBench's S to
paper presets, the single-grid, batch and stream configurations of bench.py);
``draw`` gives further ones, mostly of odd sizes.
"""
import math

import numpy as np
import torch

from npbench_gb300 import stencils
from npbench_gb300.batch import Batch

_DTYPES = {"float64": torch.float64, "float32": torch.float32}


def listed():
    return [
        # NPBench's S preset, the smallest call: 48 half-sweeps of a 25^3 grid,
        # rows of 25 elements (no 16-byte alignment), launch latency.
        {"name": "heat_3d_25_f64", "kind": "heat_3d", "n0": 25, "n1": 25, "n2": 25, "tsteps": 25,
         "dtype": "float64"},
        # The headline single-grid run: both arrays beyond the L2.
        {"name": "heat_3d_256_f64", "kind": "heat_3d", "n0": 256, "n1": 256, "n2": 256,
         "tsteps": 100, "dtype": "float64"},
        # A request of the served stream: binary32 (70% of it), three unequal
        # sides, rows that are no 16-byte multiple.
        {"name": "heat_3d_ragged_f32", "kind": "heat_3d", "n0": 211, "n1": 173, "n2": 301,
         "tsteps": 100, "dtype": "float32"},
        # The single-grid 2D run: 1000^2, 100 steps, resident in the L2.
        {"name": "jacobi_2d_1000_f64", "kind": "jacobi_2d", "n0": 1000, "n1": 1000,
         "tsteps": 100, "dtype": "float64"},
        # A 2D request of the served stream in binary32, odd sides.
        {"name": "jacobi_2d_ragged_f32", "kind": "jacobi_2d", "n0": 1403, "n1": 1177,
         "tsteps": 200, "dtype": "float32"},
        # NPBench's paper preset: a small array and very many steps.
        {"name": "jacobi_1d_32000_f64", "kind": "jacobi_1d", "n": 32000, "tsteps": 4000,
         "dtype": "float64"},
        # NPBench's paper presets of the weather stencils.
        {"name": "hdiff_256x256x160", "kind": "hdiff", "n0": 256, "n1": 256, "n2": 160},
        {"name": "vadv_256x256x160", "kind": "vadv", "n0": 256, "n1": 256, "n2": 160},
        # NPBench's paper preset: three fields, 500 steps.
        {"name": "fdtd_2d_1000x1200_f64", "kind": "fdtd_2d", "n0": 1000, "n1": 1200, "tsteps": 500,
         "dtype": "float64"},
        # NPBench's paper preset: a small grid, 700 steps of 50 pressure iterations.
        {"name": "cavity_flow_101", "kind": "cavity_flow", "n0": 101, "n1": 101, "nt": 700,
         "nit": 50},
        # NPBench's M preset: steps until the flow has settled.
        {"name": "channel_flow_121", "kind": "channel_flow", "n0": 121, "n1": 121, "nit": 10},
        # A planned batch of uneven grids, half binary32, with the binary64 guard.
        {"name": "batch_32_grids", "kind": "batch", "grids": 32, "shapes": 1},
    ]


def _between(rng, lo, hi):
    """A whole number, spread evenly over the range or, where it spans more than a factor of
    ten, over its logarithm."""
    if hi > 10 * lo:
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return rng.randint(lo, hi)


def draw(rng):
    kind = rng.choice(["heat_3d", "heat_3d", "jacobi_2d", "jacobi_2d", "jacobi_1d", "hdiff", "vadv",
                       "fdtd_2d", "cavity_flow", "channel_flow", "batch"])
    if kind == "heat_3d":
        dtype = rng.choice(["float64", "float32"])
        top = 250 if dtype == "float64" else 320
        return {"kind": kind, "n0": _between(rng, 25, top), "n1": _between(rng, 25, top),
                "n2": _between(rng, 25, top), "tsteps": rng.randint(20, 100), "dtype": dtype}
    if kind == "jacobi_2d":
        return {"kind": kind, "n0": _between(rng, 128, 3000), "n1": _between(rng, 128, 3000),
                "tsteps": rng.randint(20, 200), "dtype": rng.choice(["float64", "float32"])}
    if kind == "jacobi_1d":
        return {"kind": kind, "n": _between(rng, 3200, 34000), "tsteps": rng.randint(800, 4000),
                "dtype": rng.choice(["float64", "float64", "float32"])}
    if kind == "hdiff":
        return {"kind": kind, "n0": _between(rng, 64, 384), "n1": _between(rng, 64, 256),
                "n2": _between(rng, 60, 160)}
    if kind == "vadv":
        return {"kind": kind, "n0": _between(rng, 60, 256), "n1": _between(rng, 60, 256),
                "n2": rng.choice([40, 60, 80, 160, _between(rng, 40, 160)])}
    if kind == "fdtd_2d":
        return {"kind": kind, "n0": _between(rng, 200, 1000), "n1": _between(rng, 220, 1200),
                "tsteps": _between(rng, 20, 500), "dtype": rng.choice(["float64", "float64", "float32"])}
    if kind == "cavity_flow":
        return {"kind": kind, "n0": _between(rng, 61, 201), "n1": _between(rng, 61, 201),
                "nt": _between(rng, 25, 400), "nit": _between(rng, 5, 50)}
    if kind == "channel_flow":
        return {"kind": kind, "n0": _between(rng, 61, 161), "n1": _between(rng, 61, 161),
                "nit": _between(rng, 5, 20)}
    return {"kind": kind, "grids": _between(rng, 8, 32), "shapes": rng.randint(2, 1 << 30)}


def _specs(case):
    """The batch's grids: sides log-uniform in 64 .. 2048, alternating precision, 10 .. 500 steps."""
    rng = np.random.default_rng(case["shapes"])
    sides = np.exp(rng.uniform(math.log(64), math.log(2048), (case["grids"], 2))).round().astype(int)
    steps = rng.integers(10, 501, case["grids"])
    return [((int(a), int(b)), torch.float32 if g % 2 else torch.float64, int(t))
            for g, ((a, b), t) in enumerate(zip(sides, steps))]


def _uniform(gen, *shape):
    return torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64)


def _cfd_fields(case, gen):
    """A fluid at rest (p = 0 in the cavity, 1 in the channel) with a small seeded disturbance: in the
    channel small against what the force adds in a step, so that the flow speeds up from the start."""
    ny, nx = case["n0"], case["n1"]
    size, base = (1e-6, 1.0) if case["kind"] == "channel_flow" else (1e-3, 0.0)
    u = size * _uniform(gen, ny, nx)
    v = size * (_uniform(gen, ny, nx) - 0.5)
    p = base + size * _uniform(gen, ny, nx)
    dx, dy = 2 / (nx - 1), 2 / (ny - 1)
    return {"u0": u, "v0": v, "p0": p, "dx": dx, "dy": dy, "dt": .1 / ((nx - 1) * (ny - 1)),
            "rho": 1.0, "nu": 0.1, "F": 1.0}


def _inputs(case, seed):
    """The fields a program has on the GPU before the call."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind in ("heat_3d", "jacobi_2d"):
        # U[0, 1), the configurations' initial fields; Heat-3D starts with B a copy of A.
        dt = _DTYPES[case["dtype"]]
        shape = [case[k] for k in ("n0", "n1", "n2") if k in case]
        A = _uniform(gen, *shape).to(dt)
        return {"A": A, "B": A.clone() if kind == "heat_3d" else _uniform(gen, *shape).to(dt)}
    if kind == "jacobi_1d":
        # NPBench's ramps (i+2)/N and (i+3)/N, roughened.
        n, dt = case["n"], _DTYPES[case["dtype"]]
        i = torch.arange(n, device="cuda", dtype=torch.float64)
        return {"A": ((i + 2) / n * (0.5 + 0.5 * _uniform(gen, n))).to(dt),
                "B": ((i + 3) / n * (0.5 + 0.5 * _uniform(gen, n))).to(dt)}
    if kind == "hdiff":
        I, J, K = case["n0"], case["n1"], case["n2"]
        return {"in": _uniform(gen, I + 4, J + 4, K), "out": torch.zeros(I, J, K, device="cuda",
                                                                        dtype=torch.float64),
                "coeff": _uniform(gen, I, J, K)}
    if kind == "vadv":
        I, J, K = case["n0"], case["n1"], case["n2"]
        return {"us0": _uniform(gen, I, J, K), "u": _uniform(gen, I, J, K),
                "wcon": _uniform(gen, I + 1, J, K), "up": _uniform(gen, I, J, K),
                "ut": _uniform(gen, I, J, K), "dtr": 3. / 20.}
    if kind == "fdtd_2d":
        # NPBench's fields i(j+1)/NX, i(j+2)/NY, i(j+3)/NX and source i, roughened.
        nx, ny, T, dt = case["n0"], case["n1"], case["tsteps"], _DTYPES[case["dtype"]]
        i = torch.arange(nx, device="cuda", dtype=torch.float64)[:, None]
        j = torch.arange(ny, device="cuda", dtype=torch.float64)[None, :]
        rough = lambda f: (f * (0.5 + 0.5 * _uniform(gen, nx, ny))).to(dt)  # noqa: E731
        return {"ex": rough(i * (j + 1) / nx), "ey": rough(i * (j + 2) / ny),
                "hz": rough(i * (j + 3) / nx),
                "fict": torch.arange(T, device="cuda", dtype=torch.float64).to(dt)}
    if kind in ("cavity_flow", "channel_flow"):
        return _cfd_fields(case, gen)
    return {"grids": [(_uniform(gen, *shape).to(dt), _uniform(gen, *shape).to(dt), t)
                      for shape, dt, t in _specs(case)]}


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    if case["kind"] == "vadv":
        s["us"] = torch.empty_like(s["us0"])
    elif case["kind"] in ("cavity_flow", "channel_flow"):
        for f in "uvp":
            s[f] = torch.empty_like(s[f + "0"])
    elif case["kind"] == "batch":
        s["batch"] = Batch(s["grids"], guard=True)
    return s


def run(s):
    """One call.  Time loops go on from where the fields are; where a call's work or its results
    would change with that (the solve's tendency, the flows), it starts from the same fields again."""
    c = s["case"]
    kind = c["kind"]
    if kind == "heat_3d":
        stencils.heat_3d_kernel(c["tsteps"], s["A"], s["B"])
        return s["A"], s["B"]
    if kind == "jacobi_2d":
        stencils.jacobi_2d_kernel(c["tsteps"], s["A"], s["B"])
        return s["A"], s["B"]
    if kind == "jacobi_1d":
        stencils.jacobi_1d_kernel(c["tsteps"], s["A"], s["B"])
        return s["A"], s["B"]
    if kind == "hdiff":
        stencils.hdiff(s["in"], s["out"], s["coeff"])
        return s["out"]
    if kind == "vadv":
        s["us"].copy_(s["us0"])  # the dycore's tendency of this step
        stencils.vadv(s["us"], s["u"], s["wcon"], s["up"], s["ut"], s["dtr"])
        return s["us"]
    if kind == "fdtd_2d":
        stencils.fdtd_2d_kernel(c["tsteps"], s["ex"], s["ey"], s["hz"], s["fict"])
        return s["ex"], s["ey"], s["hz"]
    if kind in ("cavity_flow", "channel_flow"):
        for f in "uvp":
            s[f].copy_(s[f + "0"])
        if kind == "cavity_flow":
            stencils.cavity_flow(c["n1"], c["n0"], c["nt"], c["nit"], s["u"], s["v"], s["dt"], s["dx"],
                                 s["dy"], s["p"], s["rho"], s["nu"])
            return s["u"], s["v"], s["p"]
        steps = stencils.channel_flow(c["nit"], s["u"], s["v"], s["dt"], s["dx"], s["dy"], s["p"],
                                      s["rho"], s["nu"], s["F"])
        return s["u"], s["v"], s["p"], steps
    s["batch"].launch(graph=True)
    return [x for g in s["grids"] for x in g[:2]]


def work(case):
    """Bytes: every field read once and every result written once (a time loop needs no more, if it
    keeps its grid on the chip); flops: the reference's operations."""
    kind = case["kind"]
    size = 8 if case.get("dtype", "float64") == "float64" else 4
    if kind == "heat_3d":
        n = case["n0"] * case["n1"] * case["n2"]
        return {"bytes": 4 * n * size, "flops": 13 * 2 * (case["tsteps"] - 1) * n}
    if kind == "jacobi_2d":
        n = case["n0"] * case["n1"]
        return {"bytes": 4 * n * size, "flops": 5 * 2 * (case["tsteps"] - 1) * n}
    if kind == "jacobi_1d":
        return {"bytes": 4 * case["n"] * size, "flops": 3 * 2 * (case["tsteps"] - 1) * case["n"]}
    if kind == "hdiff":
        I, J, K = case["n0"], case["n1"], case["n2"]
        return {"bytes": 8 * K * ((I + 4) * (J + 4) + 2 * I * J), "flops": 20 * I * J * K}
    if kind == "vadv":
        return {"bytes": 8 * 6 * case["n0"] * case["n1"] * case["n2"],
                "flops": 25 * case["n0"] * case["n1"] * case["n2"]}
    if kind == "fdtd_2d":
        n = case["n0"] * case["n1"]
        return {"bytes": 6 * n * size, "flops": 11 * case["tsteps"] * n}
    if kind in ("cavity_flow", "channel_flow"):
        n = case["n0"] * case["n1"]
        steps = case.get("nt", 950)  # the channel settles after about that many
        return {"bytes": 6 * n * 8, "flops": steps * n * (7 * case["nit"] + 60)}
    got = {"bytes": 0, "flops": 0}
    for shape, dt, t in _specs(case):
        n = shape[0] * shape[1]
        got["bytes"] += 4 * n * (8 if dt == torch.float64 else 4)
        got["flops"] += 5 * 2 * (t - 1) * n
    return got


# ------------------------------------------------------------------ the same in plain 64-bit torch


def _jacobi_2d(T, A, B):
    for s, d in [(A, B), (B, A)] * (T - 1):
        d[1:-1, 1:-1] = 0.2 * (s[1:-1, 1:-1] + s[1:-1, :-2] + s[1:-1, 2:] + s[2:, 1:-1] + s[:-2, 1:-1])
    return A, B


def _heat_3d(T, A, B):
    for s, d in [(A, B), (B, A)] * (T - 1):
        c = s[1:-1, 1:-1, 1:-1]
        c2 = 2.0 * c
        r = 0.125 * (s[2:, 1:-1, 1:-1] - c2 + s[:-2, 1:-1, 1:-1])
        r += 0.125 * (s[1:-1, 2:, 1:-1] - c2 + s[1:-1, :-2, 1:-1])
        r += 0.125 * (s[1:-1, 1:-1, 2:] - c2 + s[1:-1, 1:-1, :-2])
        d[1:-1, 1:-1, 1:-1] = r + c
    return A, B


def _jacobi_1d(T, A, B):
    for s, d in [(A, B), (B, A)] * (T - 1):
        d[1:-1] = 0.33333 * (s[:-2] + s[1:-1] + s[2:])
    return A, B


def _hdiff(f, coeff):
    I, J = coeff.shape[0], coeff.shape[1]
    lap = 4.0 * f[1:I + 3, 1:J + 3] - (f[2:I + 4, 1:J + 3] + f[0:I + 2, 1:J + 3] + f[1:I + 3, 2:J + 4] +
                                       f[1:I + 3, 0:J + 2])
    r = lap[1:, 1:J + 1] - lap[:-1, 1:J + 1]
    flx = torch.where(r * (f[2:I + 3, 2:J + 2] - f[1:I + 2, 2:J + 2]) > 0, 0.0, r)
    r = lap[1:I + 1, 1:] - lap[1:I + 1, :-1]
    fly = torch.where(r * (f[2:I + 2, 2:J + 3] - f[2:I + 2, 1:J + 2]) > 0, 0.0, r)
    return f[2:I + 2, 2:J + 2] - coeff * (flx[1:] - flx[:-1] + fly[:, 1:] - fly[:, :-1])


def _vadv(us, u, wcon, up, ut, dtr):
    K = us.shape[2]
    q = [None] + [0.25 * (wcon[1:, :, k] + wcon[:-1, :, k]) * 0.5 for k in range(1, K)] + [None]
    ccol, dcol = [], []
    for k in range(K):
        corr = 0.0
        bcol = dtr
        if k > 0:
            bcol = bcol + q[k]
            corr = q[k] * (u[:, :, k - 1] - u[:, :, k])
        if k < K - 1:
            bcol = bcol - q[k + 1]
            corr = corr - q[k + 1] * (u[:, :, k + 1] - u[:, :, k])
        d = dtr * up[:, :, k] + ut[:, :, k] + us[:, :, k] + corr
        if k > 0:
            bcol = bcol + ccol[k - 1] * q[k]
            d = d + dcol[k - 1] * q[k]
        divided = 1.0 / bcol
        ccol.append(q[k + 1] * divided if k < K - 1 else None)
        dcol.append(d * divided)
    out = torch.empty_like(us)
    data = dcol[K - 1]
    out[:, :, K - 1] = dtr * (data - up[:, :, K - 1])
    for k in range(K - 2, -1, -1):
        data = dcol[k] - ccol[k] * data
        out[:, :, k] = dtr * (data - up[:, :, k])
    return out


def _fdtd_2d(T, ex, ey, hz, fict):
    for t in range(T):
        ey[0] = fict[t]
        ey[1:] -= 0.5 * (hz[1:] - hz[:-1])
        ex[:, 1:] -= 0.5 * (hz[:, 1:] - hz[:, :-1])
        hz[:-1, :-1] -= 0.7 * (ex[:-1, 1:] - ex[:-1, :-1] + ey[1:, :-1] - ey[:-1, :-1])
    return ex, ey, hz


def _flow(case, s):
    """Both flows, channel_flow with columns that wrap around."""
    wrap = case["kind"] == "channel_flow"
    u, v, p = (s[f + "0"].clone() for f in "uvp")
    dx, dy, dt, rho, nu = (s[k] for k in ("dx", "dy", "dt", "rho", "nu"))

    def east(f):
        return torch.roll(f, -1, 1) if wrap else f[:, 2:]

    def west(f):
        return torch.roll(f, 1, 1) if wrap else f[:, :-2]

    def mid(f):
        return f if wrap else f[:, 1:-1]

    def advect(f, cu, cv, pdiff, k1):
        m = mid(f)
        c = m[1:-1]
        out = c - cu * (c - west(f)[1:-1]) - cv * (c - m[:-2]) - k1 * pdiff
        return out + nu * (dt / dx ** 2 * (east(f)[1:-1] - 2 * c + west(f)[1:-1]) +
                           dt / dy ** 2 * (m[2:] - 2 * c + m[:-2]))

    steps, udiff = 0, 1.0
    while udiff > .001 if wrap else steps < case["nt"]:
        un, vn = u.clone(), v.clone()
        x1 = (east(u) - west(u))[1:-1] / (2 * dx)
        x2 = (mid(v)[2:] - mid(v)[:-2]) / (2 * dy)
        z = (mid(u)[2:] - mid(u)[:-2]) / (2 * dy) * (east(v) - west(v))[1:-1] / (2 * dx)
        b = rho * (1 / dt * (x1 + x2) - x1 ** 2 - 2 * z - x2 ** 2)
        cb = dx ** 2 * dy ** 2 / (2 * (dx ** 2 + dy ** 2)) * b
        for _ in range(case["nit"]):
            new = ((east(p) + west(p))[1:-1] * dy ** 2 + (mid(p)[2:] + mid(p)[:-2]) * dx ** 2) / \
                (2 * (dx ** 2 + dy ** 2)) - cb
            if wrap:
                p = torch.cat((new[:1], new, new[-1:]))
            else:
                new = torch.cat((new[:, :1], new, new[:, -1:]), 1)
                p = torch.cat((new[:1], new, torch.zeros_like(new[:1])))
        cu, cv = mid(un)[1:-1] * dt / dx, mid(vn)[1:-1] * dt / dy
        nu_ = advect(un, cu, cv, (east(p) - west(p))[1:-1], dt / (2 * rho * dx))
        nv_ = advect(vn, cu, cv, mid(p)[2:] - mid(p)[:-2], dt / (2 * rho * dy))
        u, v = torch.zeros_like(u), torch.zeros_like(v)
        mid(u)[1:-1] = nu_ + s["F"] * dt if wrap else nu_
        mid(v)[1:-1] = nv_
        if wrap:
            udiff = float((u.sum() - un.sum()) / u.sum())
        else:
            u[-1] = 1.0
        steps += 1
    return (u, v, p, steps) if wrap else (u, v, p)


def exact(case, seed):
    s = _inputs(case, seed)
    wide = lambda *names: [s[k].double() for k in names]  # noqa: E731
    kind = case["kind"]
    if kind == "heat_3d":
        return _heat_3d(case["tsteps"], *wide("A", "B"))
    if kind == "jacobi_2d":
        return _jacobi_2d(case["tsteps"], *wide("A", "B"))
    if kind == "jacobi_1d":
        return _jacobi_1d(case["tsteps"], *wide("A", "B"))
    if kind == "hdiff":
        return _hdiff(s["in"], s["coeff"])
    if kind == "vadv":
        return _vadv(s["us0"], s["u"], s["wcon"], s["up"], s["ut"], s["dtr"])
    if kind == "fdtd_2d":
        return _fdtd_2d(case["tsteps"], *wide("ex", "ey", "hz", "fict"))
    if kind in ("cavity_flow", "channel_flow"):
        return _flow(case, s)
    return [x for A, B, t in s["grids"] for x in _jacobi_2d(t, A.double(), B.double())]
