"""Performance cases: the work that users of the solver have it do, through the
Python package's public calls, from one step of the smallest 2D domain to the
256^3 evolving-grain run, the batched sweep, the diagnostics rows and the
learned surrogate's layers.

A case is a dict of plain values: `kind` picks the path, the rest its sizes and
options. The initial state of a solver case (c_O, c_Cr, phi and the grain order
parameters) is made here on the GPU from the seed and written into the solver
in place; static Voronoi grains come from the solver's own seeded tessellation,
which exact() restates. exact() advances the same state in 64 bits with plain
torch operations.
"""
import math
import random
import sys

import numpy as np
import torch

sys.path.insert(0, "ni-cr_oxidation_phase-field_simulation_b200")

import nicr  # noqa: E402
from nicr import surrogate  # noqa: E402

DEV = "cuda"


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # One call of one step and the fields read back: a driver that watches the 2D example domain
        # (61^2, evolving grains) step by step. Host latency and launches count here.
        {"name": "2d_61_step_and_read", "kind": "solver", "dim": 2, "nx": 61, "ny": 61, "nz": 1, "eta": 3, "grains": 0,
         "bc": "concentration", "precision": 0, "steps": 1, "read": "host"},
        # The 2D centre-seed single crystal run: 100 steps of a 128^2 domain between two looks at it.
        {"name": "2d_128_crystal", "kind": "solver", "dim": 2, "nx": 128, "ny": 128, "nz": 1, "eta": 0, "grains": 0,
         "bc": "closed", "precision": 0, "steps": 100, "read": "device"},
        # A small 3D domain with static Voronoi grains, as one point of a hand-run study.
        {"name": "3d_64_static", "kind": "solver", "dim": 3, "nx": 64, "ny": 64, "nz": 64, "eta": 0, "grains": 2,
         "bc": "concentration", "precision": 0, "steps": 20, "read": "device"},
        # The programs' default grid (151 x 101 x 101), static grains of the default diameter, drop-in arithmetic.
        {"name": "3d_default_grid_static", "kind": "solver", "dim": 3, "nx": 151, "ny": 101, "nz": 101, "eta": 0,
         "grains": 24, "bc": "concentration", "precision": 0, "steps": 10, "read": "device"},
        # Evolving grains on an odd grid that no tile divides, oxygen supplied through a fixed chemical potential.
        {"name": "3d_odd_evolving", "kind": "solver", "dim": 3, "nx": 97, "ny": 61, "nz": 75, "eta": 5, "grains": 0,
         "bc": "mu", "precision": 0, "steps": 6, "read": "device"},
        # The benchmark grid, 256^3 with 8 evolving order parameters, in both arithmetic forms.
        {"name": "3d_256_evolving", "kind": "solver", "dim": 3, "nx": 256, "ny": 256, "nz": 256, "eta": 8, "grains": 0,
         "bc": "concentration", "precision": 0, "steps": 2, "read": "device"},
        {"name": "3d_256_evolving_reciprocal", "kind": "solver", "dim": 3, "nx": 256, "ny": 256, "nz": 256, "eta": 8,
         "grains": 0, "bc": "concentration", "precision": 1, "steps": 2, "read": "device"},
        # A parameter sweep: uneven static-grain domains advanced together (the batched form).
        {"name": "sweep_20_domains", "kind": "sweep", "domains": 20, "sizes": 3, "precision": 1, "steps": 10},
        # What a run writes at each logging interval: the diagnostics and the grain statistics of the current state.
        {"name": "log_128_evolving", "kind": "log", "nx": 128, "ny": 128, "nz": 128, "eta": 8},
        # Training of the surrogate, layer by layer: the wide-input full-resolution decoder layer and a
        # half-resolution layer, forward and backward, with weights, bias and input gradients.
        {"name": "conv_train_48_16_at_128", "kind": "conv", "n": 1, "edge": 128, "cin": 48, "cout": 16},
        {"name": "conv_train_64_64_at_64", "kind": "conv", "n": 1, "edge": 64, "cin": 64, "cout": 64},
        # One proposal of the surrogate: the 3-level U-Net (32 base channels) on a 128^3 state and its rates.
        {"name": "unet_32_at_128", "kind": "unet", "n": 1, "edge": 128, "base": 32},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["solver2", "solver3", "solver3", "evolving3", "evolving3", "tiles3", "sweep", "log", "conv", "unet"])
    bc = rng.choice(["concentration", "mu", "closed"])
    if kind == "solver2":
        eta = rng.choice([0, 2, 5])
        return {"kind": "solver", "dim": 2, "nx": _log_int(rng, 40, 700), "ny": _log_int(rng, 40, 700), "nz": 1,
                "eta": eta, "grains": 0, "bc": bc, "precision": rng.choice([0, 0, 1]), "steps": rng.randint(1, 60),
                "read": rng.choice(["host", "device"])}
    if kind == "solver3":
        n = [_log_int(rng, 24, 200) for _ in range(3)]
        return {"kind": "solver", "dim": 3, "nx": n[0], "ny": n[1], "nz": n[2], "eta": 0,
                "grains": rng.choice([0, 8, 24]), "bc": bc, "precision": rng.choice([0, 0, 1]),
                "steps": rng.randint(2, 12), "read": "device"}
    if kind == "evolving3":
        n = [_log_int(rng, 24, 160) for _ in range(3)]
        return {"kind": "solver", "dim": 3, "nx": n[0], "ny": n[1], "nz": n[2], "eta": rng.randint(2, 8), "grains": 0,
                "bc": bc, "precision": rng.choice([0, 1]), "steps": rng.randint(2, 6), "read": "device"}
    if kind == "tiles3":
        return {"kind": "solver", "dim": 3, "nx": _log_int(rng, 40, 256), "ny": 16 * rng.randint(3, 16),
                "nz": 32 * rng.randint(2, 8), "eta": rng.randint(2, 8), "grains": 0, "bc": bc,
                "precision": rng.choice([0, 1]), "steps": 2, "read": "device"}
    if kind == "sweep":
        return {"kind": "sweep", "domains": rng.randint(6, 20), "sizes": rng.randint(0, 10 ** 6), "precision": rng.choice([0, 1]), "steps": rng.randint(4, 10)}
    if kind == "log":
        n = [_log_int(rng, 40, 160) for _ in range(3)]
        return {"kind": "log", "nx": n[0], "ny": n[1], "nz": n[2], "eta": rng.randint(2, 8)}
    if kind == "conv":
        edge = rng.choice([32, 64, 96])
        return {"kind": "conv", "n": rng.choice([1, 2]), "edge": edge, "cin": 16 * rng.randint(1, 6),
                "cout": rng.choice([16, 32, 64]), }
    return {"kind": "unet", "n": rng.choice([1, 2]), "edge": rng.choice([32, 64, 96]), "base": rng.choice([16, 32])}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _state(shape, neta, seed, layer_o, bulk_cr, bc):
    """A domain some way into a run: Cr with composition noise, oxygen that has entered at X = 0, oxide
    balls near the surface and, with evolving grains, order parameters that pass smoothly from grain to grain."""
    g = _gen(seed)
    nx, ny, nz = shape
    f = dict(dtype=torch.float64, device=DEV)
    x = (torch.arange(nx, **f) + 0.5).view(-1, 1, 1)
    y = (torch.arange(ny, **f) + 0.5).view(1, -1, 1)
    z = (torch.arange(nz, **f) + 0.5).view(1, 1, -1)

    def rand(*s):
        return torch.rand(*s, generator=g, **f)

    def dist2(c):
        dy, dz = y - c[1], z - c[2]
        dy = dy - ny * torch.round(dy / ny)
        dz = dz - nz * torch.round(dz / nz)
        return (x - c[0]) ** 2 + dy * dy + dz * dz

    cr = bulk_cr + 0.02 * (rand(nx, ny, nz) - 0.5)
    o = layer_o * torch.exp(-x / 6.0) * (0.5 + rand(nx, ny, nz))
    if bc == "closed":
        o = 0.2 * o
    p = torch.zeros(nx, ny, nz, **f)
    balls = 1 + (nx * ny * nz) // 100_000 if ny > 1 else 1 + (nx * nz) // 8_000
    centre = rand(min(balls, 24), 3).tolist()
    for c in centre:
        d = dist2((2.0 + c[0] * nx * 0.5, c[1] * ny, c[2] * nz))
        inside = d <= 16.0
        p[inside], o[inside], cr[inside] = 1.0, 0.56300203, 0.35677915
    eta = []
    if neta:
        k = 3 * neta
        best = torch.zeros(neta, nx, ny, nz, **f)
        total = torch.zeros(nx, ny, nz, **f)
        sites = rand(k, 3).tolist()
        low = torch.full((nx, ny, nz), math.inf, **f)
        ds = [torch.sqrt(dist2((s[0] * nx, s[1] * ny, s[2] * nz))) for s in sites]
        for d in ds:
            low = torch.minimum(low, d)
        for i, d in enumerate(ds):
            w = torch.exp(-(d - low) / 1.2)
            best[i % neta] += w
            total += w
        hp = p * p * p * (10.0 - 15.0 * p + 6.0 * p * p)
        eta = [best[i] / total * (1.0 - hp) for i in range(neta)]
    return o, cr, p, eta


def _grain_diameter(shape, n):
    nx, ny, nz = shape
    return (6.0 * nx * ny * nz / (math.pi * n)) ** (1.0 / 3.0)


def _config(case, seed):
    """The solver's configuration and the physical parameters exact() needs."""
    dim, shape = case.get("dim", 3), (case["nx"], case["ny"], case.get("nz", 1))
    neta = case["eta"]
    kw = dict(nx=shape[0], ny=shape[1], random_seed=1 + int(seed) % 100000, bc=case.get("bc", "concentration"),
              bounds="legacy", nucleation="ksp", precision=case.get("precision", 0))
    if dim == 3:
        kw["nz"] = shape[2]
    if neta:
        if dim == 3:
            kw.update(grains=1, grain_evolution=1, grain_diameter_grid=_grain_diameter(shape, 3 * neta), eta_colours=neta)
        else:
            kw.update(grains=1, grain_evolution=1, grain_diameter_grid=math.sqrt(4.0 * shape[0] * shape[1] / (math.pi * neta)))
    elif case["grains"]:
        kw.update(grains=1, grain_diameter_grid=_grain_diameter(shape, case["grains"]))
    else:
        kw.update(grains=0)
    if dim == 2 and not neta:
        kw.update(nucleation="center", radius_grid=4.0)
    return nicr.make_config(dim, **kw)


def _fill(solver, o, cr, p, eta):
    dim3 = solver.cfg.dim == 3
    for name, v in [("o", o), ("cr", cr), ("p", p)] + [("eta%d" % (i + 1), e) for i, e in enumerate(eta)]:
        solver.device_view(name, writable=True).copy_(v if dim3 else v[:, 0, :])
    torch.cuda.synchronize()


def _shape3(case):
    """(planes, rows, columns): a 2D domain is one row of columns."""
    return (case["nx"], case["ny"], case["nz"]) if case.get("dim", 3) == 3 else (case["nx"], 1, case["ny"])


def _sweep_edges(case):
    """The sizes of the sweep's domains, which the case fixes; the parameters come from the seed."""
    rng = np.random.default_rng(case["sizes"])
    return [tuple(int(e) for e in rng.choice((32, 48, 64, 80, 96), size=3)) for _ in range(case["domains"])]


def _sweep_draws(case, seed):
    rng = np.random.default_rng(int(seed))
    out = []
    for i, (nx, ny, nz) in enumerate(_sweep_edges(case)):
        out.append(dict(nx=nx, ny=ny, nz=nz, bulk_cr=float(rng.uniform(0.15, 0.30)),
                        layer_o=0.0023 * float(rng.uniform(0.5, 1.0)), ksp=1.28e-7 * 10.0 ** float(rng.uniform(-1.0, 1.0)),
                        grains=int(rng.integers(8, 33)), random_seed=1000 + i + int(seed) % 100000))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solver":
        s = nicr.Solver(_config(case, seed))
        _fill(s, *_state(_shape3(case), case["eta"], seed, 0.0023, 0.25, case["bc"]))
        s.reset_inventory()
        names = ["o", "cr", "p"] + ["eta%d" % (i + 1) for i in range(case["eta"])]
        return {"kind": kind, "s": s, "names": names, "steps": case["steps"], "read": case["read"]}
    if kind == "sweep":
        draws = _sweep_draws(case, seed)
        cfgs = [nicr.make_config(3, grains=1, grain_diameter_grid=_grain_diameter((d["nx"], d["ny"], d["nz"]), d["grains"]),
                                 bc="concentration", bounds="legacy", nucleation="ksp", precision=case["precision"],
                                 **{k: v for k, v in d.items() if k != "grains"}) for d in draws]
        b = nicr.Batch(cfgs)
        for i, d in enumerate(draws):
            _fill(b.domains[i], *_state((d["nx"], d["ny"], d["nz"]), 0, seed + i, d["layer_o"], d["bulk_cr"], "concentration"))
            b.domains[i].reset_inventory()
        return {"kind": kind, "b": b, "steps": case["steps"]}
    if kind == "log":
        s = nicr.Solver(_config(case, seed))
        _fill(s, *_state(_shape3(case), case["eta"], seed, 0.0023, 0.25, "concentration"))
        s.reset_inventory()
        return {"kind": kind, "s": s}
    g = _gen(seed)
    if kind == "conv":
        e, cin, cout = case["edge"], case["cin"], case["cout"]
        # activations after a ReLU, weights and bias of a trained layer, the gradient of the layer above
        x = torch.randn((case["n"], e, e, e, cin), generator=g, device=DEV).relu_().to(torch.bfloat16)
        w = torch.randn((cout, 27, cin), generator=g, device=DEV) * math.sqrt(2.0 / (27 * cin))
        b = 0.1 * torch.randn(cout, generator=g, device=DEV)
        dy = torch.randn((case["n"], e, e, e, cout), generator=g, device=DEV).to(torch.bfloat16)
        return {"kind": kind, "x": x.requires_grad_(), "w": w.requires_grad_(), "b": b.requires_grad_(), "dy": dy}
    torch.manual_seed(int(seed) & 0x7FFFFFFF)
    net = surrogate.unet(8, case["base"]).to(DEV)
    e = case["edge"]
    return {"kind": kind, "net": net, "x": torch.randn((case["n"], e, e, e, 8), generator=g, device=DEV)}


# ------------------------------------------------------------------ one pass
def _views(s, names):
    """The solver's current fields in place. A view is valid while its solver lives: it keeps it."""
    out = {}
    for n in names:
        out[n] = s.device_view(n)
        out[n].solver = s
    return out


def run(state):
    kind = state["kind"]
    if kind == "solver":
        s = state["s"]
        s.run(state["steps"])
        if state["read"] == "host":
            return {n: s.get(n) for n in state["names"]}
        return _views(s, state["names"])
    if kind == "sweep":
        b = state["b"]
        b.run(state["steps"])
        return [_views(d, ("o", "cr", "p")) for d in b.domains]
    if kind == "log":
        s = state["s"]
        d, g = s.diagnostics(), s.grain_stats()
        out = {k: sum(v) if isinstance(v, tuple) else v for k, v in list(d.items()) + list(g.items()) if k != "amount"}
        out["amount"] = g["amount"].sum(axis=1)
        return out
    if kind == "conv":
        y = surrogate.conv3d_act(state["x"], state["w"], state["b"])
        gx, gw, gb = torch.autograd.grad(y, (state["x"], state["w"], state["b"]), state["dy"])
        return {"y": y, "gx": gx, "gw": gw, "gb": gb}
    with torch.no_grad():
        return {"y": state["net"](state["x"])}


# ------------------------------------------------------------------ what a pass cannot do without
def _unet_layers(c1):
    c2, c3 = 2 * c1, 4 * c1
    return [(16, c1, 1), (c1, c1, 1), (c1, c2, 8), (c2, c2, 8), (c2, c3, 64), (c3, c3, 64), (c3 + c2, c2, 8), (c2, c2, 8),
            (c2 + c1, c1, 1), (c1, c1, 1), (c1, 16, 1)]


def work(case):
    kind = case["kind"]
    if kind == "solver":
        cells = case["nx"] * case["ny"] * case["nz"]
        arrays = 6 + 2 * case["eta"] + (1 if case["grains"] else 0)   # o, cr, phi, eta read and written, the static mask read
        return {"bytes": 8 * arrays * cells * case["steps"], "flops": (230 + 32 * case["eta"]) * cells * case["steps"]}
    if kind == "sweep":
        cells = sum(a * b * c for a, b, c in _sweep_edges(case))
        return {"bytes": 8 * 7 * cells * case["steps"], "flops": 230 * cells * case["steps"]}
    if kind == "log":
        cells = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 8 * (3 + case["eta"]) * cells, "flops": (60 + 30 * case["eta"]) * cells}
    vox = case["n"] * case["edge"] ** 3
    if kind == "conv":
        cin, cout = case["cin"], case["cout"]
        # x and dy read, y and dx written (16 bits), the weights and their gradient (32 bits)
        return {"bytes": 4 * vox * (cin + cout) + 8 * 27 * cin * cout, "flops": 3 * 2 * 27 * cin * cout * vox}
    flops = sum(2 * 27 * a * b * vox / s for a, b, s in _unet_layers(case["base"]))
    return {"bytes": 64 * vox + 4 * 27 * sum(a * b for a, b, _ in _unet_layers(case["base"])), "flops": flops}


# ------------------------------------------------------------------ the same in 64 bits with plain torch
def _h(p):
    return p * p * p * (10.0 - 15.0 * p + 6.0 * p * p)


def _dxp(a):
    """The next plane along X, the last one repeated (no flux through the ends)."""
    return torch.cat([a[1:], a[-1:]], 0)


def _dxm(a):
    return torch.cat([a[:1], a[:-1]], 0)


def _lap(a, dx):
    r = (_dxp(a) - 2 * a + _dxm(a)) / dx ** 2
    for ax in (1, 2):
        if a.shape[ax] > 1:
            r = r + (a.roll(-1, ax) - 2 * a + a.roll(1, ax)) / dx ** 2
    return r


def _mobility(c, hh, gb, bm, bo, factor):
    return c * ((1 - hh) * bm * (1 + (factor - 1) * gb) + hh * bo)


def _flux_div(m, mu, dx, left_face):
    """Minus the divergence of -M grad(mu) per cell; left_face: the flux through X = 0."""
    inner = -0.5 * (m[:-1] + m[1:]) * (mu[1:] - mu[:-1]) / dx
    zero = torch.zeros_like(m[:1])
    left = torch.cat([left_face if left_face is not None else zero, inner], 0)
    right = torch.cat([inner, zero], 0)
    r = (left - right) / dx
    for ax in (1, 2):
        if m.shape[ax] > 1:
            f = -0.5 * (m + m.roll(-1, ax)) * (mu.roll(-1, ax) - mu) / dx
            r = r + (f.roll(1, ax) - f) / dx
    return r


def _advance(o, cr, p, eta, gb, c, steps):
    dx, dt, L, W = c.dx, c.dt, 0.2, 1e4
    width = c.gb_fwhm_grid * dx * math.sqrt(math.pi) / (2 * math.sqrt(math.log(2.0)))
    ell = 3 * width / 8
    K, eW, A = 2 * c.eta_W * ell * ell, c.eta_W, c.eta_W
    scale = width / (8 * ell / 3)
    conc, mu_bc = c.bc == 0, c.bc == 1
    for _ in range(steps):
        if conc:
            o = torch.cat([torch.full_like(o[:1], c.layer_o), o[1:]], 0)
        if eta:
            S, pairs = torch.zeros_like(o), torch.zeros_like(o)
            for e in eta:
                pairs = pairs + S * e * e
                S = S + e * e
            gb = scale * torch.clamp(16 * pairs, max=1.0)
        hh = _h(p)
        mu_o = (1 - hh) * (12e6 * o + 3.2e6 * cr - 298432.0) + hh * (24e6 * o - 13.8e6 * cr - 8.88e6) - 2e-9 * _lap(o, dx)
        mu_cr = (1 - hh) * (1166528.60789006 * cr + 3.2e6 * o - 97045.64) + hh * (14e6 * cr - 13.8e6 * o + 2.68e6) - 1.5e-8 * _lap(cr, dx)
        m_o = _mobility(o, hh, gb, 2.21e-16, 2.21e-18, c.gb_factor_o)
        m_cr = _mobility(cr, hh, gb, 3.5436e-20, 3.5436e-21, c.gb_factor_cr)
        face = None
        if mu_bc:
            mf = _mobility(torch.full_like(o[:1], c.surface_c_ref), hh[:1], gb[:1], 2.21e-16, 2.21e-18, c.gb_factor_o)
            face = 2 * mf * (c.mu_res - mu_o[:1]) / dx
        on = o + dt * _flux_div(m_o, mu_o, dx, face)
        cn = cr + dt * _flux_div(m_cr, mu_cr, dx, None)
        fm = 6e6 * o * o + 583264.303945031 * cr * cr + 3.2e6 * o * cr - 298432.0 * o - 97045.64 * cr - 61732.2974223055
        fo = 12e6 * o * o + 7e6 * cr * cr - 13.8e6 * o * cr - 8.88e6 * o + 2.68e6 * cr + 1860990.0
        hp = 30 * p * p * (p - 1) * (p - 1)
        fp = W * (4 * p ** 3 - 6 * p * p + 2 * p) + hp * (fo - fm) - 3.4e-10 * _lap(p, dx)
        if eta:
            fp = fp + 0.5 * hp * (eW * (S - (1 - hh)) + A * S)
        pn = p - dt * L * fp
        hn = _h(pn)
        d_o = -2e-10 * ((0.56300203 - on) * hn - (0.56300203 - o) * hh) / dt
        d_cr = -2e-10 * ((0.35677915 - cn) * hn - (0.35677915 - cr) * hh) / dt
        on, cn = torch.clamp(on + d_o, 0.0, 1.0), torch.clamp(cn + d_cr, 0.0, 1.0)
        pn = torch.where(pn > 0.99999, torch.ones_like(pn), pn)
        pn = torch.where(pn < 1e-5, torch.zeros_like(pn), pn)
        new = []
        for e in eta:
            force = e * (eW * (S - (1 - hh) + 2 * (S - e * e)) + A * hh) - K * _lap(e, dx)
            new.append(e - dt * c.eta_L * force)
        o, cr, p, eta = on, cn, pn, new
    return o, cr, p, eta


def _mt19937_64(seed, count):
    """The first `count` values in [0, 1) of std::mt19937_64 through a uniform real distribution."""
    m64, n, m = (1 << 64) - 1, 312, 156
    mt = [seed & m64]
    for i in range(1, n):
        mt.append((6364136223846793005 * (mt[-1] ^ (mt[-1] >> 62)) + i) & m64)
    out = []
    while len(out) < count:
        for i in range(n):
            x = (mt[i] & 0xFFFFFFFF80000000) | (mt[(i + 1) % n] & 0x7FFFFFFF)
            mt[i] = mt[(i + m) % n] ^ (x >> 1) ^ (0xB5026F5AA96619E9 if x & 1 else 0)
        for x in mt:
            x ^= (x >> 29) & 0x5555555555555555
            x ^= (x << 17) & 0x71D67FFFEDA60000
            x ^= (x << 37) & 0xFFF7EEE000000000
            x ^= x >> 43
            out.append(float(x) / 2.0 ** 64)
    return out[:count]


def _static_mask(c):
    """The grain-boundary mask of the static Voronoi grains: a Gaussian of the distance to the nearest bisector."""
    nx, ny, nz = c.nx, c.ny, c.nz
    ng = max(1, int(round(6.0 * nx * ny * nz / (math.pi * c.grain_diameter_grid ** 3))))
    u = _mt19937_64(int(c.random_seed), 3 * ng)
    sites = [(u[3 * k] * nx, u[3 * k + 1] * ny, u[3 * k + 2] * nz) for k in range(ng)]
    f = dict(dtype=torch.float64, device=DEV)
    x = (torch.arange(nx, **f) + 0.5).view(-1, 1, 1)
    y = (torch.arange(ny, **f) + 0.5).view(1, -1, 1)
    z = (torch.arange(nz, **f) + 0.5).view(1, 1, -1)
    best = torch.full((nx, ny, nz), math.inf, **f)
    own = torch.zeros((nx, ny, nz), dtype=torch.int64, device=DEV)
    oy, oz = torch.zeros_like(best), torch.zeros_like(best)
    for k, (sx, sy, sz) in enumerate(sites):
        dy, dz = sy - y, sz - z
        dy, dz = dy - ny * torch.round(dy / ny), dz - nz * torch.round(dz / nz)
        r = (sx - x) ** 2 + dy * dy + dz * dz
        near = r < best
        best, own = torch.where(near, r, best), torch.where(near, torch.full_like(own, k), own)
        oy, oz = torch.where(near, y + dy, oy), torch.where(near, z + dz, oz)
    ox = torch.tensor([s[0] for s in sites], **f)[own]
    low = torch.full_like(best, math.inf)
    for k, (sx, sy, sz) in enumerate(sites):
        for im in (-1, 0, 1):
            for jm in (-1, 0, 1):
                gy, gz = sy + im * ny, sz + jm * nz
                r = (sx - x) ** 2 + (gy - y) ** 2 + (gz - z) ** 2
                sep = torch.sqrt((sx - ox) ** 2 + (gy - oy) ** 2 + (gz - oz) ** 2)
                d = torch.clamp((r - best) / (2 * sep), min=0.0)
                low = torch.minimum(low, torch.where((own == k) | (sep <= 1e-14), torch.full_like(d, math.inf), d))
    return torch.exp(-4 * math.log(2.0) * low * low / c.gb_fwhm_grid ** 2) if ng > 1 else torch.zeros_like(low)


def _exact_conv(x, w):
    """3x3x3 convolution of channels-last x with w[cout][27][cin], zeros outside."""
    n, d, h, wd, _ = x.shape
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    y = 0
    for t in range(27):
        i, j, k = t // 9, t // 3 % 3, t % 3
        y = y + xp[:, i:i + d, j:j + h, k:k + wd, :] @ w[:, t, :].T
    return y


def exact(case, seed):
    kind = case["kind"]
    if kind == "solver":
        c = _config(case, seed)
        o, cr, p, eta = _state(_shape3(case), case["eta"], seed, 0.0023, 0.25, case["bc"])
        gb = _static_mask(c) if case["grains"] else torch.zeros_like(o)
        o, cr, p, eta = _advance(o, cr, p, eta, gb, c, case["steps"])
        out = {"o": o, "cr": cr, "p": p}
        out.update({"eta%d" % (i + 1): e for i, e in enumerate(eta)})
        if case["dim"] == 2:
            out = {k: v[:, 0, :] for k, v in out.items()}
        return {k: v.cpu().numpy() for k, v in out.items()} if case["read"] == "host" else out
    if kind == "sweep":
        out = []
        for i, d in enumerate(_sweep_draws(case, seed)):
            c = nicr.make_config(3, grains=1, grain_diameter_grid=_grain_diameter((d["nx"], d["ny"], d["nz"]), d["grains"]),
                                 bc="concentration", bounds="legacy", **{k: v for k, v in d.items() if k != "grains"})
            o, cr, p, eta = _state((d["nx"], d["ny"], d["nz"]), 0, seed + i, d["layer_o"], d["bulk_cr"], "concentration")
            o, cr, p, _ = _advance(o, cr, p, [], _static_mask(c), c, case["steps"])
            out.append({"o": o, "cr": cr, "p": p})
        return out
    if kind == "log":
        c = _config(case, seed)
        o, cr, p, eta = _state(_shape3(case), case["eta"], seed, 0.0023, 0.25, "concentration")
        S, pairs = torch.zeros_like(o), torch.zeros_like(o)
        for e in eta:
            pairs = pairs + S * e * e
            S = S + e * e
        gb = torch.clamp(16 * pairs, max=1.0)
        metal = 1 - _h(p)
        out = {k: None for k in ("energy", "alive", "unassigned", "cells")}
        out.update(sum_O=float(o.sum()), sum_Cr=float(cr.sum()), sum_phi=float(p.sum()), sum_h=float(_h(p).sum()),
                   min_O=float(o.min()), max_O=float(o.max()), min_Cr=float(cr.min()), max_Cr=float(cr.max()),
                   min_Ni=float((1 - o - cr).min()), min_phi=float(p.min()), max_phi=float(p.max()),
                   min_eta=float(min(e.min() for e in eta)), max_eta=float(max(e.max() for e in eta)),
                   min_s2=float(S.min()), max_s2=float(S.max()), sum_s2=float(S.sum()), gb_max=float(gb.max()),
                   mask=float((metal * gb).sum()))
        out["amount"] = np.array([float(torch.where(S > 1e-24, metal * e * e / S.clamp_min(1e-300), 0 * S).sum()) for e in eta])
        return out
    if kind == "conv":
        st = prepare(case, seed)
        x, w, b, dy = (st[k].detach().double() for k in ("x", "w", "b", "dy"))
        y = _exact_conv(x, w) + b
        keep = y > 0
        gy = dy * keep
        gx = _exact_conv(gy, w.flip(1).permute(2, 1, 0))
        n, d, h, wd, _ = x.shape
        xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
        g2 = gy.reshape(-1, gy.shape[-1]).T
        gw = torch.stack([g2 @ xp[:, t // 9:t // 9 + d, t // 3 % 3:t // 3 % 3 + h, t % 3:t % 3 + wd, :].reshape(-1, x.shape[-1])
                          for t in range(27)], 1)
        return {"y": y.clamp_min(0), "gx": gx, "gw": gw, "gb": gy.sum((0, 1, 2, 3))}
    st = prepare(case, seed)
    net, x = st["net"], st["x"].double()

    def layer(m, v):
        y = _exact_conv(v, m.w.detach().double()) + m.b.detach().double()
        return y.clamp_min(0) if m.relu else y

    def pool(v):
        n, d, h, w, ch = v.shape
        return v.view(n, d // 2, 2, h // 2, 2, w // 2, 2, ch).mean(dim=(2, 4, 6))

    def up(v):
        return v.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)

    def block(seq, v):
        for m in seq:
            v = layer(m, v)
        return v

    h0 = torch.cat([x, torch.zeros(x.shape[:-1] + (8,), dtype=x.dtype, device=x.device)], -1)
    e1 = block(net.enc1, h0)
    e2 = block(net.enc2, pool(e1))
    mid = block(net.mid, pool(e2))
    d2 = block(net.dec2, torch.cat([up(mid), e2], -1))
    d1 = block(net.dec1, torch.cat([up(d2), e1], -1))
    return {"y": layer(net.head, d1)[..., :8]}
