"""The work this framework is used for, as cases that can be timed and compared.

Fluid frames (`kind` "frame", "batched" and "modules"), neighbour queries
("query"), peridynamics steps ("bar"), an elastoplastic frame ("plastic") and
the two differentiable rollouts ("pd_rollout", "pbd_rollout"), each called as a
program calls it: a context per simulation, positions and velocities kept on
the GPU and advanced in place.  A simulation restarts from its first state
every `EPISODE` passes, so that a long run stays in the same regime.

`exact` restates each path in double precision with plain torch: neighbour
sets decided on the float32 positions with the query's own roundings, all
physics in 64 bits.
"""
import math
import os
import sys

import torch
from torch.utils.checkpoint import checkpoint

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "physika-old_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import pk_torch  # noqa: E402
import pkhot  # noqa: E402

DEV = "cuda"
EPISODE = 24
GRAVITY = (0.0, -9.8, 0.0)
REST_DENSITY = 1000.0
MU, LAM = 0.05, 0.1


# ------------------------------------------------------------------ cases

def fluid(nx, ny, nz, **more):
    """A jittered block of fluid in the corner of its box: the 32k dam break's parameters."""
    case = {"kind": "frame", "nx": nx, "ny": ny, "nz": nz, "spacing": 0.005, "cap": 60, "iterations": 5,
            "dt": 1e-3, "box_x": 1.0, "viscosity": 0.0}
    case.update(more)
    return case


def solid(nx, ny, nz, **more):
    """A peridynamics block: horizon 3 spacing, 10 projection iterations."""
    case = {"kind": "bar", "nx": nx, "ny": ny, "nz": nz, "spacing": 0.004, "cap": 80, "iterations": 10,
            "dt": 1e-3, "break_stretch": 0.0}
    case.update(more)
    return case


def listed():
    return [
        # the smallest scene of the batched mix on its own: launches and latency
        dict(fluid(16, 8, 8), name="frame_1k"),
        # the 32,768-particle dam break, an interactive scene
        dict(fluid(32, 32, 32), name="frame_32k"),
        # the stock fluid model (ImplicitViscosity after the solve), a ragged size
        dict(fluid(61, 47, 53, viscosity=1.0), name="frame_152k_viscous"),
        # the 2,097,152-particle dam break of the benchmark
        dict(fluid(128, 128, 128, spacing=0.0025, cap=64, dt=5e-4, box_x=2.0), name="frame_2m"),
        # 256 uneven scenes stepped together, 1,024 to 65,536 particles each
        dict(fluid(0, 0, 0, kind="batched", scenes=256, n_min=1024, n_max=65536), name="batched_256"),
        # a scene graph's frame, module by module on the public neighbour list
        dict(fluid(64, 64, 64, kind="modules", viscosity=1.0), name="modules_262k"),
        # a query with a dynamic list for an application's own kernels, and the density on it
        dict(fluid(47, 46, 46, kind="query", cap=0), name="query_dynamic_99k"),
        # a small elastic body with a dynamic bond list
        dict(solid(37, 23, 23, cap=0), name="bar_20k"),
        # the 524,288-particle bar with fracture of the benchmark
        dict(solid(256, 64, 32, break_stretch=0.02), name="bar_524k"),
        # the elastoplastic body's frame (projection interleaved with DensityPBD, plasticity, viscosity)
        dict(solid(64, 32, 32, kind="plastic", cap=0), name="plastic_65k"),
        # gradients through elasticity and through the fluid, as an inverse problem takes them
        dict(solid(64, 32, 32, kind="pd_rollout", steps=10, every=5), name="pd_rollout_65k"),
        dict(fluid(64, 32, 32, kind="pbd_rollout", steps=10, every=5), name="pbd_rollout_65k"),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def dims(n):
        a = n ** (1.0 / 3.0)
        nx = max(2, int(round(a * rng.uniform(0.7, 1.5))))
        ny = max(2, int(round(a * rng.uniform(0.7, 1.4))))
        return nx, ny, max(2, int(round(n / (nx * ny))))

    kind = rng.choice(["frame", "frame", "frame", "batched", "modules", "query", "bar", "bar", "plastic",
                       "pd_rollout", "pbd_rollout"])
    cap = rng.choice([40, 60, 64, 73])
    if kind == "frame":
        n = log_int(1000, 1500000)
        fine = n > 200000
        return fluid(*dims(n), spacing=0.0025 if fine else 0.005, dt=5e-4 if fine else 1e-3, cap=cap,
                     iterations=rng.choice([3, 5, 8]), viscosity=rng.choice([0.0, 0.0, 1.0, 0.3]))
    if kind == "batched":
        return fluid(0, 0, 0, kind=kind, scenes=rng.randint(2, 128), n_min=rng.choice([300, 1024]),
                     n_max=log_int(4096, 65536), cap=cap, viscosity=rng.choice([0.0, 1.0]))
    if kind == "modules":
        return fluid(*dims(log_int(2000, 300000)), kind=kind, cap=rng.choice([0, cap]),
                     viscosity=rng.choice([1.0, 0.3]))
    if kind == "query":
        return fluid(*dims(log_int(1000, 500000)), kind=kind, cap=rng.choice([0, 0, cap]))
    if kind == "bar":
        return solid(*dims(log_int(2000, 300000)), cap=rng.choice([0, 80, 60]),
                     break_stretch=rng.choice([0.0, 0.02]))
    if kind == "plastic":
        return solid(*dims(log_int(4000, 65000)), kind=kind, cap=0)
    if kind == "pd_rollout":
        return solid(*dims(log_int(3000, 50000)), kind=kind, cap=rng.choice([0, 80]), steps=rng.randint(3, 10),
                     every=rng.randint(2, 6))
    return fluid(*dims(log_int(3000, 60000)), kind="pbd_rollout", cap=cap, steps=rng.randint(3, 10),
                 every=rng.randint(2, 6))


# ----------------------------------------------------------------- inputs

def is_solid(case):
    return case["kind"] in ("bar", "plastic", "pd_rollout")


def radius_of(case):
    return (3.0 if is_solid(case) else 2.5) * case["spacing"]


def bounds_of(case):
    if is_solid(case):
        return (0.0, 0.0, 0.0), tuple(case[k] * case["spacing"] + 0.2 for k in ("nx", "ny", "nz"))
    if case["kind"] == "pbd_rollout":
        return (0.0, 0.0, 0.0), (1.0, 1.0, 1.0)
    need = [1.25 * case[k] * case["spacing"] for k in ("nx", "ny", "nz")]
    return (0.0, 0.0, 0.0), (max(case["box_x"], need[0]), max(1.0, need[1]), max(1.0, need[2]))


def scene_dims(case):
    """Block sizes of a batched case: particle counts log-uniform in [n_min, n_max]."""
    g = torch.Generator().manual_seed(17)
    u = torch.rand(case["scenes"], generator=g, dtype=torch.float64)
    lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
    got = []
    for n in torch.exp(lo + u * (hi - lo)).tolist():
        a = max(1, int(round(n ** (1.0 / 3.0))))
        got.append((a, a, max(1, int(round(n / (a * a))))))
    return got


def block(nx, ny, nz, spacing, jitter, origin, gen):
    axes = [torch.arange(m, device=DEV, dtype=torch.float64) for m in (nx, ny, nz)]
    x = torch.stack(torch.meshgrid(*axes, indexing="ij"), -1).reshape(-1, 3)
    x = (x + 1.0) * spacing + torch.tensor(origin, device=DEV, dtype=torch.float64)
    u = torch.rand(x.shape, device=DEV, dtype=torch.float64, generator=gen)
    return (x + (2.0 * u - 1.0) * jitter * spacing).float()


def inputs(case, seed):
    """Positions, velocities and what else the seed decides: {"x", "v", ...}."""
    gen = torch.Generator(device=DEV).manual_seed(seed * 1000003 + 11)
    kind, s = case["kind"], case["spacing"]
    got = {}
    if kind == "batched":
        dims = scene_dims(case)
        xs = [block(*d, s, 0.1, (0.004, 0.004, 0.004), gen) for d in dims]
        counts = [x.shape[0] for x in xs]
        off = torch.tensor([0] + counts).cumsum(0)
        got["x"] = torch.cat(xs)
        got["offsets"] = off.to(torch.int32).to(DEV)
        got["scene"] = torch.repeat_interleave(torch.arange(len(dims), device=DEV), off.diff().to(DEV))
    else:
        d = (case["nx"], case["ny"], case["nz"])
        if is_solid(case):
            got["x"] = block(*d, s, 0.02, (0.1, 0.1, 0.1), gen)
        else:
            origin = (0.3, 0.3, 0.3) if kind == "pbd_rollout" else (0.004, 0.004, 0.004)
            got["x"] = block(*d, s, 0.1, origin, gen)
    n = got["x"].shape[0]
    got["v"] = 0.05 * torch.randn((n, 3), device=DEV, generator=gen)
    if kind in ("frame", "batched", "modules"):  # on its way to the floor: there within an episode
        got["v"][:, 1] -= 0.3
    if kind == "bar":  # falling, with bond stretches well below the fracture limit
        got["v"] *= 0.1
        got["v"][:, 1] -= 0.1
    if kind in ("bar", "pd_rollout"):
        got["bulk"] = 0.8e4 + 0.4e4 * torch.rand(n, device=DEV, generator=gen)
    if kind == "plastic":  # a shear flow
        y = got["x"][:, 1]
        got["v"][:, 0] += 0.5 * (y - y.mean()) / (y.max() - y.mean())
    if kind == "bar":  # the first x layer clamped, the last one pulled along x
        layer = case["ny"] * case["nz"]
        ids = torch.cat([torch.arange(layer, device=DEV), torch.arange(n - layer, n, device=DEV)])
        pull = torch.zeros((2 * layer, 3), device=DEV)
        pull[layer:, 0] = 0.05
        got["ids"], got["pull"] = ids.to(torch.int32), pull
        base = got["x"][ids]
        got["targets"] = [base + pull * (case["dt"] * (k + 1)) for k in range(EPISODE)]
    if kind in ("pd_rollout", "pbd_rollout"):
        got["target"] = got["x"] + 0.01 * s * torch.randn((n, 3), device=DEV, generator=gen)
    return got


def pbd_of(case):
    sweeps = 1 if case["kind"] == "plastic" else case["iterations"]
    return pkhot.pbd_params(radius_of(case), case["spacing"], REST_DENSITY, sweeps, case["dt"])


def yield_limits():
    phi = 60.0 / 180.0
    return (6.0 * 1e-4 * math.cos(phi) / (3.0 + math.sin(phi)) / math.sqrt(3.0),
            2.0 * math.sin(phi) / (3.0 + math.sin(phi)) / math.sqrt(3.0))


def prepare(case, seed):
    st = inputs(case, seed)
    st.pop("scene", None)
    kind, h = case["kind"], radius_of(case)
    lo, hi = bounds_of(case)
    ctx = pkhot.Context(0)
    st.update(case=case, ctx=ctx, h=h, lo=lo, hi=hi, passes=0, pbd=pbd_of(case))
    st["x0"], st["v0"] = st["x"].clone(), st["v"].clone()
    n = st["x"].shape[0]
    if kind in ("frame", "batched", "modules"):
        ctx.boundary_set_box(lo, hi, 0.005, True)
        st["rho"] = torch.empty(n, device=DEV)
    if not is_solid(case):
        st["params"] = pkhot.pbf_params(pkhot.nq_params(h, lo, hi, case["cap"]), st["pbd"], GRAVITY,
                                        boundary=kind != "pbd_rollout", viscosity=case["viscosity"])
    else:
        set_rest_shape(st)
    if kind == "query":
        st["list"] = torch.zeros(n * (case["cap"] or 96), dtype=torch.int32, device=DEV)
    if kind == "plastic":
        st["ones"] = torch.ones(n, device=DEV)
        st["A"], st["B"] = yield_limits()
    if kind == "pd_rollout":
        st["settings"] = pk_torch.RolloutSettings(horizon=h, mu=MU, lam=LAM, iterations=case["iterations"],
                                                  dt=case["dt"], steps=case["steps"],
                                                  checkpoint_every=case["every"])
    return st


def set_rest_shape(st):
    case, ctx = st["case"], st["ctx"]
    idx, el, tot = ctx.nq_build(st["x0"], st["h"], st["lo"], st["hi"], case["cap"])
    ctx.pd_init(st["x0"], idx, el, case["cap"], tot, st["h"])
    if "bulk" in st:
        ctx.pd_set_bulk(st["bulk"])


# ------------------------------------------------------------------- runs

def run(st):
    kind = st["case"]["kind"]
    if kind in ("pd_rollout", "pbd_rollout"):
        return RUNS[kind](st)
    k = st["passes"] % EPISODE
    st["passes"] += 1
    if k == 0 and st["passes"] > 1:
        st["x"].copy_(st["x0"])
        st["v"].copy_(st["v0"])
        if kind == "plastic":
            set_rest_shape(st)
    return RUNS[kind](st, k)


def run_frame(st, k):
    st["ctx"].pbf_step(st["x"], st["v"], st["params"], st["rho"])
    return {"x": st["x"], "v": st["v"], "rho": st["rho"]}


def run_batched(st, k):
    st["ctx"].pbf_step_batched(st["x"], st["v"], st["offsets"], st["params"], st["rho"])
    return {"x": st["x"], "v": st["v"], "rho": st["rho"]}


def run_modules(st, k):
    ctx, x, v, case = st["ctx"], st["x"], st["v"], st["case"]
    ctx.boundary_constrain(x, v, case["dt"])
    idx, el, tot = ctx.nq_build(x, st["h"], st["lo"], st["hi"], case["cap"])
    ctx.integrate(x, v, GRAVITY, case["dt"])
    ctx.pbd_solve(x, v, idx, el, case["cap"], tot, st["pbd"], st["rho"])
    ctx.viscosity(x, v, idx, el, case["cap"], tot, case["viscosity"], st["h"], 5, case["dt"])
    return {"x": x, "v": v, "rho": st["rho"]}


def run_query(st, k):
    ctx, x, case = st["ctx"], st["x"], st["case"]
    idx, el, tot = ctx.nq_build(x, st["h"], st["lo"], st["hi"], case["cap"])
    rho = ctx.summation_density(x, idx, el, case["cap"], tot, st["pbd"])
    st["list"][:tot].copy_(el)  # the application's own list, with room for a denser state
    return {"index": idx, "elements": st["list"], "rho": rho}


def run_bar(st, k):
    ctx, x, v, case = st["ctx"], st["x"], st["v"], st["case"]
    ctx.integrate(x, v, GRAVITY, case["dt"])
    ctx.fixed_points(x, v, st["ids"], st["targets"][k], st["pull"])
    ctx.pd_solve(x, v, st["h"], MU, LAM, case["iterations"], case["dt"], case["break_stretch"])
    ctx.fixed_points(x, v, st["ids"], st["targets"][k], st["pull"])
    return {"x": x, "v": v}


def run_plastic(st, k):
    ctx, x, v, h, dt = st["ctx"], st["x"], st["v"], st["h"], st["case"]["dt"]
    ctx.integrate(x, v, GRAVITY, dt)
    idx, el, tot = ctx.nq_build(x, h, st["lo"], st["hi"], 0)
    ctx.pd_begin(x, h, MU, LAM, dt)
    ctx.pd_compute_inverse_k(h)
    for _ in range(st["case"]["iterations"]):
        ctx.pd_enforce(x, h, MU, LAM, dt)
        ctx.pbd_solve(x, v, idx, el, 0, tot, st["pbd"])
    ctx.pd_update_velocity(x, v, dt)
    idx, el, tot = ctx.nq_build(x, h, st["lo"], st["hi"], 0)
    ctx.pd_rotate_rest_shape(x, h)
    ctx.pd_set_bulk(st["ones"])
    ctx.pd_apply_yielding(x, h, st["A"], st["B"], MU, LAM)
    ctx.pd_reconstruct_rest_shape(x, idx, el, 0, tot, h, False)
    ctx.viscosity(x, v, idx, el, 0, tot, 1.0, h, 5, dt)
    y1, y2, i1 = ctx.pd_get_yield(x.shape[0])
    return {"x": x, "v": v, "y1": y1, "y2": y2, "i1": i1}


def run_pd_rollout(st):
    x0, v0, bulk = (st[k].detach().requires_grad_() for k in ("x", "v", "bulk"))
    xt = pk_torch.pd_rollout(x0, v0, bulk, st["ctx"], st["settings"])
    loss = (xt - st["target"]).square().sum() / xt.shape[0]
    loss.backward()
    return {"x": xt.detach(), "gx": x0.grad, "gv": v0.grad, "gb": bulk.grad}


def run_pbd_rollout(st):
    x0, v0 = (st[k].detach().requires_grad_() for k in ("x", "v"))
    case = st["case"]
    xt, vt = pk_torch.pbd_rollout(x0, v0, st["ctx"], st["params"], case["steps"], case["every"])
    loss = (xt - st["target"]).square().sum() / xt.shape[0]
    loss.backward()
    return {"x": xt.detach(), "v": vt.detach(), "gx": x0.grad, "gv": v0.grad}


RUNS = {"frame": run_frame, "batched": run_batched, "modules": run_modules, "query": run_query, "bar": run_bar,
        "plastic": run_plastic, "pd_rollout": run_pd_rollout, "pbd_rollout": run_pbd_rollout}


# ------------------------------------------------- the work and tolerances

def particles(case):
    if case["kind"] != "batched":
        return case["nx"] * case["ny"] * case["nz"]
    span = math.log(case["n_max"] / case["n_min"])
    return case["scenes"] * (case["n_max"] - case["n_min"]) / max(span, 1e-9)


def work(case):
    """Bytes: state read and written once, rest shape or list once.  Flops:
    distance tests of the candidates inside the sphere's cells, and the pair
    terms of every sweep."""
    n, kind = particles(case), case["kind"]
    if is_solid(case):
        bonds = 93.0 if case["cap"] == 0 else min(case["cap"], 93.0)
        project = n * bonds * 120.0 * case["iterations"]
        rest = n * (16.0 * bonds + 40.0)  # the bond list, its rest positions, K^-1 and stiffness
        if kind == "bar":
            return {"bytes": 48.0 * n + rest, "flops": project}
        if kind == "plastic":
            pairs = n * 113.0
            return {"bytes": 48.0 * n + 2.0 * rest, "flops": project + pairs * (10 * 45.0 + 5 * 20.0 + 200.0)}
        steps = case["steps"]
        return {"bytes": 84.0 * n + rest, "flops": project * steps * 5.0}
    pairs = n * 65.0
    search = n * 65.0 * 10.0
    solve = pairs * 45.0 * case["iterations"]
    visc = pairs * 20.0 * 5 if case["viscosity"] > 0 else 0.0
    if kind == "query":
        return {"bytes": n * (12.0 + 4.0 + 4.0) + pairs * 4.0, "flops": search + pairs * 15.0}
    if kind == "modules":
        return {"bytes": 52.0 * n + pairs * 4.0, "flops": search + solve + visc}
    if kind == "pbd_rollout":
        return {"bytes": 72.0 * n, "flops": case["steps"] * (2 * (search + solve) + 3.0 * solve)}
    return {"bytes": 52.0 * n, "flops": search + solve + visc}


def tolerance(case):
    return TOLERANCE[case["kind"]]


# About four times what float32 differs by from `exact` over these ranges.  The
# velocities set it: displacements over dt of positions rounded to float32.
TOLERANCE = {
    "frame": {"rel": 5e-4, "max": 4e-3},
    "batched": {"rel": 1.2e-4, "max": 5e-3},
    "modules": {"rel": 2e-4, "max": 1.5e-3},
    "query": {"rel": 6e-7, "max": 3e-6, "differ": 0.0},  # the list itself is exact
    "bar": {"rel": 1.2e-3, "max": 0.3},  # a bond at the fracture limit breaks or not
    "plastic": {"rel": 5e-4, "max": 4e-3},
    "pd_rollout": {"rel": 3e-4, "max": 1.2e-3},
    # the clamp of lambda and the cap decide differently where a value is at their edge
    "pbd_rollout": {"rel": 8e-3, "max": 0.6},
}


# ------------------------------------------------- double precision, torch

def neighbours(x, h, cap, scene=None, chunk=1 << 18):
    """Pairs (i, j), |x_i - x_j| < h with the distance rounded in float32 as the
    query rounds it; with cap > 0 the `cap` nearest of each particle (itself
    among them).  A list of (i, j) chunks over consecutive i."""
    n = x.shape[0]
    lo = x.min(0).values.double() - 1e-9
    c = ((x.double() - lo) / (1.000001 * h)).floor().long()
    nx, ny, nz = (c.max(0).values + 1).tolist()
    key = (c[:, 2] * ny + c[:, 1]) * nx + c[:, 0]
    nkeys = nx * ny * nz
    if scene is not None:
        key = key + scene * nkeys
        nkeys *= int(scene.max()) + 1
    order = torch.argsort(key, stable=True)
    start = torch.zeros(nkeys + 1, dtype=torch.long, device=x.device)
    count = torch.bincount(key, minlength=nkeys)
    start[1:] = count.cumsum(0)
    most = int(count.max())
    h32 = torch.tensor(h, dtype=torch.float32, device=x.device)
    got = []
    for a in range(0, n, chunk):
        ids = torch.arange(a, min(a + chunk, n), device=x.device)
        xi, ci, ki = x[ids], c[ids], key[ids]
        found = []
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    cc = ci + torch.tensor([dx, dy, dz], device=x.device)
                    ok = ((cc >= 0) & (cc < torch.tensor([nx, ny, nz], device=x.device))).all(1)
                    k = (ki + (dz * ny + dy) * nx + dx).clamp(0, nkeys - 1)
                    s, e = start[k], torch.where(ok, start[k + 1], start[k])
                    for t in range(most):
                        j = order[(s + t).clamp(max=n - 1)]
                        d = xi - x[j]
                        dd = d.double()
                        d2 = (dd[:, 0] * dd[:, 0] + (d[:, 1] * d[:, 1]).double()).float()
                        d2 = (dd[:, 2] * dd[:, 2] + d2.double()).float()
                        hit = ((s + t < e) & (d2.double().sqrt().float() < h32)).nonzero()[:, 0]
                        if hit.numel():
                            found.append((ids[hit], j[hit], d2[hit]))
        i, j, d2 = (torch.cat(p) for p in zip(*found))
        at = torch.argsort((i - a) * (1 << 32) + d2.view(torch.int32).long())
        i, j = i[at], j[at]
        if cap > 0:
            per = torch.bincount(i - a, minlength=ids.numel())
            first = per.cumsum(0) - per
            keep = torch.arange(i.numel(), device=x.device) - first[i - a] < cap
            i, j = i[keep], j[keep]
        got.append((i, j))
    return got


def sums(n, lists, term, width):
    """sum over the pairs of term(i, j) at i: (n, width)."""
    out = torch.zeros((n, width), dtype=torch.float64, device=DEV)
    for i, j in lists:
        out = out.index_add(0, i, term(i, j))
    return out


def scaled_mass(case):
    """SummationDensity's mass: a lattice of the sampling distance gets the rest density."""
    d, h = case["spacing"], radius_of(case)
    half, total = int(h / d + 1.0), 0.0
    for a in range(-half, half + 1):
        for b in range(-half, half + 1):
            for c in range(-half, half + 1):
                q = math.sqrt(a * a + b * b + c * c) * d / h
                if q <= 1.0:
                    total += d ** 3 * 15.0 / (math.pi * h ** 3) * (1.0 - q) ** 3
    return REST_DENSITY * d ** 3 / total


def pair_geometry(x, i, j):
    d = x[i] - x[j]
    r2 = d.square().sum(1)
    apart = r2 > 1e-12
    r = torch.where(apart, r2, torch.ones_like(r2)).sqrt()
    return d, torch.where(apart, r, torch.zeros_like(r)), apart


def density_of(case, x, lists):
    h, m = radius_of(case), scaled_mass(case)

    def term(i, j):
        _, r, _ = pair_geometry(x, i, j)
        return (m * 15.0 / (math.pi * h ** 3) * (1.0 - r / h).clamp(min=0.0) ** 3)[:, None]

    return sums(x.shape[0], lists, term, 1)[:, 0]


def pbd_sweep(case, x, lists):
    """One DensityPBD iteration: (positions, density)."""
    h, m, n = radius_of(case), scaled_mass(case), x.shape[0]
    cw, cg = 15.0 / (math.pi * h ** 3), -45.0 / (math.pi * h ** 3)

    def gradient(i, j):
        d, r, apart = pair_geometry(x, i, j)
        q = (1.0 - r / h).clamp(min=0.0)
        g = torch.where(apart, cg * q * q, torch.zeros_like(q))
        return d / torch.where(apart, r, torch.ones_like(r))[:, None], q, g

    def term(i, j):
        u, q, g = gradient(i, j)
        return torch.cat([(m * cw * q ** 3)[:, None], (g * g)[:, None], g[:, None] * u], 1)

    s = sums(n, lists, term, 5)
    rho = s[:, 0]
    lam = -(rho - 1000.0) / (s[:, 1] + s[:, 2:].square().sum(1) + 0.1)
    lam = lam.clamp(max=0.0)
    move = torch.zeros((n, 3), dtype=torch.float64, device=DEV)
    for i, j in lists:
        u, _, g = gradient(i, j)
        p = 10.0 * ((lam[i] + lam[j]) * g)[:, None] * u
        move = move.index_add(0, i, p).index_add(0, j, -p)
    return x + move, rho


def viscosity_of(case, x, v, lists, strength):
    h, dt = radius_of(case), case["dt"]
    b, old, n = dt * strength / h, v, x.shape[0]

    def term(i, j):
        _, r, apart = pair_geometry(x, i, j)
        w = torch.where(apart, 45.0 / (13.0 * math.pi * h ** 3) * (1.0 - r / h).clamp(min=0.0), torch.zeros_like(r))
        return torch.cat([w[:, None], w[:, None] * v[j]], 1)

    for _ in range(5):
        s = sums(n, lists, term, 4)
        alone = s[:, :1] < 1e-6
        bb = torch.where(alone, torch.zeros_like(s[:, :1]), torch.full_like(s[:, :1], b))
        w = torch.where(alone, torch.ones_like(s[:, :1]), s[:, :1])
        v = old / (1.0 + bb) + s[:, 1:] / w * bb / (1.0 + bb)
    return v


def gravity64():
    return torch.tensor(GRAVITY, dtype=torch.float64, device=DEV)


def exact_fluid(case, seed):
    got = inputs(case, seed)
    x32, dt = got["x"], case["dt"]
    lists = neighbours(x32, radius_of(case), case["cap"], got.get("scene"))
    if case["kind"] == "query":
        return {"index": None, "elements": None, "rho": density_of(case, x32.double(), lists)}
    # no particle of a first state touches the box's walls
    v = got["v"].double() + dt * gravity64()
    y0 = x32.double() + dt * v
    x, rho = y0, None
    for _ in range(case["iterations"]):
        x, rho = pbd_sweep(case, x, lists)
    v = v + (x - y0) / dt
    if case["viscosity"] > 0:
        v = viscosity_of(case, x, v, lists, case["viscosity"])
    return {"x": x, "v": v, "rho": rho}


def rest_shape(case, x32):
    """Bonds (i, j), rest vectors e = rest_i - rest_j and K^-1 of every particle."""
    h = radius_of(case)
    i, j = (torch.cat(p) for p in zip(*neighbours(x32, h, case["cap"])))
    other = i != j
    i, j = i[other], j[other]
    rest = x32.double()
    e = rest[i] - rest[j]
    r = e.norm(dim=1)
    q = r / h
    w = q ** 3 * (1.0 - q * q).clamp(min=0.0)
    n = x32.shape[0]
    k = torch.zeros((n, 9), dtype=torch.float64, device=DEV)
    k = k.index_add(0, i, ((e / h)[:, :, None] * (e / h)[:, None, :] * w[:, None, None]).reshape(-1, 9))
    tw = torch.zeros(n, dtype=torch.float64, device=DEV).index_add(0, i, w)
    k = (k / torch.where(tw > 1e-6, tw, torch.ones_like(tw))[:, None]).reshape(n, 3, 3)
    val, vec = (torch.cat(p) for p in zip(*(torch.linalg.eigh(part) for part in k.split(4096))))
    val = torch.where(val.abs() > 1e-4 * h, 1.0 / val.abs(), torch.ones_like(val))
    return {"i": i, "j": j, "e": e, "r": r, "w": w, "wrr": q * (1.0 - q * q).clamp(min=0.0) / h ** 2, "tw": tw,
            "k": vec @ (val[:, :, None] * vec.transpose(1, 2)), "alive": torch.ones_like(r)}


def unit(u):
    l2 = u.square().sum(1, keepdim=True)
    ok = l2 > 1e-12
    return torch.where(ok, u / torch.where(ok, l2, torch.ones_like(l2)).sqrt(), torch.zeros_like(u))


def project(case, shape, x, x_old, bulk, tw):
    """One ElasticityModule projection iteration about x_old."""
    h, n = radius_of(case), x.shape[0]
    i, j, e, r = shape["i"], shape["j"], shape["e"], shape["r"]
    w = shape["w"] * shape["alive"]
    p = (x[j] - x[i]) / h
    outer = (p[:, :, None] * (-e / h)[:, None, :] * w[:, None, None]).reshape(-1, 9)
    f = torch.zeros((n, 9), dtype=torch.float64, device=DEV).index_add(0, i, outer)
    f = (f / tw[:, None]).reshape(n, 3, 3) @ shape["k"]
    flat = (torch.linalg.det(f) < -0.001)[:, None, None]
    f = torch.where(flat, torch.eye(3, dtype=torch.float64, device=DEV), f)
    d = x[j] - x[i]
    weight = bulk[i] * shape["wrr"] * shape["alive"] * (r > 0.01 * h)
    nf = unit((f[i] @ e[:, :, None])[:, :, 0])
    t = weight[:, None] * (MU * (d + r[:, None] * nf) + LAM * (d + r[:, None] * unit(-d)))
    ws = ((MU + LAM) * weight)[:, None]
    total = torch.zeros((n, 4), dtype=torch.float64, device=DEV)
    total = total.index_add(0, i, torch.cat([t, ws], 1)).index_add(0, j, torch.cat([-t, ws], 1))
    return x + ((x_old - x) + total[:, :3]) / (1.0 + total[:, 3:])


def weight_sums(shape):
    tw = torch.zeros_like(shape["tw"]).index_add(0, shape["i"], shape["w"] * shape["alive"])
    return torch.where(tw > 1e-6, tw, torch.ones_like(tw))


def exact_bar(case, seed):
    got = inputs(case, seed)
    dt, ids = case["dt"], got["ids"].long()
    shape = rest_shape(case, got["x"])
    v = got["v"].double() + dt * gravity64()
    x = got["x"].double() + dt * v
    x[ids], v[ids] = got["targets"][0].double(), got["pull"].double()
    if case["break_stretch"] > 0:
        length = (x[shape["i"]] - x[shape["j"]]).norm(dim=1)
        shape["alive"] = (length <= (1.0 + case["break_stretch"]) * shape["r"]).double()
    x_old, tw = x, weight_sums(shape)
    for _ in range(case["iterations"]):
        x = project(case, shape, x, x_old, got["bulk"].double(), tw)
    v = v + (x - x_old) / dt
    x, v = x.clone(), v.clone()
    x[ids], v[ids] = got["targets"][0].double(), got["pull"].double()
    return {"x": x, "v": v}


def exact_plastic(case, seed):
    """The elastic part: plasticity moves the rest shape of the frames that follow."""
    got = inputs(case, seed)
    dt, h = case["dt"], radius_of(case)
    shape = rest_shape(case, got["x"])
    v = got["v"].double() + dt * gravity64()
    x = got["x"].double() + dt * v
    lists = neighbours(x.float(), h, 0)
    ones, tw, x_old = torch.ones(x.shape[0], dtype=torch.float64, device=DEV), weight_sums(shape), x
    for _ in range(case["iterations"]):
        x = project(case, shape, x, x_old, ones, tw)
        y, _ = pbd_sweep(case, x, lists)
        v = v + (y - x) / dt
        x = y
    v = v + (x - x_old) / dt
    v = viscosity_of(case, x, v, neighbours(x.float(), h, 0), 1.0)
    return {"x": x, "v": v, "y1": None, "y2": None, "i1": None}


def exact_pd_rollout(case, seed):
    got = inputs(case, seed)
    dt = case["dt"]
    shape = rest_shape(case, got["x"])
    tw = weight_sums(shape)
    x0, v0, bulk = (got[k].double().requires_grad_() for k in ("x", "v", "bulk"))

    def step(x, v, b):
        v = v + dt * gravity64()
        y = x_old = x + dt * v
        for _ in range(case["iterations"]):
            y = checkpoint(project, case, shape, y, x_old, b, tw, use_reentrant=False)
        return y, v + (y - x_old) / dt

    x, v = x0, v0
    for _ in range(case["steps"]):
        x, v = step(x, v, bulk)
    ((x - got["target"].double()).square().sum() / x.shape[0]).backward()
    return {"x": x.detach(), "gx": x0.grad, "gv": v0.grad, "gb": bulk.grad}


def exact_pbd_rollout(case, seed):
    got = inputs(case, seed)
    dt = case["dt"]
    x0, v0 = (got[k].double().requires_grad_() for k in ("x", "v"))
    x, v = x0, v0
    for _ in range(case["steps"]):
        lists = neighbours(x.detach().float(), radius_of(case), case["cap"])
        v = v + dt * gravity64()
        y = y0 = x + dt * v
        for _ in range(case["iterations"]):
            y, _ = checkpoint(pbd_sweep, case, y, lists, use_reentrant=False)
        x, v = y, v + (y - y0) / dt
    ((x - got["target"].double()).square().sum() / x.shape[0]).backward()
    return {"x": x.detach(), "v": v.detach(), "gx": x0.grad, "gv": v0.grad}


def exact(case, seed):
    kind = case["kind"]
    if kind == "bar":
        return exact_bar(case, seed)
    if kind == "plastic":
        return exact_plastic(case, seed)
    if kind == "pd_rollout":
        return exact_pd_rollout(case, seed)
    if kind == "pbd_rollout":
        return exact_pbd_rollout(case, seed)
    return exact_fluid(case, seed)
