"""The work a user has the solver do, as cases that can be timed and compared.

Every case is one frame of a simulation (a few time steps through the public
entry points, then the readback a program does with it) or one training step
of the differentiable rollout.  The scenes are dam breaks in the unit box, as
in `sph2s_final_gb300.scenes`: a fluid lattice with seeded jitter beside the
five-layer boundary shell, support h = 2 spacings, the same constants, and a
time step in the same proportion to the spacing.

  single         Solver: one scene, symplectic Euler or XSPH
  two_scale      Solver2: coarse block with a refined slab, or the coupled
                 mode with two fixed populations
  batch          Batch: many independent scenes stepped together
  rollout        DensityFieldLoss: rollout, density loss, gradients
  batch_rollout  Batch.rollout_*: the same for every scene of a batch

`exact` restates one frame in 64 bits with plain torch: neighbours from a hash
of its own, the pair sums written out, gradients from torch.autograd.
"""
from __future__ import annotations

import math

import numpy as np
import torch

REST, BULK, VISC, SOUND, TENSION, XSPH_EPS = 1000.0, 30.0, 5.0, 88.1472, 0.8, 0.25
GRAVITY = -9.81
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def listed():
    return [
        # the smallest call: a preview scene shown after every step, where latency counts
        {"name": "single-4k", "kind": "single", "nx": 16, "ny": 16, "nz": 16, "inv": 32,
         "steps": 1, "xsph": False, "read": "positions"},
        # the 32,768-particle dam break, ten steps to a frame, every field read back
        {"name": "single-32k", "kind": "single", "nx": 32, "ny": 32, "nz": 32, "inv": 64,
         "steps": 10, "xsph": False, "read": "all"},
        # a block with no even side in a box that is no power of two of cells
        {"name": "single-odd-155k", "kind": "single", "nx": 61, "ny": 53, "nz": 48, "inv": 107,
         "steps": 4, "xsph": False, "read": "all"},
        # the XSPH integrator, a third pass over the neighbours
        {"name": "xsph-65k", "kind": "single", "nx": 32, "ny": 64, "nz": 32, "inv": 64,
         "steps": 4, "xsph": True, "read": "all"},
        # the headline scene: 128^3 particles, shown after every step
        {"name": "single-2m", "kind": "single", "nx": 128, "ny": 128, "nz": 128, "inv": 256,
         "steps": 1, "xsph": False, "read": "positions"},
        # a small refined scene, where one coarse particle's fine neighbours set the latency
        {"name": "two-scale-14k", "kind": "two_scale", "k": 24, "inv": 48, "i0": 15, "i1": 21,
         "coupled": False, "steps": 1},
        # two fixed populations side by side (the coupled project's step)
        {"name": "coupled-80k", "kind": "two_scale", "k": 43, "inv": 86, "i0": 23, "i1": 43,
         "coupled": True, "steps": 1},
        # the refined dam break: 262,144 coarse sites, 0.3 of them refined eightfold
        {"name": "two-scale-262k", "kind": "two_scale", "k": 64, "inv": 128, "i0": 45, "i1": 64,
         "coupled": False, "steps": 1},
        # a sweep over a few small scenes
        {"name": "batch-16", "kind": "batch", "scenes": 16, "n_min": 4096, "n_max": 8192,
         "steps": 20},
        # a sweep over the whole range of scene sizes, read back after a hundred steps
        {"name": "batch-32", "kind": "batch", "scenes": 32, "n_min": 4096, "n_max": 131072,
         "steps": 100},
        # one training step of the differentiable rollout
        {"name": "rollout-65k", "kind": "rollout", "nx": 32, "ny": 64, "nz": 32, "inv": 64,
         "steps": 20, "every": 10, "nodes": 32},
        # one training step for every scene of a batch
        {"name": "batch-rollout-8", "kind": "batch_rollout", "scenes": 8, "n_min": 4096,
         "n_max": 32768, "steps": 10, "every": 5, "nodes": 16},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _block(rng, n):
    """Block sides of about n particles in all, up to 1.6 to 1, and a box that holds them."""
    k = n ** (1.0 / 3.0)
    fx, fy = rng.uniform(0.75, 1.3), rng.uniform(0.75, 1.3)
    d = [max(6, round(k * fx)), max(6, round(k * fy)), max(6, round(k / (fx * fy)))]
    return d[0], d[1], d[2], round(max(d) * rng.uniform(1.3, 2.2))


def draw(rng):
    kind = rng.choice(["single", "single", "single", "two_scale", "two_scale", "batch",
                       "rollout", "batch_rollout"])
    if kind == "single":
        n = _log(rng, 600, 1.2e6)
        nx, ny, nz, inv = _block(rng, n)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "inv": inv,
                "steps": rng.randint(1, 10) if n < 2e5 else 1, "xsph": rng.random() < 0.25,
                "read": rng.choice(["positions", "all"])}
    if kind == "two_scale":
        k = round(_log(rng, 12, 60))
        i0 = rng.randint(round(0.55 * k), round(0.8 * k))
        return {"kind": kind, "k": k, "inv": round(k * rng.uniform(1.5, 2.2)), "i0": i0,
                "i1": min(k, i0 + rng.randint(3, max(3, round(0.3 * k)))),
                "coupled": rng.random() < 0.3, "steps": 1}
    if kind == "batch":
        lo = _log(rng, 1000, 16000)
        return {"kind": kind, "scenes": rng.randint(2, 30), "n_min": round(lo),
                "n_max": round(lo * rng.uniform(1.2, 4.0)), "steps": rng.randint(4, 20)}
    if kind == "rollout":
        nx, ny, nz, inv = _block(rng, _log(rng, 1000, 60000))
        t = rng.randint(6, 20)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "inv": inv, "steps": t,
                "every": rng.randint(3, t), "nodes": rng.randint(12, 32)}
    lo = _log(rng, 1000, 12000)
    return {"kind": kind, "scenes": rng.randint(2, 8), "n_min": round(lo),
            "n_max": round(lo * rng.uniform(1.2, 3.0)), "steps": rng.randint(4, 10),
            "every": rng.randint(2, 6), "nodes": rng.randint(10, 20)}


# ---- scenes ---------------------------------------------------------------

def _lattice(dims, step):
    z, y, x = np.meshgrid(*(np.arange(d, dtype=np.float64) for d in dims[::-1]), indexing="ij")
    return np.stack([x.ravel(), y.ravel(), z.ravel()], 1) * step


def _shell(inv, s, border=5):
    """The lattice points of the box grown by `border` layers that lie outside the box."""
    a = np.arange(-border, inv + border)
    out = (a < 0) | (a >= inv)
    keep = out[:, None, None] | out[None, :, None] | out[None, None, :]
    z, y, x = np.nonzero(keep)
    return np.ascontiguousarray((np.stack([x, y, z], 1) - border).astype(np.float32)
                                * np.float32(s))


def _scene(dims, inv, rng, visc=VISC, bulk=BULK):
    """A dam break as plain arrays and numbers, each number what the configuration holds."""
    s = float(np.float32(1.0 / inv))
    x = _lattice(dims, s)
    x = (x + rng.uniform(-0.01 * s, 0.01 * s, x.shape)).astype(np.float32)
    v = rng.normal(0.0, 0.1, x.shape).astype(np.float32)
    f = np.float32
    return {"x": x, "v": v, "s": s, "h": float(f(2.0 * s)), "m": float(f(REST * s ** 3)),
            "mu": float(f(visc)), "K": float(f(bulk)), "inv": inv,
            "dt": float(f(min(1e-4, 6.4e-3 * s)))}


def _config(sc):
    from sph2s_final_gb300.solver import Grid, SolverConfiguration
    grid = Grid.make_grid((0.0, 0.0, 0.0), (1.0, 1.0, 1.0), sc["h"])
    return SolverConfiguration.direct(sc["h"], sc["m"], REST, sc["K"], sc["mu"], SOUND, TENSION,
                                      grid, epsilon=XSPH_EPS)


def _block_scene(case, seed):
    return _scene((case["nx"], case["ny"], case["nz"]), case["inv"],
                  np.random.default_rng(seed))


def _batch_sides(case):
    """Lattice side of each scene: sizes spread evenly over the logarithm of the range."""
    S, a, b = case["scenes"], case["n_min"], case["n_max"]
    return [max(4, round((a * (b / a) ** ((i * 7 % S + 0.5) / S)) ** (1 / 3))) for i in range(S)]


def _batch_scenes(case, seed):
    rng = np.random.default_rng(seed)
    out = [_scene((k, k, k), 2 * k, rng, VISC * rng.uniform(0.5, 2), BULK * rng.uniform(0.5, 2))
           for k in _batch_sides(case)]
    dt = min(sc["dt"] for sc in out)
    for sc in out:
        sc["dt"] = dt
    return out


def _two_scale_scene(case, seed):
    """Coarse sites outside the slab [i0, i1) of the lattice, fine ones inside it."""
    rng = np.random.default_rng(seed)
    k, inv, i0, i1 = case["k"], case["inv"], case["i0"], case["i1"]
    s = float(np.float32(1.0 / inv))
    site = _lattice((k, k, k), 1.0)
    low = site[(site[:, 0] < i0) | (site[:, 0] >= i1)] * s
    high = (_lattice((2 * (i1 - i0), 2 * k, 2 * k), 0.5) + [i0, 0, 0]) * s
    f = np.float32
    return {"low": (low + rng.uniform(-0.01 * s, 0.01 * s, low.shape)).astype(f),
            "high": (high + rng.uniform(-0.005 * s, 0.005 * s, high.shape)).astype(f),
            "s": s, "h": float(f(2.0 * s)), "m": float(f(REST * s ** 3)), "inv": inv,
            "lo": (i0 - 0.5) * s, "hi": (i1 - 0.5) * s if i1 < k else 2.0,
            "coupled": case["coupled"], "dt": float(f(min(1e-4, 3.2e-3 * s)))}


def _target(sc, nodes):
    """The density field that a training step is to reach: the block carried on by its velocities."""
    x = torch.as_tensor(sc["x"], device=DEV).double() + 0.1 * torch.as_tensor(
        sc["v"], device=DEV).double()
    return _splat(x, _params(sc, x), _nodes(nodes), nodes).float().cpu().numpy()


def _nodes(n):
    s = float(np.float32(1.0 / n))
    return (torch.as_tensor(_lattice((n, n, n), 1.0), device=DEV) + 0.5) * s


def prepare(case, seed):
    from sph2s_final_gb300.solver import Grid, ParticleData, Solver
    kind = case["kind"]
    if kind in ("single", "rollout"):
        sc = _block_scene(case, seed)
        solver = Solver(ParticleData(sc["x"]), ParticleData(_shell(case["inv"], sc["s"])),
                        _config(sc), None if kind == "rollout" else sc["v"])
        n = solver.num_fluid
        if kind == "single":
            if case["xsph"]:
                solver.set_integrator("xsph")
            out = {"positions": torch.empty((n, 3), device="cuda")}
            if case["read"] == "all":
                out["velocities"] = torch.empty((n, 3), device="cuda")
                out["densities"] = torch.empty(n, device="cuda")
            return {"kind": kind, "solver": solver, "dt": sc["dt"], "steps": case["steps"],
                    "out": out}
        return {"kind": kind, "solver": solver, "dt": sc["dt"], "case": case,
                "v0": torch.from_numpy(sc["v"]).requires_grad_(True),
                "mu": torch.tensor(sc["mu"], requires_grad=True),
                "nodes": Grid.make_grid_dims((0, 0, 0), (case["nodes"],) * 3, 1.0 / case["nodes"]),
                "target": _target(sc, case["nodes"])}
    if kind == "two_scale":
        from sph2s_final_gb300.two_scale import Solver2, SolverConfiguration2
        sc = _two_scale_scene(case, seed)
        grids = [Grid.make_grid((0, 0, 0), (1, 1, 1), float(np.float32(h)))
                 for h in (sc["h"], 0.5 * sc["h"])]
        cfg = SolverConfiguration2.direct(sc["h"], sc["m"], REST, BULK, VISC, SOUND, TENSION,
                                          0.0125, grids[0], grids[1], refine_axis=0,
                                          refine_lo=sc["lo"], refine_hi=sc["hi"])
        cfg.mode = 1 if case["coupled"] else 0
        cap = [2 * len(sc["low"]) + 1024, 8 * len(sc["low"]) + len(sc["high"]) + 1024]
        solver = Solver2(sc["low"], sc["high"], _shell(case["inv"], sc["s"]), cfg, *cap)
        return {"kind": kind, "solver": solver, "dt": sc["dt"], "steps": case["steps"],
                "x": [torch.empty((c, 3), device="cuda") for c in cap],
                "state": [torch.empty(c, dtype=torch.int32, device="cuda") for c in cap]}
    from sph2s_final_gb300.batched import Batch
    scs = _batch_scenes(case, seed)
    batch = Batch([(sc["x"], _shell(sc["inv"], sc["s"]), _config(sc),
                    sc["v"] if kind == "batch" else None) for sc in scs])
    st = {"kind": kind, "solver": batch, "dt": scs[0]["dt"], "steps": case["steps"]}
    if kind == "batch_rollout":
        grid = Grid.make_grid_dims((0, 0, 0), (case["nodes"],) * 3, 1.0 / case["nodes"])
        st.update(v0=[sc["v"] for sc in scs], mu=[sc["mu"] for sc in scs], every=case["every"],
                  nodes=[grid] * len(scs), target=[_target(sc, case["nodes"]) for sc in scs])
    return st


def run(st):
    kind, solver = st["kind"], st["solver"]
    if kind == "single":
        solver.advance(st["dt"], st["steps"])
        for field, out in st["out"].items():
            solver.read_device(field, out.data_ptr(), "by_id")
        return st["out"]
    if kind == "two_scale":
        solver.advance(st["dt"], st["steps"])
        n = solver.counts()
        out = {}
        for r, name in enumerate(("low", "high")):
            solver.read_positions_device(r, st["x"][r].data_ptr())
            solver.read_states_device(r, st["state"][r].data_ptr())
            out[name] = st["x"][r][:n[name]]
            out[name + "_state"] = st["state"][r][:n[name]]
        return out
    if kind == "batch":
        solver.advance(st["dt"], st["steps"])
        frames = [solver.scene(k, "by_id") for k in range(solver.num_scenes)]
        return {"x": [f["x"] for f in frames], "v": [f["v"] for f in frames]}
    if kind == "rollout":
        from sph2s_final_gb300.autograd import DensityFieldLoss
        c = st["case"]
        st["v0"].grad = st["mu"].grad = None
        loss = DensityFieldLoss.apply(st["v0"], st["mu"], solver, st["dt"], c["steps"],
                                      c["every"], st["nodes"], st["target"])
        loss.backward()
        return {"loss": float(loss.detach()), "v0": st["v0"].grad, "mu": st["mu"].grad}
    solver.rollout_forward(st["v0"], st["mu"], st["dt"], st["steps"], st["every"])
    fields, loss = solver.rollout_density_loss(st["nodes"], st["target"])
    gv, gx, gmu = solver.rollout_backward()
    return {"loss": [float(v) for v in loss], "mu": [float(v) for v in gmu], "v0": gv, "x0": gx,
            "field": fields}


def _sizes(case):
    kind = case["kind"]
    if kind in ("single", "rollout"):
        return case["nx"] * case["ny"] * case["nz"]
    if kind == "two_scale":
        return case["k"] ** 2 * (case["k"] + 7 * (case["i1"] - case["i0"]))
    return sum(k ** 3 for k in _batch_sides(case))


def work(case):
    """Positions and velocities in and out once a pass, and what is read back; 33.5 neighbours within h = 2s, of which
    a step's density takes 12 flops each and its force 38 (four times that for gradients)."""
    n, kind = _sizes(case), case["kind"]
    step = 33.5 * 50.0 * (1.5 if case.get("xsph") else 1.0)
    if kind == "two_scale":  # each population meets the other near the slab
        step *= 1.5
    if kind in ("rollout", "batch_rollout"):
        return {"bytes": n * 4.0 * (6 + 6), "flops": n * case["steps"] * 4.0 * step}
    read = {"single": 7 if case.get("read") == "all" else 3, "two_scale": 4, "batch": 6}[kind]
    return {"bytes": n * 4.0 * (6 + 6 + read), "flops": n * case["steps"] * step}


# ---- the same in 64 bits --------------------------------------------------

def _expand(lo, hi):
    """Index pairs (i, j) with lo[i] <= j < hi[i]."""
    c = hi - lo
    i = torch.repeat_interleave(torch.arange(len(c), device=c.device), c)
    first = torch.cumsum(c, 0) - c
    return i, torch.arange(len(i), device=c.device) - (first - lo)[i]


def _pairs(a, b, h, sa=None, sb=None, same=False, chunk=150_000):
    """Pairs (i, j) with |a_i - b_j| < h; `same`: without i = j.  h is a number, or one number a
    scene, with sa and sb the scene of each point."""
    with torch.no_grad():
        ha, hb = (h, h) if sa is None else (h[sa][:, None], h[sb][:, None])
        ca, cb = torch.floor(a / ha).long(), torch.floor(b / hb).long()
        low = torch.minimum(ca.min(0).values, cb.min(0).values) - 1
        D = torch.maximum(ca.max(0).values, cb.max(0).values) - low + 2
        ca, cb = ca - low, cb - low
        ka = (ca[:, 2] * D[1] + ca[:, 1]) * D[0] + ca[:, 0]
        kb = (cb[:, 2] * D[1] + cb[:, 1]) * D[0] + cb[:, 0]
        if sa is not None:
            ka, kb = ka + sa * D.prod(), kb + sb * D.prod()
        kb, order = torch.sort(kb)
        got = []
        for at in range(0, len(a), chunk):
            k = ka[at:at + chunk]
            for dz in (-1, 0, 1):
                for dy in (-1, 0, 1):
                    row = k + (dz * D[1] + dy) * D[0]
                    i, j = _expand(torch.searchsorted(kb, row - 1),
                                   torch.searchsorted(kb, row + 1, right=True))
                    i, j = i + at, order[j]
                    r2 = (a[i] - b[j]).square().sum(1)
                    near = r2 < (h * h if sa is None else (h * h)[sa[i]])
                    if same:
                        near &= i != j
                    got.append(torch.stack([i[near], j[near]]))
        return torch.cat(got, 1)


def _poly6(h):
    return 315.0 / (64.0 * math.pi * h ** 9)


def _spiky(h):
    return 45.0 / (math.pi * h ** 6)


def _sum(n, i, term):
    return torch.zeros((n,) + term.shape[1:], dtype=torch.float64, device=term.device).index_add(
        0, i, term)


def _boundary(x, b, i, j, h, m):
    """Boundary acceleration: 0.02 c^2 shape(2 r / h) / r^2 x_ik, halved by the equal masses."""
    d = x[i] - b[j]
    r2 = d.square().sum(1)
    q = 2.0 * r2.sqrt() / h
    shape = torch.where(q < 2 / 3, torch.full_like(q, 2 / 3),
                        torch.where(q < 1, q * (2 - 1.5 * q), 0.5 * (2 - q) ** 2))
    c = 0.02 * float(np.float32(SOUND)) ** 2 * m / (m + m)
    return _sum(len(x), i, (c * shape / r2)[:, None] * d)


def _params(sc, x, bound=None):
    """Constants of one scene for _step."""
    one = {k: torch.full((1,), sc[k], dtype=torch.float64, device=x.device)
           for k in ("h", "m", "mu", "K")}
    return dict(one, scene=None, b=bound, bscene=None)


def _packed(scs):
    """Positions, velocities and constants of many scenes as one set of points."""
    t = lambda a: torch.as_tensor(np.concatenate(a), device=DEV)  # noqa: E731
    shells = [_shell(sc["inv"], sc["s"]) for sc in scs]
    p = {k: torch.tensor([sc[k] for sc in scs], dtype=torch.float64, device=DEV)
         for k in ("h", "m", "mu", "K")}
    p["scene"] = t([np.full(len(sc["x"]), k) for k, sc in enumerate(scs)])
    p["bscene"] = t([np.full(len(b), k) for k, b in enumerate(shells)])
    p["b"] = t(shells).double()
    return t([sc["x"] for sc in scs]).double(), t([sc["v"] for sc in scs]).double(), p


def _step(x, v, p, dt, xsph=False):
    """One step: (x', v', density at x)."""
    n, S = len(x), p["scene"]
    of = (lambda q, i: q[0]) if S is None else (lambda q, i: q[S[i]])
    h1 = p["h"][0] if S is None else p["h"]
    i, j = _pairs(x.detach(), x.detach(), h1, S, S, same=True)
    own = torch.arange(n, device=x.device)
    h, m, mu, K = (of(p[k], i) for k in ("h", "m", "mu", "K"))
    hi, mi, Ki = (of(p[k], own) for k in ("h", "m", "K"))
    tension = float(np.float32(TENSION))
    d = x[i] - x[j]
    r2 = d.square().sum(1)
    r = r2.sqrt()
    w = _poly6(h) * (h * h - r2) ** 3
    rho = mi * (_poly6(hi) * hi ** 6 + _sum(n, i, w))
    A = Ki * (rho - REST) / rho.square()
    push = m * _spiky(h) * (A[i] + A[j]) * (h - r) ** 2 / r - tension * m * w / rho[i]
    drag = mu * m * _spiky(h) * (h - r) / (rho[i] * rho[j])
    a = _sum(n, i, push[:, None] * d + drag[:, None] * (v[j] - v[i]))
    if p["b"] is not None:
        bi, bj = _pairs(x.detach(), p["b"], h1, S, p["bscene"])
        a = a + _boundary(x, p["b"], bi, bj, of(p["h"], bi), of(p["m"], bi))
    a = a + torch.tensor([0.0, float(np.float32(GRAVITY)), 0.0], dtype=torch.float64,
                         device=x.device)
    v1 = v + dt * a
    if xsph:
        v1 = v1 + XSPH_EPS * _sum(n, i, (m * w / rho[j])[:, None] * (v1[j] - v1[i]))
    return x + dt * v1, v1, rho


def _splat(x, p, nodes, n):
    """Poly6 density of the points on the nodes of each scene, (scenes * nodes) values."""
    S = p["scene"]
    scenes = 1 if S is None else len(p["h"])
    at = nodes.repeat(scenes, 1)
    sn = None if S is None else torch.arange(scenes, device=x.device).repeat_interleave(n ** 3)
    i, j = _pairs(at, x.detach(), p["h"][0] if S is None else p["h"], sn, S)
    h, m = (p["h"][0], p["m"][0]) if S is None else (p["h"][S[j]], p["m"][S[j]])
    w = m * _poly6(h) * (h * h - (at[i] - x[j]).square().sum(1)) ** 3
    return _sum(len(at), i, w)


def _exact_rollout(x, v, p, dt, steps, nodes, target, scenes):
    from torch.utils.checkpoint import checkpoint
    x.requires_grad_(True)
    v.requires_grad_(True)
    p["mu"].requires_grad_(True)
    xt, vt = x, v
    for _ in range(steps):
        xt, vt = checkpoint(lambda a, b: _step(a, b, p, dt)[:2], xt, vt, use_reentrant=False)
    field = _splat(xt, p, _nodes(nodes), nodes).view(scenes, -1)
    t = torch.as_tensor(np.stack(target), device=DEV).double().view(scenes, -1)
    loss = (field - t).square().mean(1)
    loss.sum().backward()
    return loss.detach(), field.detach(), x.grad, v.grad, p["mu"].grad


def _exact_two_scale(sc):
    """One step of both populations, outputs in the sorted order of the step (Morton order of the
    cells, computed in 32 bits as positions are).  Nothing is inside the slab's bounds yet, so
    nothing splits, and every particle keeps its state."""
    b = torch.as_tensor(_shell(sc["inv"], sc["s"]), device=DEV).double()
    h = [sc["h"], float(np.float32(0.5 * sc["h"]))]
    m = [sc["m"], float(np.float32(sc["m"] / 8))]
    x = [torch.as_tensor(sc[k][_morton_order(sc[k], h[r])], device=DEV).double()
         for r, k in enumerate(("low", "high"))]
    tension, dt = float(np.float32(TENSION)), sc["dt"]
    gravity = torch.tensor([0.0, float(np.float32(GRAVITY)), 0.0], dtype=torch.float64, device=DEV)
    W = lambda q, r2: _poly6(h[q]) * torch.clamp(h[q] ** 2 - r2, min=0) ** 3  # noqa: E731
    G = lambda q, r: _spiky(h[q]) * torch.clamp(h[q] - r, min=0) ** 2  # noqa: E731
    same = [_pairs(x[r], x[r], h[r], same=True) for r in (0, 1)]
    mixed = [_pairs(x[r], x[1 - r], h[0]) for r in (0, 1)]
    rho = []
    for r in (0, 1):
        (i, j), (k, l) = same[r], mixed[r]
        q2 = (x[r][i] - x[r][j]).square().sum(1)
        p2 = (x[r][k] - x[1 - r][l]).square().sum(1)
        rho.append(m[r] * (_poly6(h[r]) * h[r] ** 6 + _sum(len(x[r]), i, W(r, q2))) +
                   m[1 - r] * _sum(len(x[r]), k, 0.5 * (W(0, p2) + W(1, p2))))
    A = [BULK * (q - REST) / q.square() for q in rho]
    out = []
    for r in (0, 1):  # at rest: no drag in the first step
        c, n = 1 - r, len(x[r])
        (i, j), (k, l) = same[r], mixed[r]
        d, e = x[r][i] - x[r][j], x[r][k] - x[c][l]
        q2, p2 = d.square().sum(1), e.square().sum(1)
        q, p = q2.sqrt(), p2.sqrt()
        push = m[r] * (A[r][i] + A[r][j]) * G(r, q) / q - tension * m[r] * W(r, q2) / rho[r][i]
        a = _sum(n, i, push[:, None] * d)
        wt = W(c, p2) if sc["coupled"] else 0.5 * (W(0, p2) + W(1, p2))
        push = (m[c] * (A[r][k] + A[c][l]) * 0.5 * (G(0, p) + G(1, p)) / p -
                tension * m[c] * wt / rho[r][k])
        a = a + _sum(n, k, push[:, None] * e)
        bi, bj = _pairs(x[r], b, h[0])
        a = a + _boundary(x[r], b, bi, bj, h[0], m[0]) + gravity
        out.append(x[r] + dt * (dt * a))
    return {"low": out[0], "low_state": None, "high": out[1], "high_state": None}


def _morton_order(x, h):
    dim = int(np.ceil(np.float32(1.0) / np.float32(h)))
    c = np.clip((x / np.float32(h)).astype(np.int64), 0, dim - 1)
    key = np.zeros(len(x), np.int64)
    for bit in range(10):
        for axis in range(3):
            key |= ((c[:, axis] >> bit) & 1) << (3 * bit + axis)
    return np.argsort(key, kind="stable")


def exact(case, seed):
    kind = case["kind"]
    n = _sizes(case)
    if kind == "single":
        if n * case["steps"] > 4e6:
            return None
        sc = _block_scene(case, seed)
        x, v = (torch.as_tensor(sc[k], device=DEV).double() for k in ("x", "v"))
        p = _params(sc, x, torch.as_tensor(_shell(sc["inv"], sc["s"]), device=DEV).double())
        for _ in range(case["steps"]):
            x, v, rho = _step(x, v, p, sc["dt"], case["xsph"])
        out = {"positions": x, "velocities": v, "densities": rho}
        return out if case["read"] == "all" else {"positions": x}
    if kind == "two_scale":
        return _exact_two_scale(_two_scale_scene(case, seed)) if case["steps"] == 1 else None
    if kind == "rollout":
        sc = _block_scene(case, seed)
        x, v = (torch.as_tensor(sc[k], device=DEV).double() for k in ("x", "v"))
        p = _params(sc, x, torch.as_tensor(_shell(sc["inv"], sc["s"]), device=DEV).double())
        loss, _, _, gv, gmu = _exact_rollout(x, v, p, sc["dt"], case["steps"], case["nodes"],
                                             [_target(sc, case["nodes"])], 1)
        return {"loss": loss[0], "v0": gv, "mu": gmu[0]}
    if n * case["steps"] > 4e6:
        return None
    scs = _batch_scenes(case, seed)
    x, v, p = _packed(scs)
    ends = np.cumsum([len(sc["x"]) for sc in scs])[:-1].tolist()
    split = lambda a: list(torch.tensor_split(a, ends))  # noqa: E731
    if kind == "batch":
        for _ in range(case["steps"]):
            x, v, _ = _step(x, v, p, scs[0]["dt"])
        return {"x": split(x), "v": split(v)}
    loss, field, gx, gv, gmu = _exact_rollout(
        x, v, p, scs[0]["dt"], case["steps"], case["nodes"],
        [_target(sc, case["nodes"]) for sc in scs], len(scs))
    return {"loss": list(loss), "mu": list(gmu), "v0": split(gv), "x0": split(gx),
            "field": list(field)}
