"""The work that programs have this framework do, as cases that can be timed and compared.

A case is one pass through the public entry points: a start state put into the particle sets, then some
substeps (one scene, a batch of scenes, a two-phase scene, a scene with the weakly compressible block and
the velocity map) or a differentiable rollout with its gradients.  Scenes are dam breaks in a box of three
boundary layers, as in the benchmark workloads: a lattice block at the particle spacing, its rows sheared
past each other and every particle moved a little, so that cells are unevenly filled and neighbours are
out of lattice order as in a running flow, with velocities of about 1 m/s.

``exact`` restates the substep in 64-bit torch (the reference's kernel sequence, main.py:175-256).
"""
import math
import random

import numpy as np
import torch

DEV = "cuda"


# --------------------------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest call in use: the 5,000-particle 2D dam break, stepped as the time loop does it
        # (the clock, counters and energies read back after every substep)
        _case("loop2d_5k", "step", 2, 50, 100, 1, steps=4, cs=20, loop=True),
        # an ordinary 2D scene, odd sides
        _case("column2d_61k", "step", 2, 175, 351, 1, steps=2, cs=20),
        # the small 3D dam break of an interactive scene
        _case("column3d_8k", "step", 3, 20, 20, 20, steps=4, cs=50),
        # an ordinary 3D scene, ragged sides, at a long time step: the solves iterate past their floor
        _case("column3d_205k", "step", 3, 57, 61, 59, cs=10),
        # the headline dam break: 1M fluid particles in the 3 x 1.5 x 1 m tank
        _case("dambreak3d_1m", "step", 3, 100, 100, 100, cs=50),
        # the same tank at 1 / 160 m
        _case("dambreak3d_4m", "step", 3, 160, 160, 160, cs=50),
        # two-phase mixture (VFSPH, surface tension, volume-fraction update) in 2D, small
        _case("twophase2d_20k", "twophase", 2, 100, 101, 1, steps=2, cs=20),
        # the 2M-particle two-phase pair
        _case("twophase3d_2m", "twophase", 3, 100, 100, 100, cs=50),
        # the weakly compressible block and the particle-to-grid velocity map
        _case("wcsph3d_97k", "wcsph", 3, 46, 46, 46, cs=50),
        # many independent scenes of uneven size in one batch
        _case("batch64", "batch", 3, 2000, 50000, 64, cs=50),
        # gradients of a rollout: the test-sized block and the 99,452-particle one
        _case("rollout3d_2k", "rollout", 3, 13, 12, 13, steps=16, cs=20, every=8),
        _case("rollout3d_99k", "rollout", 3, 46, 46, 47, steps=8, cs=20, every=4),
    ]


def _case(name, kind, dim, a, b, c, steps=1, cs=50, loop=False, every=0):
    return {"name": name, "kind": kind, "dim": dim, "a": a, "b": b, "c": c, "steps": steps, "cs": cs,
            "loop": loop, "every": every}


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _sides(rng, dim, n):
    """Block sides with about n particles and aspect ratios between 1/2 and 2."""
    ax, az = rng.uniform(0.5, 2.0), rng.uniform(0.5, 2.0)
    if dim == 2:
        y = max(3, round((n / ax) ** 0.5))
        return max(3, round(ax * y)), y, 1
    y = max(3, round((n / (ax * az)) ** (1.0 / 3.0)))
    return max(3, round(ax * y)), y, max(3, round(az * y))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "twophase", "wcsph", "batch", "rollout"])
    dim = 3 if kind in ("batch", "rollout") else rng.choice([2, 3, 3])
    cs = 20 if dim == 2 else rng.choice([10, 20, 50])
    if kind == "batch":
        lo = int(_log(rng, 500, 5000))
        return _drawn(kind, dim, lo, int(lo * _log(rng, 2, 20)), rng.randint(2, 64), 1, 50)
    if kind == "rollout":
        a, b, c = _sides(rng, 3, _log(rng, 1000, 100000))
        steps = rng.randint(3, 8)
        return _drawn(kind, dim, a, b, c, steps, 20, every=rng.randint(2, steps))
    top = {"step": 4.0e6 if dim == 3 else 3e5, "twophase": 1.0e6 if dim == 3 else 1e5,
           "wcsph": 5e5 if dim == 3 else 1e5}[kind]
    n = _log(rng, 1500, 0.9 * top)
    a, b, c = _sides(rng, dim, n)
    return _drawn(kind, dim, a, b, c, 2 if n < 30000 else 1, cs, loop=n < 30000 and rng.random() < 0.5)


def _drawn(kind, dim, a, b, c, steps, cs, loop=False, every=0):
    d = _case("", kind, dim, a, b, c, steps, cs, loop, every)
    del d["name"]
    return d


# --------------------------------------------------------------------------------------- inputs
def _spacing(case):
    """Particle spacing: 0.02 m in 2D; in 3D 0.01 m, and finer where a block side would pass 1 m."""
    if case["dim"] == 2:
        return 0.02
    if case["kind"] == "step":
        return 0.01 if max(case["a"], case["b"], case["c"]) <= 100 else 1.0 / max(case["a"], case["b"], case["c"])
    return 0.01


def _tank(case, d, L):
    """Inner box of the scene (upper corner; the lower one is 0)."""
    if case["dim"] == 2:
        return [4 * L[0], 2 * L[1]]
    if case["kind"] == "batch":
        return [2.5 * L[0], 1.5 * L[1], L[2]]
    if case["kind"] == "rollout":
        return [1.6 * L[0], 1.5 * L[1], 1.6 * L[2]]
    x = 2 * L[0] + d if case["kind"] == "twophase" else L[0]
    return [max(3 * L[0], x + 0.5 * L[0]), 1.5 * L[1], L[2]]


def _lattice(sides, d):
    ax = [torch.arange(n, device=DEV, dtype=torch.float64) * d for n in sides]
    return torch.stack(torch.meshgrid(*ax, indexing="ij"), -1).reshape(-1, len(sides))


def _walls(lo, hi, d, layers=3):
    """Lattice points of the box [lo, hi] outside its inner part (three layers)."""
    n = [int((b - a + 1e-7) / d) for a, b in zip(lo, hi)]
    idx = torch.stack(torch.meshgrid(*[torch.arange(k, device=DEV) for k in n], indexing="ij"), -1).reshape(-1, len(n))
    top = torch.tensor(n, device=DEV) - layers
    keep = ((idx < layers) | (idx >= top)).any(1)
    return idx[keep].to(torch.float64) * d + torch.tensor(lo, device=DEV, dtype=torch.float64)


def _scene(case, seed):
    """Config dictionaries and the start state of one scene, from the case and the seed alone."""
    kind, dim = case["kind"], case["dim"]
    rng = random.Random(seed * 7919 + 17)
    gen = torch.Generator(device=DEV).manual_seed(seed * 104729 + 5)
    d = _spacing(case)
    sides = [case["a"], case["b"], case["c"]][:dim]
    L = [n * d for n in sides]
    pos = _lattice(sides, d)
    two = kind == "twophase"
    vf = torch.ones(len(pos), 1, device=DEV, dtype=torch.float64)
    if two:
        shift = torch.zeros(dim, device=DEV, dtype=torch.float64)
        shift[0] = L[0] + d
        first = torch.cat([torch.ones(len(pos)), torch.zeros(len(pos))]).to(DEV, torch.float64)
        pos = torch.cat([pos, pos + shift])
        noise = torch.rand(len(pos), generator=gen, device=DEV, dtype=torch.float64) * 0.1 - 0.05
        v0 = (first + noise).clamp(0, 1).to(torch.float32)
        vf = torch.stack([v0, 1 - v0], 1)
    # rows sheared along x (keeps the density), then a small move of every particle
    k = 2 * math.pi / (8 * d)
    ph = [rng.uniform(0, 2 * math.pi) for _ in range(8)]
    amp = 0.5 * d if kind == "rollout" else 2.0 * d
    pos[:, 0] += amp * (1 + torch.sin(k * pos[:, 1] / 3 + ph[0]))
    if dim == 3:
        pos[:, 0] += amp * (1 + torch.sin(k * pos[:, 2] / 5 + ph[1]))
    pos += (torch.rand(pos.shape, generator=gen, device=DEV, dtype=torch.float64) - 0.5) * (0.1 * d)
    pos = pos.to(torch.float32)
    # a solenoidal field of about 1 m/s and a little noise
    x = pos.to(torch.float64)
    vel = torch.stack([torch.sin(2 * math.pi * x[:, (q + 1) % dim] / L[(q + 1) % dim] + ph[2 + q])
                       for q in range(dim)], 1) * (0.1 if kind == "rollout" else 0.7)
    vel += torch.randn(vel.shape, generator=gen, device=DEV, dtype=torch.float64) * 0.02
    vel = vel.to(torch.float32)
    t = 3.5 * d
    hi = [v + t for v in _tank(case, d, L)]
    lo = [-t] * dim
    if kind in ("step", "wcsph") and dim == 3:
        hi[0] += 6 * d  # the sheared block keeps clear of the far wall
    bpos = _walls(lo, hi, d).to(torch.float32)
    rho = [1000, 500] if two else [rng.uniform(800.0, 1200.0) if kind == "batch" else 1000]
    config = {
        "arch": "gpu", "device_memory_GB": 6, "solver_type": "VFSPH" if two else "DFSPH", "solver_wc_gamma": 7,
        "solver_divergence_threshold": 1e-2, "solver_compression_threshold": 1e-3,
        "solver_iter_threshold_min": 2, "solver_iter_threshold_max": 100, "solver_if_cfl": True,
        "solver_cs": case["cs"], "solver_cfl_factor": 0.5, "solver_neighb_range": 1,
        "solver_neighb_grid_size_TO_global_part_size": 2, "solver_fbm_diffusion_term": 0.0,
        "solver_fbm_convection_term": 50.0 if two else 0.0,
        "solver_surface_tension_gamma": 0.07 if two else 0.0, "gui_res": [1080, 1080], "gui_part_zoomer": 1.0,
        "gui_fps": 30, "gui_canvas_bgcolor": [0.2, 0.2, 0.6], "gui_camera_pos": [6.0, 1.0, 0.0],
        "gui_camera_lookat": [0.0, 0.0, 0.0],
    }
    scenario = {
        "sim_env": {"global_part_size": d, "global_dynamic_viscosity": 0.01, "sim_dim": dim,
                    "sim_space_lb": [v - 10 * d for v in lo],
                    "sim_space_rt": [v + 10 * d + (0.5 * L[1] if q == 1 else 0.0) for q, v in enumerate(hi)],
                    "gravity": [0, -9.81, 0][:dim], "phase_num": len(rho), "phase_rest_density": rho,
                    "phase_color_hex": ["0x6F7DBC", "0xFA8012"][:len(rho)]},
        "fluid": {"max_part_num": len(pos), "objs": []}, "bound": {"max_part_num": len(bpos), "objs": []},
    }
    bvf = torch.zeros(len(bpos), len(rho), device=DEV)
    bvf[:, 0] = 1
    return {"config": config, "scenario": scenario, "d": d, "pos": pos, "vel": vel, "vf": vf.to(torch.float32),
            "bpos": bpos, "bvf": bvf}


def _scenes(case, seed):
    if case["kind"] != "batch":
        return [_scene(case, seed)]
    rng = random.Random(case["a"] + 31 * case["b"])  # the scenes' sizes belong to the case
    out = []
    for s in range(case["c"]):
        a, b, c = _sides(rng, 3, _log(rng, case["a"], case["b"]))
        out.append(_scene(dict(case, a=a, b=b, c=c), seed * 1009 + s))
    return out


def _fill(obj, cfg, pos, vel, vf):
    n = len(pos)
    obj.pos[:n] = pos
    if vel is not None:
        obj.vel[:n] = vel
    obj.volume_frac[:n] = vf
    obj.rest_volume[:n] = float(cfg.part_size[cfg.dim[None]])
    obj.part_num[None] = n
    obj.update_mass_all()


def prepare(case, seed):
    from tichi_sph_gb300 import sph_config
    from tichi_sph_gb300.adjoint import DiffRollout
    from tichi_sph_gb300.batch import BatchSolver, gather_scenes
    from tichi_sph_gb300.simulation import Simulation
    scenes = _scenes(case, seed)
    sims = []
    for sc in scenes:
        cfg = sph_config.Config(sc["config"], sc["scenario"])
        sim = Simulation(cfg, fbm=case["kind"] == "twophase", wcsph=case["kind"] == "wcsph",
                         map_grid=case["kind"] == "wcsph", device=DEV)
        _fill(sim.fluid, cfg, sc["pos"], sc["vel"], sc["vf"])
        _fill(sim.bound, cfg, sc["bpos"], None, sc["bvf"])
        sims.append(sim)
    sim = sims[0]
    st = {"case": case, "sim": sim}
    if case["kind"] == "batch":
        fluid, bound, nf, nb = gather_scenes(sims, device=DEV)
        st.update(sims=sims, fluid=fluid, bound=bound,
                  solver=BatchSolver([s.config for s in sims], fluid, bound, nf, nb))
    elif case["kind"] == "rollout":
        st.update(fluid=sim.fluid, bound=sim.bound)
        st["rollout"] = DiffRollout(sim.config, sim.fluid, sim.bound, case["steps"], checkpoint_every=case["every"],
                                    max_iters=16)
        gen = torch.Generator(device=DEV).manual_seed(seed + 3)
        st["v0"] = sc["vel"].clone().requires_grad_(True)
        st["mu"] = torch.tensor(0.01, requires_grad=True)
        st["seeds"] = _loss_seeds(sc, gen)
    else:
        st.update(fluid=sim.fluid, bound=sim.bound, solver=sim.solver)
    if case["kind"] != "rollout":
        f = st["fluid"]
        st["start"] = {k: getattr(f, k).clone() for k in _restored(case)}
    return st


def _loss_seeds(sc, gen):
    """Gradients of a loss on the final state: the centre of mass, the flow's energy, the density error."""
    vel = sc["vel"]
    n, dim = vel.shape
    gx = torch.full((n, dim), 0.3 / n, device=DEV)
    gv = (vel + 0.05 * torch.randn(n, dim, generator=gen, device=DEV)) / n
    gr = torch.randn(n, generator=gen, device=DEV) * (1e-4 / n)
    return gx, gv, gr


def _restored(case):
    """What a start state consists of (the mixture's fractions and masses change as well)."""
    return ["pos", "vel"] + (["volume_frac", "mass", "rest_density"] if case["kind"] == "twophase" else [])


# --------------------------------------------------------------------------------------- a pass
def run(state):
    case = state["case"]
    if case["kind"] == "rollout":
        v0, mu = state["v0"], state["mu"]
        x, v, rho = state["rollout"](v0, mu)
        gv0, gmu = torch.autograd.grad((x, v, rho), (v0, mu), grad_outputs=state["seeds"])
        return {"pos": x.detach(), "vel": v.detach(), "density": rho.detach(), "grad_v0": gv0, "grad_mu": gmu}
    f, b = state["fluid"], state["bound"]
    for k, t in state["start"].items():
        getattr(f, k).copy_(t)
    solver = state["solver"]
    read = {}
    for _ in range(case["steps"]):
        solver.substep()
        if case["kind"] == "wcsph":
            solver.map_velocity(state["sim"].grid)
        if case["loop"]:
            st = solver.stats()
            read = {k: st[k] for k in ("dt", "kinetic_energy", "potential_energy", "div_iter", "incom_iter")}
    nf, nb = f.part_num[None], b.part_num[None]
    out = {k: getattr(f, k)[:nf] for k in _OUT + (["volume_frac", "mass", "normal"] if case["kind"] == "twophase"
                                                  else ["pressure"] if case["kind"] == "wcsph" else [])}
    out.update({"bound_" + k: getattr(b, k)[:nb] for k in _BOUT})
    out["cell"] = f.neighb_cell_seq[:nf]
    out["in_cell"] = f.neighb_in_cell_seq[:nf]
    if case["kind"] == "wcsph":
        out["grid_vel"] = state["sim"].grid.vel
    out.update(read)
    return out


_OUT = ["pos", "vel", "acce_adv", "W", "sph_density", "sph_compression", "alpha", "alpha_2"]
_BOUT = ["W", "sph_density", "alpha"]


def _counts(case):
    """(fluid, boundary) particles of a case."""
    if case["kind"] == "batch":
        mean = (case["b"] - case["a"]) / math.log(max(case["b"] / case["a"], 1.0001))
        n = mean * case["c"]
        return n, 1.2 * n
    n = case["a"] * case["b"] * case["c"] * (2 if case["kind"] == "twophase" else 1)
    d = _spacing(case)
    box = [v / d + 7 for v in _tank(case, d, [s * d for s in (case["a"], case["b"], case["c"])[:case["dim"]]])]
    return n, np.prod(box) - np.prod([v - 6 for v in box])


def work(case):
    """State in and out once, and the pair terms at the solvers' floor of two iterations each."""
    n, nb = _counts(case)
    dim, steps = case["dim"], case["steps"]
    P = 2 if case["kind"] == "twophase" else 1
    pairs = 31 if dim == 3 else 12
    fb = 4 * (2 * dim + P + 3) + 4 * (3 * dim + 6 + 2) + (4 * (P + 1 + dim) if P == 2 else 0)
    bytes_ = steps * (n * fb + nb * 4 * (dim + 2 + 3))
    flops = steps * n * pairs * (50 + 4 * (32 + 28) + 40 + (120 if P == 2 else 0))
    if case["kind"] == "rollout":
        bytes_, flops = 3 * bytes_, 5 * flops
    return {"bytes": bytes_, "flops": flops}


# --------------------------------------------------------------------------------------- 64 bits
class _Par:
    """Constants of a scene, rounded to the 32 bits that they are held in."""

    def __init__(self, sc, case):
        f32 = lambda v: float(np.float32(v))  # noqa: E731
        env, cfg = sc["scenario"]["sim_env"], sc["config"]
        self.dim = dim = env["sim_dim"]
        self.d = f32(env["global_part_size"])
        self.h = f32(2 * self.d)
        self.sig = f32(8 / math.pi / self.h ** 3) if dim == 3 else f32(40 / 7 / math.pi / self.h ** 2)
        self.V = f32(math.pow(self.d, dim))
        self.mu = f32(env["global_dynamic_viscosity"])
        self.lb = np.array(env["sim_space_lb"], np.float32)
        rt = np.array(env["sim_space_rt"], np.float32)
        self.size = [int(v) for v in np.ceil((rt - self.lb) / np.float32(self.h)).astype(np.float32)]
        self.shape = tuple(int(v) for v in np.ceil((rt.astype(np.float64) - self.lb) / self.h))
        self.g = torch.tensor(np.array(env["gravity"], np.float32).astype(np.float64), device=DEV)
        self.rho = torch.tensor([f32(v) for v in env["phase_rest_density"]], device=DEV, dtype=torch.float64)
        self.div_tol, self.comp_tol = f32(cfg["solver_divergence_threshold"]), f32(cfg["solver_compression_threshold"])
        self.gamma, self.fbm_c = f32(cfg["solver_surface_tension_gamma"]), f32(cfg["solver_fbm_convection_term"])
        self.cs, self.cfl, self.vf = cfg["solver_cs"], f32(cfg["solver_cfl_factor"]), cfg["solver_type"] == "VFSPH"
        self.wc, self.two = case["kind"] == "wcsph", case["kind"] == "twophase"


def _codes(pos32, p):
    c = torch.floor((pos32 - torch.tensor(p.lb, device=DEV)) / np.float32(p.h)).to(torch.int64)
    code = c[:, 0] + c[:, 1] * p.size[0]
    return code + c[:, 2] * (p.size[0] * p.size[1]) if p.dim == 3 else code


class _Grid:
    def __init__(self, pos32, p):
        self.p = p
        self.codes, self.order = torch.sort(_codes(pos32, p), stable=True)

    def candidates(self, code, chunk=200000):
        """(i, j) chunks of the particles j in the cells around the codes."""
        p = self.p
        zs = [0] if p.dim == 2 else [-1, 0, 1]
        for c0 in range(0, len(code), chunk):
            cc = code[c0:c0 + chunk]
            I, J = [], []
            for dz in zs:
                for dy in (-1, 0, 1):
                    rc = cc + dy * p.size[0] + (dz * p.size[0] * p.size[1] if dz else 0)
                    lo = torch.searchsorted(self.codes, rc - 1)
                    cnt = torch.searchsorted(self.codes, rc + 1, right=True) - lo
                    i = torch.repeat_interleave(torch.arange(len(cc), device=DEV), cnt)
                    off = torch.arange(len(i), device=DEV) - (torch.cumsum(cnt, 0) - cnt)[i]
                    I.append(i + c0)
                    J.append(self.order[lo[i] + off])
            yield torch.cat(I), torch.cat(J)

    def within(self, pos32, other32, strict):
        I, J = [], []
        x, y = pos32.to(torch.float64), other32.to(torch.float64)
        for i, j in self.candidates(_codes(pos32, self.p)):
            r = (x[i] - y[j]).square().sum(1).sqrt()
            k = r < self.p.h
            if strict:
                k &= r > 0
            I.append(i[k])
            J.append(j[k])
        return torch.cat(I), torch.cat(J)


def _w(q, p):
    return torch.where(q <= 0.5, 6 * (q ** 3 - q ** 2) + 1, torch.where(q < 1, 2 * (1 - q) ** 3, 0 * q)) * p.sig


def _wg(q, p):
    return torch.where(q <= 0.5, 6 * (3 * q ** 2 - 2 * q), torch.where(q < 1, -6 * (1 - q) ** 2, 0 * q)) * (p.sig / p.h)


def _coh(q, p):
    t = (1 - q) ** 3 * q ** 3
    return torch.where(q <= 0.5, 2 * t - 1 / 64, torch.where(q < 1, t, 0 * q)) * (32 / math.pi / p.h ** 3)


def _add(n, i, v):
    return torch.zeros((n,) + v.shape[1:], device=DEV, dtype=torch.float64).index_add(0, i, v)


class _Pairs:
    """Geometry of the pairs (i, j), 0 < r < h."""

    def __init__(self, x, y, i, j, p):
        self.i, self.j = i, j
        self.x = x[i] - y[j]
        self.r = self.x.square().sum(1).sqrt()
        self.g = (_wg(self.r / p.h, p) / self.r)[:, None] * self.x
        self.w = _w(self.r / p.h, p)


def _sums(n, pairs, w0, V, m):
    """W, density and compression of n particles with their self term, over (pairs, volume, mass) sets."""
    W, rho, comp = w0 + 0 * m, w0 * m, w0 * V + 0 * m
    for pr, mj, Vj in pairs:
        W = W + _add(n, pr.i, pr.w)
        rho = rho + _add(n, pr.i, pr.w * mj[pr.j])
        comp = comp + _add(n, pr.i, pr.w * Vj)
    return W, rho, comp


def _substep(S, B, p, mu):
    """One substep in 64 bits: S holds pos, vel, vf, m, rho0 of the fluid, B pos, m of the boundary."""
    n, nb = len(S["pos"]), len(B["pos"])
    with torch.no_grad():
        x32, b32 = S["pos"].detach().to(torch.float32), B["pos"].to(torch.float32)
        gf, gb = _Grid(x32, p), _Grid(b32, p)
        ff, fb, bf = gf.within(x32, x32, True), gb.within(x32, b32, True), gf.within(b32, x32, True)
        vmax = S["vel"].detach().square().sum(1).sqrt().max().item()
        dt = p.d / p.cs
        if vmax > 1e-4:
            dt = min(dt, p.d / vmax * p.cfl)
    x, y, V = S["pos"], B["pos"], p.V
    m, rho0, mb = S["m"], S["rho0"], B["m"]
    ff, fb = _Pairs(x, x, *ff, p), _Pairs(x, y, *fb, p)
    w0 = _w(torch.zeros((), device=DEV, dtype=torch.float64), p)
    W, rho, comp = _sums(n, [(ff, m, V), (fb, mb, V)], w0, V, m)
    X = V + 0 * m if p.vf else m
    Xb = V + 0 * mb if p.vf else mb
    psi, psi0 = (comp, 1 + 0 * m) if p.vf else (rho, rho0)
    gff, gfb = ff.g * X[ff.j][:, None], fb.g * Xb[fb.j][:, None]
    a1 = _add(n, ff.i, gff) + _add(n, fb.i, gfb)
    a2 = _add(n, ff.i, gff.square().sum(1) / m[ff.j])
    alpha = a1.square().sum(1) / m + a2
    alpha = torch.where(alpha < 1e-4, 1e-4 + 0 * alpha, alpha)
    out = {"W": W, "sph_density": rho, "sph_compression": comp, "alpha": alpha, "alpha_2": a2}
    with torch.no_grad():
        pbf = _Pairs(y, x.detach(), *bf, p)
        if "sums" not in B:  # the boundary's own pairs do not change
            pbb = _Pairs(y, y, *gb.within(b32, b32, True), p)
            B["sums"] = _sums(nb, [(pbb, mb, V)], w0, V, mb)
        Wb = B["sums"][0] + _add(nb, pbf.i, pbf.w)
        rb = B["sums"][1] + _add(nb, pbf.i, pbf.w * m.detach()[pbf.j])
        ab = _add(nb, pbf.i, (pbf.g.square().sum(1) * X.detach()[pbf.j] ** 2) / m.detach()[pbf.j])
        out.update(bound_W=Wb, bound_sph_density=rb, bound_alpha=ab.clamp(min=1e-4))

    def solve(u, tol):
        it, c = 0, 0.0
        while it < 2 or c > tol:
            s = psi - psi0 + dt * (_add(n, ff.i, (gff * (u[ff.i] - u[ff.j])).sum(1)) +
                                   _add(n, fb.i, (gfb * u[fb.i]).sum(1)))
            s = s.clamp(min=0)
            kap = s / alpha
            c = (s / psi0).mean().item()
            f = kap[:, None] * a1 + _add(n, ff.i, (kap[ff.j] * X[ff.i])[:, None] * ff.g)
            u = u - f / (dt * m[:, None])
            it += 1
            if it > 100:
                break
        return u, it

    u, out["div_iter"] = solve(S["vel"], p.div_tol)
    mid = u
    dv = ((mid[ff.i] - mid[ff.j]) * ff.x).sum(1)
    lap = (2 * (2 + p.dim) * X[ff.j] / psi[ff.j] * dv / (0.01 * p.h ** 2 + ff.r ** 2))[:, None] * ff.g
    acc = p.g + _add(n, ff.i, lap) * (mu / rho0)[:, None]
    if p.gamma:
        nrm = -p.h * _add(n, ff.i, (X / psi)[ff.j][:, None] * ff.g)
        out["normal"] = nrm
        on = (S["vf"][:, 0].to(torch.float32) > 0.99)
        st = torch.zeros_like(acc)
        for i, j in gf.candidates(_codes(x32, p)):
            k = on[i] & on[j]
            i, j = i[k], j[k]
            xij = x[i] - x[j]
            r = xij.square().sum(1).sqrt()
            k = r > 0
            i, j, xij, r = i[k], j[k], xij[k], r[k]
            c = -p.gamma * m[j] * _coh(r / p.h, p) / r
            t = c[:, None] * xij + p.gamma * (nrm[i] - nrm[j])
            st = st.index_add(0, i, (2 * psi0[i] / (psi[i] + psi[j]))[:, None] * t)
        acc = acc + st
    u, out["incom_iter"] = solve(mid + acc * dt, p.comp_tol)
    if p.wc:
        pr = (rho0 * p.cs ** 2 / 7 * ((rho / rho0) ** 7 - 1)).clamp(min=0)
        q = pr / rho ** 2
        acc = acc - _add(n, ff.i, ((q[ff.i] + q[ff.j]) * m[ff.j])[:, None] * ff.g) \
            - _add(n, fb.i, (q[fb.i] * mb[fb.j])[:, None] * fb.g)
        u = mid + acc * dt
        out["pressure"] = pr
    vf = S["vf"]
    if p.two:
        acc, vf = _mixture(S, ff, u, mid, dt, p)
        rho0 = (vf * p.rho).sum(1)
        m = rho0 * V
    xn = x + u * dt
    out.update(pos=xn, vel=u, acce_adv=acc, volume_frac=vf, mass=m, dt=dt)
    out["kinetic_energy"] = float((0.5 * m * u.square().sum(1)).sum())
    out["potential_energy"] = float((-m * p.g[1] * (xn[:, 1] - float(p.lb[1]))).sum())
    if p.wc:
        idx = torch.stack(torch.meshgrid(*[torch.arange(k, device=DEV) for k in p.shape], indexing="ij"), -1)
        nodes = torch.tensor(p.lb, device=DEV) + idx.reshape(-1, p.dim).to(torch.float32) * np.float32(p.h)
        gv = torch.zeros(len(nodes), p.dim, device=DEV, dtype=torch.float64)
        at = nodes.to(torch.float64)
        for i, j in gf.candidates(_codes(nodes, p)):
            r = (at[i] - xn[j]).square().sum(1).sqrt()
            gv.index_add_(0, i, (X[j] / psi[j] * _w(r / p.h, p))[:, None] * u[j])
        out["grid_vel"] = gv.reshape(p.shape + (p.dim,))
    return out, {"pos": xn, "vel": u, "vf": vf, "m": m, "rho0": rho0}


def _mixture(S, ff, u, mid, dt, p):
    """The volume-fraction update: drift velocities, then passes until no fraction turns negative."""
    n, vf, rho0 = len(S["pos"]), S["vf"], S["rho0"][:, None]
    a = (u - mid) / dt
    zeta = (vf * (p.rho - rho0) / p.rho).sum(1)[:, None]
    fa = (a - zeta * p.g) / (1 - zeta)
    w = vf * p.rho
    c = torch.where(w > 1e-6, vf * (p.rho - rho0) / torch.where(w > 1e-6, w, 1 + 0 * w), 0 * w)
    drift = (c[:, :, None] * (p.g - fa)[:, None, :] + (fa - a)[:, None, :]) * dt
    flux = vf[:, :, None] * drift
    flag = torch.zeros(n, device=DEV, dtype=torch.bool)
    for _ in range(1000):
        k = ~flag[ff.i] & ~flag[ff.j]
        i, j = ff.i[k], ff.j[k]
        t = ((flux[i] + flux[j]) * ff.g[k][:, None, :]).sum(2)
        tmp = -p.fbm_c * dt * p.V * _add(n, i, t)
        neg = (vf + tmp < 0).any(1)
        flag |= neg
        if not neg.any():
            break
    return a, torch.where(flag[:, None], vf, vf + tmp)


def _start64(sc, p):
    vf = sc["vf"].to(torch.float64)
    rho0, rb = (vf * p.rho).sum(1), (sc["bvf"].to(torch.float64) * p.rho).sum(1)
    return ({"pos": sc["pos"].to(torch.float64), "vel": sc["vel"].to(torch.float64), "vf": vf, "m": rho0 * p.V,
             "rho0": rho0}, {"pos": sc["bpos"].to(torch.float64), "m": rb * p.V})


def exact(case, seed):
    outs = []
    scenes = _scenes(case, seed)
    if case["kind"] == "rollout":
        return _exact_rollout(case, scenes[0], seed)
    for sc in scenes:
        p = _Par(sc, case)
        with torch.no_grad():
            S, B = _start64(sc, p)
            for _ in range(case["steps"]):
                out, S = _substep(S, B, p, p.mu)
        outs.append(out)
    names = _OUT + (["volume_frac", "mass", "normal"] if case["kind"] == "twophase"
                    else ["pressure"] if case["kind"] == "wcsph" else []) + ["bound_" + k for k in _BOUT]
    res = {k: torch.cat([o[k] for o in outs]) for k in names}
    res["cell"] = res["in_cell"] = None
    if case["kind"] == "wcsph":
        res["grid_vel"] = outs[0]["grid_vel"]
    if case["loop"]:
        res.update({k: outs[0][k] for k in ("dt", "kinetic_energy", "potential_energy")},
                   div_iter=None, incom_iter=None)
    return res


def _exact_rollout(case, sc, seed):
    p = _Par(sc, case)
    gen = torch.Generator(device=DEV).manual_seed(seed + 3)
    gx, gv, gr = _loss_seeds(sc, gen)
    S, B = _start64(sc, p)
    v0 = S["vel"].clone().requires_grad_(True)
    mu = torch.tensor(p.mu, dtype=torch.float64, device=DEV, requires_grad=True)
    S["vel"] = v0
    for _ in range(case["steps"]):
        _, S = _substep(S, B, p, mu)
    x, v = S["pos"], S["vel"]
    with torch.no_grad():
        x32, b32 = x.detach().to(torch.float32), B["pos"].to(torch.float32)
        ff, fb = _Grid(x32, p).within(x32, x32, True), _Grid(b32, p).within(x32, b32, True)
    w0 = _w(torch.zeros((), device=DEV, dtype=torch.float64), p)
    _, rho, _ = _sums(len(x), [(_Pairs(x, x, *ff, p), S["m"], p.V), (_Pairs(x, B["pos"], *fb, p), B["m"], p.V)],
                      w0, p.V, S["m"])
    gv0, gmu = torch.autograd.grad((x, v, rho), (v0, mu), [t.to(torch.float64) for t in (gx, gv, gr)])
    return {"pos": x.detach(), "vel": v.detach(), "density": rho.detach(), "grad_v0": gv0, "grad_mu": gmu}
