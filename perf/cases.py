"""Performance cases: what users of this framework have it do, through its public API.

Three ways of driving the library, each over its range of sizes and forms:

* ``frames``   -- a resident simulation advances a few steps and its state is read
  for an output frame (the command-line program's loop over ``result_interval``);
  every pass continues where the last one stopped.
* ``coupled``  -- another program owns the state: each pass writes all of it from
  pinned host memory, advances one step and reads it back.
* ``batch``    -- an ensemble of instances advances in lockstep and every member's
  state is read.

The scenes are the framework's own: dam breaks with an elastic plate or block on
the lattice of ``fsim_case``, hydrostatic pressure, positions jittered by 1 % of the
spacing, and a divergence-free vortex in the water (up to about 1 m/s, what a
collapsing column of these sizes reaches after some hundred steps), so that
neighbour lists go stale at the rate they do in a developed flow.
"""
import math

import numpy as np
import torch

from fluidsim_gb300 import api, cases

FLUID = ("fluid_pos", "fluid_vel", "fluid_rho", "fluid_p")
SOLID = ("solid_pos", "solid_vel")
WIDTH = {"fluid_pos": 3, "fluid_vel": 3, "fluid_rho": 1, "fluid_p": 1, "solid_pos": 3, "solid_vel": 3}

_BASE = {"kind": "frames", "steps": 1, "dx": 0.01, "tx": 160, "ty": 40, "tz": 80, "fx": 40, "fy": 20, "fz": 40,
         "sx": 80, "sy": 0, "sz": 0, "snx": 4, "sny": 20, "snz": 40, "fixed": 3, "layers": 3, "dt": 1e-4, "sub": 4,
         "rho_s": 1100.0, "E": 1e6, "nu": 0.4, "viscid": True, "mixed": False, "skin": 0.15}


def _scene(name, **kw):
    c = dict(_BASE, **kw)
    c["name"] = name
    return c


def listed():
    four_m = dict(dx=0.005, tx=512, ty=128, tz=128, fx=256, fy=128, fz=128, sx=336, sz=49, snx=30, sny=30, snz=30,
                  fixed=0, dt=5e-5, rho_s=1200.0, E=5e6, nu=0.3)
    return [
        # the tests' smallest box: a step is a chain of launches with next to nothing in them
        _scene("box_frames", steps=10, tx=24, ty=16, tz=16, fx=12, fy=10, fz=12, sx=16, sz=4, snx=2, sny=8, snz=8,
               fixed=2),
        # the first benchmark configuration, written out every 20 steps
        _scene("dam_frames", steps=20),
        # the same tank driven by another program, plate inside the impact distance of the water
        _scene("dam_coupled", kind="coupled", sx=41),
        # the mixed-precision form, driven the same way, odd sizes
        _scene("dam_mixed_coupled", kind="coupled", fx=37, fy=21, fz=43, sx=38, mixed=True),
        # a soft thick block against inviscid water: the largest solid that the served stream asks for
        _scene("block_frames", steps=5, ty=60, fx=61, fy=37, fz=53, sx=62, sz=7, snx=15, sny=30, snz=60, viscid=False,
               sub=5, E=1e7),
        # neighbour lists switched off: the reference's cell walk every step (largest ensemble member)
        _scene("walk_frames", steps=5, ty=60, fx=63, fy=50, fz=79, sx=65, skin=0.0),
        # mid-size in the mixed form
        _scene("mixed_frames", steps=10, ty=81, fx=73, fy=71, fz=77, sx=74, mixed=True),
        # half a million particles, one exchange of the state per step
        _scene("half_million_coupled", kind="coupled", ty=91, fx=79, fy=81, fz=77, sx=80),
        # the largest served request
        _scene("million_frames", steps=5, ty=147, fx=91, fy=137, fz=79, sx=93, sny=60, snz=79, E=3e6),
        # the headline benchmark: 4.2 M fluid particles and a free elastic cube
        _scene("four_million_frames", steps=10, **four_m),
        # and in the mixed form
        _scene("four_million_mixed", steps=5, mixed=True, **four_m),
        # the batched ensemble: 64 tanks of 8 k to 250 k particles
        {"name": "ensemble", "kind": "batch", "members": 64, "member_seed": 2024, "lo": 8000, "hi": 250000,
         "mixed": False, "steps": 5},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    if rng.random() < 0.2:
        n = int(round(_log_uniform(rng, 2, 48)))
        return {"kind": "batch", "members": n, "member_seed": rng.randrange(1 << 20), "lo": 8000,
                "hi": rng.randrange(20000, 250001), "mixed": rng.random() < 0.25, "steps": rng.randrange(1, 6)}
    n = _log_uniform(rng, 1400, 4.0e6)
    side = n ** (1.0 / 3.0)
    fx = max(8, int(side * rng.uniform(0.8, 1.6)))
    fz = max(8, int(side * rng.uniform(0.6, 1.2)))
    fy = max(6, int(n / (fx * fz)))
    gap = rng.randrange(1, 12)
    snx, snz = rng.randrange(2, 7), max(4, min(fz, int(math.sqrt(27000 / 4.0))))
    sny = max(4, min(fy + 4, 27000 // (snx * snz), rng.randrange(8, 80)))
    dx = 0.005 if n > 1.5e6 else 0.01
    c = dict(_BASE, dx=dx, dt=1e-2 * dx, tx=fx + gap + snx + rng.randrange(8, fx + 12), ty=max(fy, sny) + 10, tz=fz + 1,
             fx=fx, fy=fy, fz=fz, sx=fx + gap, snx=snx, sny=sny, snz=snz, fixed=rng.choice((0, 2, 3)),
             layers=rng.choice((2, 3, 4)), E=_log_uniform(rng, 1e5, 3e6), nu=rng.uniform(0.3, 0.45),
             viscid=rng.random() < 0.75, mixed=rng.random() < 0.35)
    if rng.random() < 0.35 and n < 1.5e6:
        c["kind"] = "coupled"
    else:
        c["steps"] = max(1, min(20, int(3.5e7 / n), rng.randrange(2, 21)))
        if n < 4e5 and rng.random() < 0.2:
            c["skin"] = 0.0
    return c


# ------------------------------------------------------------------ scenes
def _config_and_case(c, seed):
    cfg = api.default_config()
    cfg.gravity = 9.81
    cfg.is_viscid = 1 if c["viscid"] else 0
    cfg.fluid_sound_speed, cfg.fluid_density, cfg.gamma, cfg.viscosity = 30.0, 1000.0, 7.0, 1e-3
    cfg.solid_density, cfg.youngs_modulus, cfg.poisson_ratio = c["rho_s"], c["E"], c["nu"]
    cfg.xmin = cfg.ymin = cfg.zmin = 0.0
    cfg.xmax, cfg.ymax, cfg.zmax = c["tx"] * c["dx"], c["ty"] * c["dx"], c["tz"] * c["dx"]
    cfg.dt, cfg.solid_sub_step, cfg.iend, cfg.result_interval = c["dt"], c["sub"], 1000, 1001
    cfg.smoothing_length, cfg.particle_diameter, cfg.impact_length_hsml_ratio = 1.3 * c["dx"], c["dx"], 2.0
    cfg.precision = api.PRECISION_MIXED if c["mixed"] else api.PRECISION_FP32
    cfg.neighbor_skin = c["skin"]
    case = api.Case()
    case.dx = c["dx"]
    for a, (t, f, lo, s) in enumerate((("tx", "fx", "sx", "snx"), ("ty", "fy", "sy", "sny"), ("tz", "fz", "sz", "snz"))):
        case.tank_n[a], case.fluid_n[a], case.solid_lo[a], case.solid_n[a] = c[t], c[f], c[lo], c[s]
    case.solid_fixed_layers, case.virt_layers, case.hydrostatic = c["fixed"], c["layers"], 1
    case.jitter, case.seed = 0.01, seed
    return cfg, case


def _members(c, seed):
    """(config, case) of every instance of a case."""
    if c["kind"] != "batch":
        return [_config_and_case(c, seed)]
    rng = np.random.default_rng(c["member_seed"])
    out = []
    for k in range(c["members"]):
        cfg, case = cases.ensemble_member(rng, n_range=(c["lo"], c["hi"]))
        cfg.precision = api.PRECISION_MIXED if c["mixed"] else api.PRECISION_FP32
        case.jitter, case.seed = 0.01, 1000 * seed + k
        out.append((cfg, case))
    return out


def _start_moving(sim, cfg, rng):
    """A vortex in the water that leaves its block's sides and bottom tangentially, and a
    swaying solid (zero where it is fixed)."""
    x = sim.get("fluid_pos").astype(np.float32)
    top = x.max(axis=0)
    speed = np.float32(rng.uniform(0.6, 1.0) * rng.choice((-1.0, 1.0)) * min(1.0, top[0] / top[1]) / 1.2)
    ax, ay = np.float32(math.pi) * x[:, 0] / top[0], np.float32(math.pi) * x[:, 1] / top[1]
    shear = speed * (1 + np.float32(0.2) * np.cos(2 * np.float32(math.pi) * x[:, 2] / top[2]
                                                  + np.float32(rng.uniform(0, 6.28))))
    u = np.zeros_like(x)
    u[:, 0] = shear * np.sin(ax) * np.cos(ay)
    u[:, 1] = -shear * (top[1] / top[0]) * np.cos(ax) * np.sin(ay)
    sim.set("fluid_vel", u)
    if sim.n["solid"]:
        s, free = sim.get("solid_pos"), sim.get("solid_type") == 0
        v = np.zeros_like(s)
        height = np.maximum(s[:, 1] - s[free, 1].min(), 0) / max(float(np.ptp(s[free, 1])), 1e-6)
        v[:, 0] = np.where(free, np.float32(rng.uniform(0.1, 0.3)) * height, 0)
        sim.set("solid_vel", v)


def _pinned(n, width):
    shape = (n, width) if width > 1 else (n,)
    return torch.empty(shape, dtype=torch.float32, pin_memory=torch.cuda.is_available())


def _slices(buffers, sims):
    """Per instance the (field names, pointers, byte counts) of its share of the host buffers."""
    at, out = {k: 0 for k in buffers}, []
    for sim in sims:
        names = [k for k in buffers if sim.n[k.split("_")[0]]]
        ptrs, sizes = [], []
        for k in names:
            n = 4 * WIDTH[k] * sim.n[k.split("_")[0]]
            ptrs.append(buffers[k].data_ptr() + at[k])
            sizes.append(n)
            at[k] += n
        out.append((names, ptrs, sizes))
    return out


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    sims = []
    for cfg, lattice in _members(case, seed):
        sim = api.Simulation.from_case(cfg, lattice)
        _start_moving(sim, cfg, rng)
        sims.append(sim)
    total = {s: sum(sim.n[s] for sim in sims) for s in ("fluid", "solid")}
    names = FLUID + (SOLID if total["solid"] else ())
    result = {k: _pinned(total[k.split("_")[0]], WIDTH[k]) for k in names}
    state = {"steps": case["steps"], "result": result, "reads": _slices(result, sims), "sims": sims}
    if case["kind"] == "coupled":
        # in the mixed form the pressure follows from the density and is not written
        start = {k: torch.from_numpy(sims[0].get(k)) for k in names}
        if torch.cuda.is_available():
            start = {k: v.pin_memory() for k, v in start.items()}
        state["start"] = start
        state["writes"] = _slices({k: v for k, v in start.items() if not (case["mixed"] and k == "fluid_p")}, sims)[0]
    elif case["kind"] == "batch":
        state["batch"] = api.Batch(sims)
        del state["sims"]  # the batch holds its members, and ends before they do
    return state


def run(state):
    if "batch" in state:
        batch = state["batch"]
        batch.step(state["steps"])
        for sim, read in zip(batch.sims, state["reads"]):
            sim.get_many_ptr(*read)
    else:
        sim = state["sims"][0]
        if "writes" in state:
            sim.set_many_ptr(*state["writes"])
        sim.step(state["steps"])
        sim.get_many_ptr(*state["reads"][0])
    return state["result"]


def work(case):
    """Each step reads and writes the state of every particle once (fluid 64 bytes, wall 32, solid 132 per sub-step
    and 16 per step) and evaluates every pair within the impact distance (81 neighbours on the lattice; a distance
    test of 10 and a pair term of 80 operations; deformation and force of a solid pair 110 per sub-step); a pass
    writes its results once and, where it does, reads its inputs once."""
    nbytes = flops = 0.0
    for cfg, lattice in _members(case, 0):
        nf, ns, nv = api.case_counts(lattice)
        nbytes += case["steps"] * (64.0 * nf + 32.0 * nv + ns * (16.0 + 132.0 * cfg.solid_sub_step))
        nbytes += (32.0 * nf + 24.0 * ns) * (2 if case["kind"] == "coupled" else 1)
        flops += case["steps"] * 81.0 * (90.0 * nf + 110.0 * ns * cfg.solid_sub_step)
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------ the same steps in 64 bits
class _Grid:
    """The method's cell grid over one set of particles: cells from the 32-bit positions, particles in cell order."""

    def __init__(self, lo, inverse, shape, pos):
        self.shape = shape
        c = ((pos.float() - lo) * inverse).to(torch.int64)
        c = torch.minimum(c.clamp(min=0), torch.tensor(shape, device=pos.device) - 1)
        self.at = c
        self.cell = (c[:, 0] * shape[1] + c[:, 1]) * shape[2] + c[:, 2]
        self.order = torch.argsort(self.cell)
        count = torch.bincount(self.cell, minlength=shape[0] * shape[1] * shape[2])
        self.first = torch.cat([count.new_zeros(1), torch.cumsum(count, 0)])


def _candidates(of, among, most=1 << 25):
    """(i, j) index tensors, in pieces: for every particle i of grid `of`, the particles j of `among` in the 27
    cells around i's. A particle's candidates are all in one piece."""
    nx, ny, nz = of.shape
    n = len(of.cell)
    if not n or not len(among.cell):
        return
    z0 = (of.at[:, 2] - 1).clamp(min=0)
    z1 = (of.at[:, 2] + 1).clamp(max=nz - 1) + 1
    begins, lengths = [], []
    for ox in (-1, 0, 1):
        for oy in (-1, 0, 1):
            x, y = of.at[:, 0] + ox, of.at[:, 1] + oy
            inside = (x >= 0) & (x < nx) & (y >= 0) & (y < ny)
            row = ((x * ny + y) * nz).clamp(min=0, max=(nx * ny - 1) * nz)
            b, e = among.first[row + z0], among.first[row + z1]
            begins.append(b)
            lengths.append(torch.where(inside, e - b, torch.zeros_like(b)))
    begins, lengths = torch.stack(begins, 1), torch.stack(lengths, 1)
    per = max(1, int(lengths.sum(1).max()))
    chunk = max(1, most // per)
    for s in range(0, n, chunk):
        b, l = begins[s:s + chunk].reshape(-1), lengths[s:s + chunk].reshape(-1)
        i = torch.arange(s, min(n, s + chunk), device=l.device).repeat_interleave(9).repeat_interleave(l)
        before = torch.cumsum(l, 0) - l
        k = torch.arange(len(i), device=l.device) - before.repeat_interleave(l) + b.repeat_interleave(l)
        yield i, among.order[k]


def _near(of, among, xi, xj, r2max):
    """Candidate pairs closer than the impact distance: (i, j, xj - xi, its square)."""
    for i, j in _candidates(of, among):
        d = xj[j] - xi[i]
        r2 = (d * d).sum(1)
        keep = r2 < r2max
        yield i[keep], j[keep], d[keep], r2[keep]


def _dot(a, b):
    return (a * b).sum(1)


def _unit(n):
    """Normalised rows, zero where the squared length is below 0.1."""
    l2 = _dot(n, n)
    return torch.where((l2 < 0.1)[:, None], torch.zeros_like(n), n / l2.clamp(min=1e-300).sqrt()[:, None])


def _cofactor(a):
    return torch.stack([torch.linalg.cross(a[:, 1], a[:, 2]), torch.linalg.cross(a[:, 2], a[:, 0]),
                        torch.linalg.cross(a[:, 0], a[:, 1])], 1)


class _Exact:
    """The method in 64 bits: cell pairs, Riemann fluid terms, mirrored walls, total-Lagrangian solid."""

    def __init__(self, cfg, dev):
        f = np.float32
        self.cfg = cfg
        h, dp, ratio = f(cfg.smoothing_length), f(cfg.particle_diameter), f(cfg.impact_length_hsml_ratio)
        x = np.arange(10000, dtype=f) * (ratio / f(10000))
        c1 = f(math.exp(-float(ratio) ** 2))
        total = np.add.accumulate((x * x * np.exp(-x * x) * (ratio / f(10000))).astype(f))[-1]
        pi = f(3.141593)
        coef = 1.0 / float(total * f(4) * pi - c1 * f(4) / f(3) * pi * ratio ** f(3))
        self.c1, self.c2 = float(c1), coef * float(h / dp) ** -3
        self.dw = 2 * coef * float(h / dp) ** -3 / float(h) ** 2
        self.h, self.ih2, self.r2 = float(h), float(h) ** -2, float((ratio * h) * (ratio * h))
        lo = np.array([cfg.xmin, cfg.ymin, cfg.zmin], f) - f(8) * dp
        hi = np.array([cfg.xmax, cfg.ymax, cfg.zmax], f) + f(8) * dp
        self.shape = [int((b - a) / (ratio * h)) for a, b in zip(lo, hi)]
        side = (hi - lo) / np.array(self.shape, f)
        self.lo, self.inverse = torch.tensor(lo, device=dev), torch.tensor(f(1) / side, device=dev)
        self.box = [torch.tensor(v, dtype=torch.float64, device=dev)
                    for v in ((cfg.xmin, cfg.ymin, cfg.zmin), (cfg.xmax, cfg.ymax, cfg.zmax))]
        self.g = torch.tensor([0.0, -cfg.gravity, 0.0], dtype=torch.float64, device=dev)
        e, nu = cfg.youngs_modulus, cfg.poisson_ratio
        self.lam, self.mu = e * nu / (1 - 2 * nu) / (1 + nu), e / (1 + nu) / 2
        self.cs = math.sqrt(e / (3 * (1 - 2 * nu)) / cfg.solid_density)
        # the 32-bit constants of the equation of state
        self.per_rho0 = float(f(1) / f(cfg.fluid_density))
        self.stiff = float(f(1) / (f(cfg.gamma) * f(cfg.fluid_sound_speed) ** f(-2) / f(cfg.fluid_density)))

    def grid(self, pos):
        return _Grid(self.lo, self.inverse, self.shape, pos)

    def riemann(self, sums, i, d, r2, ui, uj, rhoi, rhoj, pi, pj, limited, floor):
        """Adds the pair terms to sums = (density rate, acceleration)."""
        cfg = self.cfg
        kern = torch.exp(-r2 * self.ih2) * self.dw
        r = r2.sqrt()
        e = torch.where((r > 0)[:, None], d / r.clamp(min=1e-300)[:, None], torch.zeros_like(d))
        rs = rhoi + rhoj
        p = (rhoi * pj + rhoj * pi) / rs
        du = _dot(ui - uj, e)
        lim = (3 * du).clamp(max=cfg.fluid_sound_speed) if limited else torch.full_like(du, cfg.fluid_sound_speed)
        p = torch.where(du >= 0, p + rhoi * rhoj * du / rs * lim, p)
        if floor:
            p = p.clamp(min=0)
        star = (ui * rhoi[:, None] + uj * rhoj[:, None]) / rs[:, None]
        star = star + e * ((pi - pj) / rs / cfg.fluid_sound_speed)[:, None]
        f = -2 * p / rhoi * kern
        if cfg.is_viscid:
            f = f + 10 * cfg.viscosity * _dot(uj - ui, d) / (r2 + 0.01 * self.h ** 2) / rhoi * kern
        sums[0].index_add_(0, i, 2 * rhoi * _dot(ui - star, d) * kern)
        sums[1].index_add_(0, i, d * f[:, None])

    def clamp(self, x):
        return torch.minimum(torch.maximum(x, self.box[0]), self.box[1])

    def normals(self, x, grid):
        n = torch.zeros_like(x)
        for i, j, d, r2 in _near(grid, grid, x, x, self.r2):
            n.index_add_(0, i, -d * (torch.exp(-r2 * self.ih2) * self.dw)[:, None])
        return _unit(n)

    def step(self, s):
        cfg = self.cfg
        fx, fu, fr, fp = (s[k] for k in FLUID)
        sx, su, ref, kind, wx = s["solid_pos"], s["solid_vel"], s["ref"], s["type"], s["wall"]
        gf, gs, gw = self.grid(fx), self.grid(sx), self.grid(wx)
        # the solid's normal and the fluid pressure it feels
        sn, weight, press = self.normals(sx, gs), sx.new_zeros(len(sx)), sx.new_zeros(len(sx))
        for i, j, d, r2 in _near(gs, gf, sx, fx, self.r2):
            w = (torch.exp(-r2 * self.ih2) - self.c1) * self.c2
            weight.index_add_(0, i, w)
            press.index_add_(0, i, fp[j] * w)
        sp = torch.where(weight > 1e-6, (press / weight.clamp(min=1e-300)).clamp(min=cfg.min_pressure), press * 0)
        # walls mirror their nearest fluid particle
        wr, wp = torch.full_like(wx[:, 0], cfg.fluid_density), torch.zeros_like(wx[:, 0])
        wu = torch.zeros_like(wx)
        for i, j in _candidates(gw, gf):
            d = fx[j] - wx[i]
            r2 = (d * d).sum(1)
            best = torch.full((len(wx),), math.inf, dtype=r2.dtype, device=r2.device)
            best.scatter_reduce_(0, i, r2, "amin")
            hit = r2 == best[i]
            i, j, d = i[hit], j[hit], d[hit]
            wr[i], wp[i], wu[i] = fr[j], fp[j] - fr[j] * (d @ self.g), fu[j]
        wn = s["wall_normal"] if "wall_normal" in s else self.normals(wx, gw)
        s["wall_normal"] = wn
        wu = wu - wn * (2 * _dot(wu, wn))[:, None]
        # the fluid
        sums = (torch.zeros_like(fr), torch.zeros_like(fx))
        for i, j, d, r2 in _near(gf, gf, fx, fx, self.r2):
            self.riemann(sums, i, d, r2, fu[i], fu[j], fr[i], fr[j], fp[i], fp[j], True, False)
        for i, j, d, r2 in _near(gf, gs, fx, sx, self.r2):
            n = sn[j]
            uj = fu[i] - n * (2 * _dot(fu[i] - su[j], n))[:, None]
            self.riemann(sums, i, d, r2, fu[i], uj, fr[i], fr[i], fp[i], sp[j], False, False)
        for i, j, d, r2 in _near(gf, gw, fx, wx, self.r2):
            self.riemann(sums, i, d, r2, fu[i], wu[j], fr[i], wr[j], fp[i], wp[j], True, True)
        nx = self.clamp(fx + fu * cfg.dt)
        nu = fu + (sums[1] + self.g) * cfg.dt
        nr = (fr + sums[0] * cfg.dt).clamp(min=0.9 * cfg.fluid_density, max=1.1 * cfg.fluid_density)
        np_ = (((nr * self.per_rho0) ** cfg.gamma - 1) * self.stiff).clamp(min=cfg.min_pressure)
        speed, most = _dot(nu, nu).sqrt(), 0.3 * cfg.fluid_sound_speed
        nu = torch.where((speed > most)[:, None], nu * (most / speed.clamp(min=1e-300))[:, None], nu)
        s.update(zip(FLUID, (nx, nu, nr, np_)))
        if len(sx):
            self.solid(s, gf, gs, sn, sp)

    def solid(self, s, gf, gs, sn, sp):
        cfg, ref, dt = self.cfg, s["ref"], self.cfg.dt / self.cfg.solid_sub_step
        fx, fu, fr, fp = (s[k] for k in FLUID)
        free = (s["type"] == 0)[:, None]
        parts = [p for p in _near(gs, gs, ref, ref, self.r2)]
        i, j, dref, r2 = (torch.cat([p[k] for p in parts]) for k in range(4))
        keep = i != j
        i, j, dref, r2 = i[keep], j[keep], dref[keep], r2[keep]
        kern = torch.exp(-r2 * self.ih2) * self.dw
        eye = torch.eye(3, dtype=ref.dtype, device=ref.device)
        outer = lambda a, b: a[:, :, None] * b[:, None, :]  # noqa: E731
        shape = torch.zeros(len(ref), 3, 3, dtype=ref.dtype, device=ref.device)
        shape.index_add_(0, i, outer(dref, dref * kern[:, None]))
        flat = torch.linalg.det(shape) == 0
        linv = torch.where(flat[:, None, None], eye, torch.linalg.inv(torch.where(flat[:, None, None], eye, shape)))
        for _ in range(cfg.solid_sub_step):
            x, u = s["solid_pos"], s["solid_vel"]
            dx, du = x[j] - x[i], u[j] - u[i]
            grad = torch.zeros_like(shape).index_add_(0, i, outer(dx, dref * kern[:, None])) @ linv
            strain = (grad.transpose(1, 2) @ grad - eye) / 2
            trace = strain.diagonal(dim1=1, dim2=2).sum(1)
            stress = grad @ (2 * self.mu * strain + self.lam * trace[:, None, None] * eye)
            pl, av = stress @ linv, _cofactor(grad) @ linv
            nu = self.h * _dot(du, dx) / (_dot(dx, dx) + 0.01 * self.h ** 2)
            visc = cfg.arti_vis_alpha * nu * self.cs - cfg.arti_vis_beta * nu * nu
            a = torch.zeros_like(x)
            a.index_add_(0, i, ((pl[i] + pl[j]) @ dref[:, :, None])[:, :, 0] * (kern / cfg.solid_density)[:, None])
            a.index_add_(0, i, (av[i] @ dref[:, :, None])[:, :, 0] * (visc * kern)[:, None])
            for a_, b, d, q in _near(gs, gf, x, fx, self.r2):
                n, uf = sn[a_], fu[b]
                bounce = -2 * _dot(uf - u[a_], n)
                r = q.sqrt()
                e = torch.where((r > 0)[:, None], d / r.clamp(min=1e-300)[:, None], torch.zeros_like(d))
                rel = bounce * _dot(n, e)
                p = (fp[b] + sp[a_]) / 2
                p = torch.where(rel >= 0, p + fr[b] * rel / 2 * cfg.fluid_sound_speed, p)
                f = -2 * p / cfg.solid_density * torch.exp(-q * self.ih2) * self.dw
                a.index_add_(0, a_, d * f[:, None])
            s["solid_pos"] = torch.where(free, self.clamp(x + u * dt), x)
            s["solid_vel"] = torch.where(free, u + (a + self.g) * dt, torch.zeros_like(u))


def exact(case, seed):
    members = _members(case, seed)
    if case["steps"] * sum(api.case_counts(lattice)[0] for _, lattice in members) > 5e6:
        return None
    state = prepare(case, seed)
    sims = state["batch"].sims if "batch" in state else state["sims"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    out = {k: [] for k in state["result"]}
    for (cfg, _), sim in zip(members, sims):
        read = lambda k: torch.from_numpy(sim.get(k)).to(dev)  # noqa: E731,B023
        s = {k: read(k).double() for k in FLUID + SOLID}
        s.update(ref=read("solid_ref_pos").double(), type=read("solid_type"), wall=read("virt_pos").double())
        model = _Exact(cfg, dev)
        for _ in range(case["steps"]):
            model.step(s)
        for k in out:
            out[k].append(s[k].cpu())
    return {k: torch.cat(v) for k, v in out.items()}
