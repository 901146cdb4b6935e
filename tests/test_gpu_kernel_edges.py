"""The list build, the list sweep's lanes and the solid sub-steps at their edges.

Sizes around the ends of warps, blocks, the build's chunks and of the rule for
the lanes that share a particle (8,192 and 16,384 fluid particles); batches of
which only one member rebuilds; the mixed form's solid-fluid lists; odd and even
numbers of solid sub-steps; the conversions that read the mixed form.

The rates are held to the bound of the other per-phase tests: at most twice
the FP32 oracle's own error against FP64, plus 5e-5 of the largest value; the
mixed form's to 2e-4 of the cell walk's, the bound of tests/test_gpu_lists.py.
Everything else is compared exactly.
"""
import numpy as np
import pytest

from conftest import nerr
from fluidsim_gb300 import api, cases
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _box(fluid, tank=None, layers=3, solid=True, precision=api.PRECISION_FP32, seed=3, gap=1):
    tank = tank or (fluid[0] + 13, fluid[1] + 6, fluid[2] + 1)
    cfg = cases._config(0.01, tank, keep=True, precision=precision)
    block = (2, min(6, tank[1]), min(6, tank[2])) if solid else (0, 0, 0)
    case = cases._case(0.01, tank, fluid, (fluid[0] + gap, 0, 0), block, 2 if solid else 0, virt_layers=layers,
                       jitter=0.01, seed=seed)
    cfg, pa = cases.make((cfg, case))
    rng = np.random.default_rng(seed)
    vel = rng.uniform(-0.3, 0.3, pa.fluid_vel.shape).astype(np.float32)
    return cfg, api.ParticleArrays(pa.fluid_pos, vel, pa.fluid_rho, pa.fluid_p, pa.solid_pos, pa.solid_vel,
                                   pa.solid_ref_pos, pa.solid_type, pa.virt_pos)


SIZES = [(1, 1, 1), (1, 1, 31), (3, 11, 1), (1, 127, 1), (3, 43, 1), (16, 16, 32), (17, 16, 32), (25, 26, 25),
         (26, 26, 25)]


@pytest.mark.parametrize("fluid", SIZES)
def test_plain_rates_and_pairs(fluid):
    cfg, pa = _box(fluid)
    r64, r32 = orc.OracleSim(cfg, pa, "f64"), orc.OracleSim(cfg, pa, "f32")
    with api.Simulation(cfg, pa, device=0) as sim:
        for ph in (api.PHASE_CELL, api.PHASE_COUPLE, api.PHASE_VIRT):
            sim.phase(ph)
            r64.phase(ph)
            r32.phase(ph)
        assert np.array_equal(sim.list_counts(), sim.neighbor_counts())
        assert np.array_equal(sim.neighbor_counts(), r64.neighbor_counts())
        sim.phase(api.PHASE_FLUID)
        r64.phase(api.PHASE_FLUID)
        r32.phase(api.PHASE_FLUID)
        sim.sync()
        for f in ("fluid_drho_dt", "fluid_du_dt"):
            want = r64.get(f)
            assert nerr(sim.get(f), want) <= 2.0 * nerr(r32.get(f), want) + 5e-5, f


@pytest.mark.parametrize("fluid", [(1, 1, 1), (3, 11, 1), (16, 16, 32), (17, 16, 32), (25, 26, 25), (26, 26, 25)])
def test_mixed_rates_and_pairs(fluid):
    cfg, pa = _box(fluid, precision=api.PRECISION_MIXED)
    walk = api.Config.from_buffer_copy(cfg)
    walk.neighbor_skin = 0.0
    with api.Simulation(cfg, pa, device=0) as a, api.Simulation(walk, pa, device=0) as b:
        for ph in range(4):
            a.phase(ph)
            b.phase(ph)
            if ph == api.PHASE_CELL:
                assert np.array_equal(a.list_counts(), a.neighbor_counts())
                assert np.array_equal(a.neighbor_counts(), b.neighbor_counts())
        for f in ("fluid_drho_dt", "fluid_du_dt"):
            assert nerr(a.get(f), b.get(f).astype(np.float64)) <= 2e-4, f


def test_one_member_of_a_batch_rebuilds():
    # solids out of the fluid's reach: where they touch, the launch forms of the plain
    # form round the fluid-solid terms differently in the last bit
    specs = [_box((9, 8, 7), seed=1, gap=5), _box((20, 18, 19), seed=2, gap=5),
             _box((11, 10, 13), solid=False, seed=4)]
    fast = specs[1][1]
    fast.fluid_vel[:, 0] += 3.0
    alone, members = [], []
    for cfg, pa in specs:
        s = api.Simulation(cfg, pa, device=0)
        s.step(14)
        s.sync()
        alone.append({f: s.get(f) for f in ("fluid_pos", "fluid_vel", "fluid_p")})
        alone[-1]["builds"] = s.list_stats()["builds"]
        s.close()
        members.append(api.Simulation(cfg, pa, device=0))
    with api.Batch(members) as b:
        b.step(14)
        b.sync()
        for s, want in zip(members, alone):
            assert s.list_stats()["builds"] == want.pop("builds")
            for f, w in want.items():
                assert np.array_equal(s.get(f), w), f
    assert members[1].list_stats()["builds"] > members[0].list_stats()["builds"]
    for s in members:
        s.close()


@pytest.mark.parametrize("speed_share", [0.0, 0.75])
def test_mixed_solid_fluid_lists_equal_full_walk(speed_share):
    """The mixed form's solid sub-steps after the first walk recorded lists of
    (particle, cell code) as the plain form's do: bit for bit the full walk of every
    sub-step, at rest and with the plate at 0.75 of the allowed displacement (0.1 R)
    per sub-step, where later sub-steps fall back to the walk."""
    cfg, pa = cases.make(cases.tiny_box(precision=api.PRECISION_MIXED))
    R = float(np.sqrt(api.derive(cfg).impact_distance_square))
    shift = pa.solid_pos[:, 0].min() - pa.fluid_pos[:, 0].max() - cfg.particle_diameter
    sp, sr, sv = pa.solid_pos.copy(), pa.solid_ref_pos.copy(), np.zeros_like(pa.solid_vel)
    sp[:, 0] -= shift
    sr[:, 0] -= shift
    sv[pa.solid_type == 0, 0] = -speed_share * 0.1 * R / (cfg.dt / cfg.solid_sub_step)
    pa = api.ParticleArrays(pa.fluid_pos, pa.fluid_vel, pa.fluid_rho, pa.fluid_p, sp, sv, sr, pa.solid_type,
                            pa.virt_pos)
    out = []
    for full in (0, 1):
        c = api.Config.from_buffer_copy(cfg)
        c.solid_full_walk = full
        with api.Simulation(c, pa, device=0) as s:
            s.step(6 if speed_share == 0.0 else 1)
            s.sync()
            out.append({f: s.get(f) for f in ("solid_pos", "solid_vel", "solid_couple_dudt", "fluid_pos")})
    assert np.any(out[0]["solid_couple_dudt"] != 0.0)
    for f in out[0]:
        assert np.array_equal(out[0][f], out[1][f]), f


@pytest.mark.parametrize("sub_steps", [1, 2, 3])
def test_odd_and_even_sub_steps_equal_the_fused_launch(sub_steps):
    """The force launches advance the solid from buffer to buffer; the fused launch
    (which walks the fluid in every sub-step) updates it in place."""
    cfg, pa = cases.make(cases.tiny_box(jitter=0.01, seed=5))
    cfg.solid_sub_step = sub_steps
    out = []
    for fused in (0, 1):
        c = api.Config.from_buffer_copy(cfg)
        c.solid_fused = fused
        with api.Simulation(c, pa, device=0) as s:
            s.step(3)
            s.sync()
            out.append({f: s.get(f) for f in ("solid_pos", "solid_vel", "solid_F", "solid_PK1", "fluid_pos")})
    for f in out[0]:
        assert np.array_equal(out[0][f], out[1][f]), f


@pytest.mark.parametrize("tank", [(30, 20, 20), (300, 100, 100), (600, 150, 150)])
@pytest.mark.parametrize("skin", [0.15, 0.0])
def test_cell_starts_of_every_scan(tank, skin):
    """Cell grids of one and two chunks of the cluster scan (131,072 counts each) and
    beyond its limit (524,288): neighbour counts by the cell walk equal the oracle's."""
    cfg, pa = _box((9, 8, 7), tank=tank, layers=0)
    cfg.neighbor_skin = skin
    # particles in the last cells too: the carry across chunks counts
    pos = pa.fluid_pos.copy()
    pos[::2] += np.float32(0.01) * (np.array(tank, np.float32) - np.array([9, 8, 7], np.float32))
    pa = api.ParticleArrays(pos, pa.fluid_vel, pa.fluid_rho, pa.fluid_p, pa.solid_pos, pa.solid_vel,
                            pa.solid_ref_pos, pa.solid_type, pa.virt_pos)
    ref = orc.OracleSim(cfg, pa, "f64")
    ref.phase(api.PHASE_CELL)
    with api.Simulation(cfg, pa, device=0) as sim:
        sim.phase(api.PHASE_CELL)
        assert np.array_equal(sim.neighbor_counts(), ref.neighbor_counts())


def _host_views(sim, names, pinned, shift):
    """A float32 view per field in one host buffer, each `shift` bytes past a 16-byte boundary."""
    sizes = [int(np.prod(sim.get(k).shape)) for k in names]
    total = sum(4 * n + 32 for n in sizes)
    owner = api.PinnedBuffer((total,), np.uint8) if pinned else np.zeros(total + 64, np.uint8)
    raw = owner.array if pinned else owner
    at = -raw.ctypes.data % 16
    views = []
    for n in sizes:
        views.append(raw[at + shift:at + shift + 4 * n])
        at += (4 * n + shift + 15) // 16 * 16
    return owner, views


@pytest.mark.parametrize("precision", [api.PRECISION_FP32, api.PRECISION_MIXED])
@pytest.mark.parametrize("pinned,shift", [(True, 0), (True, 4), (True, 2), (False, 0), (False, 2)])
def test_fields_together_equal_fields_one_by_one(precision, pinned, shift):
    """Page-locked buffers move through one copy kernel (16-byte or 4-byte words), other
    buffers and odd alignments through one copy per field: the same bytes either way."""
    cfg, pa = _box((9, 7, 5), precision=precision)
    names = ("solid_vel", "fluid_p", "fluid_pos", "fluid_rho", "solid_pos", "fluid_vel")
    with api.Simulation(cfg, pa, device=0) as a, api.Simulation(cfg, pa, device=0) as b:
        for s in (a, b):
            s.step(3)
        owner, views = _host_views(a, names, pinned, shift)
        ptrs, sizes = [v.ctypes.data for v in views], [v.nbytes for v in views]
        a.get_many_ptr(names, ptrs, sizes)
        for k, v in zip(names, views):
            assert v.tobytes() == a.get(k).tobytes(), k
        # write back a moved state, together into a and one by one into b
        take = [k for k in range(len(names)) if precision == api.PRECISION_FP32 or names[k] != "fluid_p"]
        for k in take:
            if names[k] == "fluid_vel":
                views[k][:] = np.frombuffer((np.frombuffer(views[k].tobytes(), np.float32) * 2).tobytes(), np.uint8)
        a.set_many_ptr([names[k] for k in take], [ptrs[k] for k in take], [sizes[k] for k in take])
        for k in take:
            b.set(names[k], np.frombuffer(views[k].tobytes(), np.float32))
        for s in (a, b):
            s.step(2)
            s.sync()
        for k in names:
            assert np.array_equal(a.get(k), b.get(k)), k
        del views, owner


@pytest.mark.parametrize("gamma", [1.0, 7.0, 16.0, 17.0, 1.4])
def test_mixed_state_reads_round_once(gamma):
    """Densities and pressures read from the mixed form are the 64-bit values of the
    held deviation rounded once: within one last place (half of it, and 2^-44 relative
    from either side's arithmetic), over the fast range and what takes the other path.
    A position read back is what was set within one last place of it and of its offset
    (below 2^-4)."""
    cfg, pa = _box((25, 26, 25), precision=api.PRECISION_MIXED)
    cfg.gamma = gamma
    rng = np.random.default_rng(5)
    n = len(pa.fluid_rho)
    rho0 = np.float64(cfg.fluid_density)
    rho = (rho0 * (1.0 + rng.uniform(-1, 1, n) * 10.0 ** rng.uniform(-6, 0, n))).astype(np.float32)
    rho[:6] = [rho0, 0.0, 2.0 * rho0, 3.5 * rho0, np.nextafter(np.float32(rho0), np.float32(0)), np.inf]
    pos = pa.fluid_pos + rng.uniform(-1e-4, 1e-4, pa.fluid_pos.shape).astype(np.float32)
    delta = (rho.astype(np.float64) / rho0 - 1.0).astype(np.float32).astype(np.float64)
    with api.Simulation(cfg, pa, device=0) as sim:
        sim.set("fluid_rho", rho)
        sim.set("fluid_pos", pos)
        d = sim.derived()
        with np.errstate(divide="ignore"):
            p = np.maximum(np.float64(d.coefficient_rho2p) * np.expm1(np.float64(np.float32(gamma)) * np.log1p(delta)),
                           np.float64(cfg.min_pressure))
        assert (np.abs(sim.get("fluid_pos").astype(np.float64) - pos) <= np.spacing(np.abs(pos)) + 2.0 ** -28).all()
        for name, want in (("fluid_rho", rho0 * (1.0 + delta)), ("fluid_p", p)):
            want = want.astype(np.float32)
            got = sim.get(name)
            near = (got == want) | (got == np.nextafter(want, np.float32(np.inf))) \
                | (got == np.nextafter(want, np.float32(-np.inf)))
            assert near.all(), (name, got[~near][:4], want[~near][:4])
