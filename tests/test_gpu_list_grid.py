"""The neighbour lists' fine grid and the list sweep's lanes at their edges.

Sizes around the ends of warps, blocks and of the rules for the lanes that
share a particle (8,192 and 16,384 fluid particles) and for the finer list grid (262,144); list grids of every
reach (1 for small instances, 3 and, in a sparse domain, 2); batches of which only one member rebuilds;
and version-2 snapshots, whose list-grid order is no longer the present one.

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
         (26, 26, 25), (64, 64, 64), (65, 64, 64)]


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


@pytest.mark.parametrize("fluid", [(1, 1, 1), (3, 11, 1), (16, 16, 32), (17, 16, 32), (25, 26, 25), (26, 26, 25), (65, 64, 64)])
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


# (tank, fluid, walls): more than 262,144 fluid particles take a reach of 3 unless its
# cells exceed 64 per particle (0.7 M: reach 3; 24 M: reach 2)
@pytest.mark.parametrize("tank,fluid,layers", [((40, 30, 30), (20, 12, 12), 3), ((80, 70, 70), (65, 64, 64), 2),
                                               ((500, 200, 200), (65, 64, 64), 0)])
@pytest.mark.parametrize("precision", [api.PRECISION_FP32, api.PRECISION_MIXED])
def test_every_reach_finds_every_pair(tank, fluid, layers, precision):
    cfg, pa = _box(fluid, tank=tank, layers=layers, precision=precision)
    with api.Simulation(cfg, pa, device=0) as sim:
        for _ in range(4):
            sim.phase(api.PHASE_CELL)
            assert np.array_equal(sim.list_counts(), sim.neighbor_counts())
            for ph in range(1, 5):
                sim.phase(ph)
        sim.sync()


def test_one_member_of_a_batch_rebuilds():
    # solids out of the fluid's reach: where they touch, the compiler contracts the
    # plain form's fluid-solid terms of the launch forms differently in the last bit
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


def _as_version_2(snap, sim, cfg):
    """The snapshot with version 2's sizes of the list-grid arrays (contents there are not read)."""
    d, n = sim.derived(), sim.n
    Rs = np.sqrt(float(d.impact_distance_square)) * (1.0 + float(cfg.neighbor_skin))
    span = [float(d.cell_max[a]) - float(d.cell_min[a]) for a in range(3)]
    old = int(np.prod([max(1, int(np.floor(s / (Rs * 1.001)))) for s in span]))
    nf, ns, nv = n["fluid"], n["solid"], n["virt"]
    fixed = [16 * nf, 16 * nf, 4 * nf, 4 * nf, 16 * ns, 16 * ns, 16 * ns, 4 * ns, 4 * ns, 16 * nv, 16 * nv, 16 * nv,
             4 * nv, 4 * nv]
    tail = [4 * ns, 32] + ([16 * nv] if cfg.precision == api.PRECISION_MIXED else [])
    pad = lambda k: (k + 15) & ~15
    # the present list grid's cell count, from the payload that is not otherwise accounted for
    known = 512 + sum(map(pad, fixed + [16 * nf, 4 * nf, 16 * ns, 4 * ns] + tail))
    start = (len(snap) - known) // 3
    sizes = fixed + [start, 16 * nf, 4 * nf, start, 16 * ns, 4 * ns, start] + tail
    want = fixed + [4 * (d.cell_number_total + 1), 16 * nf, 4 * nf, 4 * (old + 1), 16 * ns, 4 * ns, 4 * (old + 1)] + tail
    out, at = [bytearray(snap[:512].tobytes())], 512
    for k, (have, need) in enumerate(zip(sizes, want)):
        data = snap[at:at + pad(have)].tobytes()
        out.append(data if have == need else bytes(pad(need)))
        at += pad(have)
    assert at == len(snap)
    head = out[0]
    head[8:12] = np.uint32(2).tobytes()
    return head, b"".join(bytes(x) for x in out[1:])


@pytest.mark.parametrize("precision", [api.PRECISION_FP32, api.PRECISION_MIXED])
def test_version_2_snapshots_load(precision):
    cfg, pa = _box((14, 9, 11), precision=precision)
    fields = ("fluid_pos", "fluid_vel", "fluid_rho", "solid_pos", "virt_pos", "virt_p", "virt_vel", "virt_rho")
    with api.Simulation(cfg, pa, device=0) as a:
        a.step(5)
        head, payload = _as_version_2(a.snapshot(step=5), a, cfg)
        at = head.find(np.uint64(len(a.snapshot()) - 512).tobytes(), 32, 64)  # payload_bytes of the header
        assert at > 0
        head[at:at + 8] = np.uint64(len(payload)).tobytes()
        with api.Simulation.from_snapshot(np.frombuffer(bytes(head) + payload, np.uint8), device=0) as b:
            assert b.snapshot_step == 5
            for f in fields:
                assert np.array_equal(a.get(f), b.get(f)), f
            builds = b.list_stats()["builds"]
            b.phase(api.PHASE_CELL)
            assert b.list_stats()["builds"] == builds + 1
            assert np.array_equal(b.list_counts(), b.neighbor_counts())
            a.step(3)
            for ph in range(1, 5):
                b.phase(ph)
            b.step(2)
            a.sync()
            b.sync()
            for f in ("fluid_pos", "fluid_vel", "fluid_rho", "solid_pos"):
                # the same steps, summed in another order: FP32 rounding (tests/test_gpu_lists.py)
                assert nerr(b.get(f), a.get(f).astype(np.float64)) <= 1e-5, f
