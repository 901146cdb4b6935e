"""Members of a batch equal their standalone runs bit for bit, solids in contact.

The plates touch the water and all velocities are random, so every kind of pair
term counts.  The batches reach each launch form of the sweeps (a parameter block,
an item array beyond it), members of both viscosity modes, and totals on the other
side of the rule for the lanes that share a particle (16,384 fluid particles) than
their members.
"""
import numpy as np
import pytest

from fluidsim_gb300 import api, cases

pytestmark = pytest.mark.gpu

FLUID = ("fluid_drho_dt", "fluid_du_dt", "fluid_pos", "fluid_vel", "fluid_rho", "fluid_p")
SOLID = ("solid_pos", "solid_vel", "solid_normal", "solid_couple_dudt")


def _scene(fluid, seed, precision, skin, viscid=1):
    tank = (fluid[0] + 13, fluid[1] + 6, fluid[2] + 1)
    cfg = cases._config(0.01, tank, keep=True, precision=precision)
    cfg.neighbor_skin, cfg.is_viscid = skin, viscid
    case = cases._case(0.01, tank, fluid, (fluid[0] + 1, 0, 0), (2, min(8, tank[1]), min(8, tank[2])), 2,
                       virt_layers=3, jitter=0.01, seed=seed)
    cfg, pa = cases.make((cfg, case))
    rng = np.random.default_rng(seed)
    n = pa.n_fluid
    vel = rng.uniform(-3.0, 3.0, (n, 3)).astype(np.float32)
    rho = (pa.fluid_rho * (1.0 + rng.uniform(-0.01, 0.01, n))).astype(np.float32)
    p = (pa.fluid_p + rng.uniform(-2000.0, 4000.0, n)).astype(np.float32)
    return cfg, api.ParticleArrays(pa.fluid_pos, vel, rho, p, pa.solid_pos, pa.solid_vel, pa.solid_ref_pos,
                                   pa.solid_type, pa.virt_pos)


def _state(sim):
    return {f: sim.get(f) for f in FLUID + SOLID}


@pytest.mark.parametrize("precision", [api.PRECISION_FP32, api.PRECISION_MIXED])
@pytest.mark.parametrize("skin", [0.15, 0.0])
@pytest.mark.parametrize("members", [
    [((13, 11, 12), 1), ((17, 20, 13), 0)],
    [((19, 20, 20), 1), ((20, 19, 20), 1), ((20, 20, 19), 1)],
    [((9, 8, 7), 1), ((8, 9, 7), 0)] * 35,
], ids=["two", "above the lanes' limit", "item array"])
def test_members_in_contact_equal_standalone(members, skin, precision):
    scenes = [_scene(fluid, seed, precision, skin, viscid) for seed, (fluid, viscid) in enumerate(members)]
    alone = []
    for cfg, pa in scenes:
        with api.Simulation(cfg, pa, device=0) as s:
            out = []
            for n in (1, 3):
                s.step(n)
                s.sync()
                out.append(_state(s))
            alone.append(out)
    assert any(np.any(a[0]["solid_couple_dudt"] != 0.0) for a in alone)
    sims = [api.Simulation(cfg, pa, device=0) for cfg, pa in scenes]
    with api.Batch(sims) as b:
        for k, n in enumerate((1, 3)):
            b.step(n)
            b.sync()
            for m, s in enumerate(sims):
                got = _state(s)
                for f, want in alone[m][k].items():
                    assert np.array_equal(got[f], want), (m, n, f, int((got[f] != want).sum()))
    for s in sims:
        s.close()
