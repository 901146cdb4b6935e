"""The capacity that fsim_list_stats reports is the number of entries a particle's
list is guaranteed to hold, the number beyond which a step fails."""
import math

import numpy as np
import pytest

from fluidsim_gb300 import api, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("skin", [0.05, 0.15, 0.3])
@pytest.mark.parametrize("precision", [api.PRECISION_FP32, api.PRECISION_MIXED])
def test_capacity_is_one_and_a_half_spheres(skin, precision):
    cfg, pa = cases.make(cases.tiny_box(precision=precision))
    cfg.neighbor_skin = skin
    R = math.sqrt(api.derive(cfg).impact_distance_square)
    full = 4.0 / 3.0 * 3.14159265358979 * (R * (1.0 + cfg.neighbor_skin) / cfg.particle_diameter) ** 3
    want = (math.ceil(1.5 * full) + 16 + 7) // 8 * 8  # whole groups of 8
    with api.Simulation(cfg, pa, device=0) as sim:
        assert sim.list_stats()["capacity"] == want


def test_capacity_equals_the_limit_in_the_error():
    cfg, pa = cases.make(cases.tiny_box())
    pos = pa.fluid_pos.copy()
    pos[:400] = pos[0]  # 400 particles in one place
    pos[:400] += np.random.default_rng(1).uniform(-1e-4, 1e-4, (400, 3)).astype(np.float32)
    pa = api.ParticleArrays(pos, pa.fluid_vel, pa.fluid_rho, pa.fluid_p, pa.solid_pos, pa.solid_vel,
                            pa.solid_ref_pos, pa.solid_type, pa.virt_pos)
    with api.Simulation(cfg, pa, device=0) as sim:
        sim.phase(api.PHASE_CELL)
        with pytest.raises(api.FsimError, match="more than %d neighbour-list" % sim.list_stats()["capacity"]):
            sim.sync()
