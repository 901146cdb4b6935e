"""The cluster scan of the cell counts (kb_scan_cluster): the order of its
barriers by reading its source, and its results over every number of chunks.

A block of a cluster may write another block's shared memory only once that
block is known to have started: every block has to pass a cluster barrier
before the first remote store.  Without it the store is undefined, so the order
is checked in the source and never by running a kernel without the barrier.
"""
import os
import re

import numpy as np
import pytest

from fluidsim_gb300 import api, cases
from oracle import oracle as orc

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fluidsim_gb300", "csrc")
CHUNK = 8 * 1024 * 16  # counts that the cluster takes at a time
LIMIT = 4 * CHUNK      # above it the three-pass scan runs


def _kernel_bodies(text):
    """The text of every kernel that maps another block's shared memory, comments taken out."""
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
    out = []
    for m in re.finditer(r"__global__[^{;]*\{", text):
        depth, k = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        body = text[m.end():k]
        if "map_shared_rank" in body:
            out.append(body)
    return out


def test_remote_stores_come_after_a_cluster_barrier():
    bodies = []
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu"):
            with open(os.path.join(CSRC, name)) as f:
                bodies += _kernel_bodies(f.read())
    assert bodies
    for body in bodies:
        before, after = body.split("map_shared_rank", 1)
        assert re.search(r"\.sync\(\)|\.barrier_wait\(", before), "remote access before any cluster barrier"
        assert re.search(r"\.sync\(\)", after), "no cluster barrier before the blocks leave"
        # every arrival has its wait
        assert body.count("barrier_arrive") == body.count("barrier_wait")


@pytest.mark.gpu
@pytest.mark.parametrize("tank,chunks", [((60, 40, 40), 1), ((300, 100, 100), 2), ((400, 110, 110), 3),
                                         ((460, 120, 120), 4), ((480, 130, 130), 5)])
@pytest.mark.parametrize("skin", [0.15, 0.0])
@pytest.mark.parametrize("mixed", [False, True])
def test_every_number_of_chunks(tank, chunks, skin, mixed):
    """Particles in the first and the last cells of grids of one to four chunks (the
    buffer of the blocks' totals is used again from the third on) and of the first
    size beyond the cluster scan: cell starts and neighbour counts equal the oracle's."""
    cfg = cases._config(0.01, tank, keep=True, precision=api.PRECISION_MIXED if mixed else api.PRECISION_FP32)
    case = cases._case(0.01, tank, (9, 8, 7), (10, 0, 0), (2, 6, 6), 2, virt_layers=0, jitter=0.01, seed=3)
    cfg, pa = cases.make((cfg, case))
    cfg.neighbor_skin = skin
    shift = np.float32(0.01) * (np.array(tank, np.float32) - np.array([13, 8, 7], np.float32))
    pos, spos = pa.fluid_pos.copy(), pa.solid_pos.copy()
    pos[::2] += shift
    spos[::3] += shift
    pa = api.ParticleArrays(pos, pa.fluid_vel, pa.fluid_rho, pa.fluid_p, spos, pa.solid_vel, spos.copy(),
                            pa.solid_type, pa.virt_pos)
    ref = orc.OracleSim(cfg, pa, "f32")
    ref.phase(api.PHASE_CELL)
    with api.Simulation(cfg, pa, device=0) as sim:
        ncell = sim.derived().cell_number_total
        assert -(-ncell // CHUNK) == chunks and (ncell <= LIMIT) == (chunks <= 4)
        for _ in range(2):  # the counts have to be zero again after each sort
            sim.phase(api.PHASE_CELL)
        sim.sync()
        assert np.array_equal(sim.neighbor_counts(), ref.neighbor_counts())
        for species, x in ((0, pa.fluid_pos), (1, pa.solid_pos)):
            ids = orc.cell_ids(sim.derived(), x, "f32")
            want = np.concatenate([[0], np.cumsum(np.bincount(ids, minlength=ncell))])
            start, order = sim.cells(species)
            assert np.array_equal(start, want) and np.array_equal(np.sort(ids, kind="stable"), ids[order])
