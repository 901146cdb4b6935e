"""The cluster scan of the cell counts (kb_scan_cluster): the order of its
barriers by reading its source, its results over every number of chunks, and where
it is taken instead of the three passes.

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


def _scene(tank, skin=0.15, mixed=False, solid=True, seed=3):
    """A block of water in the first and the last cells of a tank without walls."""
    cfg = cases._config(0.01, tank, keep=True, precision=api.PRECISION_MIXED if mixed else api.PRECISION_FP32)
    case = cases._case(0.01, tank, (9, 8, 7), (10, 0, 0), (2, 6, 6) if solid else (0, 0, 0), 2 if solid else 0,
                       virt_layers=0, jitter=0.01, seed=seed)
    cfg, pa = cases.make((cfg, case))
    cfg.neighbor_skin = skin
    shift = np.float32(0.01) * (np.array(tank, np.float32) - np.array([13, 8, 7], np.float32))
    pos, spos = pa.fluid_pos.copy(), pa.solid_pos.copy()
    pos[::2] += shift
    spos[::3] += shift
    return cfg, api.ParticleArrays(pos, pa.fluid_vel, pa.fluid_rho, pa.fluid_p, spos, pa.solid_vel, spos.copy(),
                                   pa.solid_type, pa.virt_pos)


@pytest.mark.gpu
@pytest.mark.parametrize("tank,chunks", [((60, 40, 40), 1), ((300, 100, 100), 2), ((400, 110, 110), 3),
                                         ((460, 120, 120), 4), ((480, 130, 130), 5)])
@pytest.mark.parametrize("skin", [0.15, 0.0])
@pytest.mark.parametrize("mixed", [False, True])
def test_every_number_of_chunks(tank, chunks, skin, mixed):
    """Grids of one to four chunks and of the first size beyond the cluster scan: cell
    starts and neighbour counts equal the oracle's."""
    cfg, pa = _scene(tank, skin, mixed)
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


SMALL, ONE, TWO, THREE, FOUR, FIVE = ((24, 16, 16), (60, 40, 40), (300, 100, 100), (400, 110, 110), (460, 120, 120),
                                      (480, 130, 130))


@pytest.mark.gpu
@pytest.mark.parametrize("tanks", [[ONE] * 4, [TWO] * 4, [THREE] * 4, [FOUR] * 4, [FOUR, ONE, THREE, TWO, SMALL],
                                   [FIVE] * 4, [SMALL] * 20],
                         ids=["one chunk", "two", "three", "four", "mixed sizes", "beyond", "many small"])
@pytest.mark.parametrize("skin", [0.15, 0.0])
def test_batches_of_every_number_of_chunks(tanks, skin):
    """Batches whose scans take clusters of one to four chunks (the buffer of the blocks'
    totals is used again from the third on), and ones that do not: members equal
    standalone runs."""
    scenes = [_scene(t, skin, solid=k != 1, seed=k) for k, t in enumerate(tanks)]
    names = ("fluid_pos", "fluid_vel", "fluid_rho", "solid_pos")
    alone = []
    for cfg, pa in scenes:
        with api.Simulation(cfg, pa, device=0) as s:
            s.step(3)
            s.sync()
            alone.append([s.get(f) for f in names] + [s.neighbor_counts()])
    sims = [api.Simulation(cfg, pa, device=0) for cfg, pa in scenes]
    with api.Batch(sims) as b:
        b.step(3)
        b.sync()
    for s, want in zip(sims, alone):
        for got, w in zip([s.get(f) for f in names] + [s.neighbor_counts()], want):
            assert np.array_equal(got, w)
        s.close()


@pytest.mark.gpu
def test_three_passes_where_they_are_faster():
    """One launch (a cluster per array) or three: one cluster walks several chunks one
    after another, so a single instance takes it for one chunk only; eight arrays of more
    take it, many short ones do not."""
    def launches(tanks):
        sims = [api.Simulation(*_scene(t), device=0) for t in tanks]
        if len(sims) == 1:
            n = sims[0].launches_per_step()
        else:
            with api.Batch(sims) as b:
                n = b.launches_per_step()
        for s in sims:
            s.close()
        return n

    one = launches([ONE])
    assert launches([SMALL]) == one
    for tanks, more in (([TWO], 2), ([FOUR], 2), ([FIVE], 2), ([FOUR] * 2, 2), ([ONE] * 8, 0), ([TWO] * 4, 0),
                        ([FOUR] * 4, 0), ([FIVE] * 4, 2), ([SMALL] * 20, 2)):
        assert launches(tanks) == one + more, (tanks, more)
