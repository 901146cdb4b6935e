"""The mixed form's positions, densities and pressures are read as FP64 forms them
from what is held, rounded once: bit for bit, NaN and infinities included.

The densities listed per exponent are states (of 17 million that FP32 densities can
reach) whose pressure lies so near the middle of two floats that a sum of two floats
alone rounds to the other one.
"""
import numpy as np
import pytest

from fluidsim_gb300 import api, cases
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

NEAR = {1.0: ("0x1.04fc8p+9", "0x1.1bef8p+9", "0x1.20548p+9", "0x1.243c8p+9", "0x1.28a18p+9", "0x1.2a958p+9"),
        2.0: ("0x1.e848p+9", "0x1.4ffp+10"), 3.0: ("0x1.e460p+9", "0x1.d8e384p+10"), 4.0: ("0x1.9bc0e8p+9",),
        6.0: ("0x1.cd1ba4p+9",), 7.0: (), 8.0: ("0x1.8dedfep+10",), 16.0: ("0x1.4b040cp+9",), 17.0: (), 1.4: ()}




@pytest.mark.parametrize("gamma", sorted(NEAR))
def test_reads_are_fp64_rounded_once(gamma):
    torch = pytest.importorskip("torch")  # FP64 functions of the same GPU
    cfg = cases._config(0.01, (38, 32, 26), precision=api.PRECISION_MIXED)
    cfg.gamma = gamma
    cfg, pa = cases.make((cfg, cases._case(0.01, (38, 32, 26), (25, 26, 25), (30, 0, 0), (2, 6, 6), 2, jitter=0.01,
                                           seed=7)))
    rng = np.random.default_rng(6)
    n = pa.n_fluid
    rho0 = np.float64(cfg.fluid_density)
    rho = (rho0 * (1.0 + rng.uniform(-1, 1, n) * 10.0 ** rng.uniform(-7, 0, n))).astype(np.float32)
    special = [float.fromhex(x) for x in NEAR[gamma]] + [rho0, 0.0, 2.0 * rho0, 3.5 * rho0, np.inf, -np.inf, np.nan, -5.0,
                                                         np.nextafter(np.float32(rho0), np.float32(0))]
    rho[:len(special)] = special
    with np.errstate(invalid="ignore"):
        delta = (rho.astype(np.float64) / rho0 - 1.0).astype(np.float32)
    with api.Simulation(cfg, pa, device=0) as sim:
        d = sim.derived()
        dt = torch.from_numpy(delta).cuda().double()
        p = np.float64(d.coefficient_rho2p) * torch.expm1(np.float64(np.float32(gamma)) * torch.log1p(dt)).cpu().numpy()
        p = np.fmax(p, np.float64(np.float32(cfg.min_pressure))).astype(np.float32)
        sim.set("fluid_rho", rho)
        together = {k: np.empty(n, np.float32) for k in ("fluid_rho", "fluid_p")}
        sim.get_many_ptr(list(together), [a.ctypes.data for a in together.values()], [4 * n] * 2)
        want_rho = (rho0 * (1.0 + delta.astype(np.float64))).astype(np.float32)
        for name, want in (("fluid_rho", want_rho), ("fluid_p", p)):
            for got in (sim.get(name), together[name]):
                bad = np.nonzero(~((got == want) | (np.isnan(got) & np.isnan(want))))[0]
                assert not len(bad), (name, [(float(rho[k]).hex(), got[k], want[k]) for k in bad[:4]])


def test_positions_are_fp64_rounded_once():
    cfg, pa = cases.make((cases._config(0.01, (90, 82, 76), precision=api.PRECISION_MIXED),
                          cases._case(0.01, (90, 82, 76), (70, 70, 70), (80, 0, 0), (2, 6, 6), 2, jitter=0.3, seed=7)))
    with api.Simulation(cfg, pa, device=0) as sim:
        d = sim.derived()
        cell = orc.cell_ids(d, pa.fluid_pos, "f32")
        ny, nz = d.cell_number[1], d.cell_number[2]
        at = np.stack([cell // (ny * nz), cell // nz % ny, cell % nz], 1).astype(np.float64)
        corner = np.array(d.cell_min, np.float64) + at * np.array(d.interval, np.float64)
        off = (pa.fluid_pos.astype(np.float64) - corner).astype(np.float32)
        want = (corner + off.astype(np.float64)).astype(np.float32)
        assert np.array_equal(sim.get("fluid_pos"), want)
