"""The ordered sweeps at the boundaries of their shapes.

Lists of 9 * per entries (a 5x5 block of cells of ``per`` particles each) on
both sides of: a producer warp's one and two rounds with six and twelve
producers (192, 384 and 768 entries), the pipelined pass of the shapes with
two, three and six (512, 576 and 960), and the lean viscosity slot's velocity
stage (768).

Fast particles whose tasks' regions outgrow every shape's stage, by cells or by
entries, and are swept in groups: in the grid of 33 x 18 cells some go 12 cells
to each side.  Each in every sweep shape, one update equal to the oracle's, bit
for bit.
"""
import numpy as np
import pytest

import nbodysimulation_experiment_gb300 as pkg
from nbodysimulation_experiment_gb300 import scenes
from nbodysimulation_experiment_gb300.simulation import DELTA_WARPS, VISC_WARPS
from oracle import state as ostate
from oracle.oracle import OracleSim

pytestmark = pytest.mark.gpu

H = float(scenes.H)
DT = float(scenes.DT)


def _crowd(nx, ny, at, per, seed):
    """nx x ny cells from cell `at` on, ``per`` particles each, and a generator."""
    rng = np.random.default_rng(seed)
    cells = np.array([(x, y) for y in range(ny) for x in range(nx)], np.float64)
    pos = (np.repeat(cells, per, 0) + rng.uniform(0.02, 0.98, (nx * ny * per, 2)) + at) * H
    return pos - (0.5 * scenes.REF_WIDTH, 0.5 * scenes.REF_HEIGHT), rng


def _check(pos, vel):
    scene = scenes.Scene("edges", scenes.REF_WIDTH, scenes.REF_HEIGHT, pos.astype(np.float32),
                         scenes.box_planes(scenes.REF_WIDTH, scenes.REF_HEIGHT), gravity=(0.0, 0.0))
    orc = OracleSim(scene.oracle_domain(OracleSim))
    scene.apply(orc)
    ref = orc.get_state()
    ref["vel"] = vel.astype(np.float32)
    gx, gy = scene.domain().grid()
    sim = pkg.Simulation(scene.domain())
    scene.apply(sim)
    st = ostate.from_reference_state(ref, gx, gy)
    sim.load_state(st)
    sim.set_adaptive_shapes(False)
    before = sim.dump_state()
    orc.set_state(ostate.to_reference_state(before))
    orc.update(DT)
    want = orc.get_state(lists=False)
    base = sim.sweep_shape()
    for k, warps in enumerate(DELTA_WARPS):
        sim.load_state(st)
        sim.set_sweep_shape((VISC_WARPS[k % 2], base[1], warps, base[3]))
        sim.update(DT)
        sim.synchronize()
        res = ostate.compare_step(before, sim.dump_state(), want)
        assert res["cells_equal"] == 1.0, (warps, res)
        for f in ("pos", "vel", "dens", "press"):
            assert res[f + "_ulp"] == 0, (warps, f, res)
    sim.close()


@pytest.mark.parametrize("per", [21, 22, 42, 43, 56, 57, 64, 65, 85, 86, 106, 107])
def test_list_lengths(per):
    pos, rng = _crowd(5, 5, (8, 6), per, per)
    _check(pos, rng.normal(0.0, 0.3, pos.shape))


@pytest.mark.parametrize("nx, ny, at, per, fast", [
    (5, 5, (14, 6), 20, 0.2),    # few particles, regions of up to the whole grid
    (7, 7, (13, 5), 100, 0.02),  # crowded: more than 4,096 entries
    (31, 16, (1, 1), 36, 0.1),   # nearly the whole grid: more than 12,288
])
def test_groups(nx, ny, at, per, fast):
    pos, rng = _crowd(nx, ny, at, per, per)
    vel = rng.normal(0.0, 0.3, pos.shape)
    some = rng.random(len(pos)) < fast
    vel[some] = rng.uniform(-1.0, 1.0, (some.sum(), 2)) * (12, 8) * (H / DT)
    _check(pos, vel)
