"""The ordered sweeps at the list lengths where their kernels change path.

A 5x5 block of cells holding ``per`` particles each gives its middle cells
lists of 9 * per entries and its edges and corners shorter ones.  One update
from that state in every sweep shape equals the oracle's, bit for bit, on
both sides of: a producer warp's one, two, three or four rounds of 32 list
entries (direct delta shapes: 7, 11 or 15 warps), the batches of 32 halves of
the ordered sum, the register-held positions and the geometry buffer of the
lean viscosity shape, and the smallest cells.
"""
import numpy as np
import pytest

import nbodysimulation_experiment_gb300 as pkg
from nbodysimulation_experiment_gb300 import scenes
from nbodysimulation_experiment_gb300.simulation import DELTA_WARPS, VISC_WARPS
from oracle import state as ostate
from oracle.oracle import OracleSim

pytestmark = pytest.mark.gpu


def _state(per, seed):
    """Oracle and canonical library state of the block (no gravity)."""
    rng = np.random.default_rng(seed)
    h = float(scenes.H)
    cells = np.array([(x, y) for y in range(5) for x in range(5)], np.float64)
    pos = (np.repeat(cells, per, 0) + rng.uniform(0.02, 0.98, (25 * per, 2)) + (8, 6)) * h
    pos -= (0.5 * scenes.REF_WIDTH, 0.5 * scenes.REF_HEIGHT)
    scene = scenes.Scene("edges", scenes.REF_WIDTH, scenes.REF_HEIGHT, pos.astype(np.float32),
                         scenes.box_planes(scenes.REF_WIDTH, scenes.REF_HEIGHT), gravity=(0.0, 0.0))
    orc = OracleSim(scene.oracle_domain(OracleSim))
    scene.apply(orc)
    ref = orc.get_state()
    ref["vel"] = rng.normal(0.0, 0.3, ref["vel"].shape).astype(np.float32)
    gx, gy = scene.domain().grid()
    return scene, orc, ostate.from_reference_state(ref, gx, gy)


@pytest.mark.parametrize("per", [1, 3, 4, 24, 25, 39, 40, 42, 43, 53, 54, 61, 78, 79, 99, 100, 107])
def test_one_update_in_every_shape(per):
    scene, orc, st = _state(per, per)
    sim = pkg.Simulation(scene.domain())
    scene.apply(sim)
    sim.load_state(st)
    sim.set_adaptive_shapes(False)
    before = sim.dump_state()
    orc.set_state(ostate.to_reference_state(before))
    orc.update(float(scenes.DT))
    want = orc.get_state(lists=False)
    base = sim.sweep_shape()
    for k, warps in enumerate(DELTA_WARPS):
        sim.load_state(st)
        sim.set_sweep_shape((VISC_WARPS[k % 2], base[1], warps, base[3]))
        sim.update(float(scenes.DT))
        sim.synchronize()
        res = ostate.compare_step(before, sim.dump_state(), want)
        assert res["cells_equal"] == 1.0, (warps, res)
        for f in ("pos", "vel", "dens", "press"):
            assert res[f + "_ulp"] == 0, (warps, f, res)
    sim.close()
