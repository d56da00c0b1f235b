"""The density pass with one warp a cell (a grid of mostly empty cells).

Up to 32 particles of a cell take one list per lane, a second 32 the other
slot of each lane.  One update of a 4x4 block of cells of ``per`` particles
each in a grid of 301,996 cells equals the oracle's bit for bit.
"""
import numpy as np
import pytest

import nbodysimulation_experiment_gb300 as pkg
from nbodysimulation_experiment_gb300 import scenes
from oracle import state as ostate
from oracle.oracle import OracleSim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per", [1, 31, 32, 33, 64, 65, 97])
def test_one_update(per):
    rng = np.random.default_rng(per)
    h = float(scenes.H)
    w, d = 22 * scenes.REF_WIDTH, 22 * scenes.REF_HEIGHT
    cells = np.array([(x, y) for y in range(4) for x in range(4)], np.float64)
    pos = (np.repeat(cells, per, 0) + rng.uniform(0.02, 0.98, (16 * per, 2)) + (8, 6)) * h - (0.5 * w, 0.5 * d)
    scene = scenes.Scene("lists", w, d, pos.astype(np.float32), scenes.box_planes(w, d), gravity=(0.0, 0.0))
    gx, gy = scene.domain().grid()
    assert gx * gy > 1728 * 152  # density_halves, csrc/sph_rules.h
    orc = OracleSim(scene.oracle_domain(OracleSim))
    scene.apply(orc)
    sim = pkg.Simulation(scene.domain())
    scene.apply(sim)
    before = sim.dump_state()
    orc.set_state(ostate.to_reference_state(before))
    orc.update(float(scenes.DT))
    sim.update(float(scenes.DT))
    sim.synchronize()
    res = ostate.compare_step(before, sim.dump_state(), orc.get_state(lists=False))
    assert res["cells_equal"] == 1.0, res
    for f in ("pos", "vel", "dens", "press"):
        assert res[f + "_ulp"] == 0, (f, res)
    sim.close()
