"""The density pass at the cell sizes where its warps' shares change.

A warp takes 32 or 64 particles of a cell (up to 32 in one, a second 32 in the
other slot of each lane, or in a second warp where the grid is small), and
lists are staged 256 entries at a time.  One update of a 4x4 block of cells of
``per`` particles each, in a grid small enough for two warps per cell and in
one large enough for one, equals the oracle's bit for bit.
"""
import numpy as np
import pytest

import nbodysimulation_experiment_gb300 as pkg
from nbodysimulation_experiment_gb300 import scenes
from oracle import state as ostate
from oracle.oracle import OracleSim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [1, 5])
@pytest.mark.parametrize("per", [1, 28, 29, 31, 32, 33, 63, 64, 65, 96, 97])
def test_one_update(per, size):
    rng = np.random.default_rng(per)
    h = float(scenes.H)
    w, d = size * scenes.REF_WIDTH, size * scenes.REF_HEIGHT
    cells = np.array([(x, y) for y in range(4) for x in range(4)], np.float64)
    pos = (np.repeat(cells, per, 0) + rng.uniform(0.02, 0.98, (16 * per, 2)) + (8, 6)) * h - (0.5 * w, 0.5 * d)
    scene = scenes.Scene("lists", w, d, pos.astype(np.float32), scenes.box_planes(w, d), gravity=(0.0, 0.0))
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
