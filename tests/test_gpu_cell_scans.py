"""The scans over cells on both sides of a tile of 4,096 positions.

One tile runs without the pass of per-tile sums; a thread takes four
consecutive positions, read one by one at a ragged end.  Two updates of
particles spread thinly over grids of 4,095, 4,096, 4,097, 8,192 and 8,195
cells, with movers, equal the oracle's bit for bit.
"""
import numpy as np
import pytest

import nbodysimulation_experiment_gb300 as pkg
from nbodysimulation_experiment_gb300 import scenes
from oracle import state as ostate
from oracle.oracle import OracleSim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gx, gy", [(63, 65), (64, 64), (17, 241), (64, 128), (55, 149)])
def test_two_updates(gx, gy):
    rng = np.random.default_rng(gx)
    h = float(scenes.H)
    w, d = (gx + 0.5) * h, (gy + 0.5) * h
    n = 1500
    pos = rng.uniform(-0.5, 0.5, (n, 2)) * (w, d)
    # The last cells of the last tile too.
    pos[:40] = (0.5 * w - 0.6 * h, 0.5 * d - 0.6 * h) + rng.uniform(-1.5, 0.0, (40, 2)) * h
    scene = scenes.Scene("scan", w, d, pos.astype(np.float32), scenes.box_planes(w, d), gravity=(0.0, -10.0))
    assert scene.domain().grid() == (gx, gy)
    orc = OracleSim(scene.oracle_domain(OracleSim))
    scene.apply(orc)
    sim = pkg.Simulation(scene.domain())
    scene.apply(sim)
    for _ in range(2):
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
