"""Spring selection on both sides of its small stage of 512 list entries.

Cells whose 3x3 block holds more entries are listed and run with the stage of
1,024.  A 4x4 block of cells of ``per`` particles, ``extra`` more in one of the
inner ones, has lists of 9 * per + extra entries there and shorter ones around;
two updates from it equal the oracle's, particles and springs, bit for bit.
"""
import numpy as np
import pytest

import nbodysimulation_experiment_gb300 as pkg
from nbodysimulation_experiment_gb300 import scenes
from oracle import state as ostate
from oracle.oracle import OracleSim

pytestmark = pytest.mark.gpu

SPRINGS = dict(yield_ratio=0.1, plasticity=0.3, stiffness=0.3, max_per_particle=16)
DT = float(scenes.DT)


def _by_id(count, partner, rest, ids):
    return {int(ids[k]): [(int(ids[partner[k, q]]), float(rest[k, q])) for q in range(count[k])]
            for k in range(len(count))}


@pytest.mark.parametrize("per, extra", [(1, 0), (30, 0), (56, 7), (56, 8), (56, 9), (80, 0), (100, 100)])
def test_two_updates(per, extra):
    rng = np.random.default_rng(per + extra)
    h = float(scenes.H)
    cells = np.array([(x, y) for y in range(4) for x in range(4)], np.float64)
    cells = np.concatenate([np.repeat(cells, per, 0), np.tile([[1.0, 1.0]], (extra, 1))])
    pos = (cells + rng.uniform(0.02, 0.98, cells.shape) + (8, 6)) * h
    pos -= (0.5 * scenes.REF_WIDTH, 0.5 * scenes.REF_HEIGHT)
    scene = scenes.Scene("stage", scenes.REF_WIDTH, scenes.REF_HEIGHT, pos.astype(np.float32),
                         scenes.box_planes(scenes.REF_WIDTH, scenes.REF_HEIGHT), gravity=(0.0, 0.0))
    sim, orc = pkg.Simulation(scene.domain()), OracleSim(scene.oracle_domain(OracleSim))
    for s in (sim, orc):
        scene.apply(s)
        s.set_springs(True, **SPRINGS)
    for step in range(2):
        before = sim.dump_state()
        cnt, part, rest = sim.dump_springs()
        orc.set_state(ostate.to_reference_state(before))
        orc.set_spring_state(cnt, np.where(part < 0, 0, part), rest, tag=before["id"])
        orc.update(DT)
        sim.update(DT)
        after = sim.dump_state()
        res = ostate.compare_step(before, after, orc.get_state(lists=False))
        assert res["cells_equal"] == 1.0 and res["pos_ulp"] == 0 and res["vel_ulp"] == 0, (step, res)
        assert _by_id(*sim.dump_springs(), after["id"]) == _by_id(*orc.get_spring_state(), before["id"]), step
    sim.close()
