"""The grid update where many particles change cell at once.

A warp sorts a cell's entering (and, in reference order, leaving) particles and
looks for each leaving one 32 places at a time.  A 5x5 block of cells of
``per`` particles each, fast enough that most of a cell's members leave and as
many enter, gives arrays, searches and sorts on both sides of 32 and 64.  The
cell arrays, in order, and the particles equal the oracle's after two updates,
in canonical and in reference order.
"""
import numpy as np
import pytest

import nbodysimulation_experiment_gb300 as pkg
from nbodysimulation_experiment_gb300 import scenes
from oracle import state as ostate
from oracle.oracle import OracleSim

pytestmark = pytest.mark.gpu

DT = float(scenes.DT)


@pytest.mark.parametrize("reference", [False, True])
@pytest.mark.parametrize("per", [1, 2, 20, 31, 32, 33, 64, 65, 90])
def test_two_updates(per, reference):
    rng = np.random.default_rng(per)
    h = float(scenes.H)
    cells = np.array([(x, y) for y in range(5) for x in range(5)], np.float64)
    pos = (np.repeat(cells, per, 0) + rng.uniform(0.02, 0.98, (25 * per, 2)) + (8, 6)) * h
    pos -= (0.5 * scenes.REF_WIDTH, 0.5 * scenes.REF_HEIGHT)
    pos = pos.astype(np.float32)
    vel = rng.normal(0.0, 0.7 * h / DT, pos.shape).astype(np.float32)
    scene = scenes.Scene("events", scenes.REF_WIDTH, scenes.REF_HEIGHT, pos[:0],
                         scenes.box_planes(scenes.REF_WIDTH, scenes.REF_HEIGHT), gravity=(0.0, 0.0),
                         max_particles=len(pos))
    orc, sim = OracleSim(scene.oracle_domain(OracleSim)), pkg.Simulation(scene.domain())
    for s in (orc, sim):
        scene.apply(s)
        # In reference order the particles are new ones, pushed off by a force.
        s.add_particles(pos, vel / np.float32(DT) if reference else None)
    if reference:
        sim.set_reference_order(True)
    else:
        ref = orc.get_state()
        ref["vel"] = vel
        sim.load_state(ostate.from_reference_state(ref, *scene.domain().grid()))
    for step in range(2):
        before = sim.dump_state()
        if not reference:
            orc.set_state(ostate.to_reference_state(before))
        orc.update(DT)
        sim.update(DT)
        after, want = sim.dump_state(), orc.get_state(lists=False)
        if reference:  # the oracle's numbers are the particles' identities
            cells_ref = ostate.reference_cells_by_id(want, np.arange(len(pos)))
            for a, b in zip(ostate.gpu_cells_by_id(after), cells_ref):
                assert np.array_equal(a, b), step
            for f in ("pos", "vel", "dens", "press"):
                assert ostate.ulp_diff(ostate.by_id(after, f), np.asarray(want[f], np.float32)) == 0, (step, f)
        else:
            res = ostate.compare_step(before, after, want)
            assert res["cells_equal"] == 1.0, (step, res)
            for f in ("pos", "vel", "dens", "press"):
                assert res[f + "_ulp"] == 0, (step, f, res)
    sim.close()
