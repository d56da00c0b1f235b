"""The first update of a scene sweeps every particle as an added one, in runs
of consecutive numbers that end at jumps in space (csrc/sph_api.cu,
extend_runs).  However the particles are ordered and in however many batches
they were added, the update equals the oracle's single-worker update bit for
bit; so do the updates after it, and one with particles added between."""
import numpy as np
import pytest

import nbodysimulation_experiment_gb300 as pkg
from nbodysimulation_experiment_gb300 import scenes
from oracle import state as ostate
from oracle.oracle import OracleSim

pytestmark = pytest.mark.gpu


def _positions(kind, n, rng):
    h = float(scenes.H)
    if kind == "rows":      # a lattice of long rows: a jump at the end of each
        side = 170
        p = scenes.jittered_lattice(side, -(-n // side), -4.6, -2.4, seed=5)[:n]
    elif kind == "short":   # rows shorter than a run
        p = scenes.jittered_lattice(9, -(-n // 9), -3.0, -2.5, spacing=h / 4, seed=6)[:n]
    elif kind == "random":  # every particle far from the one before
        p = rng.uniform((-1.5, -2.0), (1.5, 0.5), (n, 2))
    else:                   # all in one cell
        p = rng.uniform(0.31, 0.59, (n, 2))
    return np.ascontiguousarray(p, np.float32)


@pytest.mark.parametrize("kind,n", [("rows", 2500), ("rows", 171), ("short", 500), ("random", 900), ("random", 33),
                                    ("one", 100), ("one", 1)])
@pytest.mark.parametrize("batches", [1, 3, 40])
def test_first_updates_equal_the_oracle(kind, n, batches):
    rng = np.random.default_rng(n + batches)
    pos = _positions(kind, n, rng)
    scene = scenes.Scene("runs", scenes.REF_WIDTH, scenes.REF_HEIGHT, pos[:0],
                         scenes.box_planes(scenes.REF_WIDTH, scenes.REF_HEIGHT), max_particles=2 * n)
    sim, orc = pkg.Simulation(scene.domain()), OracleSim(scene.oracle_domain(OracleSim))
    scene.apply(sim)
    scene.apply(orc)
    for part in np.array_split(pos, batches):
        if len(part):
            sim.add_particles(part)
            sim.state_info()  # reaches the device batch by batch
            orc.add_particles(part)
    for step in range(3):
        before = sim.dump_state()
        orc.set_state(ostate.to_reference_state(before))
        orc.update(float(scenes.DT))
        sim.update(float(scenes.DT))
        res = ostate.compare_step(before, sim.dump_state(), orc.get_state(lists=False))
        assert res["cells_equal"] == 1.0, (step, res)
        for f in ("pos", "vel", "dens", "press"):
            assert res[f + "_ulp"] == 0, (step, f, res)
        if step == 0:
            sim.add_particles(pos[: n // 2] + np.float32(0.01))
            orc.add_particles(pos[: n // 2] + np.float32(0.01))
    sim.close()
