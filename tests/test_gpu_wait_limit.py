"""sph_set_wait_limit holds for the waits within a block too.

All particles lie in one cell, so no task waits for another one.  In the lean
viscosity shape its producer warp waits for the chain that runs its pairs
(several microseconds a particle): a limit of a nanosecond runs out there and
is reported, and the simulation goes on from a loaded state.  The wide shape
meets at barriers and has no such wait.
"""
import numpy as np
import pytest

import nbodysimulation_experiment_gb300 as pkg
from nbodysimulation_experiment_gb300 import scenes
from nbodysimulation_experiment_gb300.simulation import DELTA_WARPS, SPH_ERR_TIMEOUT, VISC_WARPS, SphError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lean", [False, True])
def test_limit_within_a_block(lean):
    h = float(scenes.H)
    pos = np.random.default_rng(1).uniform(0.1, 0.9, (300, 2)) * h + (16 * h - 5.0, 6 * h - 0.5 * scenes.REF_HEIGHT)
    scene = scenes.Scene("cell", scenes.REF_WIDTH, scenes.REF_HEIGHT, pos.astype(np.float32),
                         scenes.box_planes(scenes.REF_WIDTH, scenes.REF_HEIGHT), gravity=(0.0, 0.0))
    sim = pkg.Simulation(scene.domain())
    scene.apply(sim)
    sim.set_adaptive_shapes(False)
    dt = 1e-7  # the crowd stays in its cell
    sim.update(dt)
    st = sim.dump_state()
    assert st["cell_count"].max() == len(pos)
    base = sim.sweep_shape()
    sim.set_sweep_shape((VISC_WARPS[lean], base[1], DELTA_WARPS[0], base[3]))
    sim.update(dt)
    want = sim.dump_state()
    sim.load_state(st)
    sim.set_wait_limit(1e-9)
    sim.update(dt)
    if lean:
        with pytest.raises(SphError) as e:
            sim.synchronize()
        assert e.value.status == SPH_ERR_TIMEOUT
    else:
        sim.synchronize()
    sim.set_wait_limit(2.0)
    sim.load_state(st)
    sim.update(dt)
    got = sim.dump_state()
    for k in ("pos", "vel", "dens", "press", "id"):
        assert np.array_equal(got[k], want[k]), k
    sim.close()
