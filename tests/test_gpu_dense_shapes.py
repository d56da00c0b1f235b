"""Where dense states change the sweep shapes (sph_set_adaptive_shapes).

A crowd at rest of ``per`` particles in one cell, or in each of 3x3 cells (a
neighbour list of 9 * per): the updates run the tuned shapes below the
thresholds of each shape and the larger ones above them.
"""
import numpy as np
import pytest

import nbodysimulation_experiment_gb300 as pkg
from nbodysimulation_experiment_gb300 import scenes
from nbodysimulation_experiment_gb300.simulation import DELTA_WARPS, VISC_WARPS

pytestmark = pytest.mark.gpu

WIDE, LEAN, MID, TRI, QUAD, DENSE = DELTA_WARPS
VISC_WIDE, VISC_LEAN = VISC_WARPS


def _last_shape(per, side, visc, delta):
    h = float(scenes.H)
    cells = np.array([(x, y) for y in range(side) for x in range(side)], np.float64)
    pos = np.repeat(cells, per, 0) + np.random.default_rng(per).uniform(0.1, 0.9, (side * side * per, 2))
    pos = (pos + (16, 6)) * h - (0.5 * scenes.REF_WIDTH, 0.5 * scenes.REF_HEIGHT)
    scene = scenes.Scene("crowd", scenes.REF_WIDTH, scenes.REF_HEIGHT, pos.astype(np.float32),
                         scenes.box_planes(scenes.REF_WIDTH, scenes.REF_HEIGHT), gravity=(0.0, 0.0))
    sim = pkg.Simulation(scene.domain())
    scene.apply(sim)
    base = sim.sweep_shape()
    sim.set_sweep_shape((visc, base[1], delta, base[3]))
    for _ in range(4):  # the choice follows the update before last
        sim.update(1e-7)
    st = sim.get_stats()
    assert st.max_cell_particle_count == per and st.max_particle_neighbor_count == side * side * per
    shape = sim.last_sweep_shape()
    sim.close()
    return shape[0], shape[2]


@pytest.mark.parametrize("delta, per, want", [
    (LEAN, 85, LEAN), (LEAN, 95, MID), (LEAN, 160, DENSE),
    (TRI, 100, TRI), (TRI, 112, MID), (TRI, 160, DENSE),
    (QUAD, 126, QUAD), (QUAD, 136, MID), (QUAD, 160, DENSE),
    (MID, 140, MID), (MID, 160, DENSE),
    (WIDE, 140, WIDE), (WIDE, 160, DENSE), (DENSE, 20, DENSE), (DENSE, 160, DENSE),
])
def test_delta(delta, per, want):
    assert _last_shape(per, 1, VISC_WIDE, delta) == (VISC_WIDE, want)


@pytest.mark.parametrize("per, want", [(56, VISC_LEAN), (59, VISC_WIDE)])
def test_viscosity(per, want):
    """Lists of 504 and 531 entries."""
    assert _last_shape(per, 3, VISC_LEAN, QUAD) == (want, QUAD)
