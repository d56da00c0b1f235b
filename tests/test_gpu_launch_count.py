"""sph_kernel_launches counts every kernel of an update once.

The spring phase is four kernels (the choice with the small stage, the longer
lists, the commit, the displacements), so an update with springs counts four
more than one without, launched one by one or replayed from its graph.
"""
import pytest

import nbodysimulation_experiment_gb300 as pkg
from nbodysimulation_experiment_gb300 import scenes

pytestmark = pytest.mark.gpu

SPRING_KERNELS = 4


def _per_update(springs, graphs):
    scene = scenes.scaled_block(32)
    sim = pkg.Simulation(scene.domain())
    scene.apply(sim)
    sim.use_graphs(graphs)
    sim.set_springs(springs)
    sim.set_adaptive_shapes(False)
    counts = []
    for _ in range(6):
        before = sim.kernel_launches()
        sim.update(float(scenes.DT))
        counts.append(sim.kernel_launches() - before)
    sim.close()
    return counts


@pytest.mark.parametrize("graphs", [False, True])
def test_springs_add_their_kernels(graphs):
    plain, springs = _per_update(False, graphs), _per_update(True, graphs)
    assert [b - a for a, b in zip(plain, springs)] == [SPRING_KERNELS] * 6, (plain, springs)


def test_replay_counts_as_eager():
    assert _per_update(True, True) == _per_update(True, False)
