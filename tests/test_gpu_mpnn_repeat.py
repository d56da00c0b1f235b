"""Sums over the particles in the network's backward pass repeat bit for bit.

The last round's b2, b3, W4 and b4 depend on no sum in a varying order (the
edge layer's and the split weight products' atomics reach the others), so the
gradient of one sample gives the same bits every time.  Sizes below and above
one sweep of a row's blocks (8 blocks x 256 threads x 8 values), ragged.
"""
import numpy as np
import pytest

import nbodysimulation_experiment_gb300 as pkg
from nbodysimulation_experiment_gb300 import scenes

pytestmark = pytest.mark.gpu

SIZES = (("W1", 768), ("b1", 128), ("W2", 16384), ("b2", 128), ("W3", 128 * 144), ("b3", 128), ("W4", 256), ("b4", 2))
REPEATED = ("b2", "b3", "W4", "b4")


@pytest.mark.parametrize("n", [5, 1601, 40003])
def test_last_round_repeats(n):
    scene = scenes.block_n(n, seed=n)
    sim = pkg.Simulation(scene.domain())
    scene.apply(sim)
    for _ in range(3):
        sim.update(float(scenes.DT) / 4)
    model = pkg.Mpnn(n + 128, seed=3)
    model.capture(sim, float(scenes.DT), 4)
    grads = [model.gradient(0)[1].copy() for _ in range(12)]
    off = len(grads[0]) // 2  # two rounds of the same layout
    for name, size in SIZES:
        if name in REPEATED:
            block = [g[off:off + size] for g in grads]
            assert np.isfinite(block[0]).all() and all(np.array_equal(block[0], b) for b in block), name
        off += size
    assert off == len(grads[0])
    model.close()
    sim.close()
