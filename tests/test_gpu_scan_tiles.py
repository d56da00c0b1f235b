"""The scans over cells on a grid of more than 512 tiles of 4,096 positions.

Past that number the tiles' sums become offsets in a pass of their own, so no
block adds up all the tiles before its own: two launches more per update.  Two
updates of particles spread over 1,449 x 1,449 cells (513 tiles, the last one
and the last four positions ragged) equal the oracle's bit for bit.
"""
import numpy as np
import pytest

import nbodysimulation_experiment_gb300 as pkg
from nbodysimulation_experiment_gb300 import scenes
from oracle import state as ostate
from oracle.oracle import OracleSim

pytestmark = pytest.mark.gpu

H = float(scenes.H)
FEW = 512  # kScanFewTiles, csrc/sph_kernels.cuh


def _scene(gx, gy, pos):
    w, d = (gx + 0.5) * H, (gy + 0.5) * H
    scene = scenes.Scene("tiles", w, d, pos.astype(np.float32), scenes.box_planes(w, d), gravity=(3.0, -10.0))
    assert scene.domain().grid() == (gx, gy)
    return scene


def test_two_updates():
    from conftest import host_memory_gb
    if host_memory_gb() < 16:
        pytest.skip("the oracle's cell arrays take 9 GB")
    side, n = 1449, 4000
    rng = np.random.default_rng(side)
    half = 0.5 * (side + 0.5) * H
    pos = rng.uniform(-half, half, (n, 2))
    pos[:1000] *= 0.002                                       # a crowd in the middle
    pos[1000:1040] = half - 0.6 * H + rng.uniform(-1.5, 0.0, (40, 2)) * H  # and the last cells
    scene = _scene(side, side, pos)
    orc = OracleSim(scene.oracle_domain(OracleSim))
    scene.apply(orc)
    sim = pkg.Simulation(scene.domain())
    scene.apply(sim)
    for _ in range(2):
        before = sim.dump_state()
        orc.set_state(ostate.to_reference_state(before))
        orc.update(float(scenes.DT))
        sim.update(float(scenes.DT))
        res = ostate.compare_step(before, sim.dump_state(), orc.get_state(lists=False))
        assert res["cells_equal"] == 1.0, res
        for f in ("pos", "vel", "dens", "press"):
            assert res[f + "_ulp"] == 0, (f, res)
    sim.close()


def test_launches():
    counts = []
    for gx in (FEW, FEW + 1):
        sim = pkg.Simulation(_scene(gx, 4096, np.zeros((1, 2))).domain())
        sim.add_particle((0.0, 0.0))
        before = sim.kernel_launches()
        sim.update(float(scenes.DT))
        counts.append(sim.kernel_launches() - before)
        sim.close()
    assert counts[1] == counts[0] + 2, counts
