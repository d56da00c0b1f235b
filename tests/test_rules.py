"""The rules that divide an update's work (csrc/sph_rules.h), on the CPU."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = r"""
#include "sph_rules.h"
using namespace sphgb;
extern "C" {
struct P { float x, y; };
// The runs' ends of the particles at xy, added in batches of the given counts.
int runs(const P *xy, const int *batch, int batches, int first, float cell, int *ends) {
	AppendixRuns r;
	r.restart(first);
	for (int b = 0; b < batches; xy += batch[b++]) r.add(xy, batch[b], cell);
	for (size_t k = 0; k < r.ends.size(); ++k) ends[k] = r.ends[k];
	return (int)r.ends.size();
}
// The trials as rows of six numbers.
int trials(const int *now, const int *occV, const int *occD, int shapes, int lean, int sms, int *out) {
	const int v[2] = {occV[0], occV[1]};
	int n = 0;
	for (const SweepTrial &t : sweep_trials({now[0], now[1], now[2], now[3]}, v, occD, shapes, lean, sms)) {
		const int row[6] = {t.viscLean, t.viscBlocks, t.deltaShape, t.deltaBlocks, t.visc, t.delta};
		for (int k = 0; k < 6; ++k) out[6 * n + k] = row[k];
		++n;
	}
	return n;
}
int pick(const float *times, const int *counts, int n) {
	std::vector<std::vector<float>> t(n);
	for (int k = 0; k < n; times += counts[k++]) t[k].assign(times, times + counts[k]);
	return pick_launch(t);
}
int halves(int cells, int live, int n, int added, int sms) { return density_halves(cells, live, n, added, sms); }
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "shim.cpp").write_text(SHIM)
    so = str(d / "shim.so")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", "-I",
                           os.path.join(ROOT, "nbodysimulation_experiment_gb300", "csrc"), str(d / "shim.cpp"), "-o", so])
    return ctypes.CDLL(so)


@pytest.mark.parametrize("cells, live, n, added, want", [
    (1590, 114, 4096, 0, 1),          # the 4,096-particle dam break in its box
    (262144, 120, 4320, 0, 1),        # a small scene in a large box
    (2400, 2400, 86400, 0, 1),
    (16320, 3000, 65536, 0, 1),       # a spread-out block: few cells hold more than 32
    (16500, 16500, 594000, 0, 0),     # a full box
    (3000, 3000, 108000, 0, 0),
    (4864, 4800, 172800, 0, 0),
    (6000, 6000, 216000, 0, 1),       # a last wave nearly empty with one warp a cell
    (65280, 6000, 216000, 0, 0),
    (1048576, 120, 4320, 0, 0),       # mostly empty cells to pass over
    (1590, 0, 4096, 4096, 1),         # the same scenes' first updates
    (16500, 0, 594000, 594000, 0),
])
def test_density_halves(rules, cells, live, n, added, want):
    assert rules.halves(cells, live, n, added, 152) == want


RUN = 32
CELL = 0.3


def _runs(rules, pos, batches=None, first=0):
    pos = np.ascontiguousarray(pos, np.float32)
    batches = np.array([len(pos)] if batches is None else batches, np.int32)
    assert batches.sum() == len(pos)
    ends = np.zeros(len(pos) + 1, np.int32)
    rules.runs.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_float, ctypes.c_void_p]
    k = rules.runs(pos.ctypes.data, batches.ctypes.data, len(batches), first, CELL, ends.ctypes.data)
    ends = ends[:k] - first
    starts = np.concatenate([[0], ends[:-1]])
    assert ends[-1] == len(pos) and (ends > starts).all() and (ends - starts <= RUN).all()  # a partition
    assert k <= len(pos) // (RUN // 2) + 2  # what the run arrays hold
    return ends


def _rows(width, rows):
    y, x = np.divmod(np.arange(width * rows), width)
    return np.stack([x, y], 1) * 0.05


def test_runs_end_with_lattice_rows(rules):
    ends = _runs(rules, _rows(174, 40))
    assert set(range(174, 174 * 40, 174)) <= set(ends.tolist())
    assert len(ends) == 6 * 40


@pytest.mark.parametrize("width", [29, 30, 31, 32, 33, 61, 63, 65])
def test_runs_end_with_rows_about_as_long_as_a_run(rules, width):
    """Also where the run would be full just past the row's end."""
    ends = _runs(rules, _rows(width, 30))
    assert set(range(width, width * 29, width)) <= set(ends.tolist())


@pytest.mark.parametrize("n", [1, 31, 32, 33, 3000])
def test_runs_in_no_spatial_order_are_full(rules, n):
    """A jump at every particle ends no run early."""
    y, x = np.divmod(np.random.default_rng(n).permutation(n), 60)
    assert len(_runs(rules, np.stack([x, y], 1) * (2.1 * CELL))) == -(-n // RUN)


def test_runs_of_a_shuffled_block_are_almost_full(rules):
    """Few are near the one before by chance."""
    pos = np.random.default_rng(7).permutation(_rows(174, 174))
    assert len(_runs(rules, pos)) <= 1.05 * len(pos) / RUN


def test_runs_of_alternating_sources_are_full(rules):
    a = np.arange(500) * 0.02
    pos = np.stack([np.stack([a, a], 1), np.stack([a + 30.0, a], 1)], 1).reshape(-1, 2)
    assert len(_runs(rules, pos)) == -(-1000 // RUN)


@pytest.mark.parametrize("pos", [_rows(174, 20), _rows(33, 60), _rows(9, 100),
                                 np.random.default_rng(1).uniform(-40.0, 40.0, (1000, 2)),
                                 np.random.default_rng(2).uniform(-1.0, 1.0, (1000, 2))])
def test_runs_do_not_depend_on_the_batches(rules, pos):
    whole = _runs(rules, pos)
    n = len(pos)
    for batches in ([1] * n, [n // 3, 0, n - n // 3], [174] * (n // 174) + [n % 174]):
        assert np.array_equal(_runs(rules, pos, batches), whole)
    assert np.array_equal(_runs(rules, pos, first=12345), whole)


@pytest.mark.parametrize("width", [2, 3, 4, 5, 7, 13, 15, 16, 17, 31, 33, 47])
def test_runs_of_short_stretches_stay_within_their_number(rules, width):
    """Stretches of `width` near particles, each far from the one before."""
    k = np.arange(4000)
    _runs(rules, np.stack([k // width * 10.0 % 70.0, k % width * 0.05 + k // width * 0.01], 1))


def test_runs_of_odd_positions(rules):
    pos = np.random.default_rng(3).uniform(-1.0, 1.0, (200, 2))
    pos[50:60] = np.nan
    pos[100:110] = np.inf
    _runs(rules, pos)


@pytest.mark.parametrize("now", [(0, 608, 0, 152), (1, 152, 3, 760), (0, 7, 2, 9)])
@pytest.mark.parametrize("occ_v, occ_d", [((4, 1), (1, 8, 2, 5, 4, 1)), ((4, 3), (1, 6, 2, 1, 1, 9))])
def test_trials_number_the_distinct_launches(rules, now, occ_v, occ_d):
    i32 = ctypes.c_int
    out = (i32 * 6000)()
    n = rules.trials((i32 * 4)(*now), (i32 * 2)(*occ_v), (i32 * 6)(*occ_d), 6, 1, 152, out)
    rows = np.array(out[:6 * n]).reshape(n, 6)
    assert tuple(rows[0]) == now + (0, 0)
    # As many trials as the larger occupancy of each pair of shapes.
    assert n == 1 + sum(max(occ_v[d == 1], occ_d[d]) for d in range(6))
    want_v = {now[:2]} | {(0, 152 * k) for k in range(1, occ_v[0] + 1)} | {(1, 152 * k) for k in range(1, occ_v[1] + 1)}
    want_d = {now[2:]} | {(d, 152 * k) for d in range(6) for k in range(1, occ_d[d] + 1)}
    for launches, ids, want in ((rows[:, 0:2], rows[:, 4], want_v), (rows[:, 2:4], rows[:, 5], want_d)):
        number = {}
        for p, k in zip(map(tuple, launches), ids):
            assert number.setdefault(p, len(number)) == k
        assert set(number) == want


def _pick(rules, times):
    flat = np.array([x for t in times for x in t], np.float32)
    counts = np.array([len(t) for t in times], np.int32)
    rules.pick.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int]
    return rules.pick(flat.ctypes.data, counts.ctypes.data, len(times))


def test_pick_counts_each_launch_once(rules):
    assert _pick(rules, [[1.0] * 3, [0.97] * 3]) == 1
    assert _pick(rules, [[1.0] * 3, [0.985] * 3]) == 0               # within 2%
    assert _pick(rules, [[1.0] * 3, [0.9] * 3, [0.8] * 3, [0.79] * 3]) == 2
    # One fast draw of many does not make a launch faster, one slow draw not slower.
    many = [1.0] * 23 + [0.5]
    assert _pick(rules, [[0.99] * 3, many]) == 0
    assert _pick(rules, [[1.0] * 3, [0.9, 0.9, 5.0]]) == 1
