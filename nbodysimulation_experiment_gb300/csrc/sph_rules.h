// Rules that choose how an update's work is divided, in plain C++ for the host,
// the kernels and the tests.
#pragma once

#include <math.h>
#include <stddef.h>

#include <algorithm>
#include <utility>
#include <vector>

#ifdef __CUDACC__
#define SPH_RULE __host__ __device__ inline
#else
#define SPH_RULE inline
#endif

namespace sphgb {

// Density pass: whether two warps share a cell (k_density), for n particles in a
// grid of `cells` cells of which liveCells held particles before the update,
// `added` of the particles new (counted as 48 a cell), and a GPU of `sms` SMs with
// 32 resident warps each.  A cell's second warp has work where it holds more than
// 32 particles, so there are at most n / 33 of those.  They pay while about all
// working warps are resident at once.  Full grids, 36 particles a cell, split
// against not: 1,600 cells 41 against 59 us, 2,400 49 against 64, 3,000 70
// against 68, 16,500 264 against 252.  And while it does not cost more to pass
// over the empty cells twice: 120 occupied cells of 262,144 41 against 53 us,
// 2,400 of them 86 against 88; 120 of 1,048,576 135 against 78.  They pay again
// where one warp a cell leaves a last wave nearly empty, on nearly full grids:
// 6,000 cells 109 against 121, 7,225 125 against 131, 7,650 137 against 135.
SPH_RULE bool density_halves(int cells, int liveCells, int n, int added, int sms) {
	const int live = liveCells + added / 48, second = n / 33 < live ? n / 33 : live;
	return live + second <= 36 * sms ? cells <= 1728 * sms : live > 32 * sms && cells <= 48 * sms;
}

// Particles added since the last update are swept serially in runs of at most
// this many consecutive numbers.
constexpr int kAppendixRun = 32;

// Divides a scene's added particles, in the order they come, into runs: fewer
// than kAppendixRun of them where a particle lies far from the last one and the
// next kStretch near one another, as at the end of a lattice row.  A run across
// that jump would have a box as wide as the lattice: it would wait for, and hold
// up, every run of two rows, and its region would outgrow the sweep's stage
// (30,011 particles in rows of 174: delta sweep of the first update 26 against
// 7 ms).  Where the next ones are far again, as in a random order, another end
// only adds a run (30,000 in random order: 118 against 113 ms).  At most one run
// per sixteen particles in all, whatever their order.
class AppendixRuns {
public:
	size_t from = 0;        // the first run's first number
	std::vector<int> ends;  // where each run ends
	size_t end() const { return ends.empty() ? from : (size_t)ends.back(); }
	void restart(size_t first) {
		from = first;
		ends.clear();
		jump = first;
	}
	// `count` more particles at pos, numbers end() onwards.
	template <class V>
	void add(const V *pos, size_t count, float cellSize) {
		const size_t first = end();
		if (count == 0) return;
		if (!ends.empty()) ends.pop_back();  // the last run goes on
		size_t start = end();
		const float far = 2.0f * cellSize;
		for (size_t k = 0; k < count; ++k) {
			const size_t i = first + k;
			const bool near = i != from && fabsf(pos[k].x - lastX) <= far && fabsf(pos[k].y - lastY) <= far;
			if (!near) jump = i;
			lastX = pos[k].x;
			lastY = pos[k].y;
			// A full run ends at a jump just before, if there is one.
			const bool full = i - start == (size_t)kAppendixRun, recent = jump > start && i - jump <= kStretch;
			if (full || (recent && i - jump == kStretch && (ends.size() + 1) * (kAppendixRun / 2) <= jump - from)) {
				start = recent ? jump : i;
				ends.push_back((int)start);
			}
		}
		ends.push_back((int)(first + count));
	}

private:
	static constexpr size_t kStretch = 3;
	size_t jump = 0;  // the last particle far from the one before (none yet: from)
	float lastX = 0.0f, lastY = 0.0f;
};

// One trial of the sweep autotuner: an update in these shapes.  visc and delta
// number the sweeps' distinct launches in order of appearance.
struct SweepTrial {
	int viscLean, viscBlocks, deltaShape, deltaBlocks;
	int visc = 0, delta = 0;
};

// The trials: the current shapes, then every delta shape at every resident block
// count per SM up to the larger occupancy, each with the viscosity shape of the
// same kind (lean with lean, wide with the pipelined ones).  occV: blocks per SM
// of the wide and lean viscosity; occD: of the delta shapes.
inline std::vector<SweepTrial> sweep_trials(SweepTrial current, const int (&occV)[2], const int *occD, int deltaShapes,
                                            int leanShape, int sms) {
	std::vector<SweepTrial> trials;
	int viscs = 0, deltas = 0;
	auto add = [&](SweepTrial t) {
		t.visc = t.delta = -1;
		for (const SweepTrial &e : trials) {
			if (e.viscLean == t.viscLean && e.viscBlocks == t.viscBlocks) t.visc = e.visc;
			if (e.deltaShape == t.deltaShape && e.deltaBlocks == t.deltaBlocks) t.delta = e.delta;
		}
		if (t.visc < 0) t.visc = viscs++;
		if (t.delta < 0) t.delta = deltas++;
		trials.push_back(t);
	};
	add(current);
	for (int d = 0; d < deltaShapes; ++d) {
		const int lean = d == leanShape ? 1 : 0;
		for (int per = 1; per <= std::max(occV[lean], occD[d]); ++per)
			add({lean, std::min(per, occV[lean]) * sms, d, std::min(per, occD[d]) * sms});
	}
	return trials;
}

// The launch to keep from each launch's times: the first (the current one) unless
// another's median is faster by more than 2%.  All times of a launch count once,
// however many trials ran it: the lean viscosity, one block per SM, runs in
// eight of them, and the fastest of eight draws would be held against the only
// one of others.
inline int pick_launch(std::vector<std::vector<float>> times) {
	int best = 0;
	float bestTime = 0.0f;
	for (size_t k = 0; k < times.size(); ++k) {
		std::vector<float> &t = times[k];
		std::sort(t.begin(), t.end());
		const float median = 0.5f * (t[(t.size() - 1) / 2] + t[t.size() / 2]);
		if (k > 0 && !(median < 0.98f * bestTime)) continue;
		best = (int)k;
		bestTime = median;
	}
	return best;
}

}  // namespace sphgb
