// Rules that choose how an update's work is divided, in plain C++ for the host,
// the kernels and the tests.
#pragma once

#include <stddef.h>

#ifdef __CUDACC__
#define SPH_RULE __host__ __device__ inline
#else
#define SPH_RULE inline
#endif

namespace sphgb {

// Density pass: whether two warps share a cell (k_density), for a grid of
// `cells` cells of which liveCells held particles before the update, `added`
// particles (counted as 48 a cell) and a GPU of `sms` SMs with 32 resident warps
// each.  Two warps for each occupied cell pay while all of them are resident at
// once.  Full grids, 36 particles a cell, split against not: 1,600 cells 41
// against 59 us, 2,400 49 against 64, 3,000 70 against 68, 16,500 264 against
// 252.  And while it does not cost more to pass over the empty cells twice: 120
// occupied cells of 262,144 41 against 53 us, 2,400 of them 86 against 88; 120 of
// 1,048,576 135 against 78.  They pay again where one warp a cell leaves a last
// wave nearly empty, on nearly full grids: 6,000 cells 109 against 121, 7,225 125
// against 131, 7,650 137 against 135.
SPH_RULE bool density_halves(int cells, int liveCells, int added, int sms) {
	const int live = liveCells + added / 48;
	return live <= 16 * sms ? cells <= 1728 * sms : live > 32 * sms && cells <= 48 * sms;
}

}  // namespace sphgb
