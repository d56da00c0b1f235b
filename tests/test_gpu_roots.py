"""The straight-line square root and reciprocal (csrc/sph_math.cuh) against
CUDA's correctly rounded sqrtf and division, for every float they take: all
2^-96 <= x < 2^96, zero, and samples of everything that goes the general way
(smaller and larger values, the significands excluded from the straight line,
infinity, NaN).  The bits have to be equal."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "nbodysimulation_experiment_gb300", "csrc")

PROGRAM = r"""
#include "sph_math.cuh"
#include <cstdio>
// All bit patterns [lo, lo + n) in steps of `step`: how many differ.
__global__ void check(uint32_t lo, uint64_t n, uint32_t step, unsigned long long *off) {
	for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
		const float x = __uint_as_float(lo + (uint32_t)(i * step));
		const float want = sqrtf(x), wantInv = 1.0f / (want == 0.0f ? 1.0f : want);
		float r;
		const float inv = sphgb::root_and_inverse(x, r);
		const bool nan = want != want;
		if (nan ? r == r : __float_as_uint(r) != __float_as_uint(want)) atomicAdd(&off[0], 1ull);
		if (nan ? inv == inv : __float_as_uint(inv) != __float_as_uint(wantInv)) atomicAdd(&off[1], 1ull);
	}
}
int main() {
	unsigned long long *off, host[2] = {0, 0};
	if (cudaMalloc(&off, sizeof(host)) != cudaSuccess) return 2;
	cudaMemset(off, 0, sizeof(host));
	check<<<2048, 256>>>(31u << 23, (uint64_t)192 << 23, 1u, off);  // [2^-96, 2^96)
	check<<<2048, 256>>>(0u, (uint64_t)31 << 13, 1u << 10, off);    // zero, denormals, below
	check<<<2048, 256>>>(223u << 23, (uint64_t)33 << 13, 1u << 10, off);  // above, infinity, NaN
	if (cudaDeviceSynchronize() != cudaSuccess) return 3;
	cudaMemcpy(host, off, sizeof(host), cudaMemcpyDeviceToHost);
	printf("%llu %llu\n", host[0], host[1]);
	return 0;
}
"""


def test_every_float_of_the_range(tmp_path):
    from nbodysimulation_experiment_gb300 import _build
    src, exe = tmp_path / "roots.cu", tmp_path / "roots"
    src.write_text(PROGRAM)
    subprocess.run([_build.nvcc()] + _build.ARCH + ["-O3", "--fmad=false", "-std=c++17", "-I", CSRC, "-o", str(exe),
                                                    str(src)], check=True, capture_output=True, timeout=300)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out
    assert out.stdout.split() == ["0", "0"]
