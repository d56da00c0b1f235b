// CUDA kernels of the GB300-native Demo4 SPH step (sm_103a).
//
// One Update (NBodySimulation/demo4.cpp:286-451) runs as:
//   k_integrate     integrate forces (demo4.cpp:302-309) + per-step resets
//   k_viscosity     ordered viscosity sweep over the stale neighbour lists
//                   (demo4.cpp:223-237, sph.h:497-512)
//   k_predict       prev = x; x += v dt; new cell (demo4.cpp:329-347, sph.h:450-463)
//   k_scan_*        prefix sums of the grid update
//   k_scatter       appendix and mover lists per cell
//   k_grid_update   the reference's remove/insert grid update, event by event
//                   (demo4.cpp:341-356, 37-76)
//   k_density       density and pressure gather (demo4.cpp:208-221, sph.h:465-481)
//   k_delta         ordered double-density relaxation sweep (demo4.cpp:239-255,
//                   sph.h:483-495)
//   k_collide       body collisions + velocity + renumbering (demo4.cpp:411-450)
//
// Every kernel covers all scenes of the simulation at once (one launch per
// stage): particle numbers and cells carry their scene, whose step scalars,
// grid and bodies live in the scene table.
//
// The two pairwise passes of the reference are serial Gauss-Seidel sweeps in
// particle-number order: a particle's updates land in its neighbours
// immediately.  They are reproduced exactly by running them as dataflow
// "sweeps": a task is a run of consecutively numbered particles of one scene
// processed in order by one thread block, tasks are claimed in increasing
// order, and a task first waits (bounded) until every earlier task of its
// scene whose footprint can overlap its own has finished.  Two particles'
// footprints overlap only when their cells are at most two apart, so with
// particles numbered cell by cell in a 3x3-colour-major cell order most tasks
// are independent; tasks of different scenes never wait on each other.  All
// waits are bounded; a timeout raises kErrTimeout and an abort flag that
// releases every other wait, so a kernel always terminates.
//
// Arithmetic: the library is compiled with --fmad=false and IEEE division and
// square root, and every expression below follows the reference's operation
// order, so per-pair results are bit-identical to the reference.
#include "sph_internal.cuh"
#include "sph_kernels.cuh"
#include "sph_math.cuh"

namespace sphgb {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr uint32_t kWaitLimitIter = 1u << 24;

__device__ __forceinline__ uint64_t global_ns() {
	uint64_t t;
	asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
	return t;
}
__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p) {
	uint32_t v;
	asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
	return v;
}
__device__ __forceinline__ void st_release(uint32_t *p, uint32_t v) {
	asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned lanemask_lt() {
	unsigned m;
	asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
	return m;
}

// Diagnostics: %globaltimer stamps per task (coarse; for task ordering, not
// for sub-microsecond durations).
__device__ __forceinline__ void stamp(const SimTables &T, int sweep, int task, int slot, int lane) {
	if (T.prof != nullptr && lane == 0 && task < T.profStride)
		T.prof[((size_t)sweep * T.profStride + task) * 4 + slot] = global_ns();
}

// Converged bounded wait of a whole warp: each lane names one done flag (or
// none) and the warp polls until every named flag is set.  All lanes run the
// same loop, so a wait never leaves a warp diverged.  Gives up after
// `limitNs` (SimTables::waitLimitNs, 2 s by default) or 2^24 polls, raising
// kErrTimeout and the abort flag that ends every wait.
// A wait is the latency between two tasks of the chain, and a poll late by its
// sleep and by one load after the other: the abort flag is loaded along with
// the named ones, and the sleep stays at 32 ns instead of growing to 256
// (delta sweep of 65,536 particles among obstacles 1.465 -> 1.432 ms, 4,096
// dam break 0.708 -> 0.697, 1M block 2.299 -> 2.279; without any sleep 1.451,
// 0.695 and 2.299).
__device__ __forceinline__ void warp_wait(const uint32_t *flag, uint32_t *abortFlag, uint32_t *err,
                                          unsigned long long limitNs) {
	if (!__any_sync(kFull, flag != nullptr && ld_acquire(flag) == 0u)) return;
	const uint64_t t0 = global_ns();
	for (uint32_t it = 0; it < kWaitLimitIter; ++it) {
		uint32_t aborted;
		asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(aborted) : "l"(abortFlag) : "memory");
		const bool pending = flag != nullptr && ld_acquire(flag) == 0u;
		if (!__any_sync(kFull, pending)) return;
		if (__any_sync(kFull, aborted != 0u)) return;
		if (__any_sync(kFull, global_ns() - t0 > limitNs)) break;
		__nanosleep(32);
	}
	if ((threadIdx.x & 31) == 0) {
		atomicOr(err, kErrTimeout);
		atomicExch(abortFlag, 1u);
	}
}

// Cell of a position within its scene's grid (SPHComputeCellPos + clamp,
// sph.h:450-463): IEEE divide, truncation.
__device__ __forceinline__ int cell_of(float2 p, const StepParams &s) {
	int x = (int)((p.x + s.halfW) / s.cellSize);
	int y = (int)((p.y + s.halfH) / s.cellSize);
	x = min(max(x, 0), s.gx - 1);
	y = min(max(y, 0), s.gy - 1);
	return y * s.gx + x;
}

__device__ __forceinline__ int rect_dist(int ax0, int ay0, int ax1, int ay1, int bx0, int by0, int bx1, int by1) {
	int dx = max(0, max(ax0 - bx1, bx0 - ax1));
	int dy = max(0, max(ay0 - by1, by0 - ay1));
	return max(dx, dy);
}

}  // namespace

// ---------------------------------------------------------------------------
// Integrate forces (demo4.cpp:302-309) and reset the per-step cell tables and
// the sweeps' done flags and task counters.
__global__ void k_integrate(Totals tt, Particles P, SimTables T, uint32_t *doneV, int nDoneV, uint32_t *doneD,
                            int nDoneD) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < tt.n) {
		const StepParams &s = T.scenes[T.sceneOf[i]].p;
		float2 a = P.acc[i];
		float2 v = P.vel[i];
		a.x = s.extX + a.x;  // acceleration += gravity + externalForce
		a.y = s.extY + a.y;
		v.x = a.x * s.dt + v.x;  // velocity += acceleration * dt
		v.y = a.y * s.dt + v.y;
		P.vel[i] = v;
		P.acc[i] = make_float2(0.0f, 0.0f);
	}
	if (i < tt.ncell) {
		const SceneDev &sc = T.scenes[T.sceneOfCell[i]];
		const int local = i - sc.cellBase;
		T.enterCount[i] = 0;
		T.leaveCount[i] = 0;
		T.enterCursor[i] = 0;
		T.appCursor[i] = 0;
		const int cx = local % sc.p.gx, cy = local / sc.p.gx;
		T.bbox[4 * i + 0] = cx;
		T.bbox[4 * i + 1] = cy;
		T.bbox[4 * i + 2] = cx;
		T.bbox[4 * i + 3] = cy;
	}
	const int threads = gridDim.x * blockDim.x;
	for (int k = i; k < nDoneV; k += threads) doneV[k] = 0u;
	for (int k = i; k < nDoneD; k += threads) doneD[k] = 0u;
	if (i == 0) {
		*T.moveMax = 0;
		*T.springBig = 0;
		T.taskCounter[0] = 0;
		T.taskCounter[1] = 0;
	}
}

// ---------------------------------------------------------------------------
// Viscosity sweep.  Task t = canonical cell taskCell[t]; its particles share
// one stale neighbour list: the first (list-time) members of the 3x3 block of
// cells around it, y-major then x, each cell in array order (demo4.cpp:
// 188-201).  The block's positions and velocities are staged in shared
// memory, the task's particles are processed in number order, and the
// block's velocities are written back.  Two tasks conflict iff they belong to
// one scene and their cells are at most two apart; every task waits for the
// earlier conflicting ones.
// One task per block: the even and odd lanes of warp 0 run the ordered velocity
// chains while warps 1..3 compute the compacted pair geometry of the next
// particle (positions do not change during this pass, so the geometry of
// every particle of the task is known in advance).
// The task's particles k = 0, 1, ... sit at consecutive list slots own + k
// of one shared list.  Particle k's pairs before slot own + k - 1 (its head)
// need only what particles < k did at those slots, and particle k - 1 has
// passed them once it is past slot own + k + 1.  So the head of k runs in
// lockstep with the tail of k - 1 (its pairs after slot own + k), on the
// other lane: the two touch disjoint slots.  The middle of k (its pairs with
// k - 1 and k + 1) follows once k - 1 is finished, and k's tail runs
// beside the head of k + 1.  Each particle costs about the longer of its head
// and tail instead of its whole list, with every pair in the reference's
// order for each particle it touches.
// This is the wide shape (ViscWide); the lean one, k_viscosity_multi below,
// runs several tasks per block for throughput.  Particles with more in-range
// pairs than their geometry buffer holds run the geometry inline in the chain
// here; there they come in several segments.
template <class C>
struct ViscSmemT {
	float2 pos[kStageCap];
	float2 vel[kStageCap];
	float4 geo[3][C::kGeom];  // in-range pairs of a particle, list order: byte offset into vel, unit vector, 1 - q
	float4 idle;              // the entry of a chain without pairs: a valid slot, no direction
	int4 split[3];            // pairs, first pair of the middle, first pair of the tail
	int warpCnt[2][C::kWarps];
	int headCnt[C::kWarps], midCnt[C::kWarps];
	int task;
};

namespace {

// Source index of flat position e of NSEG consecutive segments (segment s
// starts at flat offset off[s] and at source index start[s]); selects only,
// so the arrays stay in registers.
template <int NSEG>
__device__ __forceinline__ int seg_src(int e, const int (&off)[NSEG], const int (&start)[NSEG]) {
	int src = start[0] + e;
#pragma unroll
	for (int q = 1; q < NSEG; ++q) src = (e >= off[q]) ? start[q] + (e - off[q]) : src;
	return src;
}

template <class C>
__device__ __forceinline__ void producers_sync() {
	asm volatile("bar.sync 1, %0;" ::"r"(C::kProducers) : "memory");
}

// Geometry of the particle at staged slot `slot` over the L staged entries
// (its whole list): in-range pairs in list order with their unit vectors
// and 1 - q (sph.h:497-505), and where its middle (slots slot-1..slot+1)
// and tail begin.  Run by the producer warps only, in two passes: the
// in-range entries are compacted first (slot, r, r^2), then the square roots
// and divisions run over the dense compacted list.
template <class C>
__device__ __forceinline__ void visc_geometry(ViscSmemT<C> &S, int buf, int slot, int L, const StepParams &s, int p) {
	const int lane = p & (kWarp - 1), w = p / kWarp;
	const float2 xi = S.pos[slot];
	int m = 0, parity = 0, nHead = 0, nToTail = 0;
	for (int base = 0; base < L; base += C::kProducers) {
		const int e = base + p;
		bool in = false;
		float rx = 0.f, ry = 0.f, r2 = 0.f;
		if (e < L) {
			const float2 xj = S.pos[e];
			rx = xj.x - xi.x;
			ry = xj.y - xi.y;
			r2 = rx * rx + ry * ry;
			in = r2 < s.h2 && e != slot;
		}
		nHead += (in && e < slot - 1) ? 1 : 0;
		nToTail += (in && e <= slot + 1) ? 1 : 0;
		const unsigned mask = __ballot_sync(kFull, in);
		int before = m, total = __popc(mask);
		if (C::kProducers > kWarp) {
			if (lane == 0) S.warpCnt[parity][w] = total;
			producers_sync<C>();
			total = 0;
#pragma unroll
			for (int q = 0; q < C::kWarps - 1; ++q) {
				const int c = S.warpCnt[parity][q];
				before += (q < w) ? c : 0;
				total += c;
			}
			parity ^= 1;
		}
		const int at = before + __popc(mask & lanemask_lt());
		if (in && at < C::kGeom) S.geo[buf][at] = make_float4(__int_as_float(8 * e), rx, ry, r2);
		m += total;
	}
	nHead = __reduce_add_sync(kFull, nHead);
	nToTail = __reduce_add_sync(kFull, nToTail);
	if (lane == 0) {
		S.headCnt[w] = nHead;
		S.midCnt[w] = nToTail;
	}
	if (C::kProducers > kWarp) producers_sync<C>(); else __syncwarp();
	if (p == 0) {
		int h = 0, t = 0;
#pragma unroll
		for (int q = 0; q < C::kProducers / kWarp; ++q) {
			h += S.headCnt[q];
			t += S.midCnt[q];
		}
		S.split[buf] = make_int4(m, h, t, 0);
	}
	const int mm = min(m, C::kGeom);
	for (int q = p; q < mm; q += C::kProducers) {
		const float4 g = S.geo[buf][q];
		float r;  // Vec2Length(Rij) == rij
		const float inv = root_and_inverse(g.w, r);
		const float qq = r * s.invH;
		S.geo[buf][q] = make_float4(g.x, g.y * inv, g.z * inv, 1.0f - qq);
	}
}

// One pair of a particle's viscosity chain (sph.h:497-512, demo4.cpp:231-234):
// v_i carries from pair to pair.  The impulse (f n * 0.5) * dt is computed as
// (f n) * (0.5 dt): 0.5 dt is exact and halving is exact, so both round the
// same real product once (unless |f n| < 2^-125).  Only approaching pairs
// (u > 0) exchange an impulse; `live` masks the idle steps of a shorter chain.
// The impulse is computed unconditionally and applied by predicated
// instructions, so a pair's dependent chain is ten FP32 operations and
// neither a select nor a branch ends it (a branch costs nine cycles a pair).
__device__ __forceinline__ void visc_pair(uint32_t at, float2 n, float o, float2 vj, float2 &vi, float sigma,
                                          float beta, float hdt, bool live = true) {
	const float uu = (vi.x - vj.x) * n.x + (vi.y - vj.y) * n.y;
	const float f = o * (sigma * uu + beta * (uu * uu));
	const float ix = (f * n.x) * hdt;
	const float iy = (f * n.y) * hdt;
	const float wx = ix + vj.x, wy = iy + vj.y;
	asm volatile(
	    "{\n"
	    ".reg .pred q, p;\n"
	    "setp.ne.s32 q, %8, 0;\n"
	    "setp.gt.and.f32 p, %2, 0f00000000, q;\n"
	    "@p sub.rn.f32 %0, %0, %3;\n"
	    "@p sub.rn.f32 %1, %1, %4;\n"
	    "@p st.shared.v2.f32 [%5], {%6, %7};\n"
	    "}\n"
	    : "+f"(vi.x), "+f"(vi.y)
	    : "f"(uu), "f"(ix), "f"(iy), "r"(at), "f"(wx), "f"(wy), "r"((int)live)
	    : "memory");
}

__device__ __forceinline__ uint32_t shared_addr(const void *p) {
	return (uint32_t)__cvta_generic_to_shared(p);
}
// Loads of the chains by shared-memory address, in program order with the
// stores of visc_pair.
__device__ __forceinline__ float2 lds2(uint32_t at) {
	float2 v;
	asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(at) : "memory");
	return v;
}
__device__ __forceinline__ float4 lds4(uint32_t at) {
	float4 v;
	asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
	             : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
	             : "r"(at)
	             : "memory");
	return v;
}

// The ordered chain over the len buffered pairs G[0..len) (byte offset of the
// partner's velocity, unit vector, 1 - q), in lockstep with the warp's other
// chains: all run the n >= len steps of the longest.  Steps past len are
// masked; they reload entry len - 1 (`idle`, an entry naming a valid slot,
// when there is none), so no step reads past the buffer.  Software pipeline
// in groups of four pairs: a group's partner velocities load while the group
// before it runs, its geometry one group earlier still, so neither
// shared-memory latency is on the chain.  Each slot occurs once per list and
// the chains touch disjoint slots, so a prefetched velocity is never one that
// changes meanwhile.  The loop leaves after whole pairs of groups: a branch
// costs more than the masked steps it would save.  In isolation, cycles per
// pair of 112: 53, against 68 for loads two pairs ahead and 61 for one pair's
// loads between every two pairs; ten dependent operations alone take 47.
__device__ __forceinline__ void visc_chain(const float2 *vel, const float4 *G, const float4 *idle, int len, int n,
                                           float2 &vi, float sigma, float beta, float hdt) {
	const uint32_t base = shared_addr(vel);
	uint32_t at = shared_addr(len > 0 ? G : idle);
	const uint32_t end = at + 16u * (uint32_t)max(len - 1, 0);
	float4 g[4], h[4];
	float2 v[4], w[4];
#pragma unroll
	for (int u = 0; u < 4; ++u) g[u] = lds4(min(at + 16u * u, end));
#pragma unroll
	for (int u = 0; u < 4; ++u) v[u] = lds2(base + __float_as_uint(g[u].x));
#pragma unroll
	for (int u = 0; u < 4; ++u) h[u] = lds4(min(at + 64u + 16u * u, end));
	int q = 0;
	if (((n + 7) & 7) < 4) {
		// One to four steps over a multiple of eight: a group on its own.
#pragma unroll
		for (int u = 0; u < 4; ++u)
			visc_pair(base + __float_as_uint(g[u].x), make_float2(g[u].y, g[u].z), g[u].w, v[u], vi, sigma, beta, hdt,
			          u < len);
		q = 4;
		at += 64u;
#pragma unroll
		for (int u = 0; u < 4; ++u) {
			g[u] = h[u];
			v[u] = lds2(base + __float_as_uint(g[u].x));
			h[u] = lds4(min(at + 64u + 16u * u, end));
		}
	}
	for (; q < n; q += 8) {
		at += 128u;
#pragma unroll
		for (int u = 0; u < 4; ++u) w[u] = lds2(base + __float_as_uint(h[u].x));
#pragma unroll
		for (int u = 0; u < 4; ++u)
			visc_pair(base + __float_as_uint(g[u].x), make_float2(g[u].y, g[u].z), g[u].w, v[u], vi, sigma, beta, hdt,
			          q + u < len);
#pragma unroll
		for (int u = 0; u < 4; ++u) g[u] = lds4(min(at + 16u * u, end));
#pragma unroll
		for (int u = 0; u < 4; ++u)
			visc_pair(base + __float_as_uint(h[u].x), make_float2(h[u].y, h[u].z), h[u].w, w[u], vi, sigma, beta, hdt,
			          q + 4 + u < len);
#pragma unroll
		for (int u = 0; u < 4; ++u) v[u] = lds2(base + __float_as_uint(g[u].x));
#pragma unroll
		for (int u = 0; u < 4; ++u) h[u] = lds4(min(at + 64u + 16u * u, end));
	}
}

// The whole chain of a particle with more in-range pairs than the geometry
// buffer holds, in list order, its geometry computed here.
template <class C>
__device__ __noinline__ float2 visc_inline(ViscSmemT<C> &S, int slot, int L, float h2, float invH, float sigma, float beta,
                                          float hdt, float2 vi) {
	const uint32_t base = shared_addr(S.vel);
	const float2 xi = S.pos[slot];
	for (int e = 0; e < L; ++e) {
		const float2 xj = S.pos[e];
		const float rx = xj.x - xi.x, ry = xj.y - xi.y;
		const float r2 = rx * rx + ry * ry;
		if (!(r2 < h2)) continue;
		float r;
		const float inv = root_and_inverse(r2, r);
		const float qq = r * invH;
		visc_pair(base + 8u * e, make_float2(rx * inv, ry * inv), 1.0f - qq, S.vel[e], vi, sigma, beta, hdt);
	}
	return vi;
}

__device__ __forceinline__ void visc_phase_bar(int threads) {
	__syncwarp();
	asm volatile("bar.sync 2, %0;" ::"r"(threads) : "memory");
}

// A task's chains (warp 0): even and odd lanes are the two chains, all lanes of
// a chain alike, so that nothing diverges.  cnt particles at slots
// own..own+cnt-1, particle j's geometry in buffer j % 3.  In phase k the chain
// k & 1 starts particle k: its head beside the tail of particle k - 1 on the
// other chain, then (once k - 1 is finished and stored) its middle, the pairs
// with k - 1 and k + 1.  vi is the chain's particle velocity, carried from the
// head to the tail.  A particle with more in-range pairs than the geometry
// buffer holds runs its whole chain in the middle.  Its own pair, which never
// changes a velocity (no direction), is not in the list.  One task of 36
// particles alone, 112 in-range pairs each and 65 on the longer chain: 1,934 ns,
// 4,004 cycles, per particle; 8% more with two lanes of the block's common loop,
// the self pair in the middle and no group on its own (visc_chain).
template <class C>
__device__ __forceinline__ void visc_chains(ViscSmemT<C> &S, int cnt, int own, int L, const StepParams &s) {
	const int c = threadIdx.x & 1;
	const uint32_t base = shared_addr(S.vel);
	const float sigma = s.sigma, beta = s.beta, hdt = 0.5f * s.dt;
	float2 vi = make_float2(0.0f, 0.0f);
	int tailFrom = 0, tailLen = 0;  // of the particle this chain started in the last phase
	for (int k = 0, buf = 0; k <= cnt; ++k, buf = buf == 2 ? 0 : buf + 1) {
		const bool head = (k & 1) == c;
		const int4 sp = k < cnt ? S.split[buf] : make_int4(0, 0, 0, 0);
		const float2 v0 = S.vel[own + min(k, cnt - 1)];
		const bool inl = sp.x > C::kGeom;
		vi = head ? v0 : vi;
		const int mid = head && !inl ? sp.z - sp.y : 0;
		const int len = head ? (inl ? 0 : sp.y) : tailLen;
		const float4 *G = head ? S.geo[buf] : S.geo[buf == 0 ? 2 : buf - 1] + tailFrom;
		float4 gm[2];
#pragma unroll
		for (int u = 0; u < 2; ++u) gm[u] = *(u < mid ? &S.geo[buf][sp.y + u] : &S.idle);
		visc_chain(S.vel, G, &S.idle, len, max(len, __shfl_xor_sync(kFull, len, 1)), vi, sigma, beta, hdt);
		if (!head && k >= 1) S.vel[own + k - 1] = vi;  // particle k - 1 is finished
		__syncwarp();
		if (inl) {
			if (head && (threadIdx.x & (kWarp - 1)) < 2) vi = visc_inline<C>(S, own + k, L, s.h2, s.invH, sigma, beta, hdt, vi);
			vi.x = __shfl_sync(kFull, vi.x, c);
			vi.y = __shfl_sync(kFull, vi.y, c);
		} else {
			float2 vm[2];
#pragma unroll
			for (int u = 0; u < 2; ++u) vm[u] = lds2(base + __float_as_uint(gm[u].x));
#pragma unroll
			for (int u = 0; u < 2; ++u)
				visc_pair(base + __float_as_uint(gm[u].x), make_float2(gm[u].y, gm[u].z), gm[u].w, vm[u], vi, sigma, beta,
				          hdt, u < mid);
		}
		tailFrom = sp.z;
		tailLen = inl ? 0 : sp.x - sp.z;
		visc_phase_bar(C::kWarps * kWarp);
	}
}

}  // namespace

template <class C>
__global__ void __launch_bounds__(C::kWarps * kWarp, C::kMinBlocks) k_viscosity(Totals tt, Particles P, SimTables T) {
	constexpr int kVT = C::kWarps * kWarp;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	ViscSmemT<C> &S = *reinterpret_cast<ViscSmemT<C> *>(smem_raw);
	const int tid = threadIdx.x, warp = tid / kWarp;
	const int nLive = *T.nLive;
	if (tid == 0) S.idle = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
	for (;;) {
		if (tid == 0) S.task = atomicAdd(&T.taskCounter[0], 1);
		__syncthreads();
		const int i = S.task;
		__syncthreads();
		if (i >= nLive) break;
		const int t = T.liveTask[i];
		stamp(T, 0, t, 0, tid);
		const int c = T.taskCell[t];
		const int cnt = T.cellCount[c];
		if (cnt > 0) {
			const SceneDev &sc = T.scenes[T.sceneOfCell[c]];
			const StepParams s = sc.p;
			const int base = sc.cellBase, gx = s.gx, gy = s.gy;
			const int cx = (c - base) % gx, cy = (c - base) / gx;
			// Segments of the 3x3 block in list order.
			int segStart[9], segOff[9];
			int L = 0, own = 0;
#pragma unroll
			for (int q = 0; q < 9; ++q) {
				const int x = cx + q % 3 - 1, y = cy + q / 3 - 1;
				int st = 0, nn = 0;
				if (x >= 0 && x < gx && y >= 0 && y < gy) {
					const int c2 = base + y * gx + x;
					st = T.cellStart[c2];
					nn = T.cellCount[c2];
				}
				segStart[q] = st;
				segOff[q] = L;
				if (q == 4) own = L;
				L += nn;
			}
			auto wait = [&] {
				// Earlier tasks of the scene within Chebyshev distance 2 (warp 0).
				if (warp == 0) {
					const uint32_t *flag = nullptr;
					const int x = cx + tid % 5 - 2, y = cy + tid / 5 - 2;
					if (tid < 25 && tid != 12 && x >= 0 && x < gx && y >= 0 && y < gy) {
						const int c2 = base + y * gx + x;
						const int r2 = T.taskOfCell[c2];
						if (r2 < t && T.cellCount[c2] > 0) flag = &T.done[r2];
					}
					warp_wait(flag, T.abort, T.error, T.waitLimitNs);
				}
				__syncthreads();
				stamp(T, 0, t, 1, tid);
			};
			auto stage = [&](float2 *to, const float2 *from) {
				for (int b0 = 0; b0 < L; b0 += 4 * kVT) {
					float2 v[4];
#pragma unroll
					for (int u = 0; u < 4; ++u) {
						const int e = b0 + u * kVT + tid;
						if (e < L) v[u] = __ldcg(&from[seg_src<9>(e, segOff, segStart)]);
					}
#pragma unroll
					for (int u = 0; u < 4; ++u) {
						const int e = b0 + u * kVT + tid;
						if (e < L) to[e] = v[u];
					}
				}
			};
			if (L > kStageCap) {
				if (tid == 0) atomicOr(T.error, kErrStageOverflow);
				wait();
			} else {
				// The positions, which this pass does not change, and the first
				// particle's geometry before the wait; the velocities after it.
				stage(S.pos, P.pos);
				__syncthreads();
				if (warp > 0) visc_geometry<C>(S, 0, own, L, s, tid - kWarp);
				wait();
				stage(S.vel, P.vel);
				__syncthreads();
				stamp(T, 0, t, 2, tid);
				if (warp == 0) {
					visc_chains<C>(S, cnt, own, L, s);
				} else {
					for (int k = 0, buf = 1; k <= cnt; ++k, buf = buf == 2 ? 0 : buf + 1) {
						if (k + 1 < cnt) visc_geometry<C>(S, buf, own + k + 1, L, s, tid - kWarp);
						visc_phase_bar(C::kWarps * kWarp);
					}
				}
				__syncthreads();
				for (int e = tid; e < L; e += kVT) __stcg(&P.vel[seg_src<9>(e, segOff, segStart)], S.vel[e]);
			}
			__syncthreads();
			__threadfence();
		}
		__syncthreads();
		stamp(T, 0, t, 3, tid);
		if (tid == 0 && i != T.hold[0]) st_release(&T.done[t], 1u);
	}
}

// ---------------------------------------------------------------------------
// Viscosity sweep, many chains per block (the lean shape, ViscLean): the
// same tasks, waits and arithmetic as k_viscosity, laid out for throughput.
// A block holds kSlots tasks at once.  The lanes of kChains chain warps run the
// slots' ordered velocity chains (those of a warp share one instruction
// stream), and a producer warp serves each slot: it claims a task, waits for
// the task's earlier conflicting ones, stages the velocities of its 3x3 block,
// holds the block's positions (which this pass does not change) in registers,
// and keeps the pair geometry ahead of the chain in two buffers; when the chain
// has taken the task's last particle it writes the velocities back and releases
// the task.
// The slots are decoupled: a producer publishes a segment of a particle's pairs
// (ready), the chain lane takes it when its last one ends and says so (taken);
// a particle with more pairs than a buffer holds comes in several segments.
// A chain warp runs eight pairs at a time and its lanes change segments between
// those, so no slot waits for another's longer list or for another's staging.
// (In block-wide phases of one particle each, every phase took as long as the
// longest of its chains, and longer still when some slot changed its task:
// 11,700 cycles per particle on the 1M block against 7,400 alone.)  Blocks of
// cells with more than kVelCap particles run from global memory on their
// producer warp (slot_far_task).
// Eighteen slots and two chain warps: sixteen or twenty slots, one or four
// chain warps measured 0-9% slower (a block of more than 20 warps is left 80
// registers a thread).  A turn of the chain loop takes ~600 cycles for twelve
// pairs, ~160 more when a lane changes segments.  Per update, the same shape in
// block-wide phases first: 1M block 2.60 -> 2.19 ms, 128 scenes 6.42 -> 4.53.
struct ViscDesc {
	int len;    // pairs of the segment
	int own;    // byte offset of the particle's velocity + kSegFirst, kSegLast
	float sigma, beta, hdt;
	int pad[3];
};
constexpr int kSegFirst = 1, kSegLast = 2;
template <class C>
struct ViscSlotT {
	float2 vel[C::kVelCap];   // velocities of the 3x3 block, list order
	float4 geo[2][C::kGeom];  // per buffer: in-range pairs (byte offset into vel, unit vector, 1 - q) of one segment
	float4 pad;               // consecutive slots start 16 bytes apart in the bank space
};
template <class C>
struct ViscMultiSmemT {
	ViscSlotT<C> slot[C::kSlots];
	float4 idle;  // the entry of a chain without pairs
	ViscDesc desc[C::kSlots][2];
	int segStart[C::kSlots][9], segOff[C::kSlots][9];
	uint32_t ready[C::kSlots], taken[C::kSlots];  // segments published by the producer, finished by the chain
	int exited;  // producers that found no more tasks
};

namespace {

__device__ __forceinline__ uint32_t ld_acquire_cta(const uint32_t *p) {
	uint32_t v;
	asm volatile("ld.acquire.cta.shared.u32 %0, [%1];" : "=r"(v) : "r"(shared_addr(p)) : "memory");
	return v;
}
__device__ __forceinline__ void st_release_cta(uint32_t *p, uint32_t v) {
	asm volatile("st.release.cta.shared.u32 [%0], %1;" ::"r"(shared_addr(p)), "r"(v) : "memory");
}

// Bounded wait of a producer warp until the chain has finished `count`
// segments of slot s (a segment takes some 5 us).  False when it gave up, with
// kErrTimeout and the abort flag raised, or saw the abort flag.  Polled every
// 500 ns: more often, the polling slowed the chains (2.67 against 2.88 ms on the
// 1M block), as did reading the global timer.  So waitLimitNs is counted in
// polls, as 512 ns each, and looked at with the abort flag at every eighth
// (2.18 -> 2.19 ms; at every poll 2.23).
template <class C>
__device__ __forceinline__ bool slot_taken(ViscMultiSmemT<C> &S, int s, uint32_t count, const SimTables &T) {
	for (uint32_t it = 0; it < kWaitLimitIter; ++it) {
		const bool ok = (int)(ld_acquire_cta(&S.taken[s]) - count) >= 0;
		if (__all_sync(kFull, ok)) return true;
		if ((it & 7u) == 7u) {
			if (__any_sync(kFull, ld_acquire(T.abort) != 0u)) return false;
			if ((unsigned long long)it << 9 > T.waitLimitNs) break;
		}
		__nanosleep(500);
	}
	if ((threadIdx.x & (kWarp - 1)) == 0) {
		atomicOr(T.error, kErrTimeout);
		atomicExch(T.abort, 1u);
	}
	return false;
}

// A producer warp's open segment.
struct ViscSegment {
	uint32_t seq;  // segments published so far: this one's number
	int m;         // pairs compacted into it
	int own;       // the particle's velocity offset, + kSegFirst on its first segment
};

// Publish the open segment (one warp): the square roots and divisions over
// its compacted entries (byte offset, r, r^2), then its descriptor; wait until
// the next buffer is free.  False when the wait gave up.
template <class C>
__device__ __forceinline__ bool slot_publish(ViscMultiSmemT<C> &S, int s, ViscSegment &g, bool last, float invH,
                                             const StepParams &p, const SimTables &T, int lane) {
	float4 *G = S.slot[s].geo[g.seq & 1u];
	__syncwarp();
	for (int q = lane; q < g.m; q += kWarp) {
		const float4 e = G[q];
		float r;  // Vec2Length(Rij) == rij
		const float inv = root_and_inverse(e.w, r);
		const float qq = r * invH;
		G[q] = make_float4(e.x, e.y * inv, e.z * inv, 1.0f - qq);
	}
	if (lane == 0) {
		ViscDesc &d = S.desc[s][g.seq & 1u];
		d.len = g.m;
		d.own = g.own + (last ? kSegLast : 0);
		d.sigma = p.sigma;
		d.beta = p.beta;
		d.hdt = 0.5f * p.dt;
	}
	__syncwarp();
	++g.seq;
	if (lane == 0) st_release_cta(&S.ready[s], g.seq);
	g.m = 0;
	g.own &= ~kSegFirst;
	// The next buffer held segment seq - 2.
	return g.seq < 2 || slot_taken<C>(S, s, g.seq - 1, T);
}

// One batch of 32 list entries (one per lane, at byte offset `off` of the
// block's velocities, position xj) of the particle at xi: the in-range ones
// (sph.h:497-505) join the segment in list order.
template <class C>
__device__ __forceinline__ bool slot_entries(ViscMultiSmemT<C> &S, int s, ViscSegment &g, int off, float2 xj, bool valid,
                                             float2 xi, float h2, float invH, const StepParams &p, const SimTables &T,
                                             int lane) {
	const float rx = xj.x - xi.x, ry = xj.y - xi.y;
	const float r2 = rx * rx + ry * ry;
	const bool in = valid && r2 < h2;
	const unsigned mask = __ballot_sync(kFull, in);
	const int n = __popc(mask);
	if (g.m + n > C::kGeom && !slot_publish<C>(S, s, g, false, invH, p, T, lane)) return false;
	if (in) S.slot[s].geo[g.seq & 1u][g.m + __popc(mask & lanemask_lt())] = make_float4(__int_as_float(off), rx, ry, r2);
	g.m += n;
	return true;
}

// A chain warp: lane l runs the segments of slot first + l in the order
// published, 3 U pairs per turn of the loop (U = kChainGroup) in three groups
// with a register set each: while a group runs, the next one's partner
// velocities and the next but one's geometry load.  Within a turn a lane's
// next turn is settled (this segment, the next one if this ends here and it is
// ready, or nothing), so its geometry is on its way before the turn ends; what
// depends on the finished pairs (the velocity to store, the next particle's
// own and its first partners') follows at the end, in the turns where a lane
// changes.
// The loop ends once every producer has, and each of their waits is bounded;
// after kChainTurns turns (some 80 s) it ends anyway, and a producer that still
// waits for a segment reports the timeout.
constexpr int kChainGroup = 4;
constexpr uint32_t kChainTurns = 1u << 28;
template <class C>
__device__ __forceinline__ void slot_chains(ViscMultiSmemT<C> &S, int first, int lane) {
	constexpr int kLanes = C::kSlots / C::kChains, U = kChainGroup;
	const bool mine = lane < kLanes;
	const int s = first + (mine ? lane : 0);
	const uint32_t base = shared_addr(S.slot[s].vel), geo = shared_addr(S.slot[s].geo[0]);
	const uint32_t idle = shared_addr(&S.idle);
	uint32_t at = idle, end = idle;  // a turn's first entry, the segment's last
	int left = 0, own = 0;           // pairs left at the start of a turn
	uint32_t seq = 0;                // segments begun
	bool active = false;
	float2 vi = make_float2(0.f, 0.f);
	float sigma = 0.f, beta = 0.f, hdt = 0.f;
	float4 ga[U], gb[U], gc[U];
	float2 va[U], vb[U], vc[U];
	auto geometry = [&](float4(&g)[U], uint32_t from, uint32_t to) {
#pragma unroll
		for (int u = 0; u < U; ++u) g[u] = lds4(min(from + 16u * u, to));
	};
	auto partners = [&](float2(&v)[U], const float4(&g)[U]) {
#pragma unroll
		for (int u = 0; u < U; ++u) v[u] = lds2(base + __float_as_uint(g[u].x));
	};
	auto pairs = [&](const float4(&g)[U], const float2(&v)[U], int first) {
#pragma unroll
		for (int u = 0; u < U; ++u)
			visc_pair(base + __float_as_uint(g[u].x), make_float2(g[u].y, g[u].z), g[u].w, v[u], vi, sigma, beta, hdt,
			          first + u < left);
	};
	geometry(ga, at, end);
	geometry(gb, at, end);
	partners(va, ga);
	for (uint32_t it = 0; it < kChainTurns; ++it) {
		if ((it & 15u) == 0u && !__any_sync(kFull, active)) {
			if (*(volatile int *)&S.exited == C::kSlots) break;
			__nanosleep(64);
		}
		uint32_t rdy;
		asm volatile("ld.relaxed.cta.shared.u32 %0, [%1];" : "=r"(rdy) : "r"(shared_addr(&S.ready[s])) : "memory");
		partners(vb, gb);
		geometry(gc, at + 32u * U, end);
		pairs(ga, va, 0);
		const bool fin = left <= 3 * U, sw = mine && fin && (int)(rdy - seq) > 0;
		const bool event = __any_sync(kFull, sw || (fin && active));
		int leftN = left - 3 * U;
		float4 n4 = make_float4(0.f, 0.f, 0.f, 0.f);
		float nHdt = 0.0f;
		at += 48u * U;
		if (event) {
			__threadfence_block();  // ready before the segment it announces
			const uint32_t desc = shared_addr(&S.desc[s][seq & 1u]);
			n4 = lds4(desc);
			nHdt = lds2(desc + 16u).x;
			if (fin) {
				leftN = sw ? __float_as_int(n4.x) : 0;
				at = leftN > 0 ? geo + (seq & 1u) * (uint32_t)sizeof(S.slot[0].geo[0]) : idle;
				end = at + 16u * (uint32_t)max(leftN - 1, 0);
			}
		}
		partners(vc, gc);
		geometry(ga, at, end);
		pairs(gb, vb, U);
		partners(va, ga);
		geometry(gb, at + 16u * U, end);
		pairs(gc, vc, 2 * U);
		if (event) {
			const int done = fin && active ? 1 : 0;
			asm volatile(
			    "{\n"
			    ".reg .pred p, q;\n"
			    "setp.ne.s32 q, %0, 0;\n"
			    "setp.ne.s32 p, %1, 0;\n"
			    "@p st.shared.v2.f32 [%2], {%3, %4};\n"
			    "@q st.release.cta.shared.u32 [%5], %6;\n"
			    "}\n" ::"r"(done),
			    "r"(done && (own & kSegLast) ? 1 : 0), "r"(base + (own & ~7)), "f"(vi.x), "f"(vi.y),
			    "r"(shared_addr(&S.taken[s])), "r"(seq)
			    : "memory");
			active = fin ? sw : active;
			own = sw ? __float_as_int(n4.y) : own;
			sigma = sw ? n4.z : sigma;
			beta = sw ? n4.w : beta;
			hdt = sw ? nHdt : hdt;
			const float2 nv = lds2(base + (own & ~7));
			if (sw && (own & kSegFirst)) vi = nv;
			seq += sw ? 1u : 0u;
			partners(va, ga);
		}
		left = leftN;
	}
}

// A task whose 3x3 block outgrows the slot, on its producer warp, velocities
// in global memory: per batch of 32 list entries every lane loads and
// evaluates its own, then all lanes run the ordered chain over the in-range
// ones (a partner occurs once per list, so its velocity may be loaded before
// the chain reaches it) and each lane stores its partner's new velocity.
template <class C>
__device__ __noinline__ void slot_far_task(ViscMultiSmemT<C> &S, int s, int L, int first, int cnt, const StepParams &p,
                                           float2 *vel, const float2 *__restrict__ pos, int lane) {
	int segStart[9], segOff[9];
#pragma unroll
	for (int q = 0; q < 9; ++q) {
		segStart[q] = S.segStart[s][q];
		segOff[q] = S.segOff[s][q];
	}
	const float hdt = 0.5f * p.dt;
	for (int k = 0; k < cnt; ++k) {
		const float2 xi = __ldg(&pos[first + k]);
		float2 vi = __ldcg(&vel[first + k]);
		for (int b0 = 0; b0 < L; b0 += kWarp) {
			const int e = b0 + lane;
			const int j = e < L ? seg_src<9>(e, segOff, segStart) : first;
			const float2 xj = __ldg(&pos[j]);
			float2 vj = __ldcg(&vel[j]);
			const float rx = xj.x - xi.x, ry = xj.y - xi.y;
			const float r2 = rx * rx + ry * ry;
			const bool in = e < L && r2 < p.h2;
			float r;
			const float inv = root_and_inverse(r2, r);
			const float nx = rx * inv, ny = ry * inv, o = 1.0f - r * p.invH;
			bool moved = false;
			for (unsigned mask = __ballot_sync(kFull, in); mask; mask &= mask - 1) {
				const int t = __ffs(mask) - 1;
				const float tx = __shfl_sync(kFull, nx, t), ty = __shfl_sync(kFull, ny, t), to = __shfl_sync(kFull, o, t);
				const float wx = __shfl_sync(kFull, vj.x, t), wy = __shfl_sync(kFull, vj.y, t);
				const float uu = (vi.x - wx) * tx + (vi.y - wy) * ty;
				if (uu > 0.0f) {
					const float f = to * (p.sigma * uu + p.beta * (uu * uu));
					const float ix = (f * tx) * hdt;
					const float iy = (f * ty) * hdt;
					vi.x = vi.x - ix;
					vi.y = vi.y - iy;
					if (lane == t) {
						vj = make_float2(ix + wx, iy + wy);
						moved = true;
					}
				}
			}
			if (moved) __stcg(&vel[j], vj);
		}
		__syncwarp();
		if (lane == 0) __stcg(&vel[first + k], vi);
		__syncwarp();
	}
}

// Copy the block's velocities between the slot and global memory (one warp).
template <class C>
__device__ __forceinline__ void slot_copy_vel(ViscMultiSmemT<C> &S, int s, int L, const int (&segStart)[9],
                                              const int (&segOff)[9], const Particles &P, int lane, bool in) {
	float2 *V = S.slot[s].vel;
	for (int b0 = 0; b0 < L; b0 += 4 * kWarp) {
		if (in) {
			float2 v[4];
#pragma unroll
			for (int u = 0; u < 4; ++u) {
				const int e = b0 + u * kWarp + lane;
				if (e < L) v[u] = __ldcg(&P.vel[seg_src<9>(e, segOff, segStart)]);
			}
#pragma unroll
			for (int u = 0; u < 4; ++u) {
				const int e = b0 + u * kWarp + lane;
				if (e < L) V[e] = v[u];
			}
		} else {
#pragma unroll
			for (int u = 0; u < 4; ++u) {
				const int e = b0 + u * kWarp + lane;
				if (e < L) __stcg(&P.vel[seg_src<9>(e, segOff, segStart)], V[e]);
			}
		}
	}
}

// Producer warp of slot s: tasks until none is left.
template <class C>
__device__ __forceinline__ void slot_producer(ViscMultiSmemT<C> &S, int s, const Particles &P, const SimTables &T,
                                              int nLive, int lane) {
	ViscSegment seg{0u, 0, 0};
	for (;;) {
		int i = 0;
		if (lane == 0) i = atomicAdd(&T.taskCounter[0], 1);
		i = __shfl_sync(kFull, i, 0);
		if (i >= nLive) return;
		const int t = T.liveTask[i];
		stamp(T, 0, t, 0, lane);
		const int c = T.taskCell[t];
		const SceneDev &sc = T.scenes[T.sceneOfCell[c]];
		const int base = sc.cellBase, gx = sc.p.gx, gy = sc.p.gy;
		const int cx = (c - base) % gx, cy = (c - base) / gx;
		const float h2 = sc.p.h2, invH = sc.p.invH;
		// Segments of the 3x3 block in list order (lanes 0..8, then a scan).
		int st = 0, nn = 0;
		if (lane < 9) {
			const int x = cx + lane % 3 - 1, y = cy + lane / 3 - 1;
			if (x >= 0 && x < gx && y >= 0 && y < gy) {
				const int c2 = base + y * gx + x;
				st = T.cellStart[c2];
				nn = T.cellCount[c2];
			}
		}
		int incl = nn;
#pragma unroll
		for (int o = 1; o < 16; o <<= 1) {
			const int v = __shfl_up_sync(kFull, incl, o);
			if (lane >= o) incl += v;
		}
		if (lane < 9) {
			S.segStart[s][lane] = st;
			S.segOff[s][lane] = incl - nn;
		}
		const int L = __shfl_sync(kFull, incl, 8);
		const int own = __shfl_sync(kFull, incl - nn, 4);
		const int first = __shfl_sync(kFull, st, 4), cnt = __shfl_sync(kFull, nn, 4);
		__syncwarp();
		// The block's positions do not depend on the earlier tasks.
		float2 px[C::kRegEntries];
		const bool regs = L <= C::kRegEntries * kWarp;
		int segStart[9], segOff[9];
#pragma unroll
		for (int q = 0; q < 9; ++q) {
			segStart[q] = S.segStart[s][q];
			segOff[q] = S.segOff[s][q];
		}
		if (regs) {
#pragma unroll
			for (int r = 0; r < C::kRegEntries; ++r) {
				const int e = r * kWarp + lane;
				px[r] = e < L ? __ldg(&P.pos[seg_src<9>(e, segOff, segStart)]) : make_float2(3.0e38f, 3.0e38f);
			}
		}
		// Wait for earlier tasks of the scene within Chebyshev distance 2.
		{
			const uint32_t *flag = nullptr;
			const int x = cx + lane % 5 - 2, y = cy + lane / 5 - 2;
			if (lane < 25 && lane != 12 && x >= 0 && x < gx && y >= 0 && y < gy) {
				const int c2 = base + y * gx + x;
				const int r2 = T.taskOfCell[c2];
				if (r2 < t && T.cellCount[c2] > 0) flag = &T.done[r2];
			}
			warp_wait(flag, T.abort, T.error, T.waitLimitNs);
		}
		if (__shfl_sync(kFull, lane == 0 ? ld_acquire(T.abort) : 0u, 0) != 0u) return;
		stamp(T, 0, t, 1, lane);
		if (L > kStageCap) {
			// The block does not fit: flag it and release the task untouched.
			if (lane == 0) {
				atomicOr(T.error, kErrStageOverflow);
				st_release(&T.done[t], 1u);
			}
			__syncwarp();
			continue;
		}
		if (L > C::kVelCap) {
			slot_far_task<C>(S, s, L, first, cnt, sc.p, P.vel, P.pos, lane);
		} else {
			slot_copy_vel<C>(S, s, L, segStart, segOff, P, lane, true);
			stamp(T, 0, t, 2, lane);
			float2 xi = __ldg(&P.pos[first]);
			for (int k = 0; k < cnt; ++k) {
				const float2 xn = __ldg(&P.pos[first + min(k + 1, cnt - 1)]);
				seg.own = 8 * (own + k) + kSegFirst;
				bool listed = false;
				if (regs) {
					// One segment: all of the particle's pairs, if they fit.
					float4 *G = S.slot[s].geo[seg.seq & 1u];
					int m = 0;
#pragma unroll
					for (int r = 0; r < C::kRegEntries; ++r) {
						if (r * kWarp >= L) break;
						const float rx = px[r].x - xi.x, ry = px[r].y - xi.y;
						const float r2 = rx * rx + ry * ry;
						const bool in = r2 < h2;
						const unsigned mask = __ballot_sync(kFull, in);
						const int at = m + __popc(mask & lanemask_lt());
						if (in && at < C::kGeom) G[at] = make_float4(__int_as_float(8 * (r * kWarp + lane)), rx, ry, r2);
						m += __popc(mask);
					}
					listed = m <= C::kGeom;
					if (listed) seg.m = m;
				}
				if (!listed) {
					for (int b0 = 0; b0 < L; b0 += kWarp) {
						const int e = b0 + lane;
						const float2 xj = e < L ? __ldg(&P.pos[seg_src<9>(e, segOff, segStart)]) : xi;
						if (!slot_entries<C>(S, s, seg, 8 * e, xj, e < L, xi, h2, invH, sc.p, T, lane)) return;
					}
				}
				if (!slot_publish<C>(S, s, seg, true, invH, sc.p, T, lane)) return;
				xi = xn;
			}
			if (!slot_taken<C>(S, s, seg.seq, T)) return;
			slot_copy_vel<C>(S, s, L, segStart, segOff, P, lane, false);
		}
		__threadfence();
		__syncwarp();
		stamp(T, 0, t, 3, lane);
		if (lane == 0 && i != T.hold[0]) st_release(&T.done[t], 1u);
	}
}

}  // namespace

template <class C>
__global__ void __launch_bounds__(C::kThreads, C::kMinBlocks) k_viscosity_multi(Totals tt, Particles P,
                                                                                           SimTables T) {
	extern __shared__ __align__(16) unsigned char smem_raw[];
	ViscMultiSmemT<C> &S = *reinterpret_cast<ViscMultiSmemT<C> *>(smem_raw);
	const int tid = threadIdx.x, warp = tid / kWarp, lane = tid & (kWarp - 1);
	if (tid < C::kSlots) {
		S.ready[tid] = 0;
		S.taken[tid] = 0;
	}
	if (tid == 0) {
		S.exited = 0;
		S.idle = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
	}
	__syncthreads();
	if (warp < C::kChains) {
		slot_chains<C>(S, warp * (C::kSlots / C::kChains), lane);
	} else {
		slot_producer<C>(S, warp - C::kChains, P, T, *T.nLive, lane);
		__syncwarp();
		if (lane == 0) atomicAdd(&S.exited, 1);
	}
}

// ---------------------------------------------------------------------------
// Reference order (single scene).  The reference's Update visits particles
// in its own index order, which is AddParticle order for a scene that was
// built and then stepped (demo4.cpp:223-255, 344-352).  In reference order
// the library does the same: refOrd lists the particles' numbers in
// AddParticle order; the viscosity sweep runs as tasks of kAppendixRun
// consecutive AddParticle indices (k_viscosity_ref), the delta sweep as the
// same runs over the whole scene (k_delta's run path), and the grid update
// applies each cell's events in AddParticle order.

__global__ void k_ref_order(Totals tt, Particles P, SimTables T) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= tt.n) return;
	const SceneDev &sc = T.scenes[T.sceneOf[i]];
	const int id = P.id[i];
	if (id < 0 || id >= sc.n) {
		atomicOr(T.error, kErrIndex);
		return;
	}
	T.refOrd[sc.pBase + id] = i;
}

// Bounding box (cell coordinates) of the old cells of each viscosity run:
// the cells whose canonical arrays made its particles' neighbour lists.  One
// warp per run.
__global__ void k_visc_boxes(Totals tt, Particles P, SimTables T) {
	const int a = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
	const int lane = threadIdx.x & (kWarp - 1);
	if (a >= tt.nViscRuns) return;
	const SceneDev &sc = T.scenes[0];
	const int gx = sc.p.gx;
	const int p0 = sc.pBase + a * kAppendixRun;
	const int p1 = min(sc.pBase + sc.n0, p0 + kAppendixRun);
	int bx0 = sc.p.gx, by0 = sc.p.gy, bx1 = -1, by1 = -1;
	for (int k = p0 + lane; k < p1; k += kWarp) {
		const int lc = P.cellOf[T.refOrd[k]] - sc.cellBase;
		bx0 = min(bx0, lc % gx);
		bx1 = max(bx1, lc % gx);
		by0 = min(by0, lc / gx);
		by1 = max(by1, lc / gx);
	}
	for (int o = 16; o > 0; o >>= 1) {
		bx0 = min(bx0, __shfl_xor_sync(kFull, bx0, o));
		by0 = min(by0, __shfl_xor_sync(kFull, by0, o));
		bx1 = max(bx1, __shfl_xor_sync(kFull, bx1, o));
		by1 = max(by1, __shfl_xor_sync(kFull, by1, o));
	}
	if (lane == 0) *reinterpret_cast<int4 *>(&T.viscBox[4 * a]) = make_int4(bx0, by0, bx1, by1);
}

// Viscosity sweep in reference order: one warp per task (run a: the
// canonical particles with AddParticle indices a*kAppendixRun onwards), each
// task waiting for the earlier runs whose old cells come within two cells of
// its own.  For each particle, in order, the warp walks its stale list (the
// 3x3 block of canonical cell arrays around its old cell, demo4.cpp:188-201)
// 32 entries at a time, computing the pair geometry of the in-range entries
// (sph.h:497-505), and lane 0 runs the ordered velocity chain over them
// (demo4.cpp:231-234), velocities in global memory.
__global__ void __launch_bounds__(kViscRefWarps * kWarp) k_viscosity_ref(Totals tt, Particles P, SimTables T) {
	__shared__ float4 geo[kViscRefWarps][kWarp];
	const int lane = threadIdx.x & (kWarp - 1), w = threadIdx.x / kWarp;
	const SceneDev &sc = T.scenes[0];
	const StepParams s = sc.p;
	const int base = sc.cellBase, gx = s.gx, gy = s.gy;
	const float hdt = 0.5f * s.dt;
	for (;;) {
		int a = 0;
		if (lane == 0) a = atomicAdd(&T.taskCounter[0], 1);
		a = __shfl_sync(kFull, a, 0);
		if (a >= tt.nViscRuns) break;
		const int4 box = *reinterpret_cast<const int4 *>(&T.viscBox[4 * a]);
		for (int q0 = 0; q0 < a; q0 += kWarp) {
			const int q = q0 + lane;
			const uint32_t *flag = nullptr;
			if (q < a) {
				const int4 o = *reinterpret_cast<const int4 *>(&T.viscBox[4 * q]);
				if (rect_dist(o.x, o.y, o.z, o.w, box.x, box.y, box.z, box.w) <= 2) flag = &T.done[q];
			}
			warp_wait(flag, T.abort, T.error, T.waitLimitNs);
		}
		const int p0 = sc.pBase + a * kAppendixRun;
		const int p1 = min(sc.pBase + sc.n0, p0 + kAppendixRun);
		for (int k = p0; k < p1; ++k) {
			const int i = T.refOrd[k];
			const int lc = P.cellOf[i] - base;
			const int cx = lc % gx, cy = lc / gx;
			const float2 xi = P.pos[i];
			float2 vi = __ldcg(&P.vel[i]);
			for (int q = 0; q < 9; ++q) {
				const int x = cx + q % 3 - 1, y = cy + q / 3 - 1;
				if (x < 0 || x >= gx || y < 0 || y >= gy) continue;
				const int c2 = base + y * gx + x;
				const int st = T.cellStart[c2], nn = T.cellCount[c2];
				for (int b0 = 0; b0 < nn; b0 += kWarp) {
					const int e = b0 + lane;
					bool in = false;
					if (e < nn) {
						const int j = st + e;
						const float2 xj = P.pos[j];
						const float rx = xj.x - xi.x, ry = xj.y - xi.y;
						const float r2 = rx * rx + ry * ry;
						in = r2 < s.h2;
						if (in) {
							const float r = sqrtf(r2);
							const float qq = r * s.invH;
							float len = r;  // Vec2Length(Rij) == rij
							if (len == 0.0f) len = 1.0f;
							const float inv = 1.0f / len;
							geo[w][lane] = make_float4(__int_as_float(j), rx * inv, ry * inv, 1.0f - qq);
						}
					}
					unsigned mask = __ballot_sync(kFull, in);
					__syncwarp();
					if (lane == 0) {
						while (mask) {
							const int t = __ffs(mask) - 1;
							mask &= mask - 1;
							const float4 g = geo[w][t];
							const int j = __float_as_int(g.x);
							const float2 vj = __ldcg(&P.vel[j]);
							const float2 n = make_float2(g.y, g.z);
							const float uu = (vi.x - vj.x) * n.x + (vi.y - vj.y) * n.y;
							if (uu > 0.0f) {
								const float f = g.w * (s.sigma * uu + s.beta * (uu * uu));
								const float ix = (f * n.x) * hdt;
								const float iy = (f * n.y) * hdt;
								vi.x = vi.x - ix;
								vi.y = vi.y - iy;
								__stcg(&P.vel[j], make_float2(ix + vj.x, iy + vj.y));
							}
						}
					}
					__syncwarp();
				}
			}
			if (lane == 0) __stcg(&P.vel[i], vi);
			__syncwarp();
		}
		__threadfence();
		__syncwarp();
		if (lane == 0 && a != T.hold[0]) st_release(&T.done[a], 1u);
	}
}

// ---------------------------------------------------------------------------
// Predict (demo4.cpp:329-337) and the new cell (demo4.cpp:347).  Movers
// extend the bounding box of new cells of their old cell, count as leaving
// their old cell and entering their new cell.  The one word that all movers
// share, the longest move, is read first: an atomic from each of them took
// most of the pass (1M block 54 -> 23 us, 128 scenes 120 -> 35).
__global__ void k_predict(Totals tt, Particles P, SimTables T) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= tt.n) return;
	const SceneDev &sc = T.scenes[T.sceneOf[i]];
	const float2 x = P.pos[i];
	const float2 v = P.vel[i];
	P.prev[i] = x;
	const float2 xn = make_float2(v.x * sc.p.dt + x.x, v.y * sc.p.dt + x.y);
	P.pos[i] = xn;
	const int local = cell_of(xn, sc.p);
	const int nc = sc.cellBase + local;
	T.newCell[i] = nc;
	const int oc = P.cellOf[i];
	if (nc != oc) {
		atomicAdd(&T.enterCount[nc], 1);
		atomicAdd(&T.leaveCount[oc], 1);
		const int gx = sc.p.gx;
		const int nx = local % gx, ny = local / gx;
		const int ox = (oc - sc.cellBase) % gx, oy = (oc - sc.cellBase) / gx;
		// The box holds the old cell already.
		if (nx < ox) atomicMin(&T.bbox[4 * oc + 0], nx);
		if (ny < oy) atomicMin(&T.bbox[4 * oc + 1], ny);
		if (nx > ox) atomicMax(&T.bbox[4 * oc + 2], nx);
		if (ny > oy) atomicMax(&T.bbox[4 * oc + 3], ny);
		const int move = max(abs(nx - ox), abs(ny - oy));
		if (__ldcg(T.moveMax) < move) atomicMax(T.moveMax, move);
	}
}

// ---------------------------------------------------------------------------
// The occupied canonical cells in task order (both sweeps skip empty cells):
// per-tile counts (not launched for a single tile), then the compacted list.

__global__ void __launch_bounds__(kScanThreads) k_live_reduce(Totals tt, SimTables T) {
	__shared__ int part[kScanThreads / kWarp];
	const int tile = blockIdx.x;
	int cnt = 0;
	for (int k = 0; k < kScanTile / kScanThreads; ++k) {
		const int t = tile * kScanTile + k * kScanThreads + threadIdx.x;
		if (t < tt.ncell) cnt += T.cellCount[T.taskCell[t]] > 0;
	}
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(kFull, cnt, o);
	if ((threadIdx.x & (kWarp - 1)) == 0) part[threadIdx.x / kWarp] = cnt;
	__syncthreads();
	if (threadIdx.x == 0) {
		int sum = 0;
		for (int w = 0; w < kScanThreads / kWarp; ++w) sum += part[w];
		T.liveTiles[tile] = sum;
	}
}

namespace {

// Four consecutive values of an n-element table from position r, a multiple
// of four; 0 past the end.
__device__ __forceinline__ void load_four(int (&v)[4], const int *p, int r, int n) {
	if (r + 4 <= n) {
		const int4 x = *reinterpret_cast<const int4 *>(p + r);
		v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
	} else {
#pragma unroll
		for (int k = 0; k < 4; ++k) v[k] = r + k < n ? p[r + k] : 0;
	}
}

// The running prefix from `first` over four consecutive values into a table's
// positions from r on.
__device__ __forceinline__ void store_prefix(int *p, int r, int n, int first, const int (&v)[4]) {
	const int4 x = make_int4(first, first + v[0], first + v[0] + v[1], first + v[0] + v[1] + v[2]);
	if (r + 4 <= n) {
		*reinterpret_cast<int4 *>(p + r) = x;
	} else {
		if (r < n) p[r] = x.x;
		if (r + 1 < n) p[r + 1] = x.y;
		if (r + 2 < n) p[r + 2] = x.z;
	}
}

// Block-wide exclusive scans (kScanThreads threads) of N tables, each on top of
// the `tile` tiles before this one: tiles[q * ntiles] holds the tiles' sums or,
// past kScanFewTiles of them, their offsets.  A thread brings one value of each
// table, of the last one a value of each of S consecutive parts of the tile.
// v[q] becomes the prefix; the thread of warp q's last lane returns the sum up
// to and including this tile, or this part, others 0.  One use of sums per
// kernel.
template <int N, int S>
__device__ __forceinline__ int block_exscan(int (&v)[N - 1 + S], int (*sums)[kWarp], const int *tiles, int tile,
                                            int ntiles) {
	constexpr int V = N - 1 + S;
	static_assert(kScanThreads == kWarp * kWarp && V <= kWarp, "one value per lane of the second level");
	const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
	int incl[V];
#pragma unroll
	for (int q = 0; q < V; ++q) {
		incl[q] = v[q];
#pragma unroll
		for (int o = 1; o < kWarp; o <<= 1) {
			const int t = __shfl_up_sync(kFull, incl[q], o);
			if (lane >= o) incl[q] += t;
		}
		if (lane == kWarp - 1) sums[q][warp] = incl[q];
	}
	int before = 0, total = 0;
	if (warp < N && ntiles > kScanFewTiles) {
		before = tiles[warp * ntiles + tile];
	} else if (warp < N) {
		for (int i = lane; i < tile; i += kWarp) before += tiles[warp * ntiles + i];
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(kFull, before, o);
	}
	__syncthreads();
	if (warp < V) {
		const int w = sums[warp][lane];
		int wi = w;
#pragma unroll
		for (int o = 1; o < kWarp; o <<= 1) {
			const int t = __shfl_up_sync(kFull, wi, o);
			if (lane >= o) wi += t;
		}
		sums[warp][lane] = before + wi - w;
		if (lane == kWarp - 1) sums[V][warp] = total = before + wi;
	}
	__syncthreads();
	int part = 0;  // sum of the parts before (the first one's includes the tiles before)
#pragma unroll
	for (int q = 0; q < V; ++q) {
		v[q] = sums[q][warp] + incl[q] - v[q] + part;
		if (q >= N - 1) part += sums[V][q];
	}
	return total;
}

}  // namespace

// The sums of ntiles tiles at tiles[blockIdx.x * ntiles] become the tiles'
// offsets.  For grids of more than kScanFewTiles tiles: there each block of the
// next pass would add up the sums before its own, a time that grows with the
// number of tiles for each of them (both passes of an update on 2^26 cells,
// 16,382 tiles: 2.25 ms more than with this pass; equal at 512 tiles, 3 us
// less without it at 64).
__global__ void __launch_bounds__(kScanThreads) k_tile_offsets(int *tiles, int ntiles) {
	__shared__ int sums[2][kWarp], carry;
	int *row = tiles + (size_t)blockIdx.x * ntiles;
	int before = 0;
	for (int base = 0; base < ntiles; base += 4 * kScanThreads) {
		int x[4], v[1] = {0};
		const int r = base + 4 * threadIdx.x;
#pragma unroll
		for (int k = 0; k < 4; ++k) {
			x[k] = r + k < ntiles ? row[r + k] : 0;
			v[0] += x[k];
		}
		const int total = block_exscan<1, 1>(v, sums, nullptr, 0, 1);
		if (threadIdx.x == kWarp - 1) carry = total;
		v[0] += before;
#pragma unroll
		for (int k = 0; k < 4; ++k) {
			if (r + k < ntiles) row[r + k] = v[0];
			v[0] += x[k];
		}
		__syncthreads();
		before += carry;
		__syncthreads();
	}
}

__global__ void __launch_bounds__(kScanThreads) k_live_apply(Totals tt, SimTables T) {
	__shared__ int sums[2][kWarp];
	const int tile = blockIdx.x, r = tile * kScanTile + 4 * threadIdx.x;
	int c[4], v[1] = {0};
	bool live[4];
	load_four(c, T.taskCell, r, tt.ncell);
#pragma unroll
	for (int k = 0; k < 4; ++k) {
		live[k] = r + k < tt.ncell && T.cellCount[c[k]] > 0;
		v[0] += live[k];
	}
	const int total = block_exscan<1, 1>(v, sums, T.liveTiles, tile, gridDim.x);
	if (tile == gridDim.x - 1 && threadIdx.x == kWarp - 1) *T.nLive = total;
#pragma unroll
	for (int k = 0; k < 4; ++k)
		if (live[k]) T.liveTask[v[0]++] = r + k;
}

// ---------------------------------------------------------------------------
// Exclusive scans over cells, in two passes over tiles of kScanTile positions:
// per-tile sums (not launched for a single tile), then per-tile scans, each
// block adding up the sums of the tiles before its own, or past kScanFewTiles
// reading them from a pass between (k_tile_offsets).  Three scans run
// together: the appendix counts and the entering counts in cell order, and
// the new cell counts (cellCount + appCount - leaveCount + enterCount) in
// numbering order (scenes in order, cells in colour rank).  Bound by launches
// and barriers on small grids, not by the few bytes: all values of a tile are
// scanned at once, so a block has two barriers (36 with one position at a time
// and one scan after another).  On large ones by the accesses by cell of the
// new counts: a thread takes one position in each quarter of the tile for
// them, so that a warp's are near one another, and four consecutive positions
// of the two tables in cell order (four consecutive ones of all three: 102
// against 60 us on 2048 x 2048 cells, 9.8 against 8.4 on 512 x 512).
// Together with the task list above and the task flags cleared in k_integrate
// instead of by four memsets: 451 -> 425 us per update at 256 particles,
// 1,527 -> 1,503 at 4,096 (dam break), 2,836 -> 2,816 at 65,536.

namespace {

__device__ __forceinline__ int new_count(const SimTables &T, int c) {
	return T.cellCount[c] + T.appCount[c] - T.leaveCount[c] + T.enterCount[c];
}

}  // namespace

// Pass 1: the three sums of every tile.
__global__ void __launch_bounds__(kScanThreads) k_scan_reduce(Totals tt, SimTables T) {
	__shared__ int part[3][kScanThreads / kWarp];
	const int t = blockIdx.x;
	int a = 0, e = 0, nw = 0;
	for (int k = 0; k < kScanTile / kScanThreads; ++k) {
		const int r = t * kScanTile + k * kScanThreads + threadIdx.x;
		if (r < tt.ncell) {
			a += T.appCount[r];
			e += T.enterCount[r];
			nw += new_count(T, T.numberOrder[r]);
		}
	}
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) {
		a += __shfl_xor_sync(kFull, a, o);
		e += __shfl_xor_sync(kFull, e, o);
		nw += __shfl_xor_sync(kFull, nw, o);
	}
	const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
	if (lane == 0) {
		part[0][warp] = a;
		part[1][warp] = e;
		part[2][warp] = nw;
	}
	__syncthreads();
	if (threadIdx.x < 3) {
		int sum = 0;
		for (int w = 0; w < kScanThreads / kWarp; ++w) sum += part[threadIdx.x][w];
		T.scanTiles[threadIdx.x * gridDim.x + t] = sum;
	}
}

// Pass 2: per-tile scans plus the tile offsets; writes appStart, enterOffset,
// newCount and newStart.  Also restarts the per-scene neighbour-count
// statistics (demo4.cpp:369-370).
__global__ void __launch_bounds__(kScanThreads) k_scan_apply(Totals tt, SimTables T) {
	constexpr int kParts = kScanTile / kScanThreads;
	static_assert(kParts == 4, "load_four");
	__shared__ int sums[3 + kParts][kWarp];
	const int t = blockIdx.x, r = t * kScanTile + 4 * threadIdx.x, r0 = t * kScanTile + threadIdx.x;
	int a[4], e[4], c[kParts], nw[kParts], v[2 + kParts] = {};
	load_four(a, T.appCount, r, tt.ncell);
	load_four(e, T.enterCount, r, tt.ncell);
#pragma unroll
	for (int k = 0; k < kParts; ++k) {
		const int p = r0 + k * kScanThreads;
		c[k] = p < tt.ncell ? T.numberOrder[p] : -1;
		nw[k] = v[2 + k] = c[k] >= 0 ? new_count(T, c[k]) : 0;
		v[0] += a[k];
		v[1] += e[k];
	}
	block_exscan<3, kParts>(v, sums, T.scanTiles, t, gridDim.x);
	store_prefix(T.appStart, r, tt.ncell, v[0], a);
	store_prefix(T.enterOffset, r, tt.ncell, v[1], e);
#pragma unroll
	for (int k = 0; k < kParts; ++k) {
		if (c[k] >= 0) {
			T.newCount[c[k]] = nw[k];
			T.newStart[c[k]] = v[2 + k];
		}
	}
	if (t == 0) {
		for (int sc = threadIdx.x; sc < tt.nscenes; sc += blockDim.x) {
			T.stats[4 * sc + 0] = T.scenes[sc].nbSeed;
			T.stats[4 * sc + 1] = 0;
			if (T.springTotal) T.springTotal[sc] = 0;
		}
	}
}

// Appendix members and movers into per-cell lists (order fixed later).
__global__ void k_scatter(Totals tt, Particles P, SimTables T) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= tt.n) return;
	const SceneDev &sc = T.scenes[T.sceneOf[i]];
	const int oc = P.cellOf[i];
	if (i - sc.pBase >= sc.n0) {
		const int slot = T.appStart[oc] + atomicAdd(&T.appCursor[oc], 1);
		T.appIdx[slot] = i;
	}
	const int nc = T.newCell[i];
	if (nc != oc) {
		const int slot = T.enterOffset[nc] + atomicAdd(&T.enterCursor[nc], 1);
		T.enterList[slot] = i;
	}
}

// ---------------------------------------------------------------------------
// Grid update, exactly as the reference's serial loop (demo4.cpp:344-352):
// particles in number order that changed cell are removed from the old cell
// by swap-with-last (demo4.cpp:56-76) and appended to the new one
// (demo4.cpp:37-54).  A cell's final array depends only on the order of its
// own events, so each warp replays one cell's events in number order.
// Bound by the cell with the most events: one lane's search for the leaving
// particle and its insertion sorts took 1 us an event; 32 places looked at
// once and ranks counted by all lanes, update_grid of 65,536 particles among
// obstacles 63 -> 34 us, dense 1M 258 -> 124, 1M block 119 -> 85, 128 scenes
// 274 -> 162.

struct GridWarp {
	int arr[kCellCap];
	int leave[kCellCap];
	int enter[kCellCap];
};

// Numbers sorted by their particles' AddParticle index (reference order).
__device__ void insertion_sort_by_id(int *a, int n, const int *id) {
	for (int i = 1; i < n; ++i) {
		const int v = a[i];
		const int key = id[v];
		int j = i - 1;
		while (j >= 0 && id[a[j]] > key) {
			a[j + 1] = a[j];
			--j;
		}
		a[j + 1] = v;
	}
}

// The n distinct values of a in ascending order of their keys, by one warp:
// a value's place is the number of smaller keys.  tmp has room for n.
template <class Key>
__device__ __forceinline__ void rank_sort(int *a, int *tmp, int n, int lane, Key key) {
	if (n < 2) return;
	for (int j = lane; j < n; j += kWarp) {
		const int v = a[j], k = key(v);
		int rank = 0;
		for (int i = 0; i < n; ++i) rank += key(a[i]) < k;
		tmp[rank] = v;
	}
	__syncwarp();
	for (int j = lane; j < n; j += kWarp) a[j] = tmp[j];
	__syncwarp();
}

__global__ void __launch_bounds__(kGridWarps * kWarp) k_grid_update(Totals tt, Particles P, Particles Q, SimTables T) {
	__shared__ GridWarp W[kGridWarps];
	GridWarp &S = W[threadIdx.x / kWarp];
	const int lane = threadIdx.x & (kWarp - 1);
	const int n = tt.n;
	const int warpsTotal = gridDim.x * kGridWarps;
	for (int c = blockIdx.x * kGridWarps + threadIdx.x / kWarp; c < tt.ncell; c += warpsTotal) {
		const int cs = T.cellStart[c], cc = T.cellCount[c];
		const int as = T.appStart[c], ac = T.appCount[c];
		const int eo = T.enterOffset[c], ec = T.enterCount[c];
		const int init = cc + ac;
		const int outStart = T.newStart[c], outCount = T.newCount[c];
		if (init == 0 && ec == 0) continue;
		uint32_t *stats = T.stats + 4 * T.sceneOfCell[c];
		if (init + ec > kCellCap || outCount > kCellCap) {
			// Over capacity: keep memory consistent (members in some order)
			// and report; the result of this update is not meaningful.
			if (lane == 0) {
				atomicOr(T.error, kErrCellOverflow);
				int w = 0;
				for (int j = 0; j < cc && w < outCount; ++j)
					if (T.newCell[cs + j] == c) T.newIdx[outStart + w++] = cs + j;
				for (int j = 0; j < ac && w < outCount; ++j)
					if (T.newCell[T.appIdx[as + j]] == c) T.newIdx[outStart + w++] = T.appIdx[as + j];
				for (int j = 0; j < ec && w < outCount; ++j) T.newIdx[outStart + w++] = T.enterList[eo + j];
				for (; w < outCount; ++w) T.newIdx[outStart + w] = 0;
				for (int j = 0; j < outCount; ++j) {
					const int p = T.newIdx[outStart + j];
					T.newLabel[p] = outStart + j;
					Q.pos[outStart + j] = P.pos[p];
				}
			}
			__syncwarp();
			continue;
		}
		for (int j = lane; j < cc; j += kWarp) S.arr[j] = cs + j;
		for (int j = lane; j < ac; j += kWarp) S.arr[cc + j] = T.appIdx[as + j];
		for (int j = lane; j < ec; j += kWarp) S.enter[j] = T.enterList[eo + j];
		__syncwarp();
		// Appendix members joined in number order (their AddParticle order);
		// entering particles are applied in number order, or in AddParticle
		// order in reference order.
		rank_sort(S.arr + cc, S.leave, ac, lane, [](int v) { return v; });
		if (tt.refOrder)
			rank_sort(S.enter, S.leave, ec, lane, [&](int v) { return P.id[v]; });
		else
			rank_sort(S.enter, S.leave, ec, lane, [](int v) { return v; });
		// Leaving particles, in number order (the array is sorted here); in
		// reference order they are sorted by AddParticle index below.
		int nl = 0;
		for (int base = 0; base < init; base += kWarp) {
			const int j = base + lane;
			bool lv = false;
			int p = 0;
			if (j < init) {
				p = S.arr[j];
				lv = T.newCell[p] != c;
			}
			const unsigned mask = __ballot_sync(kFull, lv);
			if (lv) S.leave[nl + __popc(mask & lanemask_lt())] = p;
			nl += __popc(mask);
		}
		__syncwarp();
		if (tt.refOrder) {
			if (lane == 0) insertion_sort_by_id(S.leave, nl, P.id);
			__syncwarp();
		}
		// The events in order, by all lanes alike; 32 places are searched at once.
		int cnt = init;
		int lo = 0x7fffffff, hi = 0;
		int a = 0, b = 0;
		while (a < nl || b < ec) {
			bool leaveFirst = b >= ec;
			if (a < nl && b < ec)
				leaveFirst = tt.refOrder ? P.id[S.leave[a]] < P.id[S.enter[b]] : S.leave[a] < S.enter[b];
			if (leaveFirst) {
				const int p = S.leave[a++];
				const int last = cnt - 1;
				int at = cnt;
				for (int base = 0; base < cnt; base += kWarp) {
					const unsigned hit = __ballot_sync(kFull, base + lane < cnt && S.arr[base + lane] == p);
					if (hit != 0) {
						at = base + __ffs(hit) - 1;
						break;
					}
				}
				if (at < cnt && at != last) {
					const int moved = S.arr[last];
					__syncwarp();
					if (lane == 0) {
						S.arr[at] = moved;
						S.arr[last] = p;
					}
				}
				--cnt;
			} else {
				if (lane == 0) S.arr[cnt] = S.enter[b];
				++cnt;
				++b;
			}
			__syncwarp();
			lo = min(lo, cnt);
			hi = max(hi, cnt);
		}
		if (lane == 0) {
			if (nl + ec > 0) {
				atomicMin(&stats[2], (uint32_t)lo);
				atomicMax(&stats[3], (uint32_t)hi);
			}
			if (cnt != outCount) atomicOr(T.error, kErrIndex);
		}
		__syncwarp();
		// The new cell arrays are the next canonical numbering: the particle
		// at position j of cell c becomes number newStart[c] + j.  Positions
		// are gathered into that order for the density and delta passes.
		for (int j = lane; j < outCount; j += kWarp) {
			int p = S.arr[j];
			if (p < 0 || p >= n) {
				atomicOr(T.error, kErrIndex);
				p = 0;
			}
			T.newIdx[outStart + j] = p;
			T.newLabel[p] = outStart + j;
			Q.pos[outStart + j] = P.pos[p];
		}
		__syncwarp();
	}
}

// Bounding box (scene-local cell coordinates) of the new cells of each
// appendix run (in reference order: of each run of the whole scene in
// AddParticle order); one warp per run.
__global__ void k_app_boxes(Totals tt, SimTables T) {
	const int a = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
	const int lane = threadIdx.x & (kWarp - 1);
	if (a >= tt.nApp) return;
	const SceneDev &sc = T.scenes[T.appScene[a]];
	const int gx = sc.p.gx;
	const int p0 = sc.pBase + T.appFrom[a], p1 = sc.pBase + T.appTo[a];
	int bx0 = sc.p.gx, by0 = sc.p.gy, bx1 = -1, by1 = -1;
	for (int k = p0 + lane; k < p1; k += kWarp) {
		const int lc = T.newCell[tt.refOrder ? T.refOrd[k] : k] - sc.cellBase;
		bx0 = min(bx0, lc % gx);
		bx1 = max(bx1, lc % gx);
		by0 = min(by0, lc / gx);
		by1 = max(by1, lc / gx);
	}
	for (int o = 16; o > 0; o >>= 1) {
		bx0 = min(bx0, __shfl_xor_sync(kFull, bx0, o));
		by0 = min(by0, __shfl_xor_sync(kFull, by0, o));
		bx1 = max(bx1, __shfl_xor_sync(kFull, bx1, o));
		by1 = max(by1, __shfl_xor_sync(kFull, by1, o));
	}
	if (lane == 0) *reinterpret_cast<int4 *>(&T.appBox[4 * a]) = make_int4(bx0, by0, bx1, by1);
}

// ---------------------------------------------------------------------------
// Density and pressure (demo4.cpp:208-221): a pure gather.  One warp per new
// cell; each lane sums the lists of up to two of the cell's particles (the 3x3
// block of the new cell arrays, demo4.cpp:183-206) in list order.  The block
// is staged in chunks of kDensChunk entries, so a warp needs little shared
// memory and many warps fit on an SM.
//
// Bound by instruction issue on large grids (1M block: 0.78 instructions per
// cycle and scheduler, DRAM 0.3 %), so a cell, or the rest of one, of at most
// 32 particles runs the loop with one list per lane instead of an empty second
// one (128 scenes 0.81 -> 0.71 ms, 1M block 0.44 -> 0.43).  With few occupied
// cells it is bound by one warp's time for its cell; there two warps share a
// cell, 32 particles each at a time: 4,096 dam break 52 -> 35 us, 65,536
// particles among obstacles 99 -> 66 us.  Where the warps of all cells are not
// resident at once, the staging done twice costs more (1M block 0.43 -> 0.49 ms):
// density_halves (sph_rules.h).

constexpr int kDensChunk = 256;
struct DensWarp {
	float2 pos[kDensChunk];
};

namespace {

// One list entry for one particle (sph.h:465-476): sums in list order.
__device__ __forceinline__ void dens_entry(float2 xj, float2 xi, float h2, float invH, float &d0, float &d1) {
	const float rx = xj.x - xi.x, ry = xj.y - xi.y;
	const float r2 = rx * rx + ry * ry;
	if (r2 < h2) {
		const float r = sqrtf(r2);
		const float term = 1.0f - r * invH;
		d0 = d0 + term * term;
		d1 = d1 + term * term * term;
	}
}

// Lists of N particles per lane, j0 + 32 n in the cell at st with cnt
// particles, over the L entries of its 3x3 block.
template <int N>
__device__ __forceinline__ void dens_lists(DensWarp &S, const Particles &Q, const int (&segOff)[9],
                                           const int (&segStart)[9], int L, int st, int j0, int cnt,
                                           const StepParams &s, int lane) {
	const float h2 = s.h2, invH = s.invH;
	float2 xi[N];
	float d0[N], d1[N];
#pragma unroll
	for (int n = 0; n < N; ++n) {
		const int j = j0 + n * kWarp;
		// Lanes without a particle use a position no entry is in range of.
		xi[n] = j < cnt ? Q.pos[st + j] : make_float2(3.0e38f, 3.0e38f);
		d0[n] = d1[n] = 0.0f;
	}
	for (int c0 = 0; c0 < L; c0 += kDensChunk) {
		const int len = min(kDensChunk, L - c0);
		__syncwarp();
		for (int e = lane; e < len; e += kWarp) S.pos[e] = Q.pos[seg_src<9>(c0 + e, segOff, segStart)];
		__syncwarp();
		int e = 0;
		for (; e + 4 <= len; e += 4) {
			float2 xj[4];
#pragma unroll
			for (int u = 0; u < 4; ++u) xj[u] = S.pos[e + u];
#pragma unroll
			for (int u = 0; u < 4; ++u)
#pragma unroll
				for (int n = 0; n < N; ++n) dens_entry(xj[u], xi[n], h2, invH, d0[n], d1[n]);
		}
		for (; e < len; ++e) {
			const float2 xj = S.pos[e];
#pragma unroll
			for (int n = 0; n < N; ++n) dens_entry(xj, xi[n], h2, invH, d0[n], d1[n]);
		}
	}
#pragma unroll
	for (int n = 0; n < N; ++n) {
		const int j = j0 + n * kWarp;
		if (j < cnt) {
			Q.dens[st + j] = make_float2(d0[n], d1[n]);
			Q.press[st + j] = make_float2(s.k * (d0[n] - s.rho0), s.kNear * d1[n]);
		}
	}
}

// The particles of cell c (cnt of them) from `first` on, 64 at a time: two
// lists per lane or, as one of a cell's two warps (kHalf), every other 32.
template <bool kHalf>
__device__ __forceinline__ void dens_cell(DensWarp &S, const Particles &Q, const SimTables &T, int c, int cnt, int first,
                                          int lane) {
	const int sid = T.sceneOfCell[c];
	const SceneDev &sc = T.scenes[sid];
	const StepParams &s = sc.p;
	const int base = sc.cellBase;
	const int cx = (c - base) % s.gx, cy = (c - base) / s.gx;
	int segStart[9], segOff[9];
	int L = 0;
#pragma unroll
	for (int q = 0; q < 9; ++q) {
		const int x = cx + q % 3 - 1, y = cy + q / 3 - 1;
		int st = 0, nn = 0;
		if (x >= 0 && x < s.gx && y >= 0 && y < s.gy) {
			const int c2 = base + y * s.gx + x;
			st = T.newStart[c2];
			nn = T.newCount[c2];
		}
		segStart[q] = st;
		segOff[q] = L;
		L += nn;
	}
	if (lane == 0 && first == 0) {
		atomicMin(&T.stats[4 * sid + 0], (uint32_t)L);
		atomicMax(&T.stats[4 * sid + 1], (uint32_t)L);
	}
	if (L > kStageCap) {
		if (lane == 0) atomicOr(T.error, kErrStageOverflow);
		return;
	}
	const int st = T.newStart[c];
	for (int g = first; g < cnt; g += 2 * kWarp) {
		if (!kHalf && cnt - g > kWarp)
			dens_lists<2>(S, Q, segOff, segStart, L, st, g + lane, cnt, s, lane);
		else
			dens_lists<1>(S, Q, segOff, segStart, L, st, g + lane, cnt, s, lane);
	}
	__syncwarp();
}

}  // namespace

__global__ void __launch_bounds__(kDensWarps * kWarp, 4) k_density(Totals tt, Particles Q, SimTables T, int added,
                                                                   int sms) {
	extern __shared__ __align__(16) unsigned char smem_raw[];
	DensWarp &S = reinterpret_cast<DensWarp *>(smem_raw)[threadIdx.x / kWarp];
	const int lane = threadIdx.x & (kWarp - 1);
	const int warpsTotal = gridDim.x * kDensWarps, first = blockIdx.x * kDensWarps + threadIdx.x / kWarp;
	if (density_halves(tt.ncell, *T.nLive, tt.n, added, sms)) {
		for (int w = first; w < 2 * tt.ncell; w += warpsTotal) {
			const int cnt = T.newCount[w >> 1];
			if (cnt > (w & 1) * kWarp) dens_cell<true>(S, Q, T, w >> 1, cnt, (w & 1) * kWarp, lane);
		}
	} else {
		for (int c = first; c < tt.ncell; c += warpsTotal) {
			const int cnt = T.newCount[c];
			if (cnt > 0) dens_cell<false>(S, Q, T, c, cnt, 0, lane);
		}
	}
}

// ---------------------------------------------------------------------------
// Delta sweep (double-density relaxation, demo4.cpp:239-255).  Tasks in
// number order per scene: canonical cells in rank order, then the scene's
// appendix in runs of kAppendixRun consecutive numbers.  A particle's list is
// the 3x3 block of NEW cells around its new cell.  A task stages the new
// cells of its bounding box grown by one, processes its particles in order,
// and writes back only cells inside its particles' 3x3 blocks.  Earlier tasks
// of the scene whose bounding boxes come within two cells are waited for.
// One task per block.  The block stages the task's region once.  A
// particle's list slots (three row ranges of the staged region and its own
// slot) are worked out for a chunk of particles at once, off the serial path.
//
// Particles are relaxed in a two-stage pipeline.  In phase k the producer
// warps scan particle k's list, compact the in-range pairs
// in list order and evaluate them (x_j += D/2), while the summer warp (the
// last) finishes particle k-1: its ordered sum dx -= D/2 and x_{k-1} += dx.
// The only pair of particle k that needs x_{k-1} after that sum is
// (k, k-1): the producers reserve its place in list order, and the summer,
// which knows from k's list ranges whether k-1 is in the list, evaluates it
// right after the sum (x_{k-1} += D/2) and keeps D/2 until the next phase,
// when it fills the reserved place before summing k.  The two roles share no
// data within a phase, so they meet only at the phase's end.  k's own (self)
// pair is kept aside (ownAfter) so that no warp sees k's position change
// before reading it.
// Particles whose lists exceed one pass drain the pipeline and run on the
// whole block in turn.
// The shapes and what each is for: sph_kernels.cuh.
// Rounds of 32 list entries a scanning warp loads at once (tri, quad, lean).
// One task of 36 particles alone, ns per particle, one round at a time and
// evaluated after the other warps' counts: 1,445, 1,148, 1,700; two at once
// 1,343, 1,080, 1,568; four 1,316, 1,046, 1,566; six 1,273, 1,086, 1,524.
constexpr int kScanBatch = 4;
constexpr int kSumPad = 32;  // +0 entries past the last half, at most one batch of the sum
template <class C>
struct DeltaSmemT {
	static constexpr int kProd = C::kProducers;         // producer warps
	static constexpr int kPass = kProd * C::kChainW;    // list entries per pipelined particle
	static constexpr int kSeqPass = C::kWarps * C::kChainW;  // list entries per pass, whole block
	static constexpr int kHalf = (kSeqPass > kPass ? kSeqPass : kPass) + 36;  // 4 past a multiple of the 32 banks
	static constexpr int kPhases = C::kPipelined ? 2 : 1;  // half buffers
	float2 pos[C::kStage];
	float4 cand[C::kWarps][C::kChainW];  // per warp: in-range candidates: slot, x_j.x, x_j.y, r2
	alignas(16) float half[kPhases][2][kHalf];  // per phase, x and y: delta * 0.5 of the in-range pairs, list order, +0 padded
	alignas(16) unsigned char wcnt8[16];      // kDirect: per warp, in-range pairs of this phase's particle
	int4 meta[2];             // per phase: pairs, reserved index of (k, k-1) or -1, own slot
	float2 ownAfter[2];       // per phase: the particle's position after its self pair
	int4 pslot[C::kPrefetch];  // prefetched per particle: row ranges' first slots, own slot (or -1)
	int4 plen[C::kPrefetch];   // row ranges' lengths
	float2 ppk[C::kPrefetch];  // pressure and near pressure
	int segOff[C::kRegion + 1];
	int segStart[C::kRegion];
	int owned[C::kRegion];
	int wcnt[C::kWarps];
	int4 groupBox;  // new cells of a group of particles whose task's region is too large, and
	int groupEnd;   // where it ends
	int task;
	int pend[kPendCap];  // dependencies still pending (wait_canonical)
	int npend;
};

namespace {

struct Region {
	int x0, y0, x1, y1, w, ncells, L;
};

// The staging table of the new cells of [x0,x1]x[y0,y1] (row-major): where each
// cell, a contiguous range of the new numbers, goes in the stage.  It depends on
// no other task.  Collective over the block; returns false (uniformly) if the
// region does not fit.
template <class C>
__device__ __forceinline__ bool stage_table(DeltaSmemT<C> &S, Region &R, const SimTables &T, const StepParams &s,
                                            int cellBase, int tid) {
	R.w = R.x1 - R.x0 + 1;
	R.ncells = R.w * (R.y1 - R.y0 + 1);
	if (R.ncells > C::kRegion) return false;
	if (tid < kWarp) {
		const int lane = tid;
		int carry = 0;
		for (int b0 = 0; b0 < R.ncells; b0 += kWarp) {
			const int q = b0 + lane;
			int nn = 0, st = 0;
			if (q < R.ncells) {
				const int c2 = cellBase + (R.y0 + q / R.w) * s.gx + (R.x0 + q % R.w);
				nn = T.newCount[c2];
				st = T.newStart[c2];
			}
			int incl = nn;
#pragma unroll
			for (int o = 1; o < kWarp; o <<= 1) {
				const int v = __shfl_up_sync(kFull, incl, o);
				if (lane >= o) incl += v;
			}
			if (q < R.ncells) {
				S.segOff[q] = carry + incl - nn;
				S.segStart[q] = st;
				S.owned[q] = 0;
			}
			carry += __shfl_sync(kFull, incl, kWarp - 1);
		}
		if (lane == 0) S.segOff[R.ncells] = carry;
	}
	__syncthreads();
	R.L = S.segOff[R.ncells];
	return R.L <= C::kStage;
}

// Stage the table's positions, a warp per cell, the loads of kStageCells cells
// (64 entries each) in flight at once.  Collective over the block.  (One entry
// per thread, its cell found by binary search over the table's offsets: 768 ns
// in the wide shape and 5.4 us in the lean one for 25 cells of 36 particles, now
// 320 ns and 2.6 us; one cell at a time 480 ns and 4.1 us; four, with registers
// spilled around the pipeline, slowed the particles by a tenth.)
constexpr int kStageCells = 2;
template <class C>
__device__ __forceinline__ void stage_positions(DeltaSmemT<C> &S, const Region &R, const Particles &Q, int tid) {
	const int lane = tid & (kWarp - 1);
	for (int q0 = tid / kWarp; q0 < R.ncells; q0 += kStageCells * C::kWarps) {
		float2 xp[kStageCells][2];
		int off[kStageCells], n[kStageCells], st[kStageCells];
#pragma unroll
		for (int u = 0; u < kStageCells; ++u) {
			const int q = min(q0 + u * C::kWarps, R.ncells - 1);
			off[u] = S.segOff[q];
			n[u] = q0 + u * C::kWarps < R.ncells ? S.segOff[q + 1] - off[u] : 0;
			st[u] = S.segStart[q];
#pragma unroll
			for (int v = 0; v < 2; ++v)
				if (v * kWarp + lane < n[u]) xp[u][v] = __ldcg(&Q.pos[st[u] + v * kWarp + lane]);
		}
#pragma unroll
		for (int u = 0; u < kStageCells; ++u) {
#pragma unroll
			for (int v = 0; v < 2; ++v)
				if (v * kWarp + lane < n[u]) S.pos[off[u] + v * kWarp + lane] = xp[u][v];
			for (int j = 2 * kWarp + lane; j < n[u]; j += kWarp) S.pos[off[u] + j] = __ldcg(&Q.pos[st[u] + j]);
		}
	}
	__syncthreads();
}

// Write the staged positions of the owned cells back, a warp per cell.
template <class C>
__device__ __forceinline__ void write_back_owned(DeltaSmemT<C> &S, const Region &R, const Particles &Q, int tid) {
	const int lane = tid & (kWarp - 1);
	for (int q = tid / kWarp; q < R.ncells; q += C::kWarps) {
		if (!S.owned[q]) continue;
		const int off = S.segOff[q], n = S.segOff[q + 1] - off, st = S.segStart[q];
		for (int j = lane; j < n; j += kWarp) __stcg(&Q.pos[st + j], S.pos[off + j]);
	}
}

// List slots of the particle with new cell nc and new number jk, whose 3x3
// block lies inside the staged region: in the row-major region the three
// cells of one block row are consecutive, so the list (y-major, then x, then
// cell order, demo4.cpp:188-201) is three contiguous ranges of slots.  Marks
// the block's cells as written back.  One thread per particle.
template <class C>
__device__ __forceinline__ void particle_slots(DeltaSmemT<C> &S, const Region &R, int nc, int jk, const StepParams &s,
                                               int cellBase, uint32_t *err, int4 &slot, int4 &len) {
	const int x = (nc - cellBase) % s.gx, y = (nc - cellBase) / s.gx;
	const int xa = max(x - 1, 0), xb = min(x + 1, s.gx - 1);
	int o[3], n[3];
#pragma unroll
	for (int r = 0; r < 3; ++r) {
		const int yy = y + r - 1;
		o[r] = 0;
		n[r] = 0;
		if (yy >= 0 && yy < s.gy) {
			const int rq0 = (yy - R.y0) * R.w + (xa - R.x0);
			const int rq1 = rq0 + (xb - xa);
			o[r] = S.segOff[rq0];
			n[r] = S.segOff[rq1 + 1] - o[r];
			for (int q = rq0; q <= rq1; ++q) S.owned[q] = 1;
		}
	}
	const int ownSeg = (y - R.y0) * R.w + (x - R.x0);
	const int inCell = jk - S.segStart[ownSeg];
	int own = S.segOff[ownSeg] + inCell;
	if (inCell < 0 || inCell >= S.segOff[ownSeg + 1] - S.segOff[ownSeg]) {
		atomicOr(err, kErrIndex);
		own = -1;
	}
	slot = make_int4(o[0], o[1], o[2], own);
	const int L = n[0] + n[1] + n[2];
	len = make_int4(n[0], n[1], n[2], (L + DeltaSmemT<C>::kProd - 1) / DeltaSmemT<C>::kProd);
}

// delta * 0.5 of one in-range pair (sph.h:483-495 with demo4.cpp:250-251):
// particle at xk with pressures pk, neighbour at xj, r2 = |xj - xk|^2.
__device__ __forceinline__ float2 delta_half(float2 xj, float2 xk, float r2, float2 pk, const StepParams &s) {
	const float rx = xj.x - xk.x, ry = xj.y - xk.y;
	float rij;
	const float inv = root_and_inverse(r2, rij);
	const float nx = rx * inv, ny = ry * inv;
	const float term = 1.0f - rij * s.invH;
	const float d = s.dt2 * (pk.x * term + pk.y * (term * term));
	return make_float2(d * nx * 0.5f, d * ny * 0.5f);
}

// The same without a branch, for r2 = 0 or in the plain range of root_plain;
// and for any distance, out of line.
__device__ __forceinline__ float2 delta_half_line(float2 xj, float2 xk, float r2, float2 pk, const StepParams &s) {
	const float rx = xj.x - xk.x, ry = xj.y - xk.y;
	const bool zero = r2 == 0.0f;
	float len;
	const float inv = inverse_root_line(zero ? 1.0f : r2, len);
	const float rij = zero ? 0.0f : len;
	const float nx = rx * inv, ny = ry * inv;
	const float term = 1.0f - rij * s.invH;
	const float d = s.dt2 * (pk.x * term + pk.y * (term * term));
	return make_float2(d * nx * 0.5f, d * ny * 0.5f);
}
__device__ __noinline__ float2 delta_half_any(float2 xj, float2 xk, float2 pk, const StepParams &s) {
	const float rx = xj.x - xk.x, ry = xj.y - xk.y;
	return delta_half(xj, xk, rx * rx + ry * ry, pk, s);
}

// dx -= delta * 0.5 over the n buffered halves of one component, in list
// order (demo4.cpp:251), starting at dx: one dependent subtraction per pair
// (four cycles), in batches of 32 loaded at once, so that the loads' latency and
// the loop branch, exposed between batches, add a half and no more.  The buffer is padded with +0 for
// kSumPad entries past n, and dx - (+0) == dx exactly.  Two lanes take a
// component each.  In isolation 112 pairs take 685 cycles, 818 in batches of
// eight; one lane subtracting both components took 9.4 cycles a pair.
__device__ __forceinline__ float sum_halves(const float *H, int n, float dx) {
	const uint32_t h = shared_addr(H);
	for (int b = 0; b < n; b += kSumPad) {
		float4 a[kSumPad / 4];
#pragma unroll
		for (int u = 0; u < kSumPad / 4; ++u) a[u] = lds4(h + 4u * b + 16u * u);
#pragma unroll
		for (int u = 0; u < kSumPad / 4; ++u) dx = dx - a[u].x - a[u].y - a[u].z - a[u].w;
	}
	return dx;
}
__device__ __forceinline__ float comp(float2 v, int c) { return c == 0 ? v.x : v.y; }
__device__ __forceinline__ float *comp_of(float2 *v, int c) { return reinterpret_cast<float *>(v) + c; }

// Scan and compaction of one particle's list entries [p0, p0 + pl) over
// `nw` warps (this thread is warp `w` of them): each warp takes a contiguous
// range and compacts its in-range entries, in list order, into cand[w].
// Slot `skip` (or -1) is reserved whatever its distance (marked r2 = -1);
// slot `own` records the particle's unmoved position in *ownAfter.
__device__ __forceinline__ int scan_range(float4 *cand, int nw, int w, int lane, int p0, int pl, int4 sl, int len0,
                                          int l01, float2 xk, int own, int skip, const float2 *pos, float h2,
                                          float2 *ownAfter) {
	const int per = (pl + nw - 1) / nw;
	const int e0 = p0 + w * per, e1 = min(p0 + pl, e0 + per);
	// Rows start at sl.x, sl.y - len0 and sl.z - l01 of the flat list.
	const int row1 = sl.y - len0, row2 = sl.z - l01;
	int cnt = 0;
	for (int eb = e0; eb < e1; eb += kScanBatch * kWarp) {
		float2 xj[kScanBatch];
		int slot[kScanBatch];
#pragma unroll
		for (int u = 0; u < kScanBatch; ++u) {
			const int e = eb + u * kWarp + lane;
			slot[u] = e < e1 ? e + (e < len0 ? sl.x : (e < l01 ? row1 : row2)) : -1;
			xj[u] = pos[max(slot[u], 0)];
		}
#pragma unroll
		for (int u = 0; u < kScanBatch; ++u) {
			if (eb + u * kWarp >= e1) break;
			const float rx = xj[u].x - xk.x, ry = xj[u].y - xk.y;
			float r2 = rx * rx + ry * ry;
			bool in = slot[u] >= 0 && r2 < h2;
			if (slot[u] >= 0) {
				if (slot[u] == skip) {
					in = true;
					r2 = -1.0f;
				} else if (slot[u] == own) {
					*ownAfter = xj[u];  // out of range: no displacement
				}
			}
			const unsigned mk = __ballot_sync(kFull, in);
			if (in) cand[cnt + __popc(mk & lanemask_lt())] = make_float4(__int_as_float(slot[u]), xj[u].x, xj[u].y, r2);
			cnt += __popc(mk);
		}
	}
	return cnt;
}

// Relax one particle on the whole block, not pipelined (demo4.cpp:240-254):
// lists of any length, in passes of kSeqPass entries.  Thread 0 sums.
template <class C>
__device__ __forceinline__ void relax_particle(DeltaSmemT<C> &S, int4 sl, int4 ln, float2 pk, const StepParams &s,
                                               int tid) {
	constexpr int kW = C::kWarps, kPass = DeltaSmemT<C>::kSeqPass;
	const int lane = tid & (kWarp - 1), warp = tid / kWarp;
	const int own = sl.w;
	if (own < 0) return;  // index check failed (uniform)
	const int len0 = ln.x, l01 = ln.x + ln.y, L = l01 + ln.z;
	const float2 xk = S.pos[own];
	float dx = 0.0f;  // threads 0 and 1: x and y
	for (int p0 = 0; p0 < L; p0 += kPass) {
		const int pl = min(L - p0, kPass);
		const int cnt = scan_range(S.cand[warp], kW, warp, lane, p0, pl, sl, len0, l01, xk, own, -1, S.pos, s.h2,
		                           &S.ownAfter[0]);
		if (lane == 0) S.wcnt[warp] = cnt;
		__syncthreads();
		int before = 0, total = 0;
#pragma unroll
		for (int w = 0; w < kW; ++w) {
			const int c = S.wcnt[w];
			before += (w < warp) ? c : 0;
			total += c;
		}
		if (tid < kSumPad) S.half[0][0][total + tid] = S.half[0][1][total + tid] = 0.0f;
		for (int q = lane; q < cnt; q += kWarp) {
			const float4 cd = S.cand[warp][q];
			const float2 xj = make_float2(cd.y, cd.z);
			const float2 h = delta_half(xj, xk, cd.w, pk, s);
			const int slot = __float_as_int(cd.x);
			const float2 moved = make_float2(h.x + xj.x, h.y + xj.y);
			if (slot == own) S.ownAfter[0] = moved; else S.pos[slot] = moved;
			S.half[0][0][before + q] = h.x;
			S.half[0][1][before + q] = h.y;
		}
		__syncthreads();
		if (tid < 2) {
			dx = sum_halves(S.half[0][tid], total, dx);
			if (p0 + kPass >= L) *comp_of(&S.pos[own], tid) = dx + comp(S.ownAfter[0], tid);
		}
		__syncthreads();
	}
}

// Summer warp, lanes c = 0 and 1 (x and y): the ordered dx sum of the
// particle of phase buffer b, its reserved pair filled with hres (this
// component's D/2).  Returns the component of its final position.
template <class C>
__device__ __forceinline__ float finish_sum(DeltaSmemT<C> &S, int b, int c, float hres) {
	const int4 m = S.meta[b];
	float *H = S.half[b][c];
	const float xo = comp(S.ownAfter[b], c);
	if (m.y >= 0) H[m.y] = hres;
	return sum_halves(H, m.x, 0.0f) + xo;
}

template <class C>
__device__ __forceinline__ void producers_bar() {
	__syncwarp();
	asm volatile("bar.sync 1, %0;" ::"r"(DeltaSmemT<C>::kProd * kWarp) : "memory");
}

// Producers' part of phase b for particle (sl, ln, pk): everything but the
// pair with slot `prev` (the particle still being finished, or -1).
template <class C>
__device__ __forceinline__ void produce(DeltaSmemT<C> &S, int b, int4 sl, int4 ln, float2 pk, int prev,
                                        const StepParams &s, int warp, int lane) {
	constexpr int kP = DeltaSmemT<C>::kProd, R = 2;
	const int own = sl.w;
	const int len0 = ln.x, l01 = ln.x + ln.y, L = l01 + ln.z;
	const float2 xk = S.pos[own];
	if (warp == 0 && lane == 0) S.meta[b] = make_int4(0, -1, own, 0);
	const float4 *cand = S.cand[warp];
	const int cnt = scan_range(S.cand[warp], kP, warp, lane, 0, L, sl, len0, l01, xk, own, prev, S.pos, s.h2,
	                           &S.ownAfter[b]);
	if (lane == 0) S.wcnt[warp] = cnt;
	__syncwarp();
	// The candidates of the first R rounds side by side, before the counts of
	// the other warps are needed; what is left after that, one by one.
	auto apply = [&](float4 cd, float2 h) {
		const int slot = __float_as_int(cd.x);
		const float2 moved = make_float2(h.x + cd.y, h.y + cd.z);
		if (slot == own) S.ownAfter[b] = moved; else S.pos[slot] = moved;
	};
	auto place = [&](float4 cd, float2 h, int at) {
		if (cd.w < 0.0f) {
			S.meta[b].y = at;  // (k, k-1): the summer evaluates it
		} else {
			S.half[b][0][at] = h.x;
			S.half[b][1][at] = h.y;
		}
	};
	float4 cd[R];
	float2 h[R];
	bool plain = true;
#pragma unroll
	for (int i = 0; i < R; ++i) {
		cd[i] = cand[min(i * kWarp + lane, C::kChainW - 1)];
		h[i] = delta_half_line(make_float2(cd[i].y, cd[i].z), xk, cd[i].w, pk, s);
		plain = plain && (i * kWarp + lane >= cnt || cd[i].w <= 0.0f || root_plain(cd[i].w));
	}
	if (!plain) {
#pragma unroll
		for (int i = 0; i < R; ++i) h[i] = delta_half_any(make_float2(cd[i].y, cd[i].z), xk, pk, s);
	}
#pragma unroll
	for (int i = 0; i < R; ++i)
		if (i * kWarp + lane < cnt && cd[i].w >= 0.0f) apply(cd[i], h[i]);
	int before = 0, total = cnt;
	if (kP > 1) {
		producers_bar<C>();
		total = 0;
#pragma unroll
		for (int w = 0; w < kP; ++w) {
			const int c = S.wcnt[w];
			before += (w < warp) ? c : 0;
			total += c;
		}
	}
	if (warp == kP - 1) {
		S.half[b][0][total + lane] = S.half[b][1][total + lane] = 0.0f;
		if (lane == 0) S.meta[b].x = total;
	}
#pragma unroll
	for (int i = 0; i < R; ++i)
		if (i * kWarp + lane < cnt) place(cd[i], h[i], before + i * kWarp + lane);
	for (int q = R * kWarp + lane; q < cnt; q += kWarp) {
		const float4 c = cand[q];
		const float2 hh = delta_half(make_float2(c.y, c.z), xk, c.w, pk, s);
		if (c.w >= 0.0f) apply(c, hh);
		place(c, hh, before + q);
	}
}

// Direct form of produce (kDirect): warp w takes a contiguous range of the
// list, entry `at[i]` (a staged slot, or -1) of this thread in round i of R,
// and evaluates it without compacting first, so the square root and the
// division run beside the counting and only the halves' places wait for the
// other warps' counts.  R is a compile-time number: a uniform branch per round
// costs as much as the round's arithmetic.  One task of 36 particles with 324
// list entries (wide shape, alone) takes a fifth longer per particle when every
// warp compacts first.
template <class C, int R>
__device__ __forceinline__ void produce_direct(DeltaSmemT<C> &S, int b, const int *at, int own, float2 pk, int prev,
                                               uint4 below, const StepParams &s, int warp, int lane) {
	constexpr int kP = DeltaSmemT<C>::kProd;
	static_assert(kP <= 16 && C::kChainW < 256, "a phase's counts are one 16-byte word");
	const float2 xk = S.pos[own];
	float2 xj[R], h[R];
	unsigned mask[R];
	bool in[R];
	int cnt = 0;
	bool plain = true;
	if (warp == 0 && lane == 0) S.meta[b] = make_int4(0, -1, own, 0);
#pragma unroll
	for (int i = 0; i < R; ++i) xj[i] = S.pos[max(at[i], 0)];
#pragma unroll
	for (int i = 0; i < R; ++i) {
		const float rx = xj[i].x - xk.x, ry = xj[i].y - xk.y;
		const float r2 = rx * rx + ry * ry;
		// (k, k-1) keeps its place whatever its distance: the summer
		// evaluates it.
		in[i] = at[i] >= 0 && at[i] != prev && r2 < s.h2;
		mask[i] = __ballot_sync(kFull, in[i] || (at[i] >= 0 && at[i] == prev));
		cnt += __popc(mask[i]);
		h[i] = delta_half_line(xj[i], xk, r2, pk, s);
		plain = plain && (!in[i] || r2 == 0.0f || root_plain(r2));
	}
	if (!plain) {
#pragma unroll
		for (int i = 0; i < R; ++i) h[i] = delta_half_any(xj[i], xk, pk, s);
	}
	if (lane == 0) S.wcnt8[warp] = (unsigned char)cnt;
#pragma unroll
	for (int i = 0; i < R; ++i) {
		const float2 moved = make_float2(h[i].x + xj[i].x, h[i].y + xj[i].y);
		if (at[i] == own) S.ownAfter[b] = in[i] ? moved : xj[i];
		else if (in[i]) S.pos[at[i]] = moved;
	}
	producers_bar<C>();
	const uint4 c4 = *reinterpret_cast<const uint4 *>(S.wcnt8);
	// Sum of the earlier warps' counts: bytes, masked once per task.
	int before = (int)(__dp4a(c4.x & below.x, 0x01010101u, 0u) + __dp4a(c4.y & below.y, 0x01010101u, 0u) +
	                   __dp4a(c4.z & below.z, 0x01010101u, 0u) + __dp4a(c4.w & below.w, 0x01010101u, 0u));
	if (warp == kP - 1) {
		const int total = before + cnt;
		S.half[b][0][total + lane] = S.half[b][1][total + lane] = 0.0f;
		if (lane == 0) S.meta[b].x = total;
	}
#pragma unroll
	for (int i = 0; i < R; ++i) {
		const int place = before + __popc(mask[i] & lanemask_lt());
		if (in[i]) {
			S.half[b][0][place] = h[i].x;
			S.half[b][1][place] = h[i].y;
		} else if (at[i] >= 0 && at[i] == prev) {
			S.meta[b].y = place;
		}
		before += __popc(mask[i]);
	}
}

// Byte mask of the counts of the warps before this one.
__device__ __forceinline__ uint4 warps_below(int warp) {
	uint32_t m[4];
#pragma unroll
	for (int q = 0; q < 4; ++q) {
		const int n = min(max(warp - 4 * q, 0), 4);
		m[q] = n == 4 ? 0xffffffffu : (1u << (8 * n)) - 1u;
	}
	return make_uint4(m[0], m[1], m[2], m[3]);
}

// The list entry of lane `lane` of producer warp `warp` in round i (a staged
// slot, or -1) for the particle with row ranges sl, ln.
template <class C>
__device__ __forceinline__ int direct_slot(int4 sl, int4 ln, int warp, int lane, int i) {
	const int r = i * kWarp + lane;
	const int e = warp * ln.w + r;
	const int l01 = ln.x + ln.y;
	// Rows start at sl.x, sl.y - ln.x and sl.z - l01 of the flat list.
	const int base = e < ln.x ? sl.x : (e < l01 ? sl.y - ln.x : sl.z - l01);
	return r < ln.w && e < l01 + ln.z ? base + e : -1;
}

// Summer's part of a phase (a whole warp: even lanes take the x component,
// odd lanes the y, all of them the same way, so that nothing diverges): finish
// the previous particle `prev` (buffer b ^ 1), then evaluate the pair (k, k-1)
// of particle k (list slots sl, ln, pressures pk) if k-1 is in k's list; this
// component of its D/2 goes to hres.  What does not depend on the sum is
// loaded before it.
template <class C>
__device__ __forceinline__ void summer(DeltaSmemT<C> &S, int b, int c, int prev, int4 sl, int4 ln, float2 pk,
                                       const StepParams &s, float &hres) {
	const float2 xk = S.pos[sl.w];
	const bool inList = (prev >= sl.x && prev < sl.x + ln.x) || (prev >= sl.y && prev < sl.y + ln.y) ||
	                    (prev >= sl.z && prev < sl.z + ln.z);
	float x = finish_sum<C>(S, b ^ 1, c, hres);
	const float o = __shfl_xor_sync(kFull, x, 1);
	const float2 xp = c == 0 ? make_float2(x, o) : make_float2(o, x);
	const float rx = xp.x - xk.x, ry = xp.y - xk.y;
	const float r2 = rx * rx + ry * ry;
	const float h = comp(delta_half(xp, xk, r2, pk, s), c);
	const bool in = inList && r2 < s.h2;
	hres = in ? h : 0.0f;
	*comp_of(&S.pos[prev], c) = in ? h + x : x;
}

// Role of a warp in the pipeline: a producer's number, kProd for the summer,
// or -1 (kApart: the summer is warp 3 and the other warps of its scheduler
// stay out, so that no producer takes its issue slots).  The summer's dependent
// subtractions lose a cycle whenever another warp issues in their place: one
// task of 36 particles alone, 112 in-range pairs each, takes 569 ns, 1,178
// cycles, per particle in the wide shape; with three warps on each scheduler and
// both roles in one loop a quarter more (dense a third, quad 6%).
template <class C>
__device__ __forceinline__ int pipeline_role(int warp) {
	if (!C::kApart) return warp;
	return (warp & 3) != 3 ? (warp >> 2) * 3 + (warp & 3) : (warp == 3 ? DeltaSmemT<C>::kProd : -1);
}
template <class C>
__device__ __forceinline__ bool pipelinable(int4 sl, int4 ln) {
	return C::kPipelined && sl.w >= 0 && ln.x + ln.y + ln.z <= DeltaSmemT<C>::kPass;
}
template <class C>
__device__ __forceinline__ void phase_bar() {
	__syncwarp();
	asm volatile("bar.sync 2, %0;" ::"r"((DeltaSmemT<C>::kProd + 1) * kWarp) : "memory");
}

// One particle on the producers.
template <class C>
__device__ __forceinline__ void produce_phase(DeltaSmemT<C> &S, int b, int4 sl, int4 ln, float2 pk, int at0, int prev,
                                              uint4 below, const StepParams &s, int role, int lane) {
	if constexpr (C::kDirect) {
		constexpr int kE = C::kChainW / kWarp;
		if (ln.w <= kWarp) {
			produce_direct<C, 1>(S, b, &at0, sl.w, pk, prev, below, s, role, lane);
			return;
		}
		int at[kE];
		at[0] = at0;
#pragma unroll
		for (int i = 1; i < kE; ++i) at[i] = direct_slot<C>(sl, ln, role, lane, i);
		if (ln.w <= 2 * kWarp)
			produce_direct<C, 2>(S, b, at, sl.w, pk, prev, below, s, role, lane);
		else if (kE > 4 && ln.w <= 4 * kWarp)
			produce_direct<C, (kE > 4 ? 4 : kE)>(S, b, at, sl.w, pk, prev, below, s, role, lane);
		else
			produce_direct<C, kE>(S, b, at, sl.w, pk, prev, below, s, role, lane);
	} else {
		produce<C>(S, b, sl, ln, pk, prev, s, role, lane);
	}
}

// The pipelined particles from index i on of the chunk's n: each role loops on
// its own, meeting the others at the end of every phase, until the chunk ends
// or a particle has to run on the whole block.  Returns that index; `ph` counts
// phases and `prev` is the pending particle's slot (-1: none).
template <class C>
__device__ __forceinline__ int run_pipeline(DeltaSmemT<C> &S, int i, int n, int &ph, int &prev, float &hres, uint4 below,
                                            const StepParams &s, int role, int lane) {
	constexpr int kP = DeltaSmemT<C>::kProd;
	int4 sl = S.pslot[i], ln = S.plen[i];
	if (role < 0) {
		for (; i < n; ++i, ++ph) {
			const int4 a = S.pslot[i], l = S.plen[i];
			if (!pipelinable<C>(a, l)) break;
			prev = a.w;
		}
		return i;
	}
	float2 pk = S.ppk[i];
	int at0 = role < kP && C::kDirect ? direct_slot<C>(sl, ln, role, lane, 0) : 0;
	for (;;) {
		const int next = min(i + 1, n - 1), b = (ph & 1) % DeltaSmemT<C>::kPhases;
		const int4 slN = S.pslot[next], lnN = S.plen[next];
		const float2 pkN = S.ppk[next];
		if (role < kP) {
			produce_phase<C>(S, b, sl, ln, pk, at0, prev, below, s, role, lane);
			if (C::kDirect) at0 = direct_slot<C>(slN, lnN, role, lane, 0);
		} else if (prev >= 0) {
			summer<C>(S, b, lane & 1, prev, sl, ln, pk, s, hres);
		}
		phase_bar<C>();
		prev = sl.w;
		++ph;
		if (++i >= n || !pipelinable<C>(slN, lnN)) return i;
		sl = slN;
		ln = lnN;
		pk = pkN;
	}
}

// The longest run of particles from `k` on (at most 32) whose region, the
// bounding box of their new cells grown by one, fits the stage; at least one
// particle.  Warp 0; lane i looks at the box of the first i + 1 particles.
// Particles added in no spatial order are groups of one, each with this on the
// chain.  The first particle's region therefore is not counted (it goes in
// whatever it holds), and the last warp, which has no cell of a single
// particle's region to stage in the shapes with many warps, loads the group's
// inputs: first update of 30,000 in random order 113 -> 98 ms, of 100,000 420 ->
// 330.
template <class C>
__device__ __forceinline__ void next_group(DeltaSmemT<C> &S, int k, int p1, const int *ord, const SimTables &T,
                                           const StepParams &s, int cellBase, int tid) {
	if (tid >= kWarp) return;
	const int i = min(k + tid, p1 - 1);
	const int nc = T.newCell[ord ? ord[i] : i] - cellBase;
	int x0 = nc % s.gx, y0 = nc / s.gx, x1 = x0, y1 = y0;
#pragma unroll
	for (int o = 1; o < kWarp; o <<= 1) {
		const int a = __shfl_up_sync(kFull, x0, o), b = __shfl_up_sync(kFull, y0, o);
		const int c = __shfl_up_sync(kFull, x1, o), d = __shfl_up_sync(kFull, y1, o);
		if (tid >= o) {
			x0 = min(x0, a);
			y0 = min(y0, b);
			x1 = max(x1, c);
			y1 = max(y1, d);
		}
	}
	const int rx0 = max(x0 - 1, 0), ry0 = max(y0 - 1, 0), rx1 = min(x1 + 1, s.gx - 1), ry1 = min(y1 + 1, s.gy - 1);
	bool fits = k + tid < p1 && (rx1 - rx0 + 1) * (ry1 - ry0 + 1) <= C::kRegion;
	int entries = 0;
	if (fits && tid > 0) {
		for (int y = ry0; y <= ry1; ++y)
			for (int x = rx0; x <= rx1; ++x) entries += T.newCount[cellBase + y * s.gx + x];
		fits = entries <= C::kStage;
	}
	// Boxes grow with i, so the lanes that fit come first.
	const int n = max(__popc(__ballot_sync(kFull, fits)), 1);
	if (tid == n - 1) {
		S.groupBox = make_int4(x0, y0, x1, y1);
		S.groupEnd = k + n;
	}
}

// Process particles [p0, p1) (old numbers, or positions in AddParticle order
// mapped to old numbers by `ord`; new cells within [bx0,bx1]x[by0,by1]) in
// order, in one staged region if it fits the shape's stage, otherwise in
// groups that do (next_group; staging every particle of such a task on its own
// instead, the sweep of 128 collapsing scenes at its most crowded took 8.6 ms
// against 5.9 in the lean shape, 7.8 against 4.8 in tri).  Per-particle inputs (new
// number, pressure, list slots) are prefetched in chunks, off the serial path.
// `wait` waits for the task's dependencies: what does not need their results,
// the staging table and the first chunk's inputs and list slots, is done before
// it, off the chain from task to task (delta sweep of the 4,096 dam break 0.82 ->
// 0.72 ms per update, of 65,536 obstacles 1.62 -> 1.47).
template <class C, class W>
__device__ __forceinline__ unsigned long long relax_group(DeltaSmemT<C> &S, int p0, int p1, const int *ord, int bx0,
                                                          int by0, int bx1, int by1, const Particles &Q,
                                                          const SimTables &T, const StepParams &s, int cellBase,
                                                          int tid, W wait) {
	// Returns when the region was staged (global ns), for the task
	// timestamps (sph_profile_tasks).
	constexpr int kDT = C::kWarps * kWarp;
	constexpr int kP = DeltaSmemT<C>::kProd;
	const int warp = tid / kWarp, lane = tid & (kWarp - 1);
	Region R;
	auto grow = [&](int x0, int y0, int x1, int y1) {
		R.x0 = max(x0 - 1, 0);
		R.y0 = max(y0 - 1, 0);
		R.x1 = min(x1 + 1, s.gx - 1);
		R.y1 = min(y1 + 1, s.gy - 1);
	};
	grow(bx0, by0, bx1, by1);
	auto inputs = [&](int c0, int c1) {
		for (int k = c0 + tid; k < c1; k += kDT) {
			const int q = ord ? ord[k] : k;
			const int jk = T.newLabel[q], nc = T.newCell[q];
			S.ppk[k - c0] = Q.press[jk];
			particle_slots<C>(S, R, nc, jk, s, cellBase, T.error, S.pslot[k - c0], S.plen[k - c0]);
		}
	};
	bool staged = stage_table<C>(S, R, T, s, cellBase, tid);
	if (staged) inputs(p0, min(p1, p0 + C::kPrefetch));
	__syncthreads();
	wait();
	if (staged) stage_positions<C>(S, R, Q, tid);
	const unsigned long long tStaged = global_ns();
	const int role = pipeline_role<C>(warp);
	const uint4 below = warps_below(max(role, 0));
	int g0 = p0, g1 = p1;  // the group
	for (;;) {
		if (!staged) {
			__syncthreads();
			next_group<C>(S, g0, p1, ord, T, s, cellBase, tid);
			__syncthreads();
			const int4 box = S.groupBox;
			g1 = S.groupEnd;
			grow(box.x, box.y, box.z, box.w);
			staged = stage_table<C>(S, R, T, s, cellBase, tid);
			if (staged) {
				const int k = g0 + lane;  // a group has at most 32
				if (warp == C::kWarps - 1 && k < g1) {
					const int q = ord ? ord[k] : k;
					const int jk = T.newLabel[q], nc = T.newCell[q];
					S.ppk[k - g0] = Q.press[jk];
					particle_slots<C>(S, R, nc, jk, s, cellBase, T.error, S.pslot[k - g0], S.plen[k - g0]);
				}
				stage_positions<C>(S, R, Q, tid);
			} else if (tid == 0) {
				atomicOr(T.error, kErrStageOverflow);  // one 3x3 block alone
			}
		}
		if (staged) {
			int ph = 0, prev = -1;  // prev: slot of the particle whose sum is pending (buffer ph ^ 1), or -1
			float hres = 0.0f;      // summer: this component of D/2 of the pending particle's reserved pair
			for (int c0 = g0; c0 < g1; c0 += C::kPrefetch) {
				const int c1 = min(g1, c0 + C::kPrefetch);
				if (c0 != g0) {
					inputs(c0, c1);
					__syncthreads();
				}
				for (int k = c0; k < c1;) {
					const int4 sl = S.pslot[k - c0], ln = S.plen[k - c0];
					if (pipelinable<C>(sl, ln)) {
						k = c0 + run_pipeline<C>(S, k - c0, c1 - c0, ph, prev, hres, below, s, role, lane);
						__syncthreads();
						continue;
					}
					// Drain the pipeline, then relax this particle on the whole block.
					if (C::kPipelined && prev >= 0 && role == kP)
						*comp_of(&S.pos[prev], lane & 1) = finish_sum<C>(S, (ph & 1) ^ 1, lane & 1, hres);
					__syncthreads();
					prev = -1;
					relax_particle<C>(S, sl, ln, S.ppk[k - c0], s, tid);
					++k;
				}
				__syncthreads();
			}
			if (C::kPipelined && prev >= 0 && role == kP)
				*comp_of(&S.pos[prev], lane & 1) = finish_sum<C>(S, (ph & 1) ^ 1, lane & 1, hres);
			__syncthreads();
			write_back_owned<C>(S, R, Q, tid);
		}
		if (g1 >= p1) return tStaged;
		g0 = g1;
		staged = false;
	}
}

// One more pending dependency per thread (its done flag's index, or -1) into
// `pend`; collective over the warp.
__device__ __forceinline__ void list_pending(int r, int *pend, int *npend, int lane) {
	const unsigned m = __ballot_sync(kFull, r >= 0);
	int base = 0;
	if (lane == 0 && m != 0u) base = atomicAdd(npend, __popc(m));
	base = __shfl_sync(kFull, base, 0);
	if (r >= 0) {
		const int k = base + __popc(m & lanemask_lt());
		if (k < kPendCap) pend[k] = r;
	}
}

// Warp 0 polls the listed dependencies.
__device__ __forceinline__ void poll_pending(const int *pend, int np, const SimTables &T, int tid) {
	if (tid >= kWarp) return;
	for (int k0 = 0; k0 < np; k0 += kWarp)
		warp_wait(k0 + tid < np ? &T.done[pend[k0 + tid]] : nullptr, T.abort, T.error, T.waitLimitNs);
}

// Wait for the runs before run `a` of the scene whose boxes come within two
// cells of `box`, as wait_canonical does for cells.  Collective over the block.
template <int kDT>
__device__ __forceinline__ void wait_runs(int a, int scene, int4 box, const SimTables &T, int flag0, int *pend,
                                          int *npend, int tid) {
	if (tid == 0) *npend = 0;
	__syncthreads();
	auto near = [&](int q) {
		if (q >= a || T.appScene[q] != scene) return false;
		const int4 o = *reinterpret_cast<const int4 *>(&T.appBox[4 * q]);
		return rect_dist(o.x, o.y, o.z, o.w, box.x, box.y, box.z, box.w) <= 2;
	};
	for (int q0 = 0; q0 < a; q0 += kDT) {
		const int q = q0 + tid;
		list_pending(near(q) && ld_acquire(&T.done[flag0 + q]) == 0u ? flag0 + q : -1, pend, npend, tid & (kWarp - 1));
	}
	__syncthreads();
	const int np = *npend;
	if (np > kPendCap) {
		for (int q0 = 0; q0 < a; q0 += kDT)
			warp_wait(near(q0 + tid) ? &T.done[flag0 + q0 + tid] : nullptr, T.abort, T.error, T.waitLimitNs);
	} else {
		poll_pending(pend, np, T, tid);
	}
	__syncthreads();
}

// Wait for canonical tasks of the scene (old cells) near [bx0,bx1]x[by0,by1]
// whose new-cell bounding boxes come within two cells of it and whose task
// index is below `limit`.  Collective over the block.  The block first
// collects the dependencies not yet done (one acquire load each) into
// `pend`; then warp 0 alone polls them while the other warps wait at the
// barrier, so a waiting block adds one warp's polling to the memory system
// rather than every warp's (in crowded states many blocks wait at once, and
// their polling starved the running tasks' loads).  If more than kPendCap
// are pending, every warp polls its share of the window as well.
template <int kDT>
__device__ __forceinline__ void wait_canonical(int bx0, int by0, int bx1, int by1, int moveMax, int limit,
                                               int selfCell, const SimTables &T, const StepParams &s,
                                               int cellBase, int *pend, int *npend, int tid) {
	const int rad = 2 + moveMax;
	const int x0 = max(bx0 - rad, 0), x1 = min(bx1 + rad, s.gx - 1);
	const int y0 = max(by0 - rad, 0), y1 = min(by1 + rad, s.gy - 1);
	const int w = x1 - x0 + 1;
	const int total = w * (y1 - y0 + 1);
	const int lane = tid & (kWarp - 1);
	if (tid == 0) *npend = 0;
	__syncthreads();
	for (int q0 = 0; q0 < total; q0 += kDT) {
		const int q = q0 + tid;
		int r = -1;
		if (q < total) {
			const int c2 = cellBase + (y0 + q / w) * s.gx + (x0 + q % w);
			const int r2 = T.taskOfCell[c2];
			if (c2 != selfCell && r2 < limit && T.cellCount[c2] > 0) {
				const int4 b = *reinterpret_cast<const int4 *>(&T.bbox[4 * c2]);
				if (rect_dist(b.x, b.y, b.z, b.w, bx0, by0, bx1, by1) <= 2 && ld_acquire(&T.done[r2]) == 0u) r = r2;
			}
		}
		list_pending(r, pend, npend, lane);
	}
	__syncthreads();
	const int np = *npend;
	if (np > kPendCap) {
		// Too many to list: every warp polls its share of the window.
		for (int q0 = 0; q0 < total; q0 += kDT) {
			const int q = q0 + tid;
			const uint32_t *flag = nullptr;
			if (q < total) {
				const int c2 = cellBase + (y0 + q / w) * s.gx + (x0 + q % w);
				const int r2 = T.taskOfCell[c2];
				if (c2 != selfCell && r2 < limit && T.cellCount[c2] > 0) {
					const int4 b = *reinterpret_cast<const int4 *>(&T.bbox[4 * c2]);
					if (rect_dist(b.x, b.y, b.z, b.w, bx0, by0, bx1, by1) <= 2) flag = &T.done[r2];
				}
			}
			warp_wait(flag, T.abort, T.error, T.waitLimitNs);
		}
	} else {
		poll_pending(pend, np, T, tid);
	}
	__syncthreads();
}

}  // namespace

template <class C>
__global__ void __launch_bounds__(C::kWarps * kWarp, C::kMinBlocks) k_delta(Totals tt, Particles Q, SimTables T) {
	constexpr int kDT = C::kWarps * kWarp;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	DeltaSmemT<C> &S = *reinterpret_cast<DeltaSmemT<C> *>(smem_raw);
	const int tid = threadIdx.x;
	const int nLive = tt.refOrder ? 0 : *T.nLive;
	const int ntask = nLive + tt.nApp;
	const int moveMax = *T.moveMax;
	const int *ord = tt.refOrder ? T.refOrd : nullptr;
	for (;;) {
		if (tid == 0) S.task = atomicAdd(&T.taskCounter[1], 1);
		__syncthreads();
		const int i = S.task;
		__syncthreads();
		if (i >= ntask) break;
		// Task index (done flag): canonical cell task, or ncell + appendix run.
		const int t = i < nLive ? T.liveTask[i] : tt.ncell + (i - nLive);
		stamp(T, 1, t, 0, tid);
		if (i < nLive) {
			const int c = T.taskCell[t];
			const int p0 = T.cellStart[c], cnt = T.cellCount[c];
			if (cnt > 0) {
				const SceneDev &sc = T.scenes[T.sceneOfCell[c]];
				const StepParams s = sc.p;
				const int4 b = *reinterpret_cast<const int4 *>(&T.bbox[4 * c]);
				const unsigned long long staged =
				    relax_group<C>(S, p0, p0 + cnt, nullptr, b.x, b.y, b.z, b.w, Q, T, s, sc.cellBase, tid, [&] {
					    wait_canonical<kDT>(b.x, b.y, b.z, b.w, moveMax, t, c, T, s, sc.cellBase, S.pend, &S.npend,
					                        tid);
					    stamp(T, 1, t, 1, tid);
				    });
				if (T.prof != nullptr && tid == 0 && t < T.profStride)
					T.prof[((size_t)1 * T.profStride + t) * 4 + 2] = staged;
				__syncthreads();
				__threadfence();
			}
		} else {
			// Appendix run: particles added since the last update, after all
			// canonical tasks; it waits for the earlier runs of its scene
			// whose new cells come within two cells of its own.  In reference
			// order every task is such a run, over the whole scene in
			// AddParticle order.
			const int a = t - tt.ncell;
			const int scene = T.appScene[a];
			const SceneDev &sc = T.scenes[scene];
			const StepParams s = sc.p;
			const int base = sc.cellBase;
			const int p0 = sc.pBase + T.appFrom[a], p1 = sc.pBase + T.appTo[a];
			const int4 box = *reinterpret_cast<const int4 *>(&T.appBox[4 * a]);
			const int bx0 = box.x, by0 = box.y, bx1 = box.z, by1 = box.w;
			relax_group<C>(S, p0, p1, ord, bx0, by0, bx1, by1, Q, T, s, base, tid, [&] {
				if (!tt.refOrder)
					wait_canonical<kDT>(bx0, by0, bx1, by1, moveMax, tt.ncell, -1, T, s, base, S.pend, &S.npend, tid);
				wait_runs<kDT>(a, scene, box, T, tt.ncell, S.pend, &S.npend, tid);
			});
			__syncthreads();
			__threadfence();
		}
		__syncthreads();
		stamp(T, 1, t, 3, tid);
		if (tid == 0 && i != T.hold[1]) st_release(&T.done[t], 1u);
	}
}

// Collisions (demo4.cpp:411-444, sph.h:514-681), velocity (demo4.cpp:446-450)
// and the renumbering into canonical order: the particle at position j of
// new cell c gets number newStart[c] + j.

namespace {

__device__ __forceinline__ float2 v2(float x, float y) { return make_float2(x, y); }

__device__ __forceinline__ float2 normalize2(float2 v) {
	float len = sqrtf(v.x * v.x + v.y * v.y);
	if (len == 0.0f) len = 1.0f;
	const float inv = 1.0f / len;
	return v2(v.x * inv, v.y * inv);
}

__device__ void solve_plane(float2 &p, const Body &b, const StepParams &s) {
	const float2 pp = v2(b.ax * b.r, b.ay * b.r);
	const float2 d = v2(p.x - pp.x, p.y - pp.y);
	const float proj = d.x * b.ax + d.y * b.ay;
	if (proj <= s.radius) {
		const float pen = s.radius - proj;
		p = v2(b.ax * pen + p.x, b.ay * pen + p.y);
	}
}

__device__ void solve_circle(float2 &p, const Body &b, const StepParams &s) {
	const float both = b.r + s.radius;
	const float2 d = v2(p.x - b.ax, p.y - b.ay);
	const float d2 = d.x * d.x + d.y * d.y;
	if (d2 <= both * both) {
		if (fabsf(d2) > 0.0f) {
			const float dist = sqrtf(d2);
			const float inv = 1.0f / dist;
			const float2 nrm = v2(d.x * inv, d.y * inv);
			const float pen = both - dist;
			p = v2(nrm.x * pen + p.x, nrm.y * pen + p.y);
		}
	}
}

__device__ void solve_segment(float2 &p, const Body &b, const StepParams &s) {
	const float both = s.margin + s.radius;
	const float2 a = v2(b.ax, b.ay), bb = v2(b.bx, b.by);
	const float2 e = v2(bb.x - a.x, bb.y - a.y);
	const float u = e.x * (bb.x - p.x) + e.y * (bb.y - p.y);
	const float v = e.x * (p.x - a.x) + e.y * (p.y - a.y);
	float2 closest, nrm;
	if (v <= 0.0f) {
		closest = a;
		const float2 d = v2(p.x - closest.x, p.y - closest.y);
		if (d.x * d.x + d.y * d.y > both * both) return;
		nrm = normalize2(v2(p.x - closest.x, p.y - closest.y));
	} else if (u <= 0.0f) {
		closest = bb;
		const float2 d = v2(p.x - closest.x, p.y - closest.y);
		if (d.x * d.x + d.y * d.y > both * both) return;
		nrm = normalize2(v2(p.x - closest.x, p.y - closest.y));
	} else {
		const float den = e.x * e.x + e.y * e.y;
		const float inv = 1.0f / den;
		closest = v2((a.x * u + bb.x * v) * inv, (a.y * u + bb.y * v) * inv);
		const float2 d = v2(p.x - closest.x, p.y - closest.y);
		if (d.x * d.x + d.y * d.y > both * both) return;
		nrm = v2(-e.y, e.x);
		if (nrm.x * (p.x - a.x) + nrm.y * (p.y - a.y) < 0.0f) nrm = v2(-nrm.x, -nrm.y);
		nrm = normalize2(nrm);
	}
	const float2 dp = v2(p.x - closest.x, p.y - closest.y);
	const float dist = nrm.x * dp.x + nrm.y * dp.y;
	const float pen = both - dist;
	p = v2(nrm.x * pen + p.x, nrm.y * pen + p.y);
}

// FindMTVCirclePolygon + SPHSolvePolygonCollision (sph.h:600-681), keeping
// the reference's Vec2DistanceSquared, which squares the product of the
// coordinate differences (vecmath.h:292-296).
__device__ void solve_polygon(float2 &p, const Body &b, const StepParams &s) {
	const float radius = s.margin + s.radius;
	const int n = b.vertexCount;
	if (n <= 0 || n > kMaxPoly) return;
	int edge = 0;
	float2 normal = v2(0.f, 0.f);
	float separation = -3.40282347e+38f;
	for (int k = 0; k < n; ++k) {
		const int k2 = (k + 1) % n;
		const float2 a = v2(b.verts[2 * k], b.verts[2 * k + 1]);
		const float2 c = v2(b.verts[2 * k2], b.verts[2 * k2 + 1]);
		const float2 ab = v2(c.x - a.x, c.y - a.y);
		const float2 nn = normalize2(v2(1.0f * ab.y, -1.0f * ab.x));
		const float sep = nn.x * (p.x - a.x) + nn.y * (p.y - a.y);
		if (sep > radius) return;
		if (sep > separation) {
			normal = nn;
			separation = sep;
			edge = k;
		}
	}
	const int e2 = (edge + 1) % n;
	const float2 v1 = v2(b.verts[2 * edge], b.verts[2 * edge + 1]);
	const float2 v2p = v2(b.verts[2 * e2], b.verts[2 * e2 + 1]);
	float2 mtv;
	if (separation < 1.1920929e-07f) {
		const float pen = radius - separation;
		mtv = v2(normal.x * pen, normal.y * pen);
	} else {
		const float u1 = (p.x - v1.x) * (v2p.x - v1.x) + (p.y - v1.y) * (v2p.y - v1.y);
		const float u2 = (p.x - v2p.x) * (v1.x - v2p.x) + (p.y - v2p.y) * (v1.y - v2p.y);
		if (u1 <= 0.0f) {
			const float f = (v1.x - p.x) * (v1.y - p.y);
			if (f * f > radius * radius) return;
			const float2 d = v2(p.x - v1.x, p.y - v1.y);
			const float2 nn = normalize2(d);
			const float pen = radius - (nn.x * d.x + nn.y * d.y);
			mtv = v2(nn.x * pen, nn.y * pen);
		} else if (u2 <= 0.0f) {
			const float f = (v2p.x - p.x) * (v2p.y - p.y);
			if (f * f > radius * radius) return;
			const float2 d = v2(p.x - v2p.x, p.y - v2p.y);
			const float2 nn = normalize2(d);
			const float pen = radius - (nn.x * d.x + nn.y * d.y);
			mtv = v2(nn.x * pen, nn.y * pen);
		} else {
			const float2 mid = v2((1.0f - 0.5f) * v1.x + 0.5f * v2p.x, (1.0f - 0.5f) * v1.y + 0.5f * v2p.y);
			const float sd = (p.x - mid.x) * normal.x + (p.y - mid.y) * normal.y;
			if (sd > radius) return;
			const float pen = radius - sd;
			mtv = v2(normal.x * pen, normal.y * pen);
		}
	}
	p = v2(mtv.x + p.x, mtv.y + p.y);
}

}  // namespace

__global__ void __launch_bounds__(kCollideThreads) k_collide(Totals tt, Particles P, Particles Q, SimTables T) {
	// j: new number.  Positions, densities and pressures are already in new
	// order; the rest is gathered from the old number.
	const int j = blockIdx.x * blockDim.x + threadIdx.x;
	if (j < tt.ncell) T.appCount[j] = 0;
	if (j >= tt.n) return;
	const SceneDev &sc = T.scenes[T.sceneOf[j]];
	const StepParams &s = sc.p;
	float2 x = Q.pos[j];
	for (int b = 0; b < s.nbodies; ++b) {
		const Body &bd = T.bodies[sc.bodyBase + b];
		switch (bd.type) {
			case kBodyPlane: solve_plane(x, bd, s); break;
			case kBodyCircle: solve_circle(x, bd, s); break;
			case kBodySegment: solve_segment(x, bd, s); break;
			case kBodyPolygon: solve_polygon(x, bd, s); break;
			default: break;
		}
	}
	int o = T.newIdx[j];
	if (o < 0 || o >= tt.n) {
		atomicOr(T.error, kErrIndex);
		o = 0;
	}
	const float2 pv = P.prev[o];
	Q.pos[j] = x;
	Q.prev[j] = pv;
	Q.vel[j] = make_float2((x.x - pv.x) * s.invDt, (x.y - pv.y) * s.invDt);
	Q.acc[j] = make_float2(0.0f, 0.0f);
	Q.id[j] = P.id[o];
	Q.cellOf[j] = T.newCell[o];
}

// ---------------------------------------------------------------------------
// Learned correction of a finished update: x += h u, bodies as in the
// collision stage, velocity from the previous position (canonical numbering).
__global__ void __launch_bounds__(kCollideThreads) k_learned_finish(Totals tt, Particles P, const float2 *u,
                                                                   SimTables T) {
	const int j = blockIdx.x * blockDim.x + threadIdx.x;
	if (j >= tt.n) return;
	const SceneDev &sc = T.scenes[T.sceneOf[j]];
	const StepParams &s = sc.p;
	const float2 d = u[j];
	float2 x = P.pos[j];
	x = make_float2(x.x + s.h * d.x, x.y + s.h * d.y);
	for (int b = 0; b < s.nbodies; ++b) {
		const Body &bd = T.bodies[sc.bodyBase + b];
		switch (bd.type) {
			case kBodyPlane: solve_plane(x, bd, s); break;
			case kBodyCircle: solve_circle(x, bd, s); break;
			case kBodySegment: solve_segment(x, bd, s); break;
			case kBodyPolygon: solve_polygon(x, bd, s); break;
			default: break;
		}
	}
	const float2 pv = P.prev[j];
	P.pos[j] = x;
	P.vel[j] = make_float2((x.x - pv.x) * s.invDt, (x.y - pv.y) * s.invDt);
}

// ---------------------------------------------------------------------------
// AddParticle (demo4.cpp:142-153) for a batch of numbers [first, first+count)
// of scene `scene`: the new particles join the appendix of their cell.
__global__ void k_add(int first, int count, int scene, int firstId, const float2 *pos, const float2 *force,
                      Particles P, SimTables T) {
	const int j = blockIdx.x * blockDim.x + threadIdx.x;
	if (j >= count) return;
	const SceneDev &sc = T.scenes[scene];
	const int i = first + j;
	const float2 x = pos[j];
	P.pos[i] = x;
	P.prev[i] = x;
	P.vel[i] = make_float2(0.f, 0.f);
	P.acc[i] = force[j];
	P.dens[i] = make_float2(0.f, 0.f);
	P.press[i] = make_float2(0.f, 0.f);
	P.id[i] = firstId + j;
	if (P.springN) P.springN[i] = 0;
	T.sceneOf[i] = scene;
	const int c = sc.cellBase + cell_of(x, sc.p);
	P.cellOf[i] = c;
	const int before = atomicAdd(&T.appCount[c], 1);
	const uint32_t now = (uint32_t)(T.cellCount[c] + before + 1);
	atomicMin(&T.stats[4 * scene + 2], now);
	atomicMax(&T.stats[4 * scene + 3], now);
}

// Checks of a state given to sph_load_state, on the device (one thread per
// particle and per cell): every cell range lies within the canonical
// particles, every particle's cell and AddParticle index are in range, and
// every canonical particle lies in its cell's range, and no two particles
// share an AddParticle index (seen[] starts at zero).  Particles added since
// the last update (numbers >= n0) are counted per cell into appOut.
// verdict[0] collects failures, verdict[1] the sum of the cell counts.
__global__ void k_check_state(int n, int n0, int ncell, const int *cell, const int *start, const int *count,
                              const int *id, int *appOut, int *seen, int *verdict) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	int bad = 0;
	if (i < ncell) {
		const int st = start[i], cn = count[i];
		bad |= st < 0 || cn < 0 || (long long)st + cn > n0;
		if (!bad && cn) atomicAdd(&verdict[1], cn);
	}
	if (i < n) {
		const int c = cell[i];
		const int k = id[i];
		bad |= c < 0 || c >= ncell || k < 0 || k >= n;
		if (!bad) bad |= atomicAdd(&seen[k], 1) != 0;  // AddParticle indices are distinct
		if (!bad) {
			if (i >= n0) {
				atomicAdd(&appOut[c], 1);
			} else {
				const int st = start[c], cn = count[c];
				bad |= i < st || i >= st + cn;
			}
		}
	}
	if (bad) atomicOr(&verdict[0], 1);
}

// Scatter numbers [first, first+count) into AddParticle order for host reads.
__global__ void k_gather_by_id(int first, int count, const int *id, const float2 *src, float2 *dst) {
	const int j = blockIdx.x * blockDim.x + threadIdx.x;
	if (j >= count) return;
	const int k = id[first + j];
	if (k >= 0 && k < count) dst[k] = src[first + j];
}

template <class C>
size_t visc_smem_bytes() {
	return sizeof(ViscSmemT<C>);
}
template <class C>
size_t delta_smem_bytes() {
	return sizeof(DeltaSmemT<C>);
}
cudaError_t sweep_attributes() {
	cudaError_t e = cudaFuncSetAttribute(k_viscosity<ViscWide>, cudaFuncAttributeMaxDynamicSharedMemorySize,
	                                     (int)visc_smem_bytes<ViscWide>());
	if (e == cudaSuccess)
		e = cudaFuncSetAttribute(k_viscosity_multi<ViscLean>, cudaFuncAttributeMaxDynamicSharedMemorySize,
		                         (int)sizeof(ViscMultiSmemT<ViscLean>));
	if (e == cudaSuccess)
		e = cudaFuncSetAttribute(k_delta<DeltaWide>, cudaFuncAttributeMaxDynamicSharedMemorySize,
		                         (int)delta_smem_bytes<DeltaWide>());
	if (e == cudaSuccess)
		e = cudaFuncSetAttribute(k_delta<DeltaLean>, cudaFuncAttributeMaxDynamicSharedMemorySize,
		                         (int)delta_smem_bytes<DeltaLean>());
	if (e == cudaSuccess)
		e = cudaFuncSetAttribute(k_delta<DeltaMid>, cudaFuncAttributeMaxDynamicSharedMemorySize,
		                         (int)delta_smem_bytes<DeltaMid>());
	if (e == cudaSuccess)
		e = cudaFuncSetAttribute(k_delta<DeltaTri>, cudaFuncAttributeMaxDynamicSharedMemorySize,
		                         (int)delta_smem_bytes<DeltaTri>());
	if (e == cudaSuccess)
		e = cudaFuncSetAttribute(k_delta<DeltaQuad>, cudaFuncAttributeMaxDynamicSharedMemorySize,
		                         (int)delta_smem_bytes<DeltaQuad>());
	if (e == cudaSuccess)
		e = cudaFuncSetAttribute(k_delta<DeltaDense>, cudaFuncAttributeMaxDynamicSharedMemorySize,
		                         (int)delta_smem_bytes<DeltaDense>());
	return e;
}

cudaError_t sweep_occupancy(bool viscLean, int deltaShape, int *occV, int *occD) {
	cudaError_t e = viscLean ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(occV, k_viscosity_multi<ViscLean>,
	                                                                         ViscLean::kThreads,
	                                                                         sizeof(ViscMultiSmemT<ViscLean>))
	                         : cudaOccupancyMaxActiveBlocksPerMultiprocessor(occV, k_viscosity<ViscWide>,
	                                                                         ViscWide::kWarps * kWarp,
	                                                                         visc_smem_bytes<ViscWide>());
	if (e != cudaSuccess) return e;
	if (deltaShape == kDeltaLean)
		return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occD, k_delta<DeltaLean>, DeltaLean::kWarps * kWarp,
		                                                     delta_smem_bytes<DeltaLean>());
	if (deltaShape == kDeltaMid)
		return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occD, k_delta<DeltaMid>, DeltaMid::kWarps * kWarp,
		                                                     delta_smem_bytes<DeltaMid>());
	if (deltaShape == kDeltaTri)
		return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occD, k_delta<DeltaTri>, DeltaTri::kWarps * kWarp,
		                                                     delta_smem_bytes<DeltaTri>());
	if (deltaShape == kDeltaQuad)
		return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occD, k_delta<DeltaQuad>, DeltaQuad::kWarps * kWarp,
		                                                     delta_smem_bytes<DeltaQuad>());
	if (deltaShape == kDeltaDense)
		return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occD, k_delta<DeltaDense>, DeltaDense::kWarps * kWarp,
		                                                     delta_smem_bytes<DeltaDense>());
	return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occD, k_delta<DeltaWide>, DeltaWide::kWarps * kWarp,
	                                                     delta_smem_bytes<DeltaWide>());
}

void launch_viscosity(bool lean, int blocks, cudaStream_t st, Totals tt, Particles P, SimTables T) {
	if (lean)
		k_viscosity_multi<ViscLean>
		    <<<blocks, ViscLean::kThreads, sizeof(ViscMultiSmemT<ViscLean>), st>>>(tt, P, T);
	else
		k_viscosity<ViscWide><<<blocks, ViscWide::kWarps * kWarp, visc_smem_bytes<ViscWide>(), st>>>(tt, P, T);
}

void launch_delta(int shape, int blocks, cudaStream_t st, Totals tt, Particles Q, SimTables T) {
	if (shape == kDeltaLean)
		k_delta<DeltaLean><<<blocks, DeltaLean::kWarps * kWarp, delta_smem_bytes<DeltaLean>(), st>>>(tt, Q, T);
	else if (shape == kDeltaMid)
		k_delta<DeltaMid><<<blocks, DeltaMid::kWarps * kWarp, delta_smem_bytes<DeltaMid>(), st>>>(tt, Q, T);
	else if (shape == kDeltaTri)
		k_delta<DeltaTri><<<blocks, DeltaTri::kWarps * kWarp, delta_smem_bytes<DeltaTri>(), st>>>(tt, Q, T);
	else if (shape == kDeltaQuad)
		k_delta<DeltaQuad><<<blocks, DeltaQuad::kWarps * kWarp, delta_smem_bytes<DeltaQuad>(), st>>>(tt, Q, T);
	else if (shape == kDeltaDense)
		k_delta<DeltaDense><<<blocks, DeltaDense::kWarps * kWarp, delta_smem_bytes<DeltaDense>(), st>>>(tt, Q, T);
	else
		k_delta<DeltaWide><<<blocks, DeltaWide::kWarps * kWarp, delta_smem_bytes<DeltaWide>(), st>>>(tt, Q, T);
}
size_t dens_smem_bytes() { return sizeof(DensWarp) * kDensWarps; }

}  // namespace sphgb
