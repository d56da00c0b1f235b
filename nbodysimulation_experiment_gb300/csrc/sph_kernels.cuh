// Kernel declarations and launch shapes of the GB300 Demo4 SPH step.
#pragma once

#include "sph_internal.cuh"

namespace sphgb {

// Shapes of the two ordered sweeps (one task per block).  Wide: more warps
// per task and buffers for the largest lists the reference accepts (short
// critical path for one scene).  Lean: fewer warps and smaller buffers (more
// tasks per SM for many scenes).  Results do not depend on the shape.
struct ViscWide {
	static constexpr int kWarps = 4, kProducers = 3 * kWarp, kGeom = 512, kMinBlocks = 4;
};
// Lean viscosity: kSlots tasks per block, one block per SM; the lanes of
// kChains warps run their chains, one producer warp serves each
// (k_viscosity_multi).  A slot stages up to kVelCap list entries; its producer
// holds the positions of up to kRegEntries * 32 of them in registers.  kName:
// the number that names the shape in sph_set_sweep_shape.
struct ViscLean {
	static constexpr int kName = 5;
	static constexpr int kSlots = 18, kChains = 2, kVelCap = 768, kGeom = 160, kRegEntries = 12, kMinBlocks = 1;
	static constexpr int kThreads = (kChains + kSlots) * kWarp;
	static_assert(kSlots % kChains == 0 && kSlots / kChains <= kWarp && kGeom >= kWarp, "slots per chain warp");
};
// Delta sweep.  Pipelined shapes run kProducers producer warps and one summer
// warp per task; the others relax one particle at a time on the whole block.
// kChainW in-range pairs are buffered per warp; a particle's list is relaxed
// in the pipeline when it has at most kProducers * kChainW entries.  kName
// names the shape in sph_set_sweep_shape.  Wide: twelve producers, one block
// per SM (short per-particle latency for one scene).  Lean: two warps, not
// pipelined, smaller staging (more tasks per SM for many scenes).  kDirect: a
// producer thread evaluates the list entries it scans itself (shortest phase,
// for the shapes with many warps per task); otherwise the in-range entries are
// compacted first (fewest square roots and divisions, for the shapes with two
// or three producer warps: evaluated directly, tri took 1,853 ns per particle
// of one task alone against 1,445, quad 1,234 against 1,148).  kApart: the
// summer has its scheduler to itself (pipeline_role).  kDenseCell: particles in
// the fullest cell from which the mid shape is faster (choose_shapes).
struct DeltaWide {
	static constexpr int kName = 12;
	static constexpr int kWarps = 16, kProducers = 12, kStage = kDeltaStageCap, kChainW = 96, kPrefetch = 128, kMinBlocks = 1;
	static constexpr int kRegion = kRegionCells;
	static constexpr bool kPipelined = true, kDirect = true, kApart = true;
};
struct DeltaLean {
	static constexpr int kName = 2, kDenseCell = 90;
	static constexpr int kWarps = 2, kProducers = 1, kStage = 1760, kChainW = 192, kPrefetch = 64, kMinBlocks = 8;
	static constexpr int kRegion = kRegionCells;
	static constexpr bool kPipelined = false, kDirect = false, kApart = false;
};
// Mid: pipelined, six producers, two blocks per SM (mid-size scenes, where
// more tasks run at once than one block per SM holds).
struct DeltaMid {
	static constexpr int kName = 8;
	static constexpr int kWarps = 8, kProducers = 6, kStage = kDeltaStageCap, kChainW = 160, kPrefetch = 128, kMinBlocks = 2;
	static constexpr int kRegion = 256;
	static constexpr bool kPipelined = true, kDirect = true, kApart = true;
};
// Small pipelined shapes for large scenes, where the sweep is bound by how
// many tasks run at once rather than by one task's latency: two (tri) or
// three (quad) producer warps and the summer warp, several blocks per SM.
struct DeltaTri {
	static constexpr int kName = 3, kDenseCell = 108;
	static constexpr int kWarps = 3, kProducers = 2, kStage = 2000, kChainW = 256, kPrefetch = 64, kMinBlocks = 5;
	static constexpr int kRegion = kRegionCells;
	static constexpr bool kPipelined = true, kDirect = false, kApart = false;
};
struct DeltaQuad {
	static constexpr int kName = 4, kDenseCell = 132;
	static constexpr int kWarps = 4, kProducers = 3, kStage = 3072, kChainW = 192, kPrefetch = 128, kMinBlocks = 4;
	static constexpr int kRegion = kRegionCells;
	static constexpr bool kPipelined = true, kDirect = false, kApart = true;
};
// Dense: pipelined, twelve producers, one block per SM, a 12,288-entry stage,
// for crowded states where a task's region (the bounding box of its
// particles' new cells, grown by one) outgrows the other shapes' stages and
// their tasks would be staged again for every group of particles that fits.
struct DeltaDense {
	static constexpr int kName = 16;
	static constexpr int kWarps = 16, kProducers = 12, kStage = kDeltaDenseStageCap, kChainW = 96, kPrefetch = 128, kMinBlocks = 1;
	static constexpr int kRegion = 400;
	static constexpr bool kPipelined = true, kDirect = true, kApart = true;
};
// Delta shapes by index (sph_set_sweep_shape names them by kName).
constexpr int kDeltaShapes = 6;
constexpr int kDeltaWide = 0, kDeltaLean = 1, kDeltaMid = 2, kDeltaTri = 3, kDeltaQuad = 4, kDeltaDense = 5;
constexpr int delta_shape_warps(int shape) {
	return shape == kDeltaLean    ? DeltaLean::kName
	       : shape == kDeltaMid   ? DeltaMid::kName
	       : shape == kDeltaTri   ? DeltaTri::kName
	       : shape == kDeltaQuad  ? DeltaQuad::kName
	       : shape == kDeltaDense ? DeltaDense::kName
	                              : DeltaWide::kName;
}
constexpr int kDensWarps = 8;
constexpr int kViscRefWarps = 4;  // reference-order viscosity sweep: one task per warp
constexpr int kGridWarps = 4;
constexpr int kScanThreads = 1024;
constexpr int kScanTile = 4 * kScanThreads;  // scan positions per block
// Grids of more tiles take a pass over the tiles' sums (k_tile_offsets, which
// has the figures).
constexpr int kScanFewTiles = 512;
constexpr int kElemThreads = 256;  // elementwise kernels
constexpr int kCollideThreads = 256;
constexpr int kSpringWarps = 4;

struct DensWarp;

// The two ordered sweeps in a chosen shape (lean or wide), and their set-up.
cudaError_t sweep_attributes();
cudaError_t sweep_occupancy(bool viscLean, int deltaShape, int *occV, int *occD);
// The fullest cell's particles past which dense states leave a delta shape for
// the mid one; 0: they do not (wide, mid, dense).
inline uint32_t delta_dense_cell(int shape) {
	return shape == kDeltaLean   ? DeltaLean::kDenseCell
	       : shape == kDeltaTri  ? DeltaTri::kDenseCell
	       : shape == kDeltaQuad ? DeltaQuad::kDenseCell
	                             : 0;
}
void launch_viscosity(bool lean, int blocks, cudaStream_t st, Totals tt, Particles P, SimTables T);
void launch_delta(int shape, int blocks, cudaStream_t st, Totals tt, Particles Q, SimTables T);
size_t dens_smem_bytes();

__global__ void k_integrate(Totals tt, Particles P, SimTables T, uint32_t *doneV, int nDoneV, uint32_t *doneD,
                            int nDoneD);
__global__ void k_ref_order(Totals tt, Particles P, SimTables T);
__global__ void k_visc_boxes(Totals tt, Particles P, SimTables T);
__global__ void k_viscosity_ref(Totals tt, Particles P, SimTables T);
__global__ void k_predict(Totals tt, Particles P, SimTables T);
__global__ void k_live_reduce(Totals tt, SimTables T);
__global__ void k_tile_offsets(int *tiles, int ntiles);
__global__ void k_live_apply(Totals tt, SimTables T);
__global__ void k_scan_reduce(Totals tt, SimTables T);
__global__ void k_scan_apply(Totals tt, SimTables T);
__global__ void k_scatter(Totals tt, Particles P, SimTables T);
__global__ void k_grid_update(Totals tt, Particles P, Particles Q, SimTables T);
__global__ void k_app_boxes(Totals tt, SimTables T);
__global__ void k_density(Totals tt, Particles Q, SimTables T, int added, int sms);
__global__ void k_collide(Totals tt, Particles P, Particles Q, SimTables T);
__global__ void k_add(int first, int count, int scene, int firstId, const float2 *pos, const float2 *force,
                      Particles P, SimTables T);
__global__ void k_gather_by_id(int first, int count, const int *id, const float2 *src, float2 *dst);
__global__ void k_check_state(int n, int n0, int ncell, const int *cell, const int *start, const int *count,
                              const int *id, int *appOut, int *seen, int *verdict);
__global__ void k_check_springs(int n, const int *cnt, const int *partner, int *verdict);
__global__ void k_clean_springs(int n, const int *cnt, const int *partner, const float *rest, int *cntOut,
                                int *partnerOut, float *restOut);
__global__ void k_particle_colors(int first, int count, const int *id, const float2 *dens, const float2 *press,
                                  const float2 *vel, float rho0, float4 *out);
__global__ void k_splat_points(int first, int count, const int *id, const float2 *pos, const float2 *dens,
                               const float2 *press, const float2 *vel, float rho0, float halfW, float halfH,
                               float sx, float sy, int width, int height, unsigned long long *keys);
__global__ void k_keys_to_rgba8(int pixels, const unsigned long long *keys, uint32_t *rgba);
void launch_springs_select(int blocks, cudaStream_t st, const Totals &tt, const Particles &P, const Particles &Q,
                           const SimTables &T);
void launch_springs_select_listed(int blocks, cudaStream_t st, const Totals &tt, const Particles &P,
                                  const Particles &Q, const SimTables &T);
bool configure_springs_select();
__global__ void k_springs_commit(Totals tt, Particles Q, SimTables T);
__global__ void k_springs_apply(Totals tt, Particles Q, SimTables T);
__global__ void k_learned_z0(int n, int np, const float2 *pos, const float2 *prev, float invH, float2 *z0);
__global__ void k_learned_finish(Totals tt, Particles P, const float2 *u, SimTables T);
constexpr int kErrThreads = 256;  // judge's reduction: threads per block
constexpr int kErrBlocks = 512;   // and at most this many blocks
__global__ void k_density_error(int n, const float2 *dens, float rho0, double *partial);
__global__ void k_density_error_total(int blocks, const double *partial, double *out);
__global__ void k_scatter_by_id(int n, const float2 *pos, const int *id, float2 *byId);
__global__ void k_learned_target(int n, const float2 *byId, const int *ids, const float2 *xstar, float invH,
                                 float2 *target);

}  // namespace sphgb
