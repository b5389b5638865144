// C ABI of the batched (mixed element type and order) explicit DG residual: dgpu_batch_* in include/dgpu.h.
//
// Volumes are grouped by (element type, p): tensor-product groups (QUAD/HEX, factored operators,
// dgpu_batched.cuh) first, then dense-operator groups (TET/WEDGE/PYR, dgpu_dense.cuh). They are stored group by
// group on the device; the caller's state stays in volume-list order and is permuted on upload/download. Faces
// are renumbered internally by increasing q_f so that each face order's nodes form one range. Each RK stage runs
// as one launch per group and per face order ("plain"), as three persistent launches over all groups ("fused"),
// or as the plain launches on parallel graph branches ("branches"); a whole step is replayed from a captured CUDA
// graph. dgpu_batch_autotune times the elements-per-CTA candidates of every group and the three forms on the
// actual mesh and keeps the fastest.
#include <cuda_runtime.h>

#include <algorithm>
#include <stdio.h>
#include <string>
#include <vector>

#include "../../include/dgpu.h"
#include "dgpu_batched_ns.cuh"
#include "dgpu_dense.cuh"
#include "dgpu_host_ops.h"

using namespace dgpu;

// Compiled once for the host code (DGPU_PART 0) and once per part, each of which defines one of the functions below, that
// set a context's launchers.
#ifndef DGPU_PART
#error "compile with -DDGPU_PART=0..4"
#endif
cudaError_t dgpu_batch_bind_2d(dgpu_batch* c);                  // part 1: every PDE
cudaError_t dgpu_batch_bind_3d_advection_roe(dgpu_batch* c);    // part 2: advection, Euler with Roe-Pike
cudaError_t dgpu_batch_bind_3d_lf(dgpu_batch* c);               // part 3: Euler with Lax-Friedrichs
cudaError_t dgpu_batch_bind_3d_ns(dgpu_batch* c);               // part 4: Navier-Stokes on top of Euler

namespace dgpu {

constexpr int kBranches = 16;   // streams of the branch form

struct GroupLaunch {
	cudaError_t (*vol)(dgpu_batch*, int g, bool gll_in) = nullptr;
	cudaError_t (*lift)(dgpu_batch*, int g, int mode, double dt, int stage, int want_max) = nullptr;
	cudaError_t (*conv)(dgpu_batch*, int g, bool to_gl) = nullptr;
	// Navier-Stokes: the gradient and the volume kernels of the group (TP groups only)
	cudaError_t (*ns_grad)(dgpu_batch*, int g, bool gll_in) = nullptr;
	cudaError_t (*ns_vol)(dgpu_batch*, int g, bool gll_in) = nullptr;
	int E_max = 0;
	bool dense = false;
	int idx = 0;        // index among the TP or among the dense groups
};

}  // namespace dgpu

struct dgpu_batch {
	int d = 0, nv = 0, pde = 0, flux = 0, positivity = 0;
	double b_adv[3] = {0, 0, 0};
	int n_tp = 0, n_dense = 0, n_all = 0, n_vol = 0, n_face = 0;
	std::vector<int> caller_to_internal;   // caller group -> internal group (TP first, then dense)
	std::vector<BGroup> hgroups;           // TP groups
	std::vector<DGroup> hdgroups;          // dense groups
	std::vector<BatchOps> hops;
	std::vector<GroupLaunch> gl;           // internal groups
	std::vector<int> order;                // sorted element -> list index
	std::vector<long long> list_off;       // list index -> offset in the caller's state
	std::vector<long long> sorted_off;     // sorted element -> offset in the device state
	// the source term (dgpu_batch_set_source): the caller's cubature-node offsets, and per dense group its cv0
	// (n_vc x n_vs) and every volume's w J at its nodes (group-sorted), for the projection cv0^T diag(w J) s
	std::vector<long long> list_vc_off;
	std::vector<std::vector<double>> dense_cv0_h, dense_wJ_h;
	double* source = nullptr;              // state layout (group-sorted), or null
	size_t ns = 0;
	// device
	BatchOps* d_ops = nullptr;
	BGroup* d_groups = nullptr;
	DGroup* d_dgroups = nullptr;
	std::vector<void*> dense_bufs;         // per dense group: operators, face operators, offsets, 1/J
	int4* d_elf = nullptr;
	long long* d_fbase = nullptr;
	int *d_nc = nullptr, *d_nc_inv = nullptr;   // right-trace gather permutation per face node and its inverse, or null
	int* d_node_face = nullptr;
	double *gmet = nullptr, *inv_wJ = nullptr, *fgeo = nullptr;
	double *u = nullptr, *ug = nullptr, *u0 = nullptr, *rhs = nullptr, *vol_gl = nullptr;
	double *traces = nullptr, *nnf = nullptr;
	// Navier-Stokes (BR2): kept volume gradient, gradient traces, jumps and each side's own lifting at the faces
	bool navier_stokes = false;
	NsPhys ns_phys = {0.0, 1.0, 1.0, kViscosityConstant, 0.0};
	double *ns_gv = nullptr, *ns_gtr = nullptr, *ns_dw = nullptr, *ns_y = nullptr;
	cudaError_t (*ns_nodes)(dgpu_batch*, bool face) = nullptr;   // the jump (false) or face (true) kernel
	int* d_fbc = nullptr;                  // boundary faces (null without any): code per internal face, -1 inside
	double* d_fext = nullptr;              // their exterior state, [NV][NF_f] at NV fbase[f]
	BcData bc_data = {0.0, 0.0, 0.0, 0.0};
	unsigned long long* max_bits = nullptr;
	int* err_flag = nullptr;
	unsigned long long* n_corr = nullptr;
	long long qnode[kQMax + 2] = {0};      // face nodes of order q_f: [qnode[q_f], qnode[q_f + 1])
	BTile* d_tiles = nullptr;
	int n_tiles = 0, fused_blocks_vol = 0, fused_blocks_lift = 0, fused_blocks_lift_nomax = 0, fused_blocks_face = 0;
	size_t fused_vol_smem = 0, fused_lift_smem = 0;
	cudaError_t (*fused_vol)(dgpu_batch*, bool gll_in) = nullptr;
	cudaError_t (*fused_lift)(dgpu_batch*, int mode, double dt, int stage, int want_max) = nullptr;
	// form 3: the stage kernel's grid per mode (residual, RK stage with max |rhs|, without), its barrier words
	int stage_blocks[3] = {0, 0, 0};
	unsigned* d_bar = nullptr;
	unsigned long long barrier_ns = kBarrierLimitNs;   // bound of each grid-barrier wait
	cudaError_t (*stage_launch)(dgpu_batch*, bool rhs_mode, double dt, int stage, int want_max) = nullptr;
	cudaError_t (*face_nodes)(dgpu_batch*, long long lo, long long hi, int blocks) = nullptr;
	// execution
	cudaStream_t stream = nullptr;
	bool own_stream = false;
	bool coef_valid = true, gl_valid = false;
	// 0: one launch per group and face order; 1: fused persistent launches; 2: as 0 on parallel branches;
	// 3: the whole stage in one cooperative persistent launch
	int mode = 0;
	cudaStream_t aux[kBranches] = {nullptr};
	cudaEvent_t ev_fork = nullptr, ev_join[kBranches] = {nullptr};
	bool use_graphs = true;
	cudaGraphExec_t graph[4][2] = {};   // [mode][want_max]
	double graph_dt[4][2] = {};
	long long graph_launches[4][2] = {};   // kernels per replay
	long long launches = 0;
	std::string err;

	BParams params() const
	{
		BParams P;
		for (int k = 0; k < 3; ++k)
			P.b_adv[k] = b_adv[k];
		P.n_groups = n_tp;
		P.dgroups = d_dgroups;
		P.ops = d_ops;
		P.groups = d_groups;
		P.elf = d_elf;
		P.fbase = d_fbase;
		P.nc = d_nc;
		P.nc_inv = d_nc_inv;
		P.gmet = gmet;
		P.inv_wJ = inv_wJ;
		P.fgeo = fgeo;
		P.traces = traces;
		P.nnf = nnf;
		P.vol_gl = vol_gl;
		P.max_bits = max_bits;
		P.err_flag = err_flag;
		P.n_corr = n_corr;
		P.fbc = d_fbc;
		P.fext = d_fext;
		P.bc_data = bc_data;
		P.source = source;
		if (navier_stokes) {
			P.ns_gv = ns_gv;
			P.ns_gtr = ns_gtr;
			P.ns_dw = ns_dw;
			P.ns_y = ns_y;
			P.ns = ns_phys;
			P.ns_eta = 1.01 * 2 * d;   // PENALTY_SCALING * NFMAX (compute_face_rlhs_dg_T.c:273-295)
		}
		return P;
	}
	int group_n_vol(int g) const { return gl[g].dense ? hdgroups[gl[g].idx].n_vol : hgroups[gl[g].idx].n_vol; }
	int group_E(int g) const { return gl[g].dense ? hdgroups[gl[g].idx].E : hgroups[gl[g].idx].E; }
};

namespace {

thread_local std::string g_batch_error;

[[maybe_unused]] dgpu_status bfail(dgpu_batch* c, dgpu_status st, const std::string& m)
{
	if (c)
		c->err = m;
	else
		g_batch_error = m;
	return st;
}

#define BATCH_CUDA(ctx, call)                                                                              \
	do {                                                                                                   \
		cudaError_t e_ = (call);                                                                           \
		if (e_ != cudaSuccess)                                                                             \
			return bfail((ctx), DGPU_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));        \
	} while (0)

// Lets a kernel take `bytes` of dynamic shared memory. The limit belongs to the process, not to a context, so every context
// sets the same one, all that the device has for the kernel: one of its own size would take it away from a context with
// larger groups.
template <typename K>
cudaError_t allow_smem(K* kernel, size_t bytes)
{
	int dev = 0, most = 0;
	cudaFuncAttributes a;
	cudaError_t e = cudaGetDevice(&dev);
	if (e == cudaSuccess)
		e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
	if (e == cudaSuccess)
		e = cudaFuncGetAttributes(&a, kernel);
	if (e != cudaSuccess)
		return e;
	most -= (int)a.sharedSizeBytes;
	return bytes > (size_t)most ? cudaErrorInvalidValue
	                            : cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
}

template <int D, int Q, int NV>
size_t bvol_smem(int E) { return sizeof(BatchOps) + (size_t)E * BSmem<D, Q, NV>::VOL * sizeof(double); }
template <int D, int Q, int NV>
size_t blift_smem(int E) { return sizeof(BatchOps) + (size_t)E * BSmem<D, Q, NV>::LIFT * sizeof(double); }
template <int D, int Q, int NV>
size_t bconv_smem(int E) { return sizeof(BatchOps) + (size_t)E * 3 * NV * TPShape<D, Q>::N * sizeof(double); }
[[maybe_unused]] size_t dvol_smem(int, const DGroup& G, int E) { return (size_t)E * G.vol_per_e * sizeof(double); }
[[maybe_unused]] size_t dlift_smem(int, const DGroup& G, int E) { return (size_t)E * G.lift_per_e * sizeof(double); }

// Whole warps, and at least four (eight in 3D, where a face has q times the columns): the faces' interpolation between
// orders takes every thread of the CTA. 3D from four to eight: mixed types 18^3, 4 steps, 13.07 -> 12.73 ms.
template <int D>
int threads_for(int E, int N)
{
	return std::max(((E * N + 31) / 32) * 32, D == 3 ? 256 : 128);
}

[[maybe_unused]] RkArgs rk_args(const dgpu_batch* c, double dt, int stage, int want_max)
{
	RkArgs rk;
	rk.u = c->ug;
	rk.u0 = c->u0;
	rk.rhs = c->rhs;
	rk.dt = dt;
	rk.stage = stage;
	rk.positivity = c->positivity;
	rk.want_max = want_max;
	return rk;
}

// ---- tensor-product groups ----
template <int D, int Q, int NV, int PDE>
cudaError_t launch_bvol(dgpu_batch* c, int g, bool gll_in)
{
	const int t = c->gl[g].idx;
	const BGroup& G = c->hgroups[t];
	if (G.n_vol == 0)
		return cudaSuccess;
	const int blocks = (G.n_vol + G.E - 1) / G.E, thr = threads_for<D>(G.E, TPShape<D, Q>::N);
	if (gll_in)
		bvol_group_kernel<D, Q, NV, PDE, true><<<blocks, thr, bvol_smem<D, Q, NV>(G.E), c->stream>>>(c->params(), t, c->u);
	else
		bvol_group_kernel<D, Q, NV, PDE, false><<<blocks, thr, bvol_smem<D, Q, NV>(G.E), c->stream>>>(c->params(), t, c->ug);
	c->launches++;
	return cudaGetLastError();
}

template <int D, int Q, int NV>
cudaError_t launch_blift(dgpu_batch* c, int g, int mode, double dt, int stage, int want_max)
{
	const int t = c->gl[g].idx;
	const BGroup& G = c->hgroups[t];
	if (G.n_vol == 0)
		return cudaSuccess;
	const int blocks = (G.n_vol + G.E - 1) / G.E, thr = threads_for<D>(G.E, TPShape<D, Q>::N);
	const RkArgs rk = rk_args(c, dt, stage, want_max);
	if (mode == kModeRhs)
		blift_group_kernel<D, Q, NV, kModeRhs><<<blocks, thr, blift_smem<D, Q, NV>(G.E), c->stream>>>(c->params(), t, rk);
	else if (want_max)
		blift_group_kernel<D, Q, NV, kModeRkGl><<<blocks, thr, blift_smem<D, Q, NV>(G.E), c->stream>>>(c->params(), t, rk);
	else
		blift_group_kernel<D, Q, NV, kModeRkGlNoMax><<<blocks, thr, blift_smem<D, Q, NV>(G.E), c->stream>>>(
			c->params(), t, rk);
	c->launches++;
	return cudaGetLastError();
}

template <int D, int Q, int NV>
cudaError_t launch_bconv(dgpu_batch* c, int g, bool to_gl)
{
	const int t = c->gl[g].idx;
	const BGroup& G = c->hgroups[t];
	if (G.n_vol == 0)
		return cudaSuccess;
	const int blocks = (G.n_vol + G.E - 1) / G.E, thr = threads_for<D>(G.E, TPShape<D, Q>::N);
	if (to_gl)
		bconvert_group_kernel<D, Q, NV, true><<<blocks, thr, bconv_smem<D, Q, NV>(G.E), c->stream>>>(c->params(), t, c->u, c->ug);
	else
		bconvert_group_kernel<D, Q, NV, false><<<blocks, thr, bconv_smem<D, Q, NV>(G.E), c->stream>>>(c->params(), t, c->ug, c->u);
	c->launches++;
	return cudaGetLastError();
}

// ---- dense groups ----
template <int D, int NV, int PDE>
cudaError_t launch_dvol(dgpu_batch* c, int g, bool gll_in)
{
	const int t = c->gl[g].idx;
	const DGroup& G = c->hdgroups[t];
	if (G.n_vol == 0)
		return cudaSuccess;
	const int blocks = (G.n_vol + G.E - 1) / G.E;
	dvol_group_kernel<D, NV, PDE><<<blocks, 256, dvol_smem(NV, G, G.E), c->stream>>>(c->params(), t,
	                                                                                  gll_in ? c->u : c->ug);
	c->launches++;
	return cudaGetLastError();
}

template <int NV>
cudaError_t launch_dlift(dgpu_batch* c, int g, int mode, double dt, int stage, int want_max)
{
	const int t = c->gl[g].idx;
	const DGroup& G = c->hdgroups[t];
	if (G.n_vol == 0)
		return cudaSuccess;
	const int blocks = (G.n_vol + G.E - 1) / G.E;
	const RkArgs rk = rk_args(c, dt, stage, want_max);
	if (mode == kModeRhs)
		dlift_group_kernel<NV, kModeRhs><<<blocks, 256, dlift_smem(NV, G, G.E), c->stream>>>(c->params(), t, rk);
	else
		dlift_group_kernel<NV, kModeRkGl><<<blocks, 256, dlift_smem(NV, G, G.E), c->stream>>>(c->params(), t, rk);
	c->launches++;
	return cudaGetLastError();
}

// the RK state of a dense group is its coefficient vector: u <-> ug is a copy of the group's range
[[maybe_unused]] cudaError_t copy_dense(dgpu_batch* c, int g, bool to_gl)
{
	const DGroup& G = c->hdgroups[c->gl[g].idx];
	if (G.n_vol == 0)
		return cudaSuccess;
	const size_t n = (size_t)G.n_vol * c->nv * G.n_vs;
	const double* src = to_gl ? c->u : c->ug;
	double* dst = to_gl ? c->ug : c->u;
	return cudaMemcpyAsync(dst + G.state_off, src + G.state_off, n * sizeof(double), cudaMemcpyDeviceToDevice,
	                       c->stream);
}

// ---- all groups ----
template <int D, int NV, int PDE, int FLUX>
cudaError_t launch_face_nodes(dgpu_batch* c, long long lo, long long hi, int blocks)
{
	if (hi <= lo)
		return cudaSuccess;
	if (blocks <= 0)
		blocks = (int)std::min<long long>((hi - lo + 255) / 256, 1ll << 30);
	bface_nodes_kernel<D, NV, PDE, FLUX><<<blocks, 256, 0, c->stream>>>(c->params(), c->d_node_face, lo, hi);
	c->launches++;
	return cudaGetLastError();
}

template <int D, int NV, int PDE>
cudaError_t launch_fused_vol(dgpu_batch* c, bool gll_in)
{
	if (gll_in)
		bvol_fused_kernel<D, NV, PDE, true><<<c->fused_blocks_vol, 256, c->fused_vol_smem, c->stream>>>(
			c->params(), c->d_tiles, c->n_tiles, c->u);
	else
		bvol_fused_kernel<D, NV, PDE, false><<<c->fused_blocks_vol, 256, c->fused_vol_smem, c->stream>>>(
			c->params(), c->d_tiles, c->n_tiles, c->ug);
	c->launches++;
	return cudaGetLastError();
}

template <int D, int NV>
cudaError_t launch_fused_lift(dgpu_batch* c, int mode, double dt, int stage, int want_max)
{
	const RkArgs rk = rk_args(c, dt, stage, want_max);
	if (mode == kModeRhs)
		blift_fused_kernel<D, NV, kModeRhs><<<c->fused_blocks_lift, 256, c->fused_lift_smem, c->stream>>>(
			c->params(), c->d_tiles, c->n_tiles, rk);
	else if (want_max)
		blift_fused_kernel<D, NV, kModeRkGl><<<c->fused_blocks_lift, 256, c->fused_lift_smem, c->stream>>>(
			c->params(), c->d_tiles, c->n_tiles, rk);
	else
		blift_fused_kernel<D, NV, kModeRkGlNoMax><<<c->fused_blocks_lift_nomax, 256, c->fused_lift_smem,
		                                            c->stream>>>(c->params(), c->d_tiles, c->n_tiles, rk);
	c->launches++;
	return cudaGetLastError();
}

// Form 3: the stage kernel, cooperatively (all CTAs resident: the grid barriers between its phases complete).
template <int D, int NV, int PDE, int FLUX>
cudaError_t launch_stage(dgpu_batch* c, bool rhs_mode, double dt, int stage, int want_max)
{
	cudaError_t e = cudaMemsetAsync(c->d_bar, 0, 2 * sizeof(unsigned), c->stream);
	if (e != cudaSuccess)
		return e;
	BParams P = c->params();
	RkArgs rk = rk_args(c, dt, stage, want_max);
	const BTile* tiles = c->d_tiles;
	int n_tiles = c->n_tiles;
	const double* u = rhs_mode ? c->u : c->ug;
	const int* node_face = c->d_node_face;
	long long n_nodes = c->qnode[kQMax + 1];
	unsigned* bar = c->d_bar;
	unsigned long long limit_ns = c->barrier_ns;
	void* args[] = {&P, &tiles, &n_tiles, &u, &node_face, &n_nodes, &rk, &bar, &limit_ns};
	const void* k;
	int blocks;
	if (rhs_mode) {
		k = (const void*)bstage_kernel<D, NV, PDE, FLUX, kModeRhs, true>;
		blocks = c->stage_blocks[0];
	} else if (want_max) {
		k = (const void*)bstage_kernel<D, NV, PDE, FLUX, kModeRkGl, false>;
		blocks = c->stage_blocks[1];
	} else {
		k = (const void*)bstage_kernel<D, NV, PDE, FLUX, kModeRkGlNoMax, false>;
		blocks = c->stage_blocks[2];
	}
	if (blocks < 1)
		return cudaErrorCooperativeLaunchTooLarge;
	e = cudaLaunchCooperativeKernel(k, dim3(blocks), dim3(256), args,
	                                std::max(c->fused_vol_smem, c->fused_lift_smem), c->stream);
	c->launches++;
	return e;
}

// The stage kernel's attributes and its grid: every SM times the CTAs that fit on one (the cooperative limit).
template <int D, int NV, int PDE, int FLUX>
cudaError_t bind_stage(dgpu_batch* c, int sms)
{
	const size_t smem = std::max(c->fused_vol_smem, c->fused_lift_smem);
	const void* ks[3] = {(const void*)bstage_kernel<D, NV, PDE, FLUX, kModeRhs, true>,
	                     (const void*)bstage_kernel<D, NV, PDE, FLUX, kModeRkGl, false>,
	                     (const void*)bstage_kernel<D, NV, PDE, FLUX, kModeRkGlNoMax, false>};
	for (int m = 0; m < 3; ++m) {
		cudaError_t e = allow_smem(ks[m], smem);
		if (e != cudaSuccess)
			return e;
		int per_sm = 0;
		if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ks[m], 256, smem)) != cudaSuccess)
			return e;
		c->stage_blocks[m] = sms * per_sm;
	}
	c->stage_launch = launch_stage<D, NV, PDE, FLUX>;
	return cudaSuccess;
}

template <int D, int Q, int NV, int PDE>
cudaError_t bind_tp_group(dgpu_batch* c, int g)
{
	GroupLaunch& L = c->gl[g];
	L.vol = launch_bvol<D, Q, NV, PDE>;
	L.lift = launch_blift<D, Q, NV>;
	L.conv = launch_bconv<D, Q, NV>;
	L.E_max = std::max(1, 256 / TPShape<D, Q>::N);
	const int E = L.E_max;
	cudaError_t e;
	if ((e = allow_smem(bvol_group_kernel<D, Q, NV, PDE, true>, bvol_smem<D, Q, NV>(E))))
		return e;
	if ((e = allow_smem(bvol_group_kernel<D, Q, NV, PDE, false>, bvol_smem<D, Q, NV>(E))))
		return e;
	if ((e = allow_smem(blift_group_kernel<D, Q, NV, kModeRhs>, blift_smem<D, Q, NV>(E))))
		return e;
	if ((e = allow_smem(blift_group_kernel<D, Q, NV, kModeRkGl>, blift_smem<D, Q, NV>(E))))
		return e;
	if ((e = allow_smem(blift_group_kernel<D, Q, NV, kModeRkGlNoMax>, blift_smem<D, Q, NV>(E))))
		return e;
	if ((e = allow_smem(bconvert_group_kernel<D, Q, NV, true>, bconv_smem<D, Q, NV>(E))))
		return e;
	if ((e = allow_smem(bconvert_group_kernel<D, Q, NV, false>, bconv_smem<D, Q, NV>(E))))
		return e;
	// the fused kernels need the largest of the groups' shared memory
	c->fused_vol_smem = std::max(c->fused_vol_smem, bvol_smem<D, Q, NV>(E));
	c->fused_lift_smem = std::max(c->fused_lift_smem, blift_smem<D, Q, NV>(E));
	return cudaSuccess;
}

template <int D, int NV, int PDE, int FLUX>
cudaError_t bind_all(dgpu_batch* c)
{
	size_t dvol_max = 0, dlift_max = 0;
	for (int g = 0; g < c->n_all; ++g) {
		cudaError_t e = cudaSuccess;
		if (c->gl[g].dense) {
			const DGroup& G = c->hdgroups[c->gl[g].idx];
			c->gl[g].vol = launch_dvol<D, NV, PDE>;
			c->gl[g].lift = launch_dlift<NV>;
			c->gl[g].conv = copy_dense;
			c->gl[g].E_max = G.E;
			dvol_max = std::max(dvol_max, dvol_smem(NV, G, G.E));
			dlift_max = std::max(dlift_max, dlift_smem(NV, G, G.E));
			c->fused_vol_smem = std::max(c->fused_vol_smem, sizeof(BatchOps) + dvol_smem(NV, G, G.E_fused));
			c->fused_lift_smem = std::max(c->fused_lift_smem, sizeof(BatchOps) + dlift_smem(NV, G, G.E_fused));
			continue;
		}
		switch (c->hgroups[c->gl[g].idx].q) {
		case 2: e = bind_tp_group<D, 2, NV, PDE>(c, g); break;
		case 3: e = bind_tp_group<D, 3, NV, PDE>(c, g); break;
		case 4: e = bind_tp_group<D, 4, NV, PDE>(c, g); break;
		default: e = bind_tp_group<D, 5, NV, PDE>(c, g); break;
		}
		if (e != cudaSuccess)
			return e;
	}
	cudaError_t e;
	if (c->n_dense > 0) {
		if ((e = allow_smem(dvol_group_kernel<D, NV, PDE>, dvol_max)))
			return e;
		if ((e = allow_smem(dlift_group_kernel<NV, kModeRhs>, dlift_max)))
			return e;
		if ((e = allow_smem(dlift_group_kernel<NV, kModeRkGl>, dlift_max)))
			return e;
	}
	c->fused_vol = launch_fused_vol<D, NV, PDE>;
	c->fused_lift = launch_fused_lift<D, NV>;
	c->face_nodes = launch_face_nodes<D, NV, PDE, FLUX>;
	if ((e = allow_smem(bvol_fused_kernel<D, NV, PDE, true>, c->fused_vol_smem)))
		return e;
	if ((e = allow_smem(bvol_fused_kernel<D, NV, PDE, false>, c->fused_vol_smem)))
		return e;
	if ((e = allow_smem(blift_fused_kernel<D, NV, kModeRhs>, c->fused_lift_smem)))
		return e;
	if ((e = allow_smem(blift_fused_kernel<D, NV, kModeRkGl>, c->fused_lift_smem)))
		return e;
	if ((e = allow_smem(blift_fused_kernel<D, NV, kModeRkGlNoMax>, c->fused_lift_smem)))
		return e;
	// persistent grids: as many CTAs as fit on the device at once
	int dev = 0, sms = 0, per_sm = 0;
	cudaGetDevice(&dev);
	cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bvol_fused_kernel<D, NV, PDE, false>, 256, c->fused_vol_smem);
	c->fused_blocks_vol = std::max(1, std::min(c->n_tiles, sms * std::max(1, per_sm)));
	cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, blift_fused_kernel<D, NV, kModeRkGl>, 256, c->fused_lift_smem);
	c->fused_blocks_lift = std::max(1, std::min(c->n_tiles, sms * std::max(1, per_sm)));
	cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, blift_fused_kernel<D, NV, kModeRkGlNoMax>, 256,
	                                              c->fused_lift_smem);
	c->fused_blocks_lift_nomax = std::max(1, std::min(c->n_tiles, sms * std::max(1, per_sm)));
	c->fused_blocks_face = (int)std::max<long long>(1, std::min<long long>((c->qnode[kQMax + 1] + 255) / 256,
	                                                                       (long long)sms * 8));
	if ((e = bind_stage<D, NV, PDE, FLUX>(c, sms)) != cudaSuccess)
		return e;
	return cudaGetLastError();
}

// ---- Navier-Stokes (dgpu_batched_ns.cuh) ----
template <int D, int Q, int NV>
size_t bns_smem(int E)
{
	return sizeof(BatchOps) + (size_t)E * BnsSmem<D, Q, NV>::MAX * sizeof(double);
}

template <int D, int Q, int NV>
cudaError_t launch_bns(dgpu_batch* c, int g, bool gll_in, bool volume)
{
	const int t = c->gl[g].idx;
	const BGroup& G = c->hgroups[t];
	if (G.n_vol == 0)
		return cudaSuccess;
	const int blocks = (G.n_vol + G.E_ns - 1) / G.E_ns, thr = threads_for<D>(G.E_ns, TPShape<D, Q>::N);
	const size_t sm = bns_smem<D, Q, NV>(G.E_ns);
	const double* u = gll_in ? c->u : c->ug;
	if (volume) {
		if (gll_in)
			bns_volume_group_kernel<D, Q, NV, true><<<blocks, thr, sm, c->stream>>>(c->params(), t, u);
		else
			bns_volume_group_kernel<D, Q, NV, false><<<blocks, thr, sm, c->stream>>>(c->params(), t, u);
	} else {
		if (gll_in)
			bns_grad_group_kernel<D, Q, NV, true><<<blocks, thr, sm, c->stream>>>(c->params(), t, u);
		else
			bns_grad_group_kernel<D, Q, NV, false><<<blocks, thr, sm, c->stream>>>(c->params(), t, u);
	}
	c->launches++;
	return cudaGetLastError();
}

template <int D, int Q, int NV>
cudaError_t launch_bns_grad(dgpu_batch* c, int g, bool gll_in) { return launch_bns<D, Q, NV>(c, g, gll_in, false); }
template <int D, int Q, int NV>
cudaError_t launch_bns_vol(dgpu_batch* c, int g, bool gll_in) { return launch_bns<D, Q, NV>(c, g, gll_in, true); }

template <int D, int NV, int FLUX>
cudaError_t launch_bns_nodes(dgpu_batch* c, bool face)
{
	const long long n = c->qnode[kQMax + 1];
	if (n == 0)
		return cudaSuccess;
	if (face) {
		const int blocks = (int)std::min<long long>((n + 127) / 128, 1ll << 30);
		bns_face_kernel<D, NV, FLUX><<<blocks, 128, 0, c->stream>>>(c->params(), c->d_node_face, n);
	} else {
		const int blocks = (int)std::min<long long>((n + 255) / 256, 1ll << 30);
		bns_jump_kernel<D, NV><<<blocks, 256, 0, c->stream>>>(c->params(), c->d_node_face, n);
	}
	c->launches++;
	return cudaGetLastError();
}

// The Navier-Stokes launchers of every group: elements per CTA as for Euler, fewer where the gradient and volume
// bodies' shared memory (state, D gradient or flux components, face values) would exceed 110 KB per CTA.
template <int D, int Q, int NV>
cudaError_t bind_ns_group(dgpu_batch* c, int g)
{
	GroupLaunch& L = c->gl[g];
	L.ns_grad = launch_bns_grad<D, Q, NV>;
	L.ns_vol = launch_bns_vol<D, Q, NV>;
	constexpr int N = TPShape<D, Q>::N;
	const int by_smem = (int)((110 * 1024 - sizeof(BatchOps)) / (BnsSmem<D, Q, NV>::MAX * sizeof(double)));
	const int E = std::max(1, std::min(256 / N, by_smem));
	c->hgroups[L.idx].E_ns = E;
	const int sm = (int)bns_smem<D, Q, NV>(E);
	cudaError_t e;
	if ((e = allow_smem(bns_grad_group_kernel<D, Q, NV, true>, sm)))
		return e;
	if ((e = allow_smem(bns_grad_group_kernel<D, Q, NV, false>, sm)))
		return e;
	if ((e = allow_smem(bns_volume_group_kernel<D, Q, NV, true>, sm)))
		return e;
	return allow_smem(bns_volume_group_kernel<D, Q, NV, false>, sm);
}

template <int D, int FLUX>
cudaError_t bind_ns(dgpu_batch* c)
{
	constexpr int NV = D + 2;
	for (int g = 0; g < c->n_all; ++g) {
		cudaError_t e;
		switch (c->hgroups[c->gl[g].idx].q) {
		case 2: e = bind_ns_group<D, 2, NV>(c, g); break;
		case 3: e = bind_ns_group<D, 3, NV>(c, g); break;
		case 4: e = bind_ns_group<D, 4, NV>(c, g); break;
		default: e = bind_ns_group<D, 5, NV>(c, g); break;
		}
		if (e != cudaSuccess)
			return e;
	}
	c->ns_nodes = launch_bns_nodes<D, NV, FLUX>;
	return cudaSuccess;
}

}  // namespace

#if DGPU_PART == 1
cudaError_t dgpu_batch_bind_2d(dgpu_batch* c)
{
	if (c->pde == DGPU_PDE_ADVECTION)
		return bind_all<2, 1, kAdvection, kUpwind>(c);
	const bool roe = c->flux == DGPU_NUM_FLUX_ROE_PIKE;
	const cudaError_t e = roe ? bind_all<2, 4, kEuler, kRoePike>(c) : bind_all<2, 4, kEuler, kLaxFriedrichs>(c);
	if (e != cudaSuccess || !c->navier_stokes)   // Navier-Stokes: the lift and conversion kernels are the Euler ones
		return e;
	return roe ? bind_ns<2, kRoePike>(c) : bind_ns<2, kLaxFriedrichs>(c);
}
#elif DGPU_PART == 2
cudaError_t dgpu_batch_bind_3d_advection_roe(dgpu_batch* c)
{
	return c->pde == DGPU_PDE_ADVECTION ? bind_all<3, 1, kAdvection, kUpwind>(c) : bind_all<3, 5, kEuler, kRoePike>(c);
}
#elif DGPU_PART == 3
cudaError_t dgpu_batch_bind_3d_lf(dgpu_batch* c) { return bind_all<3, 5, kEuler, kLaxFriedrichs>(c); }
#elif DGPU_PART == 4
cudaError_t dgpu_batch_bind_3d_ns(dgpu_batch* c)
{
	return c->flux == DGPU_NUM_FLUX_ROE_PIKE ? bind_ns<3, kRoePike>(c) : bind_ns<3, kLaxFriedrichs>(c);
}
#else   // the host code, to the end of the file

namespace {

cudaError_t bind(dgpu_batch* c)
{
	if (c->d == 2)
		return dgpu_batch_bind_2d(c);
	const bool lf = c->pde != DGPU_PDE_ADVECTION && c->flux != DGPU_NUM_FLUX_ROE_PIKE;
	const cudaError_t e = lf ? dgpu_batch_bind_3d_lf(c) : dgpu_batch_bind_3d_advection_roe(c);
	return e != cudaSuccess || !c->navier_stokes ? e : dgpu_batch_bind_3d_ns(c);
}

void drop_graphs(dgpu_batch* c)
{
	for (auto& gm : c->graph)
		for (auto& g : gm)
			if (g) {
				cudaGraphExecDestroy(g);
				g = nullptr;
			}
}

void free_batch(dgpu_batch* c)
{
	drop_graphs(c);
	void* ptrs[] = {c->d_nc, c->d_nc_inv, c->d_ops, c->d_groups, c->d_dgroups, c->d_elf, c->d_fbase, c->d_node_face, c->gmet, c->inv_wJ,
	                c->fgeo, c->u, c->ug, c->u0, c->rhs, c->vol_gl, c->traces, c->nnf, c->max_bits, c->err_flag, c->d_bar,
	                c->n_corr, c->d_tiles, c->d_fbc, c->d_fext, c->ns_gv, c->ns_gtr, c->ns_dw, c->ns_y, c->source};
	for (void* p : ptrs)
		if (p)
			cudaFree(p);
	for (void* p : c->dense_bufs)
		if (p)
			cudaFree(p);
	if (c->own_stream && c->stream)
		cudaStreamDestroy(c->stream);
	for (int j = 0; j < kBranches; ++j) {
		if (c->aux[j])
			cudaStreamDestroy(c->aux[j]);
		if (c->ev_join[j])
			cudaEventDestroy(c->ev_join[j]);
	}
	if (c->ev_fork)
		cudaEventDestroy(c->ev_fork);
}

template <typename T>
cudaError_t upload_vec(T** dst, const std::vector<T>& src)
{
	cudaError_t e = cudaMalloc((void**)dst, std::max<size_t>(1, src.size()) * sizeof(T));
	if (e != cudaSuccess || src.empty())
		return e;
	return cudaMemcpy(*dst, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice);
}

// Form 2: the calls launch(i) run on the branch streams, forked from and joined back into the context's stream
// (under stream capture: parallel branches of the graph).
template <typename F>
dgpu_status on_branches(dgpu_batch* c, int n_items, F launch)
{
	cudaStream_t main = c->stream;
	BATCH_CUDA(c, cudaEventRecord(c->ev_fork, main));
	int j = 0;
	for (int i = 0; i < n_items; ++i) {
		cudaStream_t br = c->aux[j % kBranches];
		BATCH_CUDA(c, cudaStreamWaitEvent(br, c->ev_fork, 0));
		c->stream = br;
		const long long before = c->launches;
		cudaError_t e = launch(i);
		c->stream = main;
		BATCH_CUDA(c, e);
		if (c->launches == before)   // nothing launched (empty group or face order): no branch
			continue;
		BATCH_CUDA(c, cudaEventRecord(c->ev_join[j % kBranches], br));
		BATCH_CUDA(c, cudaStreamWaitEvent(main, c->ev_join[j % kBranches], 0));
		++j;
	}
	return DGPU_OK;
}

// One residual on the coefficients (TP: GLL), or one RK stage on the RK state (TP: GL nodal values).
dgpu_status enqueue_stage(dgpu_batch* c, bool rhs_mode, double dt, int stage, int want_max)
{
	const int lmode = rhs_mode ? kModeRhs : kModeRkGl;
	if (c->navier_stokes) {   // forms 0 and 2: gradient | jump | volume | face | lift
		dgpu_status st;
		auto phase = [&](auto launch) -> dgpu_status {
			if (c->mode == 2)
				return on_branches(c, c->n_all, launch);
			for (int g = 0; g < c->n_all; ++g)
				BATCH_CUDA(c, launch(g));
			return DGPU_OK;
		};
		if ((st = phase([&](int g) { return c->gl[g].ns_grad(c, g, rhs_mode); })) != DGPU_OK)
			return st;
		BATCH_CUDA(c, c->ns_nodes(c, false));
		if ((st = phase([&](int g) { return c->gl[g].ns_vol(c, g, rhs_mode); })) != DGPU_OK)
			return st;
		BATCH_CUDA(c, c->ns_nodes(c, true));
		return phase([&](int g) { return c->gl[g].lift(c, g, lmode, dt, stage, want_max); });
	}
	if (c->mode == 3) {
		BATCH_CUDA(c, c->stage_launch(c, rhs_mode, dt, stage, want_max));
	} else if (c->mode == 1) {
		BATCH_CUDA(c, c->fused_vol(c, rhs_mode));
		BATCH_CUDA(c, c->face_nodes(c, 0, c->qnode[kQMax + 1], c->fused_blocks_face));
		BATCH_CUDA(c, c->fused_lift(c, lmode, dt, stage, want_max));
	} else if (c->mode == 2) {
		dgpu_status st;
		if ((st = on_branches(c, c->n_all, [&](int g) { return c->gl[g].vol(c, g, rhs_mode); })) != DGPU_OK)
			return st;
		if ((st = on_branches(c, kQMax - 1, [&](int i) {
			     return c->face_nodes(c, c->qnode[i + 2], c->qnode[i + 3], 0);
		     })) != DGPU_OK)
			return st;
		if ((st = on_branches(c, c->n_all,
		                      [&](int g) { return c->gl[g].lift(c, g, lmode, dt, stage, want_max); })) != DGPU_OK)
			return st;
	} else {
		for (int g = 0; g < c->n_all; ++g)
			BATCH_CUDA(c, c->gl[g].vol(c, g, rhs_mode));
		for (int qf = 2; qf <= kQMax; ++qf)
			BATCH_CUDA(c, c->face_nodes(c, c->qnode[qf], c->qnode[qf + 1], 0));
		for (int g = 0; g < c->n_all; ++g)
			BATCH_CUDA(c, c->gl[g].lift(c, g, lmode, dt, stage, want_max));
	}
	return DGPU_OK;
}

dgpu_status ensure_coef(dgpu_batch* c)
{
	if (!c->coef_valid) {
		for (int g = 0; g < c->n_all; ++g)
			BATCH_CUDA(c, c->gl[g].conv(c, g, false));
		c->coef_valid = true;
	}
	return DGPU_OK;
}

dgpu_status ensure_gl(dgpu_batch* c)
{
	if (!c->gl_valid) {
		for (int g = 0; g < c->n_all; ++g)
			BATCH_CUDA(c, c->gl[g].conv(c, g, true));
		c->gl_valid = true;
	}
	return DGPU_OK;
}

dgpu_status read_max(dgpu_batch* c, double* max_rhs)
{
	if (!max_rhs)
		return DGPU_OK;
	unsigned long long bits = 0;
	BATCH_CUDA(c, cudaMemcpyAsync(&bits, c->max_bits, sizeof bits, cudaMemcpyDeviceToHost, c->stream));
	BATCH_CUDA(c, cudaStreamSynchronize(c->stream));
	memcpy(max_rhs, &bits, sizeof(double));
	return DGPU_OK;
}

dgpu_status upload_group_tiles(dgpu_batch* c)
{
	if (!c->hgroups.empty())
		BATCH_CUDA(c, cudaMemcpyAsync(c->d_groups, c->hgroups.data(), c->hgroups.size() * sizeof(BGroup),
		                              cudaMemcpyHostToDevice, c->stream));
	if (!c->hdgroups.empty())
		BATCH_CUDA(c, cudaMemcpyAsync(c->d_dgroups, c->hdgroups.data(), c->hdgroups.size() * sizeof(DGroup),
		                              cudaMemcpyHostToDevice, c->stream));
	BATCH_CUDA(c, cudaStreamSynchronize(c->stream));
	return DGPU_OK;
}

void set_group_E(dgpu_batch* c, int g, int E)
{
	if (c->gl[g].dense)
		c->hdgroups[c->gl[g].idx].E = E;
	else
		c->hgroups[c->gl[g].idx].E = E;
}

// Elements per CTA of the per-group kernels. A large group fills its CTAs (256 nodes); a group too small to give every
// one of the device's SMs two of those is split further, down to a warp of a QUAD/HEX group or one dense volume: its kernels are chains
// of dependent steps, so idle SMs cost more than half-empty CTAs.
void default_tiles(dgpu_batch* c)
{
	int dev = 0, sms = 0;
	cudaGetDevice(&dev);
	cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	for (int g = 0; g < c->n_all; ++g) {
		const int n_vol = c->group_n_vol(g);
		int E = c->gl[g].E_max, N = 32;
		if (!c->gl[g].dense) {
			const int q = c->hgroups[c->gl[g].idx].q;
			N = c->d == 2 ? q * q : q * q * q;
		}
		while (E > 1 && n_vol < E * 2 * sms && (E / 2) * N >= 32)
			E /= 2;
		set_group_E(c, g, E);
	}
}

int type_faces(int t)
{
	return t == DGPU_TRI ? 3 : (t == DGPU_TET ? 4 : (t == DGPU_HEX ? 6 : (t == DGPU_QUAD ? 4 : 5)));
}

// ---- creation ----
struct GroupIn {
	bool dense;
	const dgpu_tp_operators* tp;
	const dgpu_dense_operators* dn;
};

template <typename T>
cudaError_t upload_vec(T** dst, const std::vector<T>& src);

// Uploads an operator in fixed point, entry (i, j) of `rows` x `cols` row-major from w, transposed or not.
cudaError_t upload_fix(dgpu_batch* c, const double* w, int rows, int cols, bool transposed, int s, const FixW** out)
{
	std::vector<FixW> x((size_t)rows * cols);
	for (int i = 0; i < rows; ++i)
		for (int j = 0; j < cols; ++j)
			x[transposed ? (size_t)j * rows + i : (size_t)i * cols + j] = fix_entry(w[(size_t)i * cols + j], s);
	FixW* d = nullptr;
	const cudaError_t e = upload_vec(&d, x);
	if (e == cudaSuccess) {
		c->dense_bufs.push_back(d);
		*out = d;
	}
	return e;
}

// Largest row sum of |w| (column sum when by_col), and largest entry.
double abs_sum(const double* w, int rows, int cols, bool by_col, double* mx)
{
	std::vector<double> s(by_col ? cols : rows, 0.0);
	for (int i = 0; i < rows; ++i)
		for (int j = 0; j < cols; ++j) {
			const double a = fabs(w[(size_t)i * cols + j]);
			s[by_col ? j : i] += a;
			*mx = std::max(*mx, a);
		}
	return *std::max_element(s.begin(), s.end());
}

// Scale of an operator of fix_dot: |W| < 2^61 and sum |W| <= 2^66.
int dense_shift(double sum, double mx) { return fix_shift(sum, 2.0 * mx, 66); }

// The fixed-point operators of a dense group (dgpu_fix.cuh), each at the largest scale its sums allow; none if one of them
// has no such form.
cudaError_t upload_fix_ops(dgpu_batch* c, const dgpu_dense_operators* op, int d, const std::vector<double>& Minv,
                           const std::vector<double>& fops, const std::vector<long long>& foff, DGroup* G)
{
	const int nvs = op->n_vs, nvc = op->n_vc;
	const size_t nl = (size_t)G->n_lvc * G->n_lvs, nt = (size_t)G->n_tvc * G->n_tvs;
	G->fix = fix_usable(op->cv0_vs_vc, (size_t)nvc * nvs) && fix_usable(op->cv1_vs_vc, (size_t)d * nvc * nvs) &&
	         fix_usable(Minv.data(), Minv.size()) && fix_usable(fops.data(), fops.size()) &&
	         fix_even_basis(op->cv0_vs_vc, nvc, nvs, nvs);
	if (G->prism)
		G->fix = G->fix && fix_usable(op->tri_cv0, nt) && fix_usable(op->tri_cv1, 2 * nt) &&
		         fix_usable(op->line_cv0, nl) && fix_usable(op->line_cv1, nl);
	if (!G->fix)
		return cudaSuccess;
	cudaError_t e;
	double m = 0.0;
	G->s_cv0 = dense_shift(abs_sum(op->cv0_vs_vc, nvc, nvs, false, &m), m);
	if ((e = upload_fix(c, op->cv0_vs_vc, nvc, nvs, true, G->s_cv0, &G->xcv0)))
		return e;
	m = 0.0;
	G->s_cv1 = dense_shift(abs_sum(op->cv1_vs_vc, d * nvc, nvs, true, &m), m);
	if ((e = upload_fix(c, op->cv1_vs_vc, d * nvc, nvs, false, G->s_cv1, &G->xcv1)))
		return e;
	m = 0.0;
	G->s_minv = dense_shift(abs_sum(Minv.data(), nvs, nvs, false, &m), m);
	if ((e = upload_fix(c, Minv.data(), nvs, nvs, true, G->s_minv, &G->xminv)))
		return e;
	// face operators: one scale for the traces (rows) and the lifting (columns, every face's largest)
	double mf = 0.0, trace = 0.0, lift = 0.0;
	for (int lf = 0; lf < op->n_lf; ++lf) {
		double col = 0.0;
		for (int o = 0; o < op->n_ord; ++o)
			for (int pf = 1; pf < kQMax; ++pf) {
				const int k = (lf * op->n_ord + o) * kQMax + pf;
				if (!op->cv0_vs_fc[k] || op->n_fc[k] < 1)
					continue;
				trace = std::max(trace, abs_sum(op->cv0_vs_fc[k], op->n_fc[k], nvs, false, &mf));
				col = std::max(col, abs_sum(op->cv0_vs_fc[k], op->n_fc[k], nvs, true, &mf));
			}
		lift += col;
	}
	G->s_f = dense_shift(std::max(trace, lift), mf);
	std::vector<FixW> xT(fops.size()), xL(fops.size());
	for (int lf = 0; lf < op->n_lf; ++lf)
		for (int o = 0; o < op->n_ord; ++o)
			for (int pf = 1; pf < kQMax; ++pf) {
				const long long off = foff[(lf * op->n_ord + o) * (kQMax + 1) + pf + 1];
				const int n = op->n_fc[(lf * op->n_ord + o) * kQMax + pf];
				if (off < 0)
					continue;
				for (int i = 0; i < n; ++i)
					for (int a = 0; a < nvs; ++a) {
						const FixW w = fix_entry(fops[off + (size_t)i * nvs + a], G->s_f);
						xL[off + (size_t)i * nvs + a] = w;
						xT[off + (size_t)a * n + i] = w;
					}
			}
	FixW *dT = nullptr, *dL = nullptr;
	if ((e = upload_vec(&dT, xT)))
		return e;
	c->dense_bufs.push_back(dT);
	if ((e = upload_vec(&dL, xL)))
		return e;
	c->dense_bufs.push_back(dL);
	G->xfT = dT;
	G->xfL = dL;
	if (!G->prism)
		return cudaSuccess;
	const int ntc = G->n_tvc, ntv = G->n_tvs, nlc = G->n_lvc, nlv = G->n_lvs;
	double mt = 0.0, ml = 0.0, mt1 = 0.0, ml1 = 0.0;
	const double t0 = std::max(abs_sum(op->tri_cv0, ntc, ntv, false, &mt), abs_sum(op->tri_cv0, ntc, ntv, true, &mt));
	const double l0 = std::max(abs_sum(op->line_cv0, nlc, nlv, false, &ml), abs_sum(op->line_cv0, nlc, nlv, true, &ml));
	G->s_t0 = fix_shift(t0, mt, 62);
	G->s_l0 = fix_shift(l0, ml, 62);
	// the last sum takes tri1 products of the x and y parts at s_t1 and line1 products of the z part at s_t1 + s_l0 - s_t0
	const double r = ldexp(1.0, G->s_l0 - G->s_t0);
	const double t1 = abs_sum(op->tri_cv1, 2 * ntc, ntv, true, &mt1), l1 = abs_sum(op->line_cv1, nlc, nlv, true, &ml1);
	G->s_t1 = dense_shift(t1 + r * l1, std::max(mt1, r * ml1));
	if ((e = upload_fix(c, op->tri_cv0, ntc, ntv, false, G->s_t0, &G->xt0)) ||
	    (e = upload_fix(c, op->tri_cv0, ntc, ntv, true, G->s_t0, &G->xt0T)) ||
	    (e = upload_fix(c, op->tri_cv1, 2 * ntc, ntv, false, G->s_t1, &G->xt1)) ||
	    (e = upload_fix(c, op->line_cv0, nlc, nlv, false, G->s_l0, &G->xl0)))
		return e;
	return upload_fix(c, op->line_cv1, nlc, nlv, false, G->s_t1 + G->s_l0 - G->s_t0, &G->xl1);
}

dgpu_status create_impl(const dgpu_physics* phys, const std::vector<GroupIn>& gin, const int* vol_group,
                        const dgpu_mesh* mesh, const int* face_ord, dgpu_batch** out)
{
	g_batch_error.clear();
	if (!phys || gin.empty() || !vol_group || !mesh || !out)
		return bfail(nullptr, DGPU_ERR_INVALID_ARGUMENT, "NULL argument");
	*out = nullptr;
	const int d = phys->d;
	if (d != 2 && d != 3)
		return bfail(nullptr, DGPU_ERR_UNSUPPORTED, "d must be 2 or 3");
	const bool ns_pde = phys->pde == DGPU_PDE_NAVIER_STOKES;
	if (phys->pde == DGPU_PDE_ADVECTION ? phys->num_flux != DGPU_NUM_FLUX_UPWIND
	                                    : ((phys->pde != DGPU_PDE_EULER && !ns_pde) ||
	                                       (phys->num_flux != DGPU_NUM_FLUX_ROE_PIKE &&
	                                        phys->num_flux != DGPU_NUM_FLUX_LAX_FRIEDRICHS)))
		return bfail(nullptr, DGPU_ERR_UNSUPPORTED,
		             "advection/upwind or Euler, Navier-Stokes/Roe-Pike, Lax-Friedrichs only");
	if (ns_pde && ((phys->viscosity != DGPU_VISCOSITY_CONSTANT && phys->viscosity != DGPU_VISCOSITY_SUTHERLAND) ||
	               !(phys->mu >= 0.0) || !(phys->Pr > 0.0) ||
	               (phys->viscosity == DGPU_VISCOSITY_SUTHERLAND && !(phys->r_s > 0.0))))
		return bfail(nullptr, DGPU_ERR_INVALID_ARGUMENT,
		             "Navier-Stokes needs a viscosity model, mu >= 0, Pr > 0 (and r_s > 0 for Sutherland's law)");
	if (ns_pde && phys->dTdn != 0.0 && phys->viscosity != DGPU_VISCOSITY_CONSTANT)
		return bfail(nullptr, DGPU_ERR_UNSUPPORTED, "a diabatic wall flux (dTdn != 0) needs constant viscosity");
	if (mesh->n_volumes < 1 || mesh->n_faces < 1 || !mesh->metrics_vc || !mesh->jacobian_det_vc ||
	    !mesh->face_vol || !mesh->face_lf || !mesh->normals_fc || !mesh->jacobian_det_fc)
		return bfail(nullptr, DGPU_ERR_INVALID_ARGUMENT, "incomplete mesh");
	int dev = 0, n_dev = 0;
	if (cudaGetDeviceCount(&n_dev) != cudaSuccess || n_dev < 1)
		return bfail(nullptr, DGPU_ERR_NO_DEVICE, "no CUDA device");
	cudaGetDevice(&dev);
	cudaDeviceProp prop;
	if (cudaGetDeviceProperties(&prop, dev) != cudaSuccess || prop.major * 10 + prop.minor != 103)
		return bfail(nullptr, DGPU_ERR_NO_DEVICE, "device is not compute capability 10.3 (sm_103a build)");

	dgpu_batch* c = new dgpu_batch();
	c->d = d;
	c->pde = phys->pde;
	c->flux = phys->num_flux;
	c->nv = (phys->pde != DGPU_PDE_ADVECTION ? d + 2 : 1);
	c->positivity = (phys->pde != DGPU_PDE_ADVECTION && phys->positivity) ? 1 : 0;
	c->navier_stokes = ns_pde;
	if (ns_pde)
		c->ns_phys = NsPhys{phys->mu, phys->Pr, phys->r_s, phys->viscosity,
		                    -phys->mu * (kGamma / kGm1 * phys->r_s) / phys->Pr * phys->dTdn};
	for (int k = 0; k < 3; ++k)
		c->b_adv[k] = phys->b_adv[k];
	c->n_vol = mesh->n_volumes;
	c->n_face = mesh->n_faces;
	const int nv = c->nv, nV = c->n_vol, nF = c->n_face, nG = (int)gin.size();
	auto reject = [&](dgpu_status st, std::string m) {   // by value: m may be the context's own message
		free_batch(c);
		delete c;
		return bfail(nullptr, st, m);
	};

	// ---- groups: TP first (caller order), then dense (caller order) ----
	c->caller_to_internal.assign(nG, -1);
	std::vector<int> internal_to_caller;
	for (int pass = 0; pass < 2; ++pass)
		for (int g = 0; g < nG; ++g)
			if (gin[g].dense == (pass == 1)) {
				GroupLaunch L;
				L.dense = gin[g].dense;
				L.idx = L.dense ? c->n_dense++ : c->n_tp++;
				c->caller_to_internal[g] = (int)c->gl.size();
				internal_to_caller.push_back(g);
				c->gl.push_back(L);
			}
	c->n_all = nG;
	c->hgroups.resize(c->n_tp);
	c->hops.resize(c->n_tp);
	c->hdgroups.resize(c->n_dense);
	if (c->navier_stokes && c->n_dense > 0)
		return reject(DGPU_ERR_UNSUPPORTED, "Navier-Stokes in the batched context takes QUAD/HEX groups only");
	std::vector<int> g_q(nG), g_nvs(nG), g_nvc(nG), g_type(nG);   // per internal group
	std::vector<std::vector<double>> w(nG);                         // volume cubature weights per node
	std::vector<const dgpu_dense_operators*> dops(c->n_dense);
	for (int ig = 0; ig < nG; ++ig) {
		const GroupIn& in = gin[internal_to_caller[ig]];
		if (!in.dense) {
			if (!in.tp)
				return reject(DGPU_ERR_INVALID_ARGUMENT, "NULL operator set");
			const dgpu_tp_operators& o = *in.tp;
			if ((d == 2 && o.elem_type != DGPU_QUAD) || (d == 3 && o.elem_type != DGPU_HEX) || o.p < 1 ||
			    o.p > kQMax - 1)
				return reject(DGPU_ERR_UNSUPPORTED, "TP groups must be QUAD (d=2) or HEX (d=3) with p in 1..4");
			if (!o.cv0_vs_vc || !o.cv1_vs_vc || !o.cv0_vs_fc || !o.w_vc)
				return reject(DGPU_ERR_INVALID_ARGUMENT, "NULL operator");
			if (c->positivity && (!o.ccSB0_vs_vs || !o.ccBS0_vs_vs))
				return reject(DGPU_ERR_INVALID_ARGUMENT, "positivity needs ccSB0/ccBS0");
			const int q = o.p + 1, t = c->gl[ig].idx;
			for (int h = 0; h < ig; ++h)
				if (!c->gl[h].dense && g_q[h] == q)
					return reject(DGPU_ERR_INVALID_ARGUMENT, "two TP groups with the same p");
			memset(&c->hops[t], 0, sizeof(BatchOps));
			if (!derive_tp_ops(&o, d, &c->hops[t].t))
				return reject(DGPU_ERR_INVALID_ARGUMENT, "cv0_vs_vc is singular");
			// GL(q) Lagrange at GL(qf) nodes for every face order qf >= q
			double xq[kQMax], xf[kQMax];
			gauss_legendre_nodes(q, xq);
			for (int qf = q; qf <= kQMax; ++qf) {
				gauss_legendre_nodes(qf, xf);
				for (int i = 0; i < qf; ++i)
					for (int a = 0; a < q; ++a)
						c->hops[t].Iup[qf][i][a] = lagrange_value(xq, q, a, xf[i]);
				// rows (interpolation) and columns (its transpose) of one scale
				double sum = 0.0, mx = 0.0;
				for (int i = 0; i < qf; ++i) {
					double r = 0.0;
					for (int a = 0; a < q; ++a) {
						r += fabs(c->hops[t].Iup[qf][i][a]);
						mx = std::max(mx, fabs(c->hops[t].Iup[qf][i][a]));
					}
					sum = std::max(sum, r);
				}
				for (int a = 0; a < q; ++a) {
					double r = 0.0;
					for (int i = 0; i < qf; ++i)
						r += fabs(c->hops[t].Iup[qf][i][a]);
					sum = std::max(sum, r);
				}
				c->hops[t].sI[qf] = fix_shift(sum, mx, 62);
				for (int i = 0; i < qf; ++i)
					for (int a = 0; a < q; ++a)
						c->hops[t].fI[qf][i][a] = fix_entry(c->hops[t].Iup[qf][i][a], c->hops[t].sI[qf]);
			}
			c->hgroups[t].q = q;
			const int N = (d == 2 ? q * q : q * q * q);
			g_q[ig] = q;
			g_nvs[ig] = g_nvc[ig] = N;
			g_type[ig] = o.elem_type;
			w[ig].resize(N);
			for (int n = 0; n < N; ++n) {
				int r = n;
				double x = 1.0;
				for (int k = 0; k < d; ++k) {
					x *= o.w_vc[r % q];
					r /= q;
				}
				w[ig][n] = x;
			}
		} else {
			const dgpu_dense_operators* op = in.dn;
			if (!op)
				return reject(DGPU_ERR_INVALID_ARGUMENT, "NULL operator set");
			if (d == 2 ? op->elem_type != DGPU_TRI
			           : (op->elem_type != DGPU_TET && op->elem_type != DGPU_WEDGE && op->elem_type != DGPU_PYR))
				return reject(DGPU_ERR_UNSUPPORTED, "dense groups must be TRI (d = 2) or TET, WEDGE, PYR (d = 3)");
			if (op->p < 1 || op->p > kQMax - 1 || op->n_vs < 1 || op->n_vc < 1 || op->n_vs > 1024 ||
			    op->n_vc > 4096 || op->n_lf != type_faces(op->elem_type) || op->n_ord < 1 || op->n_ord > kMaxOrd ||
			    !op->cv0_vs_vc || !op->cv1_vs_vc || !op->w_vc || !op->n_fc || !op->cv0_vs_fc || !op->w_fc)
				return reject(DGPU_ERR_INVALID_ARGUMENT, "incomplete dense operator set");
			if (c->positivity && (!op->ccSB0_vs_vs || !op->ccBS0_vs_vs))
				return reject(DGPU_ERR_INVALID_ARGUMENT, "positivity needs the Bezier maps of every dense group");
			const int t = c->gl[ig].idx;
			dops[t] = op;
			g_q[ig] = op->p + 1;
			g_nvs[ig] = op->n_vs;
			g_nvc[ig] = op->n_vc;
			g_type[ig] = op->elem_type;
			w[ig].assign(op->w_vc, op->w_vc + op->n_vc);
			DGroup& G = c->hdgroups[t];
			memset(&G, 0, sizeof G);
			G.n_vs = op->n_vs;
			G.n_vc = op->n_vc;
			G.n_lf = op->n_lf;
			G.n_ord = op->n_ord;
			G.vol_per_e = DSmem::vol(nv, G.n_vs, G.n_vc);
			G.nff_max = 1;
			for (int k = 0; k < op->n_lf * op->n_ord * kQMax; ++k)
				if (op->cv0_vs_fc[k])
					G.nff_max = std::max(G.nff_max, op->n_fc[k]);
			G.lift_per_e = DSmem::lift(nv, G.n_vs, G.n_lf, G.nff_max);
			if (op->elem_type == DGPU_WEDGE && op->tri_cv0 && op->tri_cv1 && op->line_cv0 && op->line_cv1) {
				const int ntv = op->n_tri_vs, ntc = op->n_tri_vc, nlv = op->n_line_vs, nlc = op->n_line_vc;
				if (ntv < 1 || ntc < 1 || nlv < 1 || nlc < 1 || ntv * nlv != op->n_vs || ntc * nlc != op->n_vc)
					return reject(DGPU_ERR_INVALID_ARGUMENT, "WEDGE factor sizes do not match n_vs / n_vc");
				// the factors must reproduce the dense operators
				double scale = 0.0, diff = 0.0;
				for (int rz = 0; rz < nlc; ++rz)
					for (int rt = 0; rt < ntc; ++rt)
						for (int c0 = 0; c0 < nlv; ++c0)
							for (int t = 0; t < ntv; ++t) {
								const size_t rr = (size_t)rz * ntc + rt, cc = (size_t)c0 * ntv + t;
								const size_t ti = (size_t)rt * ntv + t, li = (size_t)rz * nlv + c0;
								const double ref[4] = {op->cv0_vs_vc[rr * op->n_vs + cc],
								                       op->cv1_vs_vc[(0 * (size_t)op->n_vc + rr) * op->n_vs + cc],
								                       op->cv1_vs_vc[(1 * (size_t)op->n_vc + rr) * op->n_vs + cc],
								                       op->cv1_vs_vc[(2 * (size_t)op->n_vc + rr) * op->n_vs + cc]};
								const double fac[4] = {op->line_cv0[li] * op->tri_cv0[ti],
								                       op->line_cv0[li] * op->tri_cv1[ti],
								                       op->line_cv0[li] * op->tri_cv1[(size_t)ntc * ntv + ti],
								                       op->line_cv1[li] * op->tri_cv0[ti]};
								for (int k = 0; k < 4; ++k) {
									scale = std::max(scale, fabs(ref[k]));
									diff = std::max(diff, fabs(ref[k] - fac[k]));
								}
							}
				if (!(diff <= 1e-12 * scale))
					return reject(DGPU_ERR_INVALID_ARGUMENT, "the WEDGE factors do not reproduce the dense operators");
				// longer factors (no cubature in use has them) run as dense operators
				G.prism = std::max(std::max(ntv, ntc), std::max(nlv, nlc)) <= 32 ? 1 : 0;
				G.n_tvs = ntv;
				G.n_tvc = ntc;
				G.n_lvs = nlv;
				G.n_lvc = nlc;
				if (G.prism)
					G.vol_per_e += DSmem::prism_tmp(nv, ntv, ntc, nlv, nlc);
			}
			G.E = std::max(1, 256 / op->n_vc);
			while (G.E > 1 && (size_t)G.E * std::max(G.vol_per_e, G.lift_per_e) * 8 > 96 * 1024)
				G.E /= 2;
			G.E_fused = G.E;
			// (without the block exponents; a lift beyond its bound would take faces of a thousand nodes)
			if ((size_t)(G.vol_per_e - nv - 1) * 8 > 200 * 1024 || (size_t)G.lift_per_e * 8 > 216 * 1024)
				return reject(DGPU_ERR_UNSUPPORTED, "dense operator set too large for one volume per CTA");
		}
	}
	// ---- volumes: group-sorted order, offsets ----
	std::vector<int> count(nG, 0), vg(nV);
	for (int v = 0; v < nV; ++v) {
		if (vol_group[v] < 0 || vol_group[v] >= nG)
			return reject(DGPU_ERR_INVALID_ARGUMENT, "vol_group out of range");
		vg[v] = c->caller_to_internal[vol_group[v]];
		count[vg[v]]++;
	}
	c->list_off.resize(nV + 1);
	std::vector<long long>& list_vc_off = c->list_vc_off;
	list_vc_off.resize(nV + 1);
	long long so = 0, vco = 0;
	for (int v = 0; v < nV; ++v) {
		c->list_off[v] = so;
		list_vc_off[v] = vco;
		so += (long long)nv * g_nvs[vg[v]];
		vco += g_nvc[vg[v]];
	}
	c->list_off[nV] = so;
	list_vc_off[nV] = vco;
	c->ns = (size_t)so;
	c->order.resize(nV);
	std::vector<int> sorted_pos(nV);
	std::vector<long long> g_elem0(nG), g_state(nG), g_gmet(nG), g_wj(nG);
	{
		long long elem = 0, st_off = 0, gm_off = 0, wj_off = 0;
		std::vector<int> next(nG);
		for (int g = 0; g < nG; ++g) {   // internal order
			g_elem0[g] = elem;
			g_state[g] = st_off;
			g_gmet[g] = gm_off;
			g_wj[g] = wj_off;
			next[g] = (int)elem;
			elem += count[g];
			st_off += (long long)count[g] * nv * g_nvs[g];
			gm_off += (long long)count[g] * d * d * g_nvc[g];
			if (!c->gl[g].dense)
				wj_off += (long long)count[g] * g_nvc[g];
		}
		for (int v = 0; v < nV; ++v) {
			const int p = next[vg[v]]++;
			c->order[p] = v;
			sorted_pos[v] = p;
		}
	}
	for (int g = 0; g < nG; ++g) {
		if (c->gl[g].dense) {
			DGroup& G = c->hdgroups[c->gl[g].idx];
			G.n_vol = count[g];
			G.elem0 = g_elem0[g];
			G.state_off = g_state[g];
			G.gmet_off = g_gmet[g];
		} else {
			BGroup& G = c->hgroups[c->gl[g].idx];
			G.n_vol = count[g];
			G.elem0 = g_elem0[g];
			G.state_off = g_state[g];
			G.gmet_off = g_gmet[g];
			G.wj_off = g_wj[g];
			G.E = std::max(1, 256 / g_nvs[g]);
		}
	}
	c->sorted_off.resize(nV);
	std::vector<double> gmet, inv_wJ;
	std::vector<std::vector<double>> inv_J(c->n_dense);
	// curved (non-affine) dense volumes: their group keeps a per-volume M^-1, formed from w J at every node
	std::vector<char> dense_curved(c->n_dense, 0);
	std::vector<std::vector<double>> dense_wJ(c->n_dense);
	for (int g = 0; g < nG; ++g) {
		const int N = g_nvc[g];
		for (int e = 0; e < count[g]; ++e) {
			const int p = (int)g_elem0[g] + e, v = c->order[p];
			c->sorted_off[p] = g_state[g] + (long long)e * nv * g_nvs[g];
			const double* m = mesh->metrics_vc + list_vc_off[v] * d * d;
			const double* J = mesh->jacobian_det_vc + list_vc_off[v];
			for (int j = 0; j < d; ++j)
				for (int i = 0; i < d; ++i)
					for (int n = 0; n < N; ++n)
						gmet.push_back(w[g][n] * m[n + (size_t)N * (i + d * j)]);
			for (int n = 0; n < N; ++n)
				if (!(J[n] > 0.0))
					return reject(DGPU_ERR_INVALID_ARGUMENT, "non-positive jacobian_det_vc");
			if (c->gl[g].dense) {
				const int t = c->gl[g].idx;
				for (int n = 1; n < N; ++n)
					if (fabs(J[n] - J[0]) > 1e-12 * J[0])
						dense_curved[t] = 1;
				inv_J[t].push_back(1.0 / J[0]);
				for (int n = 0; n < N; ++n)
					dense_wJ[t].push_back(w[g][n] * J[n]);
			} else {
				for (int n = 0; n < N; ++n)
					inv_wJ.push_back(1.0 / (w[g][n] * J[n]));
			}
		}
	}
	// ---- faces: order p_f = max of the sides; internal face ids by increasing q_f ----
	std::vector<int> face_q(nF), face_nfc(nF);
	int n_bnd = 0;
	for (int f = 0; f < nF; ++f) {
		int qf = 0;
		const int ns_f = (mesh->face_vol[2 * f + 1] < 0) ? 1 : 2;   // a boundary face has side 0 only
		if (ns_f == 1) {
			if (!mesh->bc_fc || !mesh->bc_state_fc)
				return reject(DGPU_ERR_INVALID_ARGUMENT, "boundary faces need bc_fc and bc_state_fc");
			const int code = mesh->bc_fc[f] % kBcStepSC;
			if (code < 0 || (c->navier_stokes ? !bc_is_navier_stokes(code)
			                       : (c->pde == DGPU_PDE_EULER ? !bc_is_euler(code) : !bc_is_advection_upwind(code))))
				return reject(DGPU_ERR_UNSUPPORTED,
				              "BC code " + std::to_string(mesh->bc_fc[f]) + " is not provided for this pde");
			if ((code == kBcBackPressure || code == kBcTotalTP) && !mesh->bc_data)
				return reject(DGPU_ERR_INVALID_ARGUMENT, "back pressure / total TP faces need bc_data");
			++n_bnd;
		}
		for (int s = 0; s < ns_f; ++s) {
			const int v = mesh->face_vol[2 * f + s], lf = mesh->face_lf[2 * f + s];
			if (v < 0 || v >= nV || lf < 0 || lf >= type_faces(g_type[vg[v]]))
				return reject(DGPU_ERR_INVALID_ARGUMENT, "bad face connectivity");
			qf = std::max(qf, g_q[vg[v]]);
		}
		face_q[f] = qf;
		int nfc = -1;
		for (int s = 0; s < ns_f; ++s) {
			const int v = mesh->face_vol[2 * f + s], lf = mesh->face_lf[2 * f + s], g = vg[v];
			const int ord = face_ord ? face_ord[2 * f + s] : 0;
			int n_s;
			if (c->gl[g].dense) {
				const dgpu_dense_operators* op = dops[c->gl[g].idx];
				if (ord < 0 || ord >= op->n_ord)
					return reject(DGPU_ERR_INVALID_ARGUMENT, "face_ord out of range");
				const int k = (lf * op->n_ord + ord) * kQMax + (qf - 1);
				if (!op->cv0_vs_fc[k] || op->n_fc[k] < 1)
					return reject(DGPU_ERR_INVALID_ARGUMENT, "missing dense face operator");
				n_s = op->n_fc[k];
			} else {
				if (ord != 0)
					return reject(DGPU_ERR_UNSUPPORTED, "QUAD/HEX volumes must see their faces unpermuted (face_ord 0)");
				n_s = (d == 2 ? qf : qf * qf);
			}
			if (nfc >= 0 && n_s != nfc)
				return reject(DGPU_ERR_INVALID_ARGUMENT, "the two sides of a face have different face node counts");
			nfc = n_s;
		}
		face_nfc[f] = nfc;
	}
	std::vector<long long> caller_fc_off(nF + 1);   // the caller's face-node offsets (face-list order)
	caller_fc_off[0] = 0;
	for (int f = 0; f < nF; ++f)
		caller_fc_off[f + 1] = caller_fc_off[f] + face_nfc[f];
	std::vector<int> by_q(nF);                      // internal face id -> caller face
	for (int f = 0; f < nF; ++f)
		by_q[f] = f;
	std::stable_sort(by_q.begin(), by_q.end(), [&](int a, int b) { return face_q[a] < face_q[b]; });
	std::vector<int> internal_face(nF);
	std::vector<long long> fbase(nF + 1);
	std::vector<int> node_face;
	long long fb = 0;
	int cur_q = 0;
	for (int k = 0; k < nF; ++k) {
		const int f = by_q[k];
		internal_face[f] = k;
		while (cur_q < face_q[f])
			c->qnode[++cur_q] = fb;
		fbase[k] = fb;
		for (int i = 0; i < face_nfc[f]; ++i)
			node_face.push_back(k);
		fb += face_nfc[f];
	}
	while (cur_q <= kQMax)
		c->qnode[++cur_q] = fb;
	fbase[nF] = fb;
	std::vector<int4> elf((size_t)nV * kMaxLf, int4{-1, -1, -1, 0});
	// the right-trace gather permutation of every interior face (get_operator__nc_fc_T(1, face),
	// compute_face_rlhs_T.c:133-146) in the internal face-node layout, and its inverse for side 1's lift; both stay
	// off the device when every face's is the identity
	std::vector<int> nc_int, nc_inv_int;
	bool nc_identity = true;
	if (mesh->nc_fc) {
		nc_int.resize(fb);
		nc_inv_int.resize(fb);
		for (int f = 0; f < nF; ++f) {
			const long long b0 = fbase[internal_face[f]];
			const int nff = face_nfc[f];
			const bool interior = mesh->face_vol[2 * f + 1] >= 0;
			for (int i = 0; i < nff; ++i)
				nc_inv_int[b0 + i] = -1;
			for (int i = 0; i < nff; ++i) {
				const int j = interior ? mesh->nc_fc[caller_fc_off[f] + i] : i;
				if (j < 0 || j >= nff || nc_inv_int[b0 + j] != -1)
					return reject(DGPU_ERR_INVALID_ARGUMENT, "nc_fc of face " + std::to_string(f) +
					                                         " is not a permutation of its face nodes");
				nc_int[b0 + i] = j;
				nc_inv_int[b0 + j] = i;
				nc_identity = nc_identity && j == i;
			}
		}
	}
	for (int f = 0; f < nF; ++f) {
		const int ns_f = (mesh->face_vol[2 * f + 1] < 0) ? 1 : 2;
		for (int s = 0; s < ns_f; ++s) {
			const int v = mesh->face_vol[2 * f + s], lf = mesh->face_lf[2 * f + s];
			int4& slot = elf[(size_t)sorted_pos[v] * kMaxLf + lf];
			if (slot.x != -1)
				return reject(DGPU_ERR_INVALID_ARGUMENT, "a volume face appears twice in the face list");
			slot = int4{internal_face[f], s, face_q[f], face_ord ? face_ord[2 * f + s] : 0};
		}
	}
	for (int p = 0; p < nV; ++p)
		for (int lf = 0; lf < type_faces(g_type[vg[c->order[p]]]); ++lf)
			if (elf[(size_t)p * kMaxLf + lf].x < 0)
				return reject(DGPU_ERR_INVALID_ARGUMENT, "a volume face is missing from the face list");
	// face weights at the canonical nodes: the side-0 volume's face rule (TP: GL, the caller's weights when a TP
	// group of that order exists)
	double wq[kQMax + 1][kQMax] = {{0}};
	bool have_q[kQMax + 1] = {false};
	for (int g = 0; g < nG; ++g)
		if (!c->gl[g].dense) {
			const dgpu_tp_operators* o = gin[internal_to_caller[g]].tp;
			for (int a = 0; a < g_q[g]; ++a)
				wq[g_q[g]][a] = o->w_vc[a];
			have_q[g_q[g]] = true;
		}
	for (int q = 1; q <= kQMax; ++q)
		if (!have_q[q]) {   // GL weights 2 / ((1 - x^2) P_q'(x)^2)
			double x[kQMax];
			gauss_legendre_nodes(q, x);
			for (int a = 0; a < q; ++a) {
				double pp, dp;
				legendre(q, x[a], &pp, &dp);
				wq[q][a] = 2.0 / ((1.0 - x[a] * x[a]) * dp * dp);
			}
		}
	std::vector<double> fgeo((size_t)(d + 1) * fb);
	for (int f = 0; f < nF; ++f) {
		const int qf = face_q[f], nff = face_nfc[f];
		const long long base = (d + 1) * fbase[internal_face[f]];
		const int v0 = mesh->face_vol[2 * f], lf0 = mesh->face_lf[2 * f], g0 = vg[v0];
		const double* wf_dense = nullptr;
		if (c->gl[g0].dense) {
			wf_dense = dops[c->gl[g0].idx]->w_fc[lf0 * kQMax + (qf - 1)];
			if (!wf_dense)
				return reject(DGPU_ERR_INVALID_ARGUMENT, "missing dense face weights");
		}
		for (int i = 0; i < nff; ++i) {
			const double wf = wf_dense ? wf_dense[i] : (d == 2 ? wq[qf][i] : wq[qf][i % qf] * wq[qf][i / qf]);
			for (int k = 0; k < d; ++k)
				fgeo[base + (size_t)k * nff + i] = mesh->normals_fc[(caller_fc_off[f] + i) * d + k];
			fgeo[base + (size_t)d * nff + i] = wf * mesh->jacobian_det_fc[caller_fc_off[f] + i];
		}
	}
	// boundary faces: code per internal face and the exterior state in the internal face-node layout
	std::vector<int> fbc;
	std::vector<double> fext;
	if (n_bnd > 0) {
		fbc.assign(nF, -1);
		fext.assign((size_t)nv * fb, 0.0);
		for (int f = 0; f < nF; ++f) {
			if (mesh->face_vol[2 * f + 1] >= 0)
				continue;
			const int k = internal_face[f], nff = face_nfc[f];
			fbc[k] = mesh->bc_fc[f] % kBcStepSC;
			for (int i = 0; i < nff; ++i)
				for (int var = 0; var < nv; ++var)
					fext[(size_t)nv * fbase[k] + (size_t)var * nff + i] =
						mesh->bc_state_fc[(caller_fc_off[f] + i) * nv + var];
		}
		if (mesh->bc_data)
			c->bc_data = BcData{mesh->bc_data[0], mesh->bc_data[1], mesh->bc_data[2], mesh->bc_data[3]};
	}
	// fused tiles: full CTAs per group (TP: 256 / q^d volumes; dense: E_fused)
	std::vector<BTile> tiles;
	for (int g = 0; g < nG; ++g) {
		const bool dn = c->gl[g].dense;
		const int E = dn ? c->hdgroups[c->gl[g].idx].E_fused : std::max(1, 256 / g_nvs[g]);
		if (!dn)
			c->hgroups[c->gl[g].idx].first_tile = (int)tiles.size();
		const int tg = dn ? c->n_tp + c->gl[g].idx : c->gl[g].idx;
		for (int e0 = 0; e0 < count[g]; e0 += E)
			tiles.push_back(BTile{tg, e0});
	}
	c->n_tiles = (int)tiles.size();

	// ---- device ----
#define B_TRY(call)                                                                                  \
	do {                                                                                             \
		cudaError_t e_ = (call);                                                                     \
		if (e_ != cudaSuccess)                                                                       \
			return reject(DGPU_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));        \
	} while (0)
	B_TRY(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
	c->own_stream = true;
	for (int j = 0; j < kBranches; ++j) {
		B_TRY(cudaStreamCreateWithFlags(&c->aux[j], cudaStreamNonBlocking));
		B_TRY(cudaEventCreateWithFlags(&c->ev_join[j], cudaEventDisableTiming));
	}
	B_TRY(cudaEventCreateWithFlags(&c->ev_fork, cudaEventDisableTiming));
	const size_t ns = c->ns;
	B_TRY(cudaMalloc((void**)&c->u, ns * sizeof(double)));
	B_TRY(cudaMalloc((void**)&c->ug, ns * sizeof(double)));
	B_TRY(cudaMalloc((void**)&c->u0, ns * sizeof(double)));
	B_TRY(cudaMalloc((void**)&c->rhs, ns * sizeof(double)));
	B_TRY(cudaMalloc((void**)&c->vol_gl, ns * sizeof(double)));
	B_TRY(cudaMalloc((void**)&c->traces, (size_t)2 * nv * fb * sizeof(double)));
	B_TRY(cudaMalloc((void**)&c->nnf, (size_t)nv * fb * sizeof(double)));
	if (c->navier_stokes) {
		B_TRY(cudaMalloc((void**)&c->ns_gv, (size_t)d * ns * sizeof(double)));
		B_TRY(cudaMalloc((void**)&c->ns_gtr, (size_t)2 * d * nv * fb * sizeof(double)));
		B_TRY(cudaMalloc((void**)&c->ns_dw, (size_t)nv * fb * sizeof(double)));
		B_TRY(cudaMalloc((void**)&c->ns_y, (size_t)2 * d * nv * fb * sizeof(double)));
		B_TRY(cudaMemset(c->ns_gtr, 0, (size_t)2 * d * nv * fb * sizeof(double)));
		B_TRY(cudaMemset(c->ns_y, 0, (size_t)2 * d * nv * fb * sizeof(double)));
	}
	B_TRY(cudaMalloc((void**)&c->max_bits, sizeof(unsigned long long)));
	B_TRY(cudaMalloc((void**)&c->err_flag, sizeof(int)));
	B_TRY(cudaMalloc((void**)&c->d_bar, 2 * sizeof(unsigned)));
	B_TRY(cudaMemset(c->d_bar, 0, 2 * sizeof(unsigned)));
	B_TRY(cudaMalloc((void**)&c->n_corr, sizeof(unsigned long long)));
	B_TRY(cudaMemset(c->u, 0, ns * sizeof(double)));
	B_TRY(cudaMemset(c->traces, 0, (size_t)2 * nv * fb * sizeof(double)));
	B_TRY(cudaMemset(c->nnf, 0, (size_t)nv * fb * sizeof(double)));
	B_TRY(cudaMemset(c->max_bits, 0, sizeof(unsigned long long)));
	B_TRY(cudaMemset(c->err_flag, 0, sizeof(int)));
	B_TRY(cudaMemset(c->n_corr, 0, sizeof(unsigned long long)));
	// dense groups: operators, M_ref^-1, face operator table, 1/J
	for (int t = 0; t < c->n_dense; ++t) {
		const dgpu_dense_operators* op = dops[t];
		DGroup& G = c->hdgroups[t];
		const int nvs = op->n_vs, nvc = op->n_vc;
		std::vector<double> cv0(op->cv0_vs_vc, op->cv0_vs_vc + (size_t)nvc * nvs);
		c->dense_cv0_h.push_back(cv0);
		c->dense_wJ_h.push_back(dense_wJ[t]);
		std::vector<double> cv1(op->cv1_vs_vc, op->cv1_vs_vc + (size_t)d * nvc * nvs);
		std::vector<double> M((size_t)nvs * nvs, 0.0), Minv((size_t)nvs * nvs);
		for (int a = 0; a < nvs; ++a)
			for (int b = 0; b < nvs; ++b) {
				double s = 0.0;
				for (int r = 0; r < nvc; ++r)
					s += cv0[(size_t)r * nvs + a] * op->w_vc[r] * cv0[(size_t)r * nvs + b];
				M[(size_t)a * nvs + b] = s;
			}
		if (!host_invert(nvs, M.data(), Minv.data()))
			return reject(DGPU_ERR_INVALID_ARGUMENT, "singular reference mass matrix of a dense group");
		// an orthonormal basis: M_ref = I to rounding, so M^-1 = 1/J without the n_vs^2 product
		double off_id = 0.0;
		for (int a = 0; a < nvs; ++a)
			for (int b = 0; b < nvs; ++b)
				off_id = std::max(off_id, fabs(M[(size_t)a * nvs + b] - (a == b ? 1.0 : 0.0)));
		G.minv_identity = off_id <= 1e-13 ? 1 : 0;
		std::vector<double> fops;
		std::vector<long long> foff((size_t)kMaxLf * kMaxOrd * (kQMax + 1), -1);
		for (int lf = 0; lf < op->n_lf; ++lf)
			for (int o = 0; o < op->n_ord; ++o)
				for (int pf = 1; pf < kQMax; ++pf) {
					const int k = (lf * op->n_ord + o) * kQMax + pf;
					if (!op->cv0_vs_fc[k] || op->n_fc[k] < 1)
						continue;
					foff[(lf * op->n_ord + o) * (kQMax + 1) + pf + 1] = (long long)fops.size();
					fops.insert(fops.end(), op->cv0_vs_fc[k], op->cv0_vs_fc[k] + (size_t)op->n_fc[k] * nvs);
				}
		double *d_cv0 = nullptr, *d_cv1 = nullptr, *d_minv = nullptr, *d_fops = nullptr, *d_ij = nullptr;
		long long* d_foff = nullptr;
		B_TRY(upload_vec(&d_cv0, cv0));
		c->dense_bufs.push_back(d_cv0);
		B_TRY(upload_vec(&d_cv1, cv1));
		c->dense_bufs.push_back(d_cv1);
		B_TRY(upload_vec(&d_minv, Minv));
		c->dense_bufs.push_back(d_minv);
		B_TRY(upload_vec(&d_fops, fops));
		c->dense_bufs.push_back(d_fops);
		B_TRY(upload_vec(&d_foff, foff));
		c->dense_bufs.push_back(d_foff);
		B_TRY(upload_vec(&d_ij, inv_J[t]));
		c->dense_bufs.push_back(d_ij);
		if (c->positivity) {
			double *d_sb = nullptr, *d_bs = nullptr;
			B_TRY(upload_vec(&d_sb, std::vector<double>(op->ccSB0_vs_vs, op->ccSB0_vs_vs + (size_t)nvs * nvs)));
			c->dense_bufs.push_back(d_sb);
			B_TRY(upload_vec(&d_bs, std::vector<double>(op->ccBS0_vs_vs, op->ccBS0_vs_vs + (size_t)nvs * nvs)));
			c->dense_bufs.push_back(d_bs);
			G.ccSB0 = d_sb;
			G.ccBS0 = d_bs;
			// FP32 pre-filter: the map in FP32 and its rounding bound, (n_vs + 2) 2^-23 max_m sum_a |ccSB0[m][a]|
			// (inputs and map entries rounded to FP32, n_vs-term FP32 sums), doubled
			std::vector<float> sbf((size_t)nvs * nvs);
			double row_max = 0.0;
			for (int m = 0; m < nvs; ++m) {
				double r = 0.0;
				for (int a = 0; a < nvs; ++a) {
					sbf[(size_t)m * nvs + a] = (float)op->ccSB0_vs_vs[(size_t)m * nvs + a];
					r += fabs(op->ccSB0_vs_vs[(size_t)m * nvs + a]);
				}
				row_max = std::max(row_max, r);
			}
			float* d_sbf = nullptr;
			B_TRY(upload_vec(&d_sbf, sbf));
			c->dense_bufs.push_back(d_sbf);
			G.ccSB0f = d_sbf;
			G.pos_err = (float)(2.0 * (nvs + 2) * ldexp(1.0, -23) * row_max);
		}
		B_TRY(upload_fix_ops(c, op, d, Minv, fops, foff, &G));
		G.cv0 = d_cv0;
		G.cv1 = d_cv1;
		G.minv = d_minv;
		G.fops = d_fops;
		G.fop_off = d_foff;
		G.inv_J = d_ij;
		G.minv_vol = nullptr;
		if (dense_curved[t] && G.n_vol > 0) {
			// a group with a curved volume: M^-1 = (cv0^T diag(w J) cv0)^-1 for each of its volumes
			// (constructor_inverse_mass_T, volume_solver_T.c:115-145), formed on the device once
			const size_t smem = dense_minv_smem(nvs);
			if (smem > 227 * 1024)
				return reject(DGPU_ERR_UNSUPPORTED, "curved dense group too large for the mass-matrix inversion");
			double *d_wj = nullptr, *d_mv = nullptr;
			B_TRY(upload_vec(&d_wj, dense_wJ[t]));
			B_TRY(cudaMalloc((void**)&d_mv, (size_t)G.n_vol * nvs * nvs * sizeof(double)));
			c->dense_bufs.push_back(d_mv);
			B_TRY(allow_smem(dense_minv_kernel, smem));
			dense_minv_kernel<<<G.n_vol, 128, smem, c->stream>>>(d_cv0, d_wj, nvs, nvc, G.n_vol, d_mv);
			B_TRY(cudaGetLastError());
			B_TRY(cudaStreamSynchronize(c->stream));
			B_TRY(cudaFree(d_wj));
			G.minv_vol = d_mv;
		}
	}
	B_TRY(upload_vec(&c->d_ops, c->hops));
	B_TRY(upload_vec(&c->d_groups, c->hgroups));
	B_TRY(upload_vec(&c->d_dgroups, c->hdgroups));
	B_TRY(upload_vec(&c->d_elf, elf));
	B_TRY(upload_vec(&c->d_fbase, fbase));
	if (!nc_identity) {
		B_TRY(upload_vec(&c->d_nc, nc_int));
		B_TRY(upload_vec(&c->d_nc_inv, nc_inv_int));
	}
	B_TRY(upload_vec(&c->d_node_face, node_face));
	B_TRY(upload_vec(&c->gmet, gmet));
	B_TRY(upload_vec(&c->inv_wJ, inv_wJ));
	B_TRY(upload_vec(&c->fgeo, fgeo));
	B_TRY(upload_vec(&c->d_tiles, tiles));
	if (n_bnd > 0) {
		B_TRY(upload_vec(&c->d_fbc, fbc));
		B_TRY(upload_vec(&c->d_fext, fext));
	}
	B_TRY(bind(c));
#undef B_TRY
	default_tiles(c);
	const dgpu_status ts = upload_group_tiles(c);   // bind set every group's E_ns
	if (ts != DGPU_OK)
		return reject(ts, c->err);
	*out = c;
	return DGPU_OK;
}

}  // namespace

extern "C" {

dgpu_status dgpu_batch_create(const dgpu_physics* phys, int n_groups, const dgpu_tp_operators* ops,
                              const int* vol_group, const dgpu_mesh* mesh, dgpu_batch** out)
{
	if (!ops || n_groups < 1)
		return bfail(nullptr, DGPU_ERR_INVALID_ARGUMENT, "NULL argument");
	std::vector<GroupIn> gin(n_groups);
	for (int g = 0; g < n_groups; ++g)
		gin[g] = GroupIn{false, &ops[g], nullptr};
	return create_impl(phys, gin, vol_group, mesh, nullptr, out);
}

dgpu_status dgpu_batch_create_groups(const dgpu_physics* phys, int n_groups, const dgpu_group* groups,
                                     const int* vol_group, const dgpu_mesh* mesh, const int* face_ord,
                                     dgpu_batch** out)
{
	if (!groups || n_groups < 1)
		return bfail(nullptr, DGPU_ERR_INVALID_ARGUMENT, "NULL argument");
	std::vector<GroupIn> gin(n_groups);
	for (int g = 0; g < n_groups; ++g) {
		if ((groups[g].tp == nullptr) == (groups[g].dense == nullptr))
			return bfail(nullptr, DGPU_ERR_INVALID_ARGUMENT, "each group needs exactly one of tp / dense");
		gin[g] = GroupIn{groups[g].dense != nullptr, groups[g].tp, groups[g].dense};
	}
	return create_impl(phys, gin, vol_group, mesh, face_ord, out);
}

dgpu_status dgpu_batch_destroy(dgpu_batch* c)
{
	if (!c)
		return DGPU_ERR_INVALID_ARGUMENT;
	if (c->stream)
		cudaStreamSynchronize(c->stream);
	free_batch(c);
	delete c;
	return DGPU_OK;
}

const char* dgpu_batch_last_error(const dgpu_batch* c) { return c ? c->err.c_str() : g_batch_error.c_str(); }

dgpu_status dgpu_batch_state_size(const dgpu_batch* c, size_t* n)
{
	if (!c || !n)
		return DGPU_ERR_INVALID_ARGUMENT;
	*n = c->ns;
	return DGPU_OK;
}

dgpu_status dgpu_batch_set_source(dgpu_batch* c, const double* source_vc)
{
	if (!c)
		return DGPU_ERR_INVALID_ARGUMENT;
	if (!source_vc) {
		if (c->source) {
			BATCH_CUDA(c, cudaStreamSynchronize(c->stream));
			cudaFree(c->source);
			c->source = nullptr;
			drop_graphs(c);
		}
		return DGPU_OK;
	}
	// per sorted element: a TP volume's source is its GL nodal values (added after 1/(w J)); a dense volume's is
	// tw0_vt_vc (J s) = cv0^T diag(w J) s (added before M^-1)
	const int nv = c->nv;
	std::vector<double> h(c->ns, 0.0);
	for (int g = 0; g < c->n_all; ++g) {
		const bool dense = c->gl[g].dense;
		const int t = c->gl[g].idx;
		const long long elem0 = dense ? c->hdgroups[t].elem0 : c->hgroups[t].elem0;
		const int n_vol = c->group_n_vol(g);
		for (int e = 0; e < n_vol; ++e) {
			const long long p = elem0 + e;
			const int v = c->order[p];
			const double* src = source_vc + c->list_vc_off[v] * nv;
			double* o = h.data() + c->sorted_off[p];
			if (!dense) {
				std::copy(src, src + (c->list_off[v + 1] - c->list_off[v]), o);
				continue;
			}
			const int nvs = c->hdgroups[t].n_vs, nvc = c->hdgroups[t].n_vc;
			const double* cv0 = c->dense_cv0_h[t].data();
			const double* wJ = c->dense_wJ_h[t].data() + (size_t)e * nvc;
			for (int k = 0; k < nv; ++k)
				for (int m = 0; m < nvs; ++m) {
					double a = 0.0;
					for (int n = 0; n < nvc; ++n)
						a += cv0[(size_t)n * nvs + m] * (wJ[n] * src[n + (size_t)nvc * k]);
					o[(size_t)k * nvs + m] = a;
				}
		}
	}
	if (!c->source) {
		BATCH_CUDA(c, cudaStreamSynchronize(c->stream));
		BATCH_CUDA(c, cudaMalloc((void**)&c->source, c->ns * sizeof(double)));
		drop_graphs(c);   // captured steps hold the kernels' parameters, the source pointer among them
	}
	BATCH_CUDA(c, cudaMemcpyAsync(c->source, h.data(), c->ns * sizeof(double), cudaMemcpyHostToDevice, c->stream));
	BATCH_CUDA(c, cudaStreamSynchronize(c->stream));
	return DGPU_OK;
}

dgpu_status dgpu_batch_upload_state(dgpu_batch* c, const double* sol)
{
	if (!c || !sol)
		return DGPU_ERR_INVALID_ARGUMENT;
	std::vector<double> h(c->ns);
	for (int p = 0; p < c->n_vol; ++p) {
		const int v = c->order[p];
		std::copy(sol + c->list_off[v], sol + c->list_off[v + 1], h.begin() + c->sorted_off[p]);
	}
	BATCH_CUDA(c, cudaMemcpyAsync(c->u, h.data(), c->ns * sizeof(double), cudaMemcpyHostToDevice, c->stream));
	BATCH_CUDA(c, cudaStreamSynchronize(c->stream));
	c->coef_valid = true;
	c->gl_valid = false;
	return DGPU_OK;
}

static dgpu_status download_perm(dgpu_batch* c, const double* dev, double* sol)
{
	std::vector<double> h(c->ns);
	BATCH_CUDA(c, cudaMemcpyAsync(h.data(), dev, c->ns * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
	BATCH_CUDA(c, cudaStreamSynchronize(c->stream));
	for (int p = 0; p < c->n_vol; ++p) {
		const int v = c->order[p];
		std::copy(h.begin() + c->sorted_off[p], h.begin() + c->sorted_off[p] + (c->list_off[v + 1] - c->list_off[v]),
		          sol + c->list_off[v]);
	}
	return DGPU_OK;
}

dgpu_status dgpu_batch_download_state(dgpu_batch* c, double* sol)
{
	if (!c || !sol)
		return DGPU_ERR_INVALID_ARGUMENT;
	dgpu_status st = ensure_coef(c);
	if (st != DGPU_OK)
		return st;
	return download_perm(c, c->u, sol);
}

dgpu_status dgpu_batch_download_rhs(dgpu_batch* c, double* rhs)
{
	if (!c || !rhs)
		return DGPU_ERR_INVALID_ARGUMENT;
	return download_perm(c, c->rhs, rhs);
}

// The device error flag: 1 when the positivity limiter met a negative average, kErrBarrier when a grid barrier of
// the stage kernel (form 3) gave up waiting.
static dgpu_status check_flag(dgpu_batch* c)
{
	if (!c->positivity && c->mode != 3)
		return DGPU_OK;
	int flag = 0;
	BATCH_CUDA(c, cudaMemcpyAsync(&flag, c->err_flag, sizeof flag, cudaMemcpyDeviceToHost, c->stream));
	BATCH_CUDA(c, cudaStreamSynchronize(c->stream));
	if (flag == kErrBarrier) {   // reported once: the next launch starts from zeroed barrier words
		BATCH_CUDA(c, cudaMemsetAsync(c->err_flag, 0, sizeof(int), c->stream));
		BATCH_CUDA(c, cudaStreamSynchronize(c->stream));
		return bfail(c, DGPU_ERR_CUDA, "stage kernel: a grid barrier timed out");
	}
	if (flag)
		return bfail(c, DGPU_ERR_POSITIVITY, "average density or pressure below EPS_PHYS");
	return DGPU_OK;
}

dgpu_status dgpu_batch_compute_rhs(dgpu_batch* c, double* max_rhs)
{
	if (!c)
		return DGPU_ERR_INVALID_ARGUMENT;
	dgpu_status st = ensure_coef(c);
	if (st != DGPU_OK)
		return st;
	if ((st = enqueue_stage(c, true, 0.0, 0, 1)) != DGPU_OK)
		return st;
	if (c->mode == 3 && (st = check_flag(c)) != DGPU_OK)
		return st;
	return read_max(c, max_rhs);
}

dgpu_status dgpu_batch_ssp_rk3_steps(dgpu_batch* c, double dt, int n_steps, double* max_rhs)
{
	if (!c || n_steps < 0 || !(dt == dt))
		return DGPU_ERR_INVALID_ARGUMENT;
	dgpu_status st = ensure_gl(c);
	if (st != DGPU_OK)
		return st;
	const int wm = max_rhs ? 1 : 0;
	for (int s = 0; s < n_steps; ++s) {
		const int want = (wm && s == n_steps - 1) ? 1 : 0;
		if (!c->use_graphs) {
			for (int stage = 0; stage < 3 && st == DGPU_OK; ++stage)
				st = enqueue_stage(c, false, dt, stage, (want && stage == 2) ? 1 : 0);
			if (st != DGPU_OK)
				return st;
			continue;
		}
		cudaGraphExec_t& gx = c->graph[c->mode][want];
		if (!gx || c->graph_dt[c->mode][want] != dt) {
			if (gx) {
				cudaGraphExecDestroy(gx);
				gx = nullptr;
			}
			cudaGraph_t g;
			BATCH_CUDA(c, cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
			const long long before = c->launches;
			for (int stage = 0; stage < 3 && st == DGPU_OK; ++stage)
				st = enqueue_stage(c, false, dt, stage, (want && stage == 2) ? 1 : 0);
			c->graph_launches[c->mode][want] = c->launches - before;
			c->launches = before;
			cudaError_t ec = cudaStreamEndCapture(c->stream, &g);
			if (st != DGPU_OK)
				return st;
			BATCH_CUDA(c, ec);
			cudaError_t ei = cudaGraphInstantiate(&gx, g, 0);
			cudaGraphDestroy(g);
			BATCH_CUDA(c, ei);
			c->graph_dt[c->mode][want] = dt;
		}
		BATCH_CUDA(c, cudaGraphLaunch(gx, c->stream));
		c->launches += c->graph_launches[c->mode][want];
	}
	if (n_steps > 0)
		c->coef_valid = false;
	if ((st = check_flag(c)) != DGPU_OK)
		return st;
	return read_max(c, max_rhs);
}

dgpu_status dgpu_batch_set_mode(dgpu_batch* c, int form)
{
	if (!c || form < 0 || form > 3)
		return DGPU_ERR_INVALID_ARGUMENT;
	if (c->navier_stokes && (form == 1 || form == 3))
		return bfail(c, DGPU_ERR_UNSUPPORTED, "Navier-Stokes runs in forms 0 and 2");
	c->mode = form;
	return DGPU_OK;
}

dgpu_status dgpu_batch_set_barrier_timeout(dgpu_batch* c, double seconds)
{
	if (!c || !(seconds > 0.0) || !(seconds <= 60.0))
		return DGPU_ERR_INVALID_ARGUMENT;
	c->barrier_ns = (unsigned long long)(seconds * 1e9);
	drop_graphs(c);   // captured stages hold the bound among their kernel parameters
	return DGPU_OK;
}

dgpu_status dgpu_batch_set_group_tile(dgpu_batch* c, int group, int elements_per_cta)
{
	if (!c || group < 0 || group >= c->n_all)
		return DGPU_ERR_INVALID_ARGUMENT;
	const int g = c->caller_to_internal[group];
	if (elements_per_cta < 1 || elements_per_cta > c->gl[g].E_max)
		return DGPU_ERR_INVALID_ARGUMENT;
	set_group_E(c, g, elements_per_cta);
	dgpu_status st = upload_group_tiles(c);
	drop_graphs(c);
	return st;
}

dgpu_status dgpu_batch_autotune(dgpu_batch* c, double dt, int reps, char* report, size_t report_len)
{
	if (!c || reps < 1 || !(dt == dt))
		return DGPU_ERR_INVALID_ARGUMENT;
	std::string rep;
	// keep the state, the residual and the correction count: tuning runs steps and residuals on them
	const bool coef_was = c->coef_valid, gl_was = c->gl_valid;
	double* saved = nullptr;
	unsigned long long n_corr0 = 0;
	BATCH_CUDA(c, cudaMalloc((void**)&saved, 2 * c->ns * sizeof(double)));
	BATCH_CUDA(c, cudaMemcpyAsync(saved, coef_was ? c->u : c->ug, c->ns * sizeof(double), cudaMemcpyDeviceToDevice,
	                              c->stream));
	BATCH_CUDA(c, cudaMemcpyAsync(saved + c->ns, c->rhs, c->ns * sizeof(double), cudaMemcpyDeviceToDevice,
	                              c->stream));
	BATCH_CUDA(c, cudaMemcpyAsync(&n_corr0, c->n_corr, sizeof n_corr0, cudaMemcpyDeviceToHost, c->stream));
	BATCH_CUDA(c, cudaStreamSynchronize(c->stream));
	dgpu_status st = ensure_gl(c);
	if (st != DGPU_OK) {
		cudaFree(saved);
		return st;
	}
	cudaEvent_t e0, e1;
	cudaEventCreate(&e0);
	cudaEventCreate(&e1);
	auto time_group = [&](int g) -> float {
		float best = 0.f;
		for (int r = 0; r < reps + 1; ++r) {
			cudaEventRecord(e0, c->stream);
			c->gl[g].vol(c, g, false);
			c->gl[g].lift(c, g, kModeRhs, 0.0, 0, 1);
			cudaEventRecord(e1, c->stream);
			cudaEventSynchronize(e1);
			float ms = 0.f;
			cudaEventElapsedTime(&ms, e0, e1);
			if (r > 0)
				best = (r == 1 || ms < best) ? ms : best;
		}
		return best;
	};
	c->mode = 0;
	for (int g = 0; g < c->n_all; ++g) {
		if (c->group_n_vol(g) == 0 || c->navier_stokes)   // Navier-Stokes: the lifts keep the Euler default
			continue;
		int bestE = c->group_E(g);
		float bestT = -1.f;
		for (int E = c->gl[g].E_max; E >= 1; E /= 2) {
			set_group_E(c, g, E);
			upload_group_tiles(c);
			const float t = time_group(g);
			char line[160];
			if (c->gl[g].dense)
				snprintf(line, sizeof line, "dense group n_vs=%d n_vc=%d E=%d: %.4f ms\n",
				         c->hdgroups[c->gl[g].idx].n_vs, c->hdgroups[c->gl[g].idx].n_vc, E, t);
			else
				snprintf(line, sizeof line, "group q=%d E=%d: %.4f ms\n", c->hgroups[c->gl[g].idx].q, E, t);
			rep += line;
			if (bestT < 0.f || t < bestT) {
				bestT = t;
				bestE = E;
			}
			if (E == 1)
				break;
		}
		set_group_E(c, g, bestE);
	}
	if ((st = upload_group_tiles(c)) != DGPU_OK) {
		cudaFree(saved);
		return st;
	}
	drop_graphs(c);
	// the three forms on RK steps (graph-replayed unless graphs are off)
	static const char* names[4] = {"plain", "fused", "branches", "stage"};
	float tmode[4] = {0.f, 0.f, 0.f, 0.f};
	int best = 0;
	for (int m = 0; m < 4; ++m) {
		if (c->navier_stokes && (m == 1 || m == 3)) {   // forms 0 and 2 only
			tmode[m] = 1e30f;
			continue;
		}
		c->mode = m;
		if ((st = dgpu_batch_ssp_rk3_steps(c, dt, 1, nullptr)) != DGPU_OK)
			break;
		cudaEventRecord(e0, c->stream);
		if ((st = dgpu_batch_ssp_rk3_steps(c, dt, reps, nullptr)) != DGPU_OK)
			break;
		cudaEventRecord(e1, c->stream);
		cudaEventSynchronize(e1);
		cudaEventElapsedTime(&tmode[m], e0, e1);
		char line[128];
		snprintf(line, sizeof line, "%s: %.4f ms per RK3 step\n", names[m], tmode[m] / reps);
		rep += line;
		if (tmode[m] < tmode[best])
			best = m;
	}
	c->mode = best;
	cudaMemcpyAsync(coef_was ? c->u : c->ug, saved, c->ns * sizeof(double), cudaMemcpyDeviceToDevice, c->stream);
	cudaMemcpyAsync(c->rhs, saved + c->ns, c->ns * sizeof(double), cudaMemcpyDeviceToDevice, c->stream);
	cudaMemcpyAsync(c->n_corr, &n_corr0, sizeof n_corr0, cudaMemcpyHostToDevice, c->stream);
	cudaStreamSynchronize(c->stream);
	cudaFree(saved);
	cudaEventDestroy(e0);
	cudaEventDestroy(e1);
	c->coef_valid = coef_was;
	c->gl_valid = coef_was ? false : gl_was;
	if (report && report_len)
		snprintf(report, report_len, "%s", rep.c_str());
	return st;
}

dgpu_status dgpu_batch_set_graphs(dgpu_batch* c, int enable)
{
	if (!c || (enable != 0 && enable != 1))
		return DGPU_ERR_INVALID_ARGUMENT;
	c->use_graphs = enable != 0;
	return DGPU_OK;
}

dgpu_status dgpu_batch_get_mode(const dgpu_batch* c, int* form)
{
	if (!c || !form)
		return DGPU_ERR_INVALID_ARGUMENT;
	*form = c->mode;
	return DGPU_OK;
}

dgpu_status dgpu_batch_kernel_launches(const dgpu_batch* c, long long* n)
{
	if (!c || !n)
		return DGPU_ERR_INVALID_ARGUMENT;
	*n = c->launches;
	return DGPU_OK;
}

dgpu_status dgpu_batch_set_stream(dgpu_batch* c, void* stream)
{
	if (!c)
		return DGPU_ERR_INVALID_ARGUMENT;
	BATCH_CUDA(c, cudaStreamSynchronize(c->stream));
	if (c->own_stream)
		cudaStreamDestroy(c->stream);
	c->own_stream = false;
	c->stream = (cudaStream_t)stream;
	drop_graphs(c);
	return DGPU_OK;
}

dgpu_status dgpu_batch_positivity_corrections(dgpu_batch* c, long long* n)
{
	if (!c || !n)
		return DGPU_ERR_INVALID_ARGUMENT;
	unsigned long long v = 0;
	BATCH_CUDA(c, cudaMemcpyAsync(&v, c->n_corr, sizeof v, cudaMemcpyDeviceToHost, c->stream));
	BATCH_CUDA(c, cudaStreamSynchronize(c->stream));
	*n = (long long)v;
	return DGPU_OK;
}

}  // extern "C"

#endif   // DGPU_PART == 0
