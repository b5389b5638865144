// Batched explicit DG residual over a mesh of several (element type, p) groups (QUAD or HEX, p = 1..4 mixed).
//
// Elements are stored group by group. A face between volumes of orders p_L and p_R is integrated with the face
// cubature of order p_f = max(p_L, p_R) (the reference's face order, face_solver.c:123-132): each volume
// writes its trace at the face's q_f = p_f + 1 GL points (tangential interpolation from its own q GL points when
// q_f > q), the face kernel evaluates the numerical flux there, and each volume applies the transpose of that
// interpolation before its lift. With q_f = q this reduces to the single-order kernels of dgpu_tp.cuh.
//
// Every kernel body is a __device__ function of (D, Q, ...) with a runtime number of elements per CTA, called
// either by one kernel launch per group ("plain per-group" form) or by one persistent kernel that walks a tile
// list covering all groups and dispatches on each tile's Q ("fused" form).
#pragma once

#include "dgpu_tp.cuh"

namespace dgpu {

constexpr int kMaxLf = 6;       // element-face slots per volume in elf (HEX has the most faces)
constexpr int kMaxOrd = 8;      // face orientations (QUAD faces)

struct BatchOps {
	TPOps t;
	double Iup[kQMax + 1][kQMax][kQMax];   // Iup[qf][i][a]: GL(q) Lagrange a at GL(qf) node i, qf >= q
	FixW fI[kQMax + 1][kQMax][kQMax];      // Iup in fixed point (dgpu_fix.cuh), as a 1D pass in both directions
	int sI[kQMax + 3];                     // its scales
};
static_assert(sizeof(BatchOps) % 8 == 0, "BatchOps is copied to shared memory as doubles");

struct BGroup {
	int q, n_vol, E;          // order+1, volumes, elements per CTA of the per-group form
	int first_tile;           // first tile of this group in the fused tile list
	int E_ns;                 // elements per CTA of the Navier-Stokes gradient and volume kernels
	long long elem0;          // first element (group-sorted element index)
	long long state_off;      // offset of the group's first element in state-sized arrays
	long long gmet_off;       // ... in the metric array
	long long wj_off;         // ... in the 1/(wJ) array
};

// A non-tensor-product (dense-operator) group: TET, WEDGE or PYR volumes of one p (kernels in dgpu_dense.cuh).
struct DGroup {
	int n_vs, n_vc, n_lf, n_ord;
	int n_vol, E, E_fused;      // volumes; volumes per CTA of the per-group and of the fused kernels
	long long elem0;            // first element (group-sorted index)
	long long state_off;        // in state-sized arrays
	long long gmet_off;         // per element D*D*n_vc doubles of w * metrics, component j*D+i
	const double* cv0;          // n_vc x n_vs
	const double* cv1;          // D x n_vc x n_vs
	const double* minv;         // n_vs x n_vs (M_ref^-1)
	const double* inv_J;        // per element 1 / J
	const double* minv_vol;     // per element n_vs x n_vs M^-1 when the group has a curved volume, else null
	const double* fops;         // face operator table
	const long long* fop_off;   // [(lf * n_ord + ord) * (kQMax + 1) + q_f] -> offset in fops, -1 if absent
	int vol_per_e, lift_per_e;  // shared memory per volume (doubles) of the volume and lift bodies
	int minv_identity;          // M_ref is the identity to rounding (orthonormal basis): M^-1 = 1/J
	int prism;                  // WEDGE with TRI x LINE factors: sum-factorised volume term
	int n_tvs, n_tvc, n_lvs, n_lvc;
	const double* ccSB0;        // n_vs x n_vs: coefficients -> Bezier coefficients (positivity), or null
	const double* ccBS0;        // n_vs x n_vs: Bezier -> coefficients
	const float* ccSB0f;        // ccSB0 in FP32 (the limiter's pre-filter)
	float pos_err;              // bound on |b_fp32 - b| / max |s| of the pre-filter's Bezier coefficients
	// Fixed-point forms (dgpu_fix.cuh), W = w 2^s, in the order the kernels' lanes read them:
	const FixW* xcv0;           // [n_vs][n_vc], s_cv0
	const FixW* xcv1;           // [D][n_vc][n_vs], s_cv1 (summed over j and r)
	const FixW* xfT;            // face operators as trace operators: per table entry [n_vs][n_fc], s_f
	const FixW* xfL;            // ... as lifting operators: [n_fc][n_vs], s_f (summed over the faces)
	const FixW* xminv;          // [a][m], s_minv
	const FixW *xt0, *xt0T, *xt1, *xl0, *xl1;   // WEDGE factors: tri0 [rt][t] and [t][rt], tri1, line0, line1
	int s_cv0, s_cv1, s_f, s_minv, s_t0, s_l0, s_t1;   // s_l1 = s_t1 + s_l0 - s_t0 (one sum)
	int nff_max;                // face nodes of the group's largest face
	int fix;                    // 0: the operators have no fixed-point form (fix_usable): every volume keeps the FP64 loops
};

struct BParams {
	double b_adv[3];
	int n_groups;             // TP groups; dense groups follow them in the tile list (group >= n_groups)
	const DGroup* dgroups;
	const BatchOps* ops;      // [group]
	const BGroup* groups;     // [group]
	const int4* elf;          // [element][kMaxLf]: (face, side, q_f, orientation)
	const long long* fbase;   // [face + 1]: first face node of the face (faces laid out by increasing q_f)
	// right-trace gather permutation per face node (side 1's trace in side 0's node order is tR[nc[fbase + i]]) and
	// its inverse (side 1's own node j holds side 0's node nc_inv[fbase + j]); both null when every face's is the
	// identity (get_operator__nc_fc_T(1, face), compute_face_rlhs_T.c:133-146)
	const int* nc = nullptr;
	const int* nc_inv = nullptr;
	const double* gmet;
	const double* inv_wJ;
	const double* fgeo;       // [node][D+1] blocks per face: (D+1) * fbase[f] + k * NF_f + i
	double* traces;           // per face: 2 NV NF_f at 2 NV fbase[f]: [side][NV][NF_f]
	double* nnf;              // per face: NV NF_f at NV fbase[f]: [NV][NF_f]
	double* vol_gl;           // state layout
	unsigned long long* max_bits;
	int* err_flag;
	unsigned long long* n_corr;
	// boundary faces (no side-1 volume), all null on a mesh without any:
	const int* fbc;           // [face]: BC code modulo BC_STEP_SC, -1 on interior faces
	const double* fext;       // per face: NV NF_f at NV fbase[f]: [NV][NF_f] exterior state at the face nodes
	BcData bc_data;
	// Navier-Stokes (BR2, dgpu_batched_ns.cuh), all null otherwise:
	double* ns_gv = nullptr;  // per element [D][NV][N] at D * its state offset: the kept volume gradient
	double* ns_gtr = nullptr; // per face: 2 D NV NF_f at 2 D NV fbase[f]: [side][D][NV][NF_f] gradient traces
	double* ns_dw = nullptr;  // per face: NV NF_f at NV fbase[f]: w_f J_f (W_R - W_L) / 2, side-0 node order
	double* ns_y = nullptr;   // per face, as ns_gtr: each side's own lifting of X at the face nodes (own node order)
	NsPhys ns = {0.0, 1.0, 1.0, kViscosityConstant, 0.0};
	double ns_eta = 0.0;      // BR2 scaling of a face's own lifting in its face gradient
	// The test case's source term (compute_source_rhs_dg_like, compute_rlhs.c:47-57) in the state layout, or null:
	// a TP element's GL nodal values of s (M^-1 tw0_vt_vc (J s) = V^-1 s: added after 1/(w J)); a dense element's
	// tw0_vt_vc (J s) = cv0^T diag(w J) s (added before M^-1).
	const double* source = nullptr;
};

// Fused tile list entry: group and first element within the group.
struct BTile {
	int group;
	int e0;
};

// ---------------------------------------------------------------------------------------------------------------
// shared-memory sizes (doubles per element) of the bodies
template <int D, int Q, int NV>
struct BSmem {
	static constexpr int N = TPShape<D, Q>::N;
	static constexpr int NFQ = TPShape<D, Q>::NF;
	static constexpr int VX = NV * N * 2 + D * NV * N + 2 * D * NV * NFQ;    // su, st, sf, own-order traces
	static constexpr int LX = 3 * NV * N + 2 * D * NV * NFQ;                 // sa, sb, sc, face terms
	// then the element's faces (bface_table) and the block exponents (ints) of dgpu_fix.cuh
	static constexpr int VOL = VX + 6 * D + (TPSmem<D, Q, NV>::EXP + TPSmem<D, Q, NV>::AEXP + 1) / 2;
	static constexpr int LIFT = LX + 6 * D + (TPSmem<D, Q, NV>::LEXP + 1) / 2;
};

// The faces of a QUAD/HEX element, read once into shared memory (2D entries).
struct BFace {
	long long base;   // first face node
	int side, qf, pad[2];
};
static_assert(sizeof(BFace) == 24, "three doubles per face");

__device__ __forceinline__ void bface_table(const BParams& P, long long v, int n, int node, int N, BFace* t)
{
	for (int lf = node; lf < n; lf += N) {
		const int4 fd = P.elf[v * kMaxLf + lf];
		t[lf].base = P.fbase[fd.x];
		t[lf].side = fd.y;
		t[lf].qf = fd.z;
	}
}

// ---------------------------------------------------------------------------------------------------------------
// Volume term + traces at each face's order
// ---------------------------------------------------------------------------------------------------------------
template <int D, int Q, int NV, int PDE, bool GLL_IN>
__device__ void bvol_body(const BParams& P, const BatchOps* sops, const BGroup& G, int e0, int E,
                          const double* __restrict__ u, double* base)
{
	constexpr int N = TPShape<D, Q>::N, NFQ = TPShape<D, Q>::NF;
	constexpr int PER_E = BSmem<D, Q, NV>::VOL, XE = TPSmem<D, Q, NV>::EXP, AE = TPSmem<D, Q, NV>::AEXP;
	const int tid = threadIdx.x;
	const int n_here = min(E, G.n_vol - e0);
	const int e = tid / N, node = tid % N;
	const bool active = e < n_here;
	double* su = base + e * PER_E;
	double* st = su + NV * N;
	double* sf = st + NV * N;
	double* str = sf + D * NV * N;   // [lf][NV][NFQ]
	BFace* tab = reinterpret_cast<BFace*>(su + BSmem<D, Q, NV>::VX);
	int* sx = reinterpret_cast<int*>(base + BSmem<D, Q, NV>::VX + 6 * D);   // element 0's exponents, 2 PER_E ints apart
	double W[NV];
	if (active) {
		const double* ublk = u + G.state_off + (long long)(e0 + e) * NV * N + node;
#pragma unroll
		for (int k = 0; k < NV; ++k)
			W[k] = ublk[k * N];
		for (int i = node; i < XE + AE; i += N)
			sx[e * 2 * PER_E + i] = 0;
		bface_table(P, G.elem0 + e0 + e, 2 * D, node, N, tab);
	}
	__syncthreads();
	if (GLL_IN)
		tp_apply_fix<D, Q, NV, true>(W, su, st, sops->t.fB, sops->t.sB, sops->t.B, sops->t.fix, e, node, active, sx + XE, 2 * PER_E);
	double fr[D][NV];
	if (active) {
		double g[D * D];
		const double* gm = P.gmet + G.gmet_off + (long long)(e0 + e) * D * D * N;
#pragma unroll
		for (int c = 0; c < D * D; ++c)
			g[c] = gm[c * N + node];
		tp_flux<D, NV, PDE>(P.b_adv, W, g, fr);
	}
	int eb[2 * NV];
	const bool ok = tp_stage_volume<D, Q, NV>(W, fr, sops->t.fix, e, node, active, su, sf, sx, 2 * PER_E, eb);
	if (active) {
		// traces at this element's own GL points: written out where the face has them (q_f == Q), kept as limbs (or as
		// doubles out of range) where the face's order is higher
		double out[NV];
		for (int it = node; it < 2 * D * NFQ; it += N) {
			const int lf = it / NFQ, t = it % NFQ;
			if (tab[lf].qf == Q) {
				tp_trace<D, Q, NV>(&sops->t, su, eb, ok, lf, t, out);
				double* dst = P.traces + 2 * NV * tab[lf].base + (long long)tab[lf].side * NV * NFQ;
#pragma unroll
				for (int k = 0; k < NV; ++k)
					dst[k * NFQ + t] = out[k];
			} else if (kFixed<NV> && ok) {
				int stride, b0;
				tp_face_line<D, Q>(lf, t, b0, stride);
				const int2* xu = reinterpret_cast<const int2*>(su) + b0;
#pragma unroll
				for (int k = 0; k < NV; ++k) {
					FixAcc s = {0, 0};
#pragma unroll
					for (int m = 0; m < Q; ++m)
						fix_mac(s, sops->t.fT[lf & 1][m], xu[k * N + m * stride]);
					reinterpret_cast<int2*>(str)[(lf * NV + k) * NFQ + t] = fix_limbs(s.h * 4 + (s.m >> 28));
				}
			} else {
				tp_trace<D, Q, NV>(&sops->t, su, eb, ok, lf, t, out);
#pragma unroll
				for (int k = 0; k < NV; ++k)
					str[(lf * NV + k) * NFQ + t] = out[k];
			}
		}
		// volume term in GL space
		tp_derivative<D, Q, NV>(&sops->t, sf, eb, ok, node, out);
		double* vg = P.vol_gl + G.state_off + (long long)(e0 + e) * NV * N;
#pragma unroll
		for (int k = 0; k < NV; ++k)
			vg[k * N + node] = out[k];
	}
	if (active && node == 0)
		sx[e * 2 * PER_E + XE] = ok;   // for the threads of the CTA that interpolate this element's traces
	__syncthreads();
	{
		// the traces of the higher-order faces: tangential interpolation Q -> q_f, separable in 3D. A thread takes one
		// (element, face, variable, i0) column, contracts the first tangential direction once per b and reuses the Q
		// partial sums for all q_f outputs i1. In fixed point, the block exponent rising by each pass's 62 - s.
		constexpr int NI = 2 * D * NV * kQMax;
		for (int t = tid; t < n_here * NI; t += blockDim.x) {
			const int e = t / NI, it = t % NI;
			const double* str = base + e * PER_E + 2 * NV * N + D * NV * N;
			const BFace* tab = reinterpret_cast<const BFace*>(base + e * PER_E + BSmem<D, Q, NV>::VX);
			const int lf = it / (NV * kQMax), k = it / kQMax % NV, i0 = it % kQMax, qf = tab[lf].qf;
			if (qf == Q || i0 >= qf)
				continue;
			const bool ok = kFixed<NV> && sx[e * 2 * PER_E + XE] != 0;
			const int nff = (D == 2 ? qf : qf * qf);
			double* dst = P.traces + 2 * NV * tab[lf].base + (long long)tab[lf].side * NV * nff + k * nff + i0;
			if (ok) {
				const int2* src = reinterpret_cast<const int2*>(str) + (lf * NV + k) * NFQ;
				const FixW* I0 = sops->fI[qf][i0];
				const int sI = sops->sI[qf];
				const int e1 = fix_block(sx[e * 2 * PER_E + k]) + 62 - sops->t.sT;
				if (D == 2) {
					FixAcc s = {0, 0};
#pragma unroll
					for (int a = 0; a < Q; ++a)
						fix_mac(s, I0[a], src[a]);
					dst[0] = fix_to_double(fix_sum(s), fix_scale(e1, sI));
				} else {
					int2 r[Q];
#pragma unroll
					for (int b = 0; b < Q; ++b) {
						FixAcc s = {0, 0};
#pragma unroll
						for (int a = 0; a < Q; ++a)
							fix_mac(s, I0[a], src[a + Q * b]);
						r[b] = fix_limbs(s.h * 4 + (s.m >> 28));
					}
					for (int i1 = 0; i1 < qf; ++i1) {
						FixAcc s = {0, 0};
#pragma unroll
						for (int b = 0; b < Q; ++b)
							fix_mac(s, sops->fI[qf][i1][b], r[b]);
						dst[qf * i1] = fix_to_double(fix_sum(s), fix_scale(e1 + 62 - sI, sI));
					}
				}
			} else {
				const double* src = str + (lf * NV + k) * NFQ;
				const double(*I)[kQMax] = sops->Iup[qf];
				for (int i1 = 0; i1 < (D == 2 ? 1 : qf); ++i1) {
					double s = 0.0;
					for (int b = 0; b < (D == 2 ? 1 : Q); ++b) {
						double r = 0.0;
						for (int a = 0; a < Q; ++a)
							r = fma(I[i0][a], src[a + Q * b], r);
						s = D == 2 ? r : fma(I[i1][b], r, s);
					}
					dst[qf * i1] = s;
				}
			}
		}
	}
	__syncthreads();   // shared memory is reused by the next tile
}

// ---------------------------------------------------------------------------------------------------------------
// Face numerical flux at q_f points (faces of one q_f in [f_begin, f_end) of the face list)
// ---------------------------------------------------------------------------------------------------------------
template <int D, int NV, int PDE, int FLUX>
__device__ __forceinline__ void bface_node_rt(const BParams& P, int f, int i, int nff)
{
	const long long fb = P.fbase[f];
	const double* tL = P.traces + 2 * NV * fb;
	const double* tR = tL + NV * nff;
	double WL[NV], WR[NV], n[D];
	const double* fg = P.fgeo + (D + 1) * fb;
#pragma unroll
	for (int k = 0; k < D; ++k)
		n[k] = fg[k * nff + i];
	const int code = P.fbc ? P.fbc[f] : -1;
#pragma unroll
	for (int k = 0; k < NV; ++k)
		WL[k] = tL[k * nff + i];
	if (code < 0) {
		const int iR = P.nc ? P.nc[fb + i] : i;
#pragma unroll
		for (int k = 0; k < NV; ++k)
			WR[k] = tR[k * nff + iR];
	} else {
		// a boundary face: the boundary value of its BC from the interior trace (face_solver_T.c:203-275)
		const double* ext = P.fext + NV * fb + i;
		if constexpr (PDE == kEuler) {
			double e[NV];
#pragma unroll
			for (int k = 0; k < NV; ++k)
				e[k] = ext[k * nff];
			euler_boundary<D, double>(code, WL, e, n, WR, P.bc_data);
		} else {
			WR[0] = advection_boundary_value<D, double>(WL[0], ext[0], n, P.b_adv);
		}
	}
	const double sc = fg[D * nff + i];
	double* out = P.nnf + NV * fb;
	if constexpr (PDE == kEuler) {
		double nF[NV];
		if constexpr (FLUX == kRoePike) {
			num_flux_roe_pike<D>(WL, WR, n, nF, sc);
		} else {
			num_flux_lax_friedrichs<D>(WL, WR, n, nF, sc);
		}
#pragma unroll
		for (int k = 0; k < NV; ++k)
			out[k * nff + i] = nF[k];
	} else {
		out[i] = num_flux_upwind<D>(WL[0], WR[0], n, P.b_adv) * sc;
	}
}

// ---------------------------------------------------------------------------------------------------------------
// Lift (with the transposed tangential interpolation from q_f) + M^-1 + residual | RK stage + positivity
// ---------------------------------------------------------------------------------------------------------------
template <int D, int Q, int NV, int MODE>
__device__ void blift_body(const BParams& P, const BatchOps* sops, const BGroup& G, int e0, int E, const RkArgs& rk,
                           double* base)
{
	constexpr int N = TPShape<D, Q>::N, NFQ = TPShape<D, Q>::NF;
	constexpr int PER_E = BSmem<D, Q, NV>::LIFT;
	const int tid = threadIdx.x;
	const int n_here = min(E, G.n_vol - e0);
	const int e = tid / N, node = tid % N;
	const bool active = e < n_here;
	double* sa = base + e * PER_E;
	double* sb = sa + NV * N;
	double* sc = sb + NV * N;
	double* sg = sc + NV * N;            // [lf][NV][NFQ]: E_lf^T-side face terms at this element's points
	constexpr int SX = 2 * PER_E;
	BFace* tab = reinterpret_cast<BFace*>(sa + BSmem<D, Q, NV>::LX);
	int* sx = reinterpret_cast<int*>(base + BSmem<D, Q, NV>::LX + 6 * D);   // element 0's block exponents, SX ints apart
	const int* sscale = sx + e * SX + NV;   // FP32 scales of the positivity pre-filter
	if (active) {
		for (int i = node; i < TPSmem<D, Q, NV>::LEXP; i += N)
			sx[e * SX + i] = 0;
		bface_table(P, G.elem0 + e0 + e, 2 * D, node, N, tab);
	}
	__syncthreads();
	{
		// face terms at the element's own points: copy (q_f == Q) or transposed interpolation q_f -> Q (separable in 3D).
		// A thread takes one (element, face, variable, a) column: the face's values of the variable are one block; it
		// contracts i0 for every i1 and reuses the q_f partial sums for all Q outputs b.
		constexpr int NI = 2 * D * NV * Q;
		for (int t = tid; t < n_here * NI; t += blockDim.x) {
			const int e = t / NI, it = t % NI;
			double* sg = base + e * PER_E + 3 * NV * N;
			const BFace* tab = reinterpret_cast<const BFace*>(base + e * PER_E + BSmem<D, Q, NV>::LX);
			const int lf = it / (NV * Q), k = it / Q % NV, a = it % Q;
			const int qf = tab[lf].qf, nff = (D == 2 ? qf : qf * qf);
			const long long fb = tab[lf].base;
			const double* src = P.nnf + NV * fb + k * nff;
			const bool flip = tab[lf].side == 0;   // side 0: rhs -= ; side 1: rhs -= (-nnf)
			// side 1 reads the face flux (side 0's node order) at its own nodes through the inverse permutation
			const int* ci = (!flip && P.nc_inv) ? P.nc_inv + fb : nullptr;
			double* out = sg + (lf * NV + k) * NFQ + a;
			if (qf == Q) {
#pragma unroll
				for (int b = 0; b < (D == 2 ? 1 : Q); ++b) {
					const int i = a + Q * b;
					const double x = src[ci ? ci[i] : i];
					out[Q * b] = flip ? -x : x;
				}
				continue;
			}
			constexpr int N1 = (D == 2 ? 1 : kQMax);
			// the block exponent first (high words, all loads in flight), the values row by row after it
			int xe = 0;
#pragma unroll
			for (int i1 = 0; i1 < N1; ++i1)
#pragma unroll
				for (int i0 = 0; i0 < kQMax; ++i0) {
					const int i = i0 + qf * i1;
					if (i0 < qf && (D == 2 || i1 < qf))
						xe = max(xe, (reinterpret_cast<const int*>(src)[2 * (ci ? ci[i] : i) + 1] >> 20) & 0x7ff);
				}
			if (kFixed<NV> && fix_in_range(xe)) {
				const int eb = fix_block(xe), sI = sops->sI[qf];
				int2 r[N1];
#pragma unroll
				for (int i1 = 0; i1 < N1; ++i1) {
					double x[kQMax];
#pragma unroll
					for (int i0 = 0; i0 < kQMax; ++i0) {
						const int i = i0 + qf * i1;
						x[i0] = (i0 < qf && (D == 2 || i1 < qf)) ? src[ci ? ci[i] : i] : 0.0;
					}
					FixAcc s = {0, 0};
#pragma unroll
					for (int i0 = 0; i0 < kQMax; ++i0)
						fix_mac(s, sops->fI[qf][i0][a], fix_pack(x[i0], eb));   // entries beyond q_f are zero
					if (D == 2) {
						const double t = fix_to_double(fix_sum(s), fix_scale(eb, sI));
						out[0] = flip ? -t : t;
					}
					r[i1] = fix_limbs(s.h * 4 + (s.m >> 28));
				}
				if (D == 3) {
#pragma unroll
					for (int bb = 0; bb < Q; ++bb) {
						FixAcc s = {0, 0};
#pragma unroll
						for (int i1 = 0; i1 < N1; ++i1)
							fix_mac(s, sops->fI[qf][i1][bb], r[i1]);
						const double t = fix_to_double(fix_sum(s), fix_scale(eb + 62 - sI, sI));
						out[Q * bb] = flip ? -t : t;
					}
				}
			} else {
#pragma unroll 1
				for (int bb = 0; bb < (D == 2 ? 1 : Q); ++bb) {
					double s = 0.0;
					for (int i1 = 0; i1 < (D == 2 ? 1 : qf); ++i1) {
						double r = 0.0;
						for (int i0 = 0; i0 < qf; ++i0) {
							const int i = i0 + qf * i1;
							r = fma(sops->Iup[qf][i0][a], src[ci ? ci[i] : i], r);
						}
						s = D == 2 ? r : fma(sops->Iup[qf][i1][bb], r, s);
					}
					out[Q * bb] = flip ? -s : s;
				}
			}
		}
	}
	__syncthreads();

	constexpr int NFT = TPSmem<D, Q, NV>::NFT, NR = (NFT + N - 1) / N;
	double fv[NR][NV], Rg[NV];
	if (active) {
		const double* vg = P.vol_gl + G.state_off + (long long)(e0 + e) * NV * N;
#pragma unroll
		for (int k = 0; k < NV; ++k)
			Rg[k] = vg[k * N + node];
#pragma unroll
		for (int r = 0; r < NR; ++r) {
			const int it = node + r * N;
			if (it >= NFT)
				break;
#pragma unroll
			for (int k = 0; k < NV; ++k)
				fv[r][k] = sg[((it / NFQ) * NV + k) * NFQ + it % NFQ];
		}
	}
	tp_lift_sum<D, Q, NV>(&sops->t, sops->t.fix, fv, Rg, e, node, active, sa, sx, SX);
	if (active) {
		const double iw = P.inv_wJ[G.wj_off + (long long)(e0 + e) * N + node];
#pragma unroll
		for (int k = 0; k < NV; ++k)
			Rg[k] = mul_int(Rg[k], iw);
		if (P.source) {
			const double* sv = P.source + G.state_off + (long long)(e0 + e) * NV * N + node;
#pragma unroll
			for (int k = 0; k < NV; ++k)
				Rg[k] = add(Rg[k], sv[(long long)k * N]);
		}
	}
	__syncthreads();   // the face terms are read; sa, sb, sc are reused

	const bool need_coef = (MODE == kModeRhs) || (MODE != kModeRkGlNoMax && rk.want_max);
	unsigned long long mx = 0ull;
	double R[NV];
	if (need_coef) {
#pragma unroll
		for (int k = 0; k < NV; ++k)
			R[k] = Rg[k];
		tp_apply_fix<D, Q, NV, false>(R, sa, sb, sops->t.fBinv, sops->t.sBinv, sops->t.Binv, sops->t.fix, e, node, active,
		                              sx + 2 * NV, SX);
		if (active) {
#pragma unroll
			for (int k = 0; k < NV; ++k) {
				const unsigned long long bits = abs_bits(R[k]);
				mx = bits > mx ? bits : mx;
			}
		}
#pragma unroll
		for (int off = 16; off > 0; off >>= 1) {
			const unsigned long long o = __shfl_xor_sync(0xffffffffu, mx, off);
			mx = o > mx ? o : mx;
		}
		if ((tid & 31) == 0 && mx && P.max_bits)
			atomicMax(P.max_bits, mx);
		__syncthreads();
	}
	const long long so = G.state_off + (long long)(e0 + e) * NV * N + node;
	if constexpr (MODE == kModeRhs) {
		if (active)
#pragma unroll
			for (int k = 0; k < NV; ++k)
				rk.rhs[so + (long long)k * N] = R[k];
	} else {
		double snew[NV];
		if (active) {
#pragma unroll
			for (int k = 0; k < NV; ++k) {
				const double s = rk.u[so + (long long)k * N];
				if (rk.stage == 0)
					rk.u0[so + (long long)k * N] = s;
				snew[k] = rk_update(rk.stage, s, rk.stage == 0 ? s : rk.u0[so + (long long)k * N], rk.dt, Rg[k]);
			}
		}
		if (rk.positivity) {
			if (active)
#pragma unroll
				for (int k = 0; k < NV; ++k)
					sb[k * N + node] = snew[k];
			__syncthreads();
			float* xf = reinterpret_cast<float*>(sa);
			float* tf = xf + NV * N;
			float* tmpf = reinterpret_cast<float*>(sc);
			int sb32[NV];
#pragma unroll
			for (int k = 0; k < NV; ++k) {
				const float x = active ? (float)snew[k] : 0.f;
				if (active)
					xf[k * N + node] = x;
				sb32[k] = __float_as_int(fabsf(x));
			}
			elem_max<N, NV>(sb32, e, active, sx + NV, SX);
			__syncthreads();
			tp_apply<D, Q, NV>(xf, tf, tmpf, sops->t.SBf, node, active);
			bool safe = true;
			if (active) {
				const float err = sops->t.pos_err;
				const float rho_lo = tf[node] - err * __int_as_float(sscale[0]);
				safe = rho_lo > 1e-6f * __int_as_float(sscale[0]) + 1e-12f;
				if (safe) {
					float m2 = 0.f;
#pragma unroll
					for (int k = 0; k < D; ++k) {
						const float mk = fabsf(tf[(1 + k) * N + node]) + err * __int_as_float(sscale[1 + k]);
						m2 += mk * mk;
					}
					const float E_lo = tf[(D + 1) * N + node] - err * __int_as_float(sscale[D + 1]);
					const float ke = 0.5f * m2 / rho_lo;
					safe = 0.4f * (E_lo - ke) > 1e-5f * (fabsf(E_lo) + ke) + 1e-12f;
				}
			}
			const int unsafe = __syncthreads_or(active && !safe);
			if (unsafe) {
				int flag = 0;
				const bool corr =
					tp_positivity_exact<D, Q, NV>(sops->t.SBg, sops->t.BSg, sb, sc, sa, node, active, &flag);
				if (flag)
					atomicExch(P.err_flag, 1);
				if (corr) {
					if (node == 0)
						atomicAdd(P.n_corr, 1ull);
#pragma unroll
					for (int k = 0; k < NV; ++k)
						snew[k] = sb[k * N + node];
				}
			}
		}
		if (active)
#pragma unroll
			for (int k = 0; k < NV; ++k)
				rk.u[so + (long long)k * N] = snew[k];
	}
	__syncthreads();   // shared memory is reused by the next tile
}

// ---------------------------------------------------------------------------------------------------------------
// Kernels: per group, and fused persistent over all groups
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void load_batch_ops(BatchOps* sops, const BatchOps* g)
{
	for (int i = threadIdx.x; i < (int)(sizeof(BatchOps) / 8); i += blockDim.x)
		reinterpret_cast<double*>(sops)[i] = reinterpret_cast<const double*>(g)[i];
}

template <int D, int Q, int NV, int PDE, bool GLL_IN>
__global__ void __launch_bounds__(256) bvol_group_kernel(const BParams P, int g, const double* __restrict__ u)
{
	extern __shared__ double smem[];
	BatchOps* sops = reinterpret_cast<BatchOps*>(smem);
	const BGroup G = P.groups[g];
	load_batch_ops(sops, &P.ops[g]);
	if (blockIdx.x == 0 && threadIdx.x == 0 && P.max_bits && G.elem0 == 0)   // first non-empty group
		*P.max_bits = 0ull;
	__syncthreads();
	bvol_body<D, Q, NV, PDE, GLL_IN>(P, sops, G, blockIdx.x * G.E, G.E, u, smem + sizeof(BatchOps) / 8);
}

// Minimum CTAs per SM of the per-group lift (caps its registers): 4 for the RK stages that reduce no max |rhs|
// (64 registers: twice the resident warps of the 128-register build), 2 otherwise.
template <int MODE>
struct BLiftOccupancy { static constexpr int value = (MODE == kModeRkGlNoMax) ? 4 : 2; };

template <int D, int Q, int NV, int MODE>
__global__ void __launch_bounds__(256, BLiftOccupancy<MODE>::value) blift_group_kernel(const BParams P, int g,
                                                                                      const RkArgs rk)
{
	extern __shared__ double smem[];
	BatchOps* sops = reinterpret_cast<BatchOps*>(smem);
	const BGroup G = P.groups[g];
	load_batch_ops(sops, &P.ops[g]);
	__syncthreads();
	blift_body<D, Q, NV, MODE>(P, sops, G, blockIdx.x * G.E, G.E, rk, smem + sizeof(BatchOps) / 8);
}

template <int D, int Q, int NV, bool TO_GL>
__global__ void __launch_bounds__(256) bconvert_group_kernel(const BParams P, int g, const double* __restrict__ in,
                                                               double* __restrict__ out)
{
	extern __shared__ double smem[];
	BatchOps* sops = reinterpret_cast<BatchOps*>(smem);
	double* base = smem + sizeof(BatchOps) / 8;
	const BGroup G = P.groups[g];
	load_batch_ops(sops, &P.ops[g]);
	constexpr int N = TPShape<D, Q>::N, AE = TPSmem<D, Q, NV>::AEXP;
	constexpr int PER_E = 3 * NV * N;   // two buffers, then the block exponents
	const int E = G.E, e0 = blockIdx.x * E;
	const int e = threadIdx.x / N, node = threadIdx.x % N;
	const bool active = e < min(E, G.n_vol - e0);
	int* sx = reinterpret_cast<int*>(base + 2 * NV * N);
	const long long o = G.state_off + (long long)(e0 + e) * NV * N + node;
	double x[NV];
	if (active) {
#pragma unroll
		for (int k = 0; k < NV; ++k)
			x[k] = in[o + k * N];
		for (int i = node; i < AE; i += N)
			sx[e * 2 * PER_E + i] = 0;
	}
	__syncthreads();
	tp_apply_fix<D, Q, NV, true>(x, base + e * PER_E, base + e * PER_E + NV * N, TO_GL ? sops->t.fB : sops->t.fBinv,
	                             TO_GL ? sops->t.sB : sops->t.sBinv, TO_GL ? sops->t.B : sops->t.Binv, sops->t.fix, e, node, active,
	                             sx, 2 * PER_E);
	if (active)
#pragma unroll
		for (int k = 0; k < NV; ++k)
			out[o + k * N] = x[k];
}

}  // namespace dgpu
