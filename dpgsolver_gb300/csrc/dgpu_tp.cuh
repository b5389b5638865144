// Tensor-product (QUAD/HEX) explicit DG residual kernels for sm_103a, FP64.
//
// Formulation. The reference applies dense per-element operators (operator_T.c:96-156 -> cblas_dgemm):
//   R = M^-1 [ sum_d tw1_vt_vc[d] fr_d - sum_faces tw0_vt_fc nnf ],   M = V^T diag(w J) V,
// with V = cv0_vs_vc. On TP elements with GLL solution nodes and (p+1)-point GL cubature V = B (x) B (x) B is
// square and invertible (B = 1D GLL->GL interpolation), cv1_vs_vc[d] = Dgl_d V (GL collocation derivative,
// exact for degree p), and cv0_vs_fc[lf] = E_lf V (E_lf = GL Lagrange values at the face). Hence
//   R = V^-1 R_gl,   R_gl = diag(1/(w J)) [ sum_d Dgl_d^T (w fr_d) - sum_lf E_lf^T (w_f J_f F*) ],
// the same operator in exact arithmetic with the V^-T V^T pair cancelled: every contraction is a 1D
// sum-factorised pass of q FMAs per node, and the dense per-element M^-1 is never formed.
//
// Because the SSP-RK3 stage update is linear, V u_new = a V u0 + b (V u + dt R) = a ug0 + b (ug + dt R_gl): the
// time stepper keeps the state as GL nodal values ug = V u and never applies V or V^-1 inside a step; the
// reference's GLL coefficients are recovered (V^-1) only when the caller reads the state.
//
// Kernels:
//   tp_volume_kernel   [V u ->] ug; Euler/advection flux and metric contraction; sum_j Dgl_j^T; face traces.
//   tp_face_kernel     per face node: numerical flux of the two traces, scaled by w_f J_f.
//   tp_lift_kernel     lift of the face fluxes and diag(1/(wJ)); then either V^-1 + residual + max|rhs| (the
//                      reference's compute_rhs_dg), or the RK stage update in GL space + positivity check.
//   tp_convert_kernel  u <-> ug.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "dgpu_fix.cuh"
#include "dgpu_physics.cuh"

namespace dgpu {

constexpr int kQMax = 5;  // p <= 4

// 1D operators of one (element type, p), derived on the host from the caller's ops_tp factors.
struct TPOps {
	double B[kQMax][kQMax];     // GLL -> GL interpolation  B[m][a]
	double Binv[kQMax][kQMax];  // GL -> GLL                 Binv[a][m]
	double Dgl[kQMax][kQMax];   // GL collocation derivative Dgl[m][k] = l_k'(x_m)
	double lb[2][kQMax];        // GL Lagrange basis at r = -1 / +1
	double SBg[kQMax][kQMax];   // ccSB0 B^-1: GL nodal values -> Bezier coefficients (ccSB0: Lagrange -> Bezier, 1D)
	double BSg[kQMax][kQMax];   // B ccBS0:   Bezier coefficients -> GL nodal values
	double BT[kQMax][kQMax];    // B^T    (adjoint: V^T)
	double BinvT[kQMax][kQMax]; // Binv^T (adjoint: V^-T)
	float SBf[kQMax][kQMax];    // SBg rounded to FP32 (positivity pre-filter)
	float pos_err;              // |FP32 Bezier coefficient - exact| <= pos_err * max_i |x_i| (per variable)
	// Fixed-point forms (dgpu_fix.cuh) and their scales: W = w 2^s. Last: load_ops leaves them out where they are not used
	FixW fD[kQMax][kQMax];      // Dgl^T: fD[a][m] = Dgl[m][a], summed over the D directions
	FixW fG[kQMax][kQMax];      // Dgl, one direction (Navier-Stokes gradients)
	FixW fT[2][kQMax];          // lb as the trace operator
	FixW fU[2][kQMax];          // lb as the lifting operator, summed over the 2D faces and fOne
	FixW fOne;                  // the volume term's weight 1 in that sum
	FixW fB[kQMax][kQMax];      // B and B^-1 as 1D passes (sum |W| <= 2^62)
	FixW fBinv[kQMax][kQMax];
	FixW fBT[kQMax][kQMax];     // their transposes (adjoint)
	FixW fBinvT[kQMax][kQMax];
	int sD, sT, sU, sB, sBinv, sG, sBT, sBinvT;
	int fix;                    // 0: the operators have no fixed-point form (fix_usable): every element keeps the FP64 loops
	int pad;
};
static_assert(sizeof(TPOps) % 8 == 0 && offsetof(TPOps, fD) % 8 == 0, "TPOps is copied to shared memory as doubles");

// Whether the contractions of NV variables run in block fixed point. The advected scalar stays in FP64: its flux couples a
// line of nodes to no other one when the velocity lies along it, and a line far below its element's largest value would
// keep fewer bits than FP64 gives it. (The variables of the Euler equations are coupled by every numerical flux: see
// dgpu_fix.cuh.) On QUAD 16^2 p2 an RK step takes 22.9 us so, 26.9 in fixed point, and a residual 41.3 and 41.7; a
// residual on 128^2 p4 67 and 55.
template <int NV>
constexpr bool kFixed = NV > 1;

struct TPParams {
	int n_vol;
	int n_face;
	double b_adv[3];
	const int* vol_face;       // [v][2D]: face * 2 + side
	const double* gmet;        // [v][D*D][N]: w_vc * metrics, component j*D+i = w J dr_j/dx_i
	const double* inv_wJ;      // [v][N]: 1 / (w_vc J_vc)
	const double* fgeo;        // [f][D+1][NF]: unit normal (D) and w_fc J_f
	const int* nc;             // [f][NF] right-trace gather permutation, or nullptr (identity)
	const int* nc_inv;         // [f][NF] its inverse, or nullptr
	double* traces;            // [f][2][NV][NF]
	double* nnf;               // [f][NV][NF]
	double* vol_gl;            // [v][NV][N]
	unsigned long long* max_bits;  // max |rhs| as the bit pattern of a non-negative double
	int* err_flag;             // positivity failure flag
	unsigned long long* n_corr;    // positivity corrections applied
	// Boundary faces (no side-1 volume), or all three nullptr on a mesh without any:
	const int* bnd;            // [f] index b of the face in the boundary list, -1 for an interior face
	const int* bc_code;        // [b] BC code modulo BC_STEP_SC
	const double* bc_ext;      // [b][NV][NF] exterior (test case) conserved state at the face nodes
	BcData bc_data;            // back pressure / total temperature and pressure data
	// Navier-Stokes (BR2 second-order terms), all nullptr otherwise:
	double* ns_gtr;            // [face side][D][NV][NF] traces of the volume gradient
	const double* ns_lam;      // [face side][NF] diagonal of the face's own lifting at its nodes
	double* ns_X;              // [f][D][NV][NF] w_f J_f n (s_R - s_L) / 2, side-0 node order
	double* ns_gv;             // [v][D][NV][N] volume gradient (physical, at the GL nodes)
	NsPhys ns;                 // viscosity model and constants
	double ns_eta;             // BR2 scaling of a face's own lifting in its face gradient
	// Volume kernel on GLL coefficients only (may be null): also keep the coefficients it read and the GL values it
	// formed, so that one pass over a caller's host buffer both uploads the state and starts the RK step.
	double* keep_coef = nullptr;   // [v][NV][N]
	double* keep_gl = nullptr;     // [v][NV][N]
	// The test case's source term at the volume cubature nodes, or null (compute_source_rhs_dg_like,
	// src/simulation/solvers/compute_rlhs.c:47-57). M^-1 tw0_vt_vc (J s) = V^-1 s on the GL nodes, so it adds to the
	// GL nodal residual after the 1/(w J) scaling.
	const double* source = nullptr;   // [v][NV][N]
};

// Right-hand state of face node i of boundary face b: the boundary value of its BC from the interior trace WL.
template <int D, int NV, int PDE, typename T>
__device__ __forceinline__ void boundary_value(const TPParams& P, int b, int i, int NF, const T* WL, const double* n,
                                               T* WR)
{
	const double* ext = P.bc_ext + (size_t)b * NV * NF;
	if constexpr (PDE == kEuler) {
		double e[NV];
#pragma unroll
		for (int k = 0; k < NV; ++k)
			e[k] = ext[k * NF + i];
		euler_boundary<D, T>(P.bc_code[b], WL, e, n, WR, P.bc_data);
	} else {
		WR[0] = advection_boundary_value<D, T>(WL[0], ext[i], n, P.b_adv);
	}
}

template <int D, int Q>
struct TPShape {
	static constexpr int N = (D == 2 ? Q * Q : Q * Q * Q);
	static constexpr int NF = (D == 2 ? Q : Q * Q);
	static constexpr int E = (N >= 256 ? 1 : 256 / N);   // elements per CTA
	static constexpr int THREADS = ((E * N + 31) / 32) * 32;  // whole warps; surplus threads idle
};

// Index of the node along direction `dir`.
template <int Q>
__device__ __forceinline__ int node_coord(int node, int dir)
{
	return dir == 0 ? node % Q : (dir == 1 ? (node / Q) % Q : node / (Q * Q));
}

// One sum-factorised pass along `dir`: out[var][node] = sum_m M[a(node)][m] in[var][node with a -> m].
template <int D, int Q, int NV, typename T, typename TM>
__device__ __forceinline__ void tp_pass(const T* __restrict__ in, T* __restrict__ out, const TM (*M)[kQMax],
                                        int dir, int node)
{
	constexpr int N = TPShape<D, Q>::N;
	const int stride = (dir == 0 ? 1 : (dir == 1 ? Q : Q * Q));
	const int a = node_coord<Q>(node, dir);
	const int base = node - a * stride;
	T w[Q];
#pragma unroll
	for (int m = 0; m < Q; ++m)
		w[m] = (T)M[a][m];
#pragma unroll
	for (int v = 0; v < NV; ++v) {
		T s = 0;
#pragma unroll
		for (int m = 0; m < Q; ++m)
			s += w[m] * in[v * N + base + m * stride];
		out[v * N + node] = s;
	}
}

// The pass's result at the node alone, kept in registers.
template <int D, int Q, int NV>
__device__ __forceinline__ void tp_pass_value(const double* in, double* x, const double (*M)[kQMax], int dir, int node)
{
	constexpr int N = TPShape<D, Q>::N;
	const int stride = (dir == 0 ? 1 : (dir == 1 ? Q : Q * Q));
	const int a = node_coord<Q>(node, dir);
	const int base = node - a * stride;
#pragma unroll
	for (int v = 0; v < NV; ++v) {
		x[v] = 0.0;
#pragma unroll
		for (int m = 0; m < Q; ++m)
			x[v] += M[a][m] * in[v * N + base + m * stride];
	}
}

// The D passes of M (x) M (x) M over one element block: in -> out, `tmp` as scratch (in, out, tmp distinct).
// Every thread of the CTA must call it (it synchronises); `active` selects the threads that compute.
template <int D, int Q, int NV, typename T, typename TM>
__device__ __forceinline__ void tp_apply(const T* in, T* out, T* tmp, const TM (*M)[kQMax], int node, bool active)
{
	if (D == 2) {
		if (active) tp_pass<D, Q, NV>(in, tmp, M, 0, node);
		__syncthreads();
		if (active) tp_pass<D, Q, NV>(tmp, out, M, 1, node);
	} else {
		if (active) tp_pass<D, Q, NV>(in, out, M, 0, node);
		__syncthreads();
		if (active) tp_pass<D, Q, NV>(out, tmp, M, 1, node);
		__syncthreads();
		if (active) tp_pass<D, Q, NV>(tmp, out, M, 2, node);
	}
	__syncthreads();
}

__device__ __forceinline__ unsigned long long abs_bits(double x)
{
	return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
}

// Copies the operator set (a __grid_constant__ kernel parameter) into shared memory; the caller synchronises before use.
// The loads go through the parameter's generic address: indexed by thread, the constant port would serve the 32 addresses
// of a warp one after the other. FIX: with the fixed-point forms.
template <bool FIX = true>
__device__ __forceinline__ void load_ops(TPOps* sops, const TPOps& ops)
{
	const double* src = reinterpret_cast<const double*>(&ops);
	for (int i = threadIdx.x; i < (int)((FIX ? sizeof(TPOps) : offsetof(TPOps, fD)) / 8); i += blockDim.x) {
		double x;
		asm volatile("ld.f64 %0, [%1];" : "=d"(x) : "l"(src + i));
		reinterpret_cast<double*>(sops)[i] = x;
	}
}

// ---------------------------------------------------------------------------------------------------------------
// Volume term + traces
// ---------------------------------------------------------------------------------------------------------------
// Shared memory per element of the bodies below (doubles).
template <int D, int Q, int NV>
struct TPSmem {
	static constexpr int N = TPShape<D, Q>::N;
	static constexpr int VOL = NV * N * 2 + D * NV * N;   // su, st, sf
	static constexpr int NFT = 2 * D * TPShape<D, Q>::NF;  // face nodes of the element
	static constexpr int LIFT = 3 * NV * N;               // sa, sb, sc (at first the face terms: NV NFT <= 3 NV N)
	// block exponents (ints) per element, kept apart:
	static constexpr int AEXP = NV + (NV > 1 ? 2 : 0);    // of a change of basis: one per variable, spreads of rho and E
	static constexpr int EXP = AEXP + NV;                 // of the volume term: state, spreads, fluxes
	static constexpr int LEXP = 2 * AEXP + 2 * NV;        // of the lift: faces, FP32 scales, two changes of basis
};

// Node index of face node t of local face lf with coordinate 0 along the face's normal direction, and the stride
// along it (tangential coordinates in ascending direction order).
template <int D, int Q>
__device__ __forceinline__ void tp_face_line(int lf, int t, int& base, int& stride)
{
	const int nd = lf >> 1;
	if (D == 2) {
		stride = (nd == 0 ? 1 : Q);
		base = (nd == 0 ? t * Q : t);
	} else {
		const int t0 = t % Q, t1 = t / Q;
		stride = (nd == 0 ? 1 : (nd == 1 ? Q : Q * Q));
		base = (nd == 0 ? t0 * Q + t1 * Q * Q : (nd == 1 ? t0 + t1 * Q * Q : t0 + t1 * Q));
	}
}

// Face node index on local face lf of the line through node.
template <int D, int Q>
__device__ __forceinline__ int tp_face_node(int lf, int node)
{
	const int nd = lf >> 1;
	if (D == 2)
		return nd == 0 ? node_coord<Q>(node, 1) : node_coord<Q>(node, 0);
	const int c0 = node_coord<Q>(node, 0), c1 = node_coord<Q>(node, 1), c2 = node_coord<Q>(node, 2);
	return nd == 0 ? c1 + Q * c2 : (nd == 1 ? c0 + Q * c2 : c0 + Q * c1);
}

// Contravariant flux of W at a node with the w-weighted metric terms g.
template <int D, int NV, int PDE>
__device__ __forceinline__ void tp_flux(const double* b_adv, const double* W, const double* g, double (*fr)[NV])
{
	if constexpr (PDE == kEuler) {
		euler_flux_node<D>(W, g, fr);
	} else {
		// advection: f_i = b_i u ; fr_j = sum_i g[j][i] b_i u
#pragma unroll
		for (int j = 0; j < D; ++j) {
			double gb = 0.0;
#pragma unroll
			for (int i = 0; i < D; ++i)
				gb = fma(g[j * D + i], b_adv[i], gb);
			fr[j][0] = mul(gb, W[0]);
		}
	}
}

// tp_pass along the direction of the given stride, not unrolled (the rare FP64 path beside the fixed-point one).
template <int Q, int NV>
__device__ __noinline__ void tp_pass_rolled(const double* in, double* out, const double (*M)[kQMax], int node,
                                            int stride, int N)
{
	const int a = (node / stride) % Q;
#pragma unroll 1
	for (int k = 0; k < NV; ++k) {
		const double* x = in + k * N + node - a * stride;
		double s = 0.0;
#pragma unroll 1
		for (int m = 0; m < Q; ++m)
			s = fma(M[a][m], x[m * stride], s);
		out[k * N + node] = s;
	}
}

// M (x) .. (x) M applied to the CTA's elements in block fixed point (FP64 passes for an element out of range): x holds
// the node's values on entry and exit; buf and tmp NV N words per element, sx AEXP zeroed ints per element, stride_x ints
// apart. STATE: x is a conserved state (fix_spread); fix: TPOps::fix; FIX: false for FP64 passes throughout (sx is not
// used then). All threads of the CTA must call it; buf is free again after the next barrier.
template <int D, int Q, int NV, bool STATE, bool FIX = kFixed<NV>>
__device__ __forceinline__ void tp_apply_fix(double* x, double* buf, double* tmp, const FixW (*F)[kQMax], int sF,
                                             const double (*M)[kQMax], bool fix, int e, int node, bool active, int* sx,
                                             int stride_x)
{
	constexpr int N = TPShape<D, Q>::N, K = STATE ? TPSmem<D, Q, NV>::AEXP : NV;
	if constexpr (!FIX) {
		__syncthreads();   // buf may still be read, as before the barrier below
		if (active)
#pragma unroll
			for (int k = 0; k < NV; ++k)
				buf[k * N + node] = x[k];
		__syncthreads();
		if (active) tp_pass<D, Q, NV>(buf, tmp, M, 0, node);
		__syncthreads();
		if constexpr (D == 3) {
			if (active) tp_pass<D, Q, NV>(tmp, buf, M, 1, node);
			__syncthreads();
		}
		if (active) tp_pass_value<D, Q, NV>(D == 2 ? tmp : buf, x, M, D - 1, node);
	} else {
		int eb[K];
#pragma unroll
		for (int k = 0; k < NV; ++k)
			eb[k] = active ? fix_exponent(x[k]) : 0;
		if constexpr (K > NV) {
			eb[NV] = active ? fix_low(x[0]) : 0;
			eb[NV + 1] = active ? fix_low(x[NV - 1]) : 0;
		}
		elem_max<N, K>(eb, e, active, sx, stride_x);
		__syncthreads();
		bool ok = fix;
		if (active) {
			const int* se = sx + e * stride_x;
			if constexpr (K > NV)
				ok = ok && fix_spread(se[0], se[NV]) && fix_spread(se[NV - 1], se[NV + 1]);
#pragma unroll
			for (int k = 0; k < NV; ++k) {
				ok = ok && fix_in_range(se[k]);
				eb[k] = fix_block(se[k]);
			}
#pragma unroll
			for (int k = 0; k < NV; ++k) {
				if (ok)
					reinterpret_cast<int2*>(buf)[k * N + node] = fix_pack(x[k], eb[k]);
				else
					buf[k * N + node] = x[k];
			}
		}
		__syncthreads();
		double *src = buf, *dst = tmp;
#pragma unroll
		for (int dir = 0; dir < D - 1; ++dir) {
			if (active) {
				if (ok)
					fix_pass<D, Q, NV>(reinterpret_cast<int2*>(src), reinterpret_cast<int2*>(dst), F, dir, node);
				else   // Inf, NaN, huge values or a spread state: FP64 for this element
					tp_pass_rolled<Q, NV>(src, dst, M, node, dir == 0 ? 1 : Q, N);
			}
			__syncthreads();
			double* t = src;
			src = dst;
			dst = t;
		}
		constexpr int stride = (D == 2 ? Q : Q * Q);
		if (active) {
			if (ok) {
				const int a = node / stride, base = node % stride;
				FixW w[Q];
#pragma unroll
				for (int m = 0; m < Q; ++m)
					w[m] = F[a][m];
#pragma unroll
				for (int k = 0; k < NV; ++k) {
					FixAcc s = {0, 0};
#pragma unroll
					for (int m = 0; m < Q; ++m)
						fix_mac(s, w[m], reinterpret_cast<const int2*>(src)[k * N + base + m * stride]);
					x[k] = fix_to_double(fix_sum(s), fix_scale(eb[k] + (D - 1) * (62 - sF), sF));
				}
			} else {
				tp_pass_rolled<Q, NV>(src, dst, M, node, stride, N);
#pragma unroll
				for (int k = 0; k < NV; ++k)
					x[k] = dst[k * N + node];
			}
		}
	}
}

// The contractions of the volume term, shared by the uniform and the batched kernels: the node's state W and fluxes fr
// are staged in su (NV N words) and sf (D NV N words) of its element, in block fixed point when the element is in range
// (the return value), as doubles otherwise; eb receives the element's block exponents. sx: EXP zeroed ints per element,
// `stride` ints apart. All threads of the CTA must call it; synchronises before it returns. STATE, fix and FIX as in
// tp_apply_fix.
template <int D, int Q, int NV, bool STATE = true, bool FIX = kFixed<NV>>
__device__ __forceinline__ bool tp_stage_volume(const double* W, const double (*fr)[NV], bool fix, int e, int node, bool active,
                                                double* su, double* sf, int* sx, int stride, int* eb)
{
	constexpr int N = TPShape<D, Q>::N, XE = TPSmem<D, Q, NV>::EXP, AE = TPSmem<D, Q, NV>::AEXP;
	if constexpr (!FIX) {
		__syncthreads();   // su and sf may still be read
		if (active)
#pragma unroll
			for (int k = 0; k < NV; ++k) {
				su[k * N + node] = W[k];
#pragma unroll
				for (int j = 0; j < D; ++j)
					sf[(j * NV + k) * N + node] = fr[j][k];
			}
		__syncthreads();
		return false;
	} else {
		int x[XE];
#pragma unroll
		for (int k = 0; k < XE; ++k)
			x[k] = 0;
		if (active) {
#pragma unroll
			for (int k = 0; k < NV; ++k) {
				x[k] = fix_exponent(W[k]);
				int m = 0;
#pragma unroll
				for (int j = 0; j < D; ++j)
					m = max(m, fix_exponent(fr[j][k]));
				x[AE + k] = m;
			}
			if constexpr (STATE && AE > NV) {
				x[NV] = fix_low(W[0]);
				x[NV + 1] = fix_low(W[NV - 1]);
			}
		}
		elem_max<N, XE>(x, e, active, sx, stride);
		__syncthreads();
		bool ok = fix;
		if (active) {
			const int* se = sx + e * stride;
			if constexpr (STATE && AE > NV)
				ok = ok && fix_spread(se[0], se[NV]) && fix_spread(se[NV - 1], se[NV + 1]);
#pragma unroll
			for (int k = 0; k < NV; ++k) {
				ok = ok && fix_in_range(se[k]) && fix_in_range(se[AE + k]);
				eb[k] = fix_block(se[k]);
				eb[NV + k] = fix_block(se[AE + k]);
			}
			if (ok) {
				int2* xu = reinterpret_cast<int2*>(su);
				int2* xf = reinterpret_cast<int2*>(sf);
#pragma unroll
				for (int k = 0; k < NV; ++k) {
					xu[k * N + node] = fix_pack(W[k], eb[k]);
#pragma unroll
					for (int j = 0; j < D; ++j)
						xf[(j * NV + k) * N + node] = fix_pack(fr[j][k], eb[NV + k]);
				}
			} else {
#pragma unroll
				for (int k = 0; k < NV; ++k) {
					su[k * N + node] = W[k];
#pragma unroll
					for (int j = 0; j < D; ++j)
						sf[(j * NV + k) * N + node] = fr[j][k];
				}
			}
		}
		__syncthreads();
		return ok;
	}
}

// out[k] = sum_j Dgl_j^T (w fr_j) at the node.
template <int D, int Q, int NV, bool FIX = kFixed<NV>>
__device__ __forceinline__ void tp_derivative(const TPOps* sops, const double* sf, const int* eb, bool ok, int node,
                                              double* out)
{
	constexpr int N = TPShape<D, Q>::N;
	if (FIX && ok) {
		const int2* xf = reinterpret_cast<const int2*>(sf);
		FixAcc acc[NV];
#pragma unroll
		for (int k = 0; k < NV; ++k)
			acc[k] = {0, 0};
#pragma unroll
		for (int j = 0; j < D; ++j) {
			const int stride = (j == 0 ? 1 : (j == 1 ? Q : Q * Q));
			const int a = node_coord<Q>(node, j);
			const int b0 = node - a * stride;
#pragma unroll
			for (int m = 0; m < Q; ++m) {
				const FixW w = sops->fD[a][m];
#pragma unroll
				for (int k = 0; k < NV; ++k)
					fix_mac(acc[k], w, xf[(j * NV + k) * N + b0 + m * stride]);
			}
		}
#pragma unroll
		for (int k = 0; k < NV; ++k)
			out[k] = fix_to_double(fix_sum(acc[k]), fix_scale(eb[NV + k], sops->sD));
	} else {
#pragma unroll
		for (int k = 0; k < NV; ++k)
			out[k] = 0.0;
#pragma unroll(FIX ? 1 : D)
		for (int j = 0; j < D; ++j) {
			const int stride = (j == 0 ? 1 : (j == 1 ? Q : Q * Q));
			const int a = (node / stride) % Q;
			const double* f = sf + j * NV * N + node - a * stride;
#pragma unroll(FIX ? 1 : Q)
			for (int m = 0; m < Q; ++m)
#pragma unroll
				for (int k = 0; k < NV; ++k)
					out[k] = fma(sops->Dgl[m][a], f[k * N + m * stride], out[k]);
		}
	}
}

// K values of every node staged in an element's buffer (K N words): in block fixed point when the element is in range
// (returned), as doubles otherwise. eb: the K block exponents. STATE: fix_spread on x[0] and x[K - 1] (K + 2 exponents).
// All threads of the CTA must call it; synchronises before it returns.
template <int N, int K, bool STATE, bool FIX = kFixed<K>>
__device__ __forceinline__ bool tp_stage(const double* x, bool fix, int e, int node, bool active, double* buf, int* sx, int stride,
                                         int* eb)
{
	constexpr int KX = STATE ? K + 2 : K;
	if constexpr (!FIX) {
		__syncthreads();   // buf may still be read
		if (active)
#pragma unroll
			for (int k = 0; k < K; ++k)
				buf[k * N + node] = x[k];
		__syncthreads();
		return false;
	} else {
		int m[KX];
#pragma unroll
		for (int k = 0; k < K; ++k)
			m[k] = active ? fix_exponent(x[k]) : 0;
		if constexpr (STATE) {
			m[K] = active ? fix_low(x[0]) : 0;
			m[K + 1] = active ? fix_low(x[K - 1]) : 0;
		}
		elem_max<N, KX>(m, e, active, sx, stride);
		__syncthreads();
		bool ok = fix;
		if (active) {
			const int* se = sx + e * stride;
			if constexpr (STATE)
				ok = ok && fix_spread(se[0], se[K]) && fix_spread(se[K - 1], se[K + 1]);
#pragma unroll
			for (int k = 0; k < K; ++k) {
				ok = ok && fix_in_range(se[k]);
				eb[k] = fix_block(se[k]);
			}
#pragma unroll
			for (int k = 0; k < K; ++k)
				if (ok)
					reinterpret_cast<int2*>(buf)[k * N + node] = fix_pack(x[k], eb[k]);
				else
					buf[k * N + node] = x[k];
		}
		__syncthreads();
		return ok;
	}
}

// d[j][k] = sum_m Dgl[a][m] x of the staged values, the reference derivative in direction j at the node.
template <int D, int Q, int NV, bool FIX = kFixed<NV>>
__device__ __forceinline__ void tp_gradient(const TPOps* sops, const double* su, const int* eb, bool ok, int node,
                                            double (*d)[NV])
{
	constexpr int N = TPShape<D, Q>::N;
#pragma unroll
	for (int j = 0; j < D; ++j) {
		const int stride = (j == 0 ? 1 : (j == 1 ? Q : Q * Q));
		const int a = node_coord<Q>(node, j);
		const int b0 = node - a * stride;
		if (FIX && ok) {
			FixW w[Q];
#pragma unroll
			for (int m = 0; m < Q; ++m)
				w[m] = sops->fG[a][m];
#pragma unroll
			for (int k = 0; k < NV; ++k) {
				FixAcc s = {0, 0};
#pragma unroll
				for (int m = 0; m < Q; ++m)
					fix_mac(s, w[m], reinterpret_cast<const int2*>(su)[k * N + b0 + m * stride]);
				d[j][k] = fix_to_double(fix_sum(s), fix_scale(eb[k], sops->sG));
			}
		} else {
#pragma unroll
			for (int k = 0; k < NV; ++k)
				d[j][k] = 0.0;
#pragma unroll(FIX ? 1 : Q)
			for (int m = 0; m < Q; ++m)
#pragma unroll
				for (int k = 0; k < NV; ++k)
					d[j][k] = fma(sops->Dgl[a][m], su[k * N + b0 + m * stride], d[j][k]);
		}
	}
}

// out[k] = the trace of the staged state at node t of local face lf.
template <int D, int Q, int NV, bool FIX = kFixed<NV>>
__device__ __forceinline__ void tp_trace(const TPOps* sops, const double* su, const int* eb, bool ok, int lf, int t,
                                         double* out)
{
	constexpr int N = TPShape<D, Q>::N;
	int stride, base;
	tp_face_line<D, Q>(lf, t, base, stride);
	if (FIX && ok) {
		const int2* xu = reinterpret_cast<const int2*>(su) + base;
		FixW w[Q];
#pragma unroll
		for (int m = 0; m < Q; ++m)
			w[m] = sops->fT[lf & 1][m];
#pragma unroll
		for (int k = 0; k < NV; ++k) {
			FixAcc s = {0, 0};
#pragma unroll
			for (int m = 0; m < Q; ++m)
				fix_mac(s, w[m], xu[k * N + m * stride]);
			out[k] = fix_to_double(fix_sum(s), fix_scale(eb[k], sops->sT));
		}
	} else {
#pragma unroll
		for (int k = 0; k < NV; ++k)
			out[k] = 0.0;
#pragma unroll(FIX ? 1 : Q)
		for (int m = 0; m < Q; ++m)
#pragma unroll
			for (int k = 0; k < NV; ++k)
				out[k] = fma(sops->lb[lf & 1][m], su[k * N + base + m * stride], out[k]);
	}
}

// The lifting, shared likewise: fv holds the signed face terms of the element's face nodes node + r N (node index
// lf NF + t), Rg the node's volume term; Rg becomes volume term + sum over the faces of E_lf^T (face terms). sa: NV NFT
// words of the element, sx: NV zeroed ints per element (not used unless FIX). All threads of the CTA must call it; sa must
// not be written before the next barrier.
template <int D, int Q, int NV, bool FIX = kFixed<NV>>
__device__ __forceinline__ void tp_lift_sum(const TPOps* sops, bool fix, const double (*fv)[NV], double* Rg, int e, int node,
                                            bool active, double* sa, int* sx, int stride)
{
	constexpr int N = TPShape<D, Q>::N, NF = TPShape<D, Q>::NF, NFT = TPSmem<D, Q, NV>::NFT, NR = (NFT + N - 1) / N;
	int eb[NV];
	bool ok = FIX && fix;
	if constexpr (FIX) {
#pragma unroll
		for (int k = 0; k < NV; ++k)
			eb[k] = 0;
		if (active) {
#pragma unroll
			for (int k = 0; k < NV; ++k) {
				eb[k] = fix_exponent(Rg[k]);
#pragma unroll
				for (int r = 0; r < NR; ++r)
					if (node + r * N < NFT)
						eb[k] = max(eb[k], fix_exponent(fv[r][k]));
			}
		}
		elem_max<N, NV>(eb, e, active, sx, stride);
	}
	__syncthreads();
	if (active) {
		if constexpr (FIX) {
#pragma unroll
			for (int k = 0; k < NV; ++k) {
				ok = ok && fix_in_range(sx[e * stride + k]);
				eb[k] = fix_block(sx[e * stride + k]);
			}
		}
#pragma unroll
		for (int r = 0; r < NR; ++r) {
			const int it = node + r * N;
			if (it >= NFT)
				break;
#pragma unroll
			for (int k = 0; k < NV; ++k)
				if (ok)
					reinterpret_cast<int2*>(sa)[k * NFT + it] = fix_pack(fv[r][k], eb[k]);
				else
					sa[k * NFT + it] = fv[r][k];
		}
	}
	__syncthreads();
	if (!active)
		return;
	if (ok) {
		FixAcc acc[NV];
		const FixW one = sops->fOne;
#pragma unroll
		for (int k = 0; k < NV; ++k) {
			const int2 x = fix_pack(Rg[k], eb[k]);
			acc[k] = {(long long)one.h * x.y, (long long)one.h * x.x};   // the weight 1 has no low limb
		}
#pragma unroll
		for (int lf = 0; lf < 2 * D; ++lf) {
			const FixW w = sops->fU[lf & 1][node_coord<Q>(node, lf >> 1)];
			const int2* x = reinterpret_cast<const int2*>(sa) + lf * NF + tp_face_node<D, Q>(lf, node);
#pragma unroll
			for (int k = 0; k < NV; ++k)
				fix_mac(acc[k], w, x[k * NFT]);
		}
#pragma unroll
		for (int k = 0; k < NV; ++k)
			Rg[k] = fix_to_double(fix_sum(acc[k]), fix_scale(eb[k], sops->sU));
	} else {
#pragma unroll(FIX ? 1 : 2 * D)
		for (int lf = 0; lf < 2 * D; ++lf) {
			const double l = sops->lb[lf & 1][node_coord<Q>(node, lf >> 1)];
			const double* x = sa + lf * NF + tp_face_node<D, Q>(lf, node);
#pragma unroll
			for (int k = 0; k < NV; ++k)
				Rg[k] = fma(l, x[k * NFT], Rg[k]);
		}
	}
}

// One SSP-RK3 stage of a value (solve_explicit.c:277-295), rounding written out; the lone products on the integer pipe.
__device__ __forceinline__ double rk_update(int stage, double s, double s0, double dt, double R)
{
	if (stage == 0)
		return mad(dt, R, s);
	if (stage == 1)
		return mul_int(0.25, mad(dt, R, mad(3.0, s0, s)));
	return mul_int(1.0 / 3.0, mad(2.0, mad(dt, R, s), s0));
}

// Volume term of the CTA's E elements; per element PER_E doubles at base (su, st, sf at the start), sx the block
// exponents. The flux is FP64; the derivative and the traces contract in block fixed point (dgpu_fix.cuh): 90 of the
// 138 FP64 operations per node at q = 4 leave the FP64 pipe, which bounded the kernel. HEX 32^3 p3: 488 -> 218 us, the FP64
// pipe at 50 % and the issue slots at 57 %.
template <int D, int Q, int NV, int PDE, bool GLL_IN, int PER_E>
__device__ __forceinline__ void tp_volume_body(const TPOps* sops, bool fix, const TPParams& P, const double* __restrict__ u,
                                               int v0, int n_here, double* base, int* sx)
{
	using S = TPShape<D, Q>;
	constexpr int N = S::N, NF = S::NF, XE = TPSmem<D, Q, NV>::EXP, AE = TPSmem<D, Q, NV>::AEXP;
	const int tid = threadIdx.x;
	const int e = tid / N, node = tid % N;
	const bool active = e < n_here;
	const int v = v0 + e;
	double* su = base + e * PER_E;
	double* st = su + NV * N;
	double* sf = st + NV * N;
	double W[NV];
	if (active)
#pragma unroll
		for (int k = 0; k < NV; ++k)
			W[k] = u[((size_t)v * NV + k) * N + node];
	if constexpr (kFixed<NV>)
		for (int i = tid; i < S::E * XE + (GLL_IN ? S::E * AE : 0); i += blockDim.x)
			sx[i] = 0;
	__syncthreads();
	if (GLL_IN) {
		if (active && P.keep_coef)
#pragma unroll
			for (int k = 0; k < NV; ++k)
				P.keep_coef[((size_t)v * NV + k) * N + node] = W[k];
		tp_apply_fix<D, Q, NV, true>(W, su, st, sops->fB, sops->sB, sops->B, fix, e, node, active, sx + S::E * XE, AE);   // V u
		if (active && P.keep_gl)
#pragma unroll
			for (int k = 0; k < NV; ++k)
				P.keep_gl[((size_t)v * NV + k) * N + node] = W[k];
	}

	double fr[D][NV];
	if (active) {
		double g[D * D];
#pragma unroll
		for (int c = 0; c < D * D; ++c)
			g[c] = P.gmet[((size_t)v * D * D + c) * N + node];
		tp_flux<D, NV, PDE>(P.b_adv, W, g, fr);
	}
	int eb[2 * NV];
	const bool ok = tp_stage_volume<D, Q, NV>(W, fr, fix, e, node, active, su, sf, sx, XE, eb);
	if (!active)
		return;
	double out[NV];
	tp_derivative<D, Q, NV>(sops, sf, eb, ok, node, out);
#pragma unroll
	for (int k = 0; k < NV; ++k)
		P.vol_gl[((size_t)v * NV + k) * N + node] = out[k];
	// traces of ug on the 2D local faces
	for (int it = node; it < 2 * D * NF; it += N) {
		const int lf = it / NF, t = it % NF;
		const int fs = P.vol_face[(size_t)v * 2 * D + lf];
		double* dst = P.traces + (size_t)fs * NV * NF;
		tp_trace<D, Q, NV>(sops, su, eb, ok, lf, t, out);
#pragma unroll
		for (int k = 0; k < NV; ++k)
			dst[k * NF + t] = out[k];
	}
}

// Four CTAs per SM (64 registers, 28 bytes spilled at q = 4, whose shared memory allows no more): the FP64 flux of one CTA then overlaps the
// integer contractions of the others. HEX 32^3 p3, 5 steps: 9.33 -> 8.97 ms together with the lift's.
template <int D, int Q, int NV, int PDE, bool GLL_IN>
__global__ void __launch_bounds__(TPShape<D, Q>::THREADS, 4)
tp_volume_kernel(const __grid_constant__ TPOps ops, const TPParams P, const double* __restrict__ u)
{
	using S = TPShape<D, Q>;
	extern __shared__ double smem[];
	TPOps* sops = reinterpret_cast<TPOps*>(smem);
	load_ops<kFixed<NV>>(sops, ops);
	const int v0 = blockIdx.x * S::E;
	if (blockIdx.x == 0 && threadIdx.x == 0 && P.max_bits)
		*P.max_bits = 0ull;
	double* base = smem + sizeof(TPOps) / 8;
	constexpr int VOL = TPSmem<D, Q, NV>::VOL;
	tp_volume_body<D, Q, NV, PDE, GLL_IN, VOL>(sops, ops.fix, P, u, v0, min(S::E, P.n_vol - v0), base,
	                                           reinterpret_cast<int*>(base + S::E * VOL));
}

// ---------------------------------------------------------------------------------------------------------------
// Face numerical flux
// ---------------------------------------------------------------------------------------------------------------
// Bound by the FP64 pipe's sums and fused products (76 %); reciprocals, roots and lone products run on the integer pipe.
// Lax-Friedrichs at HEX 32^3 p3: 295 -> 122 us.
// Roe-Pike: five CTAs an SM (96 registers, 56 bytes spilled); the two pipes it uses overlap only across warps. HEX 21^3 p2 with
// boundaries: 59 us, and 60 at four CTAs (128 registers, no spills).
template <int FLUX>
struct FaceOccupancy { static constexpr int value = (FLUX == kRoePike) ? 5 : 6; };

template <int D, int Q, int NV, int PDE, int FLUX>
__global__ void __launch_bounds__(128, FaceOccupancy<FLUX>::value)
tp_face_kernel(const TPParams P)
{
	using S = TPShape<D, Q>;
	constexpr int NF = S::NF;
	const int gid = blockIdx.x * blockDim.x + threadIdx.x;
	if (gid >= P.n_face * NF)
		return;
	const int f = gid / NF, i = gid % NF;
	const int b = P.bnd ? P.bnd[f] : -1;
	const double* tL = P.traces + (size_t)(2 * f) * NV * NF;
	double WL[NV], WR[NV], n[D];
#pragma unroll
	for (int k = 0; k < NV; ++k)
		WL[k] = tL[k * NF + i];
	const double* fg = P.fgeo + (size_t)f * (D + 1) * NF;
#pragma unroll
	for (int k = 0; k < D; ++k)
		n[k] = fg[k * NF + i];
	if (b < 0) {
		const int iR = P.nc ? P.nc[(size_t)f * NF + i] : i;
		const double* tR = P.traces + (size_t)(2 * f + 1) * NV * NF;
#pragma unroll
		for (int k = 0; k < NV; ++k)
			WR[k] = tR[k * NF + iR];
	} else {
		boundary_value<D, NV, PDE, double>(P, b, i, NF, WL, n, WR);
	}
	const double sc = fg[D * NF + i];
	double* out = P.nnf + (size_t)f * NV * NF;
	if constexpr (PDE == kEuler) {
		double nF[NV];
		if constexpr (FLUX == kRoePike) {
			num_flux_roe_pike<D>(WL, WR, n, nF, sc);
		} else {
			num_flux_lax_friedrichs<D>(WL, WR, n, nF, sc);
		}
#pragma unroll
		for (int k = 0; k < NV; ++k)
			out[k * NF + i] = nF[k];
	} else {
		out[i] = num_flux_upwind<D>(WL[0], WR[0], n, P.b_adv) * sc;
	}
}

// ---------------------------------------------------------------------------------------------------------------
// Lift + M^-1 + (residual | RK stage + positivity)
// ---------------------------------------------------------------------------------------------------------------
// kModeRkGl reads rk.want_max at run time; kModeRkGlNoMax is the RK stage compiled without the max |rhs| path
// (fewer registers for the common graph-replayed stage).
// kModeRkGlOut is kModeRkGl that also writes the new state's GLL coefficients (the last stage of a step whose result
// goes back to the caller).
enum LiftMode { kModeRhs = 0, kModeRkGl = 1, kModeRkGlNoMax = 2, kModeRkGlOut = 3 };

struct RkArgs {
	double* u;         // kModeRkGl: state as GL nodal values (ug), updated in place
	double* u0;        // kModeRkGl: stage-0 copy (ug of sol_coef_p)
	double* rhs;       // kModeRhs: residual output (GLL coefficients)
	double dt;
	int stage;         // 0, 1, 2
	int positivity;
	int want_max;      // kModeRkGl: also reduce max |rhs| (needs V^-1 of the GL residual)
	double* out_coef = nullptr;   // kModeRkGlOut: V^-1 of the new state (GLL coefficients)
	double* out_host = nullptr;   // kModeRkGlOut: the same into a caller's pinned host buffer, or null
};

// enforce_positivity_highorder (solve.c:187-233) on one element held in shared memory.
// `c` holds the element's conserved state [NV][N] in the basis that `toB` maps to Bezier coefficients (`fromB`
// maps back); `b` and `tmp` are scratch [NV][N]. Returns true when this element was corrected (c then holds the
// corrected state). The reference's serial averages and minima run on one thread per element; the Bezier
// transforms are sum-factorised passes by the element's threads. All threads of the CTA must call it.
template <int D, int Q, int NV>
__device__ __noinline__ bool tp_positivity_exact(const double (*toB)[kQMax], const double (*fromB)[kQMax], double* c, double* b,
                                    double* tmp, int node, bool active, int* flag_out)
{
	constexpr int N = TPShape<D, Q>::N;
	tp_apply<D, Q, NV>(c, b, tmp, toB, node, active);
	// convert_variables c -> p per coefficient (solution_euler_T.c:173-194)
	if (active) {
		const double rho = b[node];
		const double rho_inv = 1.0 / rho;
		double rho2V2 = 0.0;
#pragma unroll
		for (int k = 0; k < D; ++k) {
			const double m = b[(1 + k) * N + node];
			rho2V2 += m * m;
			b[(1 + k) * N + node] = m * rho_inv;
		}
		b[(D + 1) * N + node] = kGm1 * (b[(D + 1) * N + node] - 0.5 * rho2V2 * rho_inv);
	}
	__syncthreads();
	int corrected = 0;
	if (active && node == 0) {
		for (int vr = 0; vr < NV; vr += NV - 1) {
			const double* vd = b + vr * N;
			double s = 0.0, mn = vd[0];
			for (int i = 0; i < N; ++i) {
				s += vd[i];
				if (vd[i] < mn)
					mn = vd[i];
			}
			const double avg = s / N;
			if (avg < kEpsPhys) {
				*flag_out = 1;
				break;
			}
			if (mn < kEpsPhys) {
				double p_ho = (avg - kEpsPhys) / (avg - mn);
				p_ho = fmax(0.0, fmin(1.0, p_ho));
				// correct_coef (solve.c:356-374)
				for (int w = 0; w < NV; ++w) {
					double* data = b + w * N;
					double aw = 0.0;
					for (int i = 0; i < N; ++i)
						aw += data[i];
					aw /= N;
					if ((w == 0 || w == NV - 1) && aw < kEpsPhys)
						aw = kEpsPhys;
					for (int i = 0; i < N; ++i)
						data[i] = p_ho * data[i] + (1 - p_ho) * aw;
				}
				corrected = 1;
			}
		}
		tmp[0] = corrected;  // broadcast through shared memory (tmp is free here)
	}
	__syncthreads();
	corrected = active ? (int)tmp[0] : 0;
	__syncthreads();
	const int any = __syncthreads_or(corrected);
	if (!any)
		return false;
	if (corrected) {
		// convert p -> c per coefficient, then back to the state's basis
		const double rho = b[node];
		double V2 = 0.0;
#pragma unroll
		for (int k = 0; k < D; ++k) {
			const double uu = b[(1 + k) * N + node];
			V2 += uu * uu;
			b[(1 + k) * N + node] = rho * uu;
		}
		b[(D + 1) * N + node] = b[(D + 1) * N + node] / kGm1 + 0.5 * rho * V2;
	}
	__syncthreads();
	tp_apply<D, Q, NV>(b, c, tmp, fromB, node, corrected != 0);
	return corrected != 0;
}

// Positivity in the RK epilogue. The exact check is the reference's FP64 computation above. It is preceded by
// an FP32 pre-filter that proves, for most elements, that the exact check cannot trigger: every FP32 Bezier
// coefficient carries an absolute error of at most pos_err * max_i |x_i| of its variable (a forward bound for D
// passes of q-term FMA dot products with FP32-rounded inputs and coefficients, computed on the host with a factor
// 2 margin); density and pressure are bounded below from those intervals, with a further relative margin of
// 1e-5 on the pressure bound for its own FP32 arithmetic. Only CTAs holding an element that fails the filter run
// the exact check, so the decisions are those of the exact FP64 check.

// Lift, 1/(wJ), then the residual (V^-1, max|rhs|) or the RK stage + positivity, for the CTA's E elements; per
// element PER_E doubles at base. FIX: false for FP64 contractions (kModeRhs: tangents).
template <int D, int Q, int NV, int MODE, int PER_E, bool FIX>
__device__ __forceinline__ void tp_lift_body(const TPOps* sops, bool fix, const TPParams& P, const RkArgs& rk, int v0,
                                             int n_here, double* base, int* sx)
{
	using S = TPShape<D, Q>;
	constexpr int N = S::N, NF = S::NF;
	const int tid = threadIdx.x;
	const int e = tid / N, node = tid % N;
	const bool active = e < n_here;
	const int v = v0 + e;
	double* sa = base + e * PER_E;
	double* sb = sa + NV * N;
	double* sc = sb + NV * N;
	constexpr int NFT = TPSmem<D, Q, NV>::NFT, NR = (NFT + N - 1) / N;
	constexpr int AE = TPSmem<D, Q, NV>::AEXP;
	const int* sscale = sx + S::E * NV + e * NV;   // FP32 scales of the positivity pre-filter
	for (int i = tid; i < S::E * TPSmem<D, Q, NV>::LEXP; i += blockDim.x)
		sx[i] = 0;
	double fv[NR][NV], Rg[NV];   // the face terms this thread stages; GL-space residual R_gl of this node
	if (active) {
#pragma unroll
		for (int k = 0; k < NV; ++k)
			Rg[k] = P.vol_gl[((size_t)v * NV + k) * N + node];
#pragma unroll
		for (int r = 0; r < NR; ++r) {
			const int it = node + r * N;
			if (it >= NFT)
				break;
			const int lf = it / NF, t = it % NF;
			const int fs = P.vol_face[(size_t)v * 2 * D + lf];
			const int f = fs >> 1, s = fs & 1;
			const int idx = (s == 1 && P.nc_inv) ? P.nc_inv[(size_t)f * NF + t] : t;
			const double* src = P.nnf + (size_t)f * NV * NF;
#pragma unroll
			for (int k = 0; k < NV; ++k) {
				// side 0: rhs -= E^T nnf ; side 1: rhs -= E^T (-nnf)   (compute_face_rlhs_T.c:297-310)
				const double x = src[k * NF + idx];
				fv[r][k] = s == 0 ? -x : x;
			}
		}
	}
	__syncthreads();   // sx is zero; sops is written by other warps
	tp_lift_sum<D, Q, NV, FIX>(sops, fix, fv, Rg, e, node, active, sa, sx, NV);
	if (active) {
		const double iw = P.inv_wJ[(size_t)v * N + node];
#pragma unroll
		for (int k = 0; k < NV; ++k)
			Rg[k] = mul_int(Rg[k], iw);
		if (P.source)
#pragma unroll
			for (int k = 0; k < NV; ++k)
				Rg[k] = add(Rg[k], P.source[((size_t)v * NV + k) * N + node]);
	}
	__syncthreads();   // the face terms are read; sa, sb, sc are reused

	const bool need_coef = (MODE == kModeRhs) || ((MODE == kModeRkGl || MODE == kModeRkGlOut) && rk.want_max);
	unsigned long long mx = 0ull;
	double R[NV];
	if (MODE != kModeRkGlNoMax && need_coef) {
		// R = V^-1 R_gl (GLL coefficients): D passes of Binv
#pragma unroll
		for (int k = 0; k < NV; ++k)
			R[k] = Rg[k];
		tp_apply_fix<D, Q, NV, false, FIX>(R, sa, sb, sops->fBinv, sops->sBinv, sops->Binv, fix, e, node, active,
		                              sx + 2 * S::E * NV, AE);
		if (active) {
#pragma unroll
			for (int k = 0; k < NV; ++k) {
				const unsigned long long bits = abs_bits(R[k]);
				mx = bits > mx ? bits : mx;
			}
		}
		// max |rhs| (compute_max_rhs_dg_like): integer max over the bit patterns of |R|
#pragma unroll
		for (int off = 16; off > 0; off >>= 1) {
			const unsigned long long o = __shfl_xor_sync(0xffffffffu, mx, off);
			mx = o > mx ? o : mx;
		}
		if ((tid & 31) == 0 && mx && P.max_bits)
			atomicMax(P.max_bits, mx);
		__syncthreads();   // sa/sb/sc are reused below
	}

	if constexpr (MODE == kModeRhs) {
		if (active) {
#pragma unroll
			for (int k = 0; k < NV; ++k)
				rk.rhs[((size_t)v * NV + k) * N + node] = R[k];
		}
		return;
	} else {
		// SSP-RK3 stage update in GL space (solve_explicit.c:277-295; linear, so V commutes with it)
		double snew[NV];
		if (active) {
			const size_t o = (size_t)v * NV * N + node;
#pragma unroll
			for (int k = 0; k < NV; ++k) {
				const double s = rk.u[o + (size_t)k * N];
				if (rk.stage == 0)
					rk.u0[o + (size_t)k * N] = s;
				snew[k] = rk_update(rk.stage, s, rk.stage == 0 ? s : rk.u0[o + (size_t)k * N], rk.dt, Rg[k]);
			}
		}
		if (rk.positivity) {
			if (active)
#pragma unroll
				for (int k = 0; k < NV; ++k)
					sb[k * N + node] = snew[k];
			__syncthreads();
			// FP32 pre-filter (sa as float [NV][N] x2, sscale per element)
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
			elem_max<N, NV>(sb32, e, active, sx + S::E * NV, NV);
			__syncthreads();
			tp_apply<D, Q, NV>(xf, tf, tmpf, sops->SBf, node, active);
			bool safe = true;
			if (active) {
				const float err = sops->pos_err;
				const float rho = tf[node];
				const float erho = err * __int_as_float(sscale[0]);
				const float rho_lo = rho - erho;
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
					const float p_lo = 0.4f * (E_lo - ke);
					const float mag = fabsf(E_lo) + ke;
					safe = p_lo > 1e-5f * mag + 1e-12f;   // NaN/Inf fail this test and go to the exact path
				}
			}
			const int unsafe = __syncthreads_or(active && !safe);
			if (unsafe) {
				int flag = 0;
				const bool corr =
					tp_positivity_exact<D, Q, NV>(sops->SBg, sops->BSg, sb, sc, sa, node, active, &flag);
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
		if (active) {
			const size_t o = (size_t)v * NV * N + node;
#pragma unroll
			for (int k = 0; k < NV; ++k)
				rk.u[o + (size_t)k * N] = snew[k];
		}
		if constexpr (MODE == kModeRkGlOut) {
			// the new state's GLL coefficients: V^-1 of the GL values (D passes of Binv)
			__syncthreads();   // sa/sb/sc are free again
			tp_apply_fix<D, Q, NV, true>(snew, sa, sb, sops->fBinv, sops->sBinv, sops->Binv, fix, e, node, active,
			                             sx + S::E * (2 * NV + AE), AE);
			if (active)
#pragma unroll
				for (int k = 0; k < NV; ++k) {
					const size_t o = ((size_t)v * NV + k) * N + node;
					rk.out_coef[o] = snew[k];
					if (rk.out_host)
						rk.out_host[o] = snew[k];
				}
		}
	}
}

// Minimum CTAs per SM of the lift kernel (caps its registers): 4 for the plain RK stage, 3 otherwise (80 registers; the
// stages spill some 280 bytes around the positivity check's call; at 2 CTAs the last stage of a step with max |rhs| took
// 449 us at HEX 32^3 p3, twice the plain one).
// Plain stages at HEX 32^3 p3: 244 us with FP64 products in the stage update, 187 to 212 with integer ones; both pipes at half.
template <int MODE>
struct LiftOccupancy { static constexpr int value = (MODE == kModeRkGlNoMax) ? 4 : 3; };   // Out: as RkGl

template <int D, int Q, int NV, int MODE, bool FIX = kFixed<NV>>
__global__ void __launch_bounds__(TPShape<D, Q>::THREADS, LiftOccupancy<MODE>::value)
tp_lift_kernel(const __grid_constant__ TPOps ops, const TPParams P, const RkArgs rk)
{
	using S = TPShape<D, Q>;
	extern __shared__ double smem[];
	TPOps* sops = reinterpret_cast<TPOps*>(smem);
	load_ops<kFixed<NV>>(sops, ops);
	const int v0 = blockIdx.x * S::E;
	constexpr int LIFT = TPSmem<D, Q, NV>::LIFT;
	double* base = smem + sizeof(TPOps) / 8;
	tp_lift_body<D, Q, NV, MODE, LIFT, FIX>(sops, ops.fix, P, rk, v0, min(S::E, P.n_vol - v0), base,
	                                   reinterpret_cast<int*>(base + S::E * LIFT));
}

// ---------------------------------------------------------------------------------------------------------------
// u (GLL coefficients) <-> ug (GL nodal values)
// ---------------------------------------------------------------------------------------------------------------
// in_copy / out_copy (either may be null): also write the input / the result there, so that one pass both moves a
// state between a caller's pinned host buffer and the device and changes its basis.
template <int D, int Q, int NV, bool TO_GL>
__global__ void __launch_bounds__(TPShape<D, Q>::THREADS)
tp_convert_kernel(const __grid_constant__ TPOps ops, int n_vol, const double* __restrict__ in, double* __restrict__ out,
                  double* __restrict__ in_copy, double* __restrict__ out_copy)
{
	using S = TPShape<D, Q>;
	constexpr int N = S::N, E = S::E;
	extern __shared__ double smem[];
	TPOps* sops = reinterpret_cast<TPOps*>(smem);
	double* base = smem + sizeof(TPOps) / 8;
	constexpr int PER_E = 2 * NV * N;
	int* sx = reinterpret_cast<int*>(base + E * PER_E);
	const int tid = threadIdx.x;
	load_ops<kFixed<NV>>(sops, ops);
	const int v0 = blockIdx.x * E;
	const int e = tid / N, node = tid % N;
	const bool active = e < min(E, n_vol - v0);
	double x[NV];
	const size_t o = (size_t)(v0 + e) * NV * N + node;
	if (active)
#pragma unroll
		for (int k = 0; k < NV; ++k) {
			x[k] = in[o + (size_t)k * N];
			if (in_copy)
				in_copy[o + (size_t)k * N] = x[k];
		}
	if constexpr (kFixed<NV>)
		for (int i = tid; i < E * TPSmem<D, Q, NV>::AEXP; i += blockDim.x)
			sx[i] = 0;
	__syncthreads();
	tp_apply_fix<D, Q, NV, true>(x, base + e * PER_E, base + e * PER_E + NV * N, TO_GL ? sops->fB : sops->fBinv,
	                       TO_GL ? sops->sB : sops->sBinv, TO_GL ? sops->B : sops->Binv, ops.fix, e, node, active, sx,
	                             TPSmem<D, Q, NV>::AEXP);
	if (active)
#pragma unroll
		for (int k = 0; k < NV; ++k) {
			out[o + (size_t)k * N] = x[k];
			if (out_copy)
				out_copy[o + (size_t)k * N] = x[k];
		}
}

}  // namespace dgpu
