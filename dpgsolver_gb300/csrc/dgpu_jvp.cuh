// Forward-mode linearisation of the residual: R(u) and the directional derivative (dR/du) du in one pass.
//
// The reference linearises its residual by complex step (compute_lhs_cmplx_step_dg,
// src/testing/support/simulation/solvers/dg/test_support_solve_dg.c:83-110): every flux routine is instantiated for
// double complex and the imaginary part of R(u + i h du) / h is the product. Here the flux routines are
// instantiated for the dual number Dual<1> (value, derivative), which gives the same product without the step h.
// Everything between the fluxes is linear (V, Dgl^T, the traces, the lift, diag(1/(wJ)), V^-1), so the tangent
// rides through those as a second set of buffers: the volume and face kernels below write the primal quantities to
// the primal parameter set P and the tangent ones to Pd, and the ordinary lift kernel in residual mode, run once on
// P and once on Pd, finishes R and (dR/du) du.
#pragma once

#include "dgpu_tp.cuh"

namespace dgpu {

// Volume term on GLL coefficients u (primal) and du (tangent): both through V, the flux as Dual<1>, the contraction and
// the traces of each in block fixed point (dgpu_fix.cuh), as in the residual's volume kernel. Per element:
// 2 x (su, st, sf) in shared memory and the block exponents of both. R and J d on a HEX 17^3 p2 mesh, Roe-Pike, from host
// buffers and back: 386 -> 353 us.
// FIXT: whether the tangent is in fixed point too. Not for the columns of a Jacobian: a unit direction's values fall by the
// product of D interpolation weights over an element, and the entries far from it would keep fewer bits (HEX p2,
// Lax-Friedrichs: median relative error of an entry 3.2e-14 in FP64, 5.9e-14 in fixed point; for directions without such
// structure there is no difference).
template <int D, int Q, int NV, int PDE, bool FIXT = kFixed<NV>>
__global__ void __launch_bounds__(TPShape<D, Q>::THREADS)
tp_jvp_volume_kernel(const __grid_constant__ TPOps ops, const TPParams P, const TPParams Pd, const double* __restrict__ u,
                     const double* __restrict__ du)
{
	using S = TPShape<D, Q>;
	constexpr int N = S::N, NF = S::NF, E = S::E;
	constexpr int VOL = TPSmem<D, Q, NV>::VOL, XE = TPSmem<D, Q, NV>::EXP, AE = TPSmem<D, Q, NV>::AEXP;
	extern __shared__ double smem[];
	TPOps* sops = reinterpret_cast<TPOps*>(smem);
	double* base = smem + sizeof(TPOps) / 8;
	int* sx = reinterpret_cast<int*>(base + 2 * E * VOL);   // per quantity: E x XE, E x AE
	load_ops<kFixed<NV>>(sops, ops);
	const int tid = threadIdx.x, v0 = blockIdx.x * E, n_here = min(E, P.n_vol - v0);
	const int e = tid / N, node = tid % N, v = v0 + e;
	const bool active = e < n_here;
	for (int i = tid; i < 2 * E * (XE + AE); i += blockDim.x)
		sx[i] = 0;
	double W[NV], dW[NV];
	if (active)
#pragma unroll
		for (int k = 0; k < NV; ++k) {
			W[k] = u[((size_t)v * NV + k) * N + node];
			dW[k] = du[((size_t)v * NV + k) * N + node];
		}
	__syncthreads();
	double* su = base + (2 * e) * VOL;
	double* st = su + NV * N;
	double* sf = st + NV * N;
	double* dsu = base + (2 * e + 1) * VOL;
	double* dst = dsu + NV * N;
	double* dsf = dst + NV * N;
	int* dsx = sx + E * (XE + AE);
	tp_apply_fix<D, Q, NV, true>(W, su, st, sops->fB, sops->sB, sops->B, ops.fix, e, node, active, sx + E * XE, AE);
	tp_apply_fix<D, Q, NV, false, FIXT>(dW, dsu, dst, sops->fB, sops->sB, sops->B, ops.fix, e, node, active, dsx + E * XE, AE);
	double fr[D][NV], dfr[D][NV];
	if (active) {
		double g[D * D];
#pragma unroll
		for (int c = 0; c < D * D; ++c)
			g[c] = P.gmet[((size_t)v * D * D + c) * N + node];
		if constexpr (PDE == kEuler) {
			Dual<1> w[NV], f[D][D + 2];
#pragma unroll
			for (int k = 0; k < NV; ++k) {
				w[k].v = W[k];
				w[k].d[0] = dW[k];
			}
			euler_flux_ref<D, Dual<1>>(w, g, f);
#pragma unroll
			for (int j = 0; j < D; ++j)
#pragma unroll
				for (int k = 0; k < NV; ++k) {
					fr[j][k] = f[j][k].v;
					dfr[j][k] = f[j][k].d[0];
				}
		} else {
			tp_flux<D, NV, PDE>(P.b_adv, W, g, fr);
			tp_flux<D, NV, PDE>(P.b_adv, dW, g, dfr);
		}
	}
	int eb[2 * NV], deb[2 * NV];
	const bool ok = tp_stage_volume<D, Q, NV>(W, fr, ops.fix, e, node, active, su, sf, sx, XE, eb);
	const bool dok = tp_stage_volume<D, Q, NV, false, FIXT>(dW, dfr, ops.fix, e, node, active, dsu, dsf, dsx, XE, deb);
	if (!active)
		return;
	double out[NV];
	tp_derivative<D, Q, NV>(sops, sf, eb, ok, node, out);
#pragma unroll
	for (int k = 0; k < NV; ++k)
		P.vol_gl[((size_t)v * NV + k) * N + node] = out[k];
	tp_derivative<D, Q, NV, FIXT>(sops, dsf, deb, dok, node, out);
#pragma unroll
	for (int k = 0; k < NV; ++k)
		Pd.vol_gl[((size_t)v * NV + k) * N + node] = out[k];
	// traces of both on the 2D local faces
	for (int it = node; it < 2 * D * NF; it += N) {
		const int lf = it / NF, t = it % NF;
		const int fs = P.vol_face[(size_t)v * 2 * D + lf];
		double* tp = P.traces + (size_t)fs * NV * NF;
		double* td = Pd.traces + (size_t)fs * NV * NF;
		tp_trace<D, Q, NV>(sops, su, eb, ok, lf, t, out);
#pragma unroll
		for (int k = 0; k < NV; ++k)
			tp[k * NF + t] = out[k];
		tp_trace<D, Q, NV, FIXT>(sops, dsu, deb, dok, lf, t, out);
#pragma unroll
		for (int k = 0; k < NV; ++k)
			td[k * NF + t] = out[k];
	}
}

// Numerical flux at every face node of the primal traces (P) and its derivative along the tangent traces (Pd). FP64-bound
// (84 %): the value half of the fluxes' lone products runs on the integer pipe. With it, and CTAs of 128 threads for the
// registers it takes (128; Roe-Pike in 3D spills 332 bytes, and three CTAs an SM, which spill none, were slower), R and J d on HEX 17^3 p2, Roe-Pike, went from 353 to 337 us.
template <int D, int Q, int NV, int PDE, int FLUX>
__global__ void __launch_bounds__(128, 4) tp_jvp_face_kernel(const TPParams P, const TPParams Pd)
{
	using S = TPShape<D, Q>;
	constexpr int NF = S::NF;
	const int gid = blockIdx.x * blockDim.x + threadIdx.x;
	if (gid >= P.n_face * NF)
		return;
	const int f = gid / NF, i = gid % NF;
	const int b = P.bnd ? P.bnd[f] : -1;
	const int iR = P.nc ? P.nc[(size_t)f * NF + i] : i;
	const size_t oL = (size_t)(2 * f) * NV * NF, oR = (size_t)(2 * f + 1) * NV * NF;
	double n[D];
	const double* fg = P.fgeo + (size_t)f * (D + 1) * NF;
#pragma unroll
	for (int k = 0; k < D; ++k)
		n[k] = fg[k * NF + i];
	const double sc = fg[D * NF + i];
	double* out = P.nnf + (size_t)f * NV * NF;
	double* dout = Pd.nnf + (size_t)f * NV * NF;
	if constexpr (PDE == kEuler) {
		Dual<1> WL[NV], WR[NV], nF[NV];
#pragma unroll
		for (int k = 0; k < NV; ++k) {
			WL[k].v = P.traces[oL + k * NF + i];
			WL[k].d[0] = Pd.traces[oL + k * NF + i];
		}
		if (b < 0) {
#pragma unroll
			for (int k = 0; k < NV; ++k) {
				WR[k].v = P.traces[oR + k * NF + iR];
				WR[k].d[0] = Pd.traces[oR + k * NF + iR];
			}
		} else {
			boundary_value<D, NV, PDE, Dual<1>>(P, b, i, NF, WL, n, WR);
		}
		if constexpr (FLUX == kRoePike)
			num_flux_roe_pike<D, Dual<1>>(WL, WR, n, nF);
		else
			num_flux_lax_friedrichs<D, Dual<1>>(WL, WR, n, nF);
#pragma unroll
		for (int k = 0; k < NV; ++k) {
			out[k * NF + i] = nF[k].v * sc;
			dout[k * NF + i] = nF[k].d[0] * sc;
		}
	} else {
		// upwind: linear in the traces, the branch set by b.n alone; the boundary value is the interior trace
		// (derivative: its tangent) or the fixed exterior state (derivative 0)
		double uR = 0.0, duR = 0.0;
		if (b < 0) {
			uR = P.traces[oR + iR];
			duR = Pd.traces[oR + iR];
		} else {
			Dual<1> uL, r;
			uL.v = P.traces[oL + i];
			uL.d[0] = Pd.traces[oL + i];
			boundary_value<D, NV, PDE, Dual<1>>(P, b, i, NF, &uL, n, &r);
			uR = r.v;
			duR = r.d[0];
		}
		out[i] = num_flux_upwind<D>(P.traces[oL + i], uR, n, P.b_adv) * sc;
		dout[i] = num_flux_upwind<D>(Pd.traces[oL + i], duR, n, P.b_adv) * sc;
	}
}

}  // namespace dgpu
