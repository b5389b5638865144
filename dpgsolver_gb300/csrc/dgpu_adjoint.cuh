// Discrete adjoint of the explicit DG residual: the vector-Jacobian product  ubar = (dR/du)^T rbar.
//
// With ug = V u, X = sum_j Dgl_j^T fr_j(ug) - sum_lf E_lf^T S_f F*(traces), R = V^-1 diag(1/(wJ)) X (the factored
// form of dgpu_tp.cuh), the transpose is applied in reverse order:
//   xbar  = diag(1/(wJ)) V^-T rbar                              (GL space)
//   ubar_g = sum_j (dfr_j/dU)^T (Dgl_j xbar)                    (volume, pointwise Jacobians by reverse mode)
//          + sum_lf E_lf^T (dF*/dW_side)^T S_f (E_R xbar_R - E_L xbar_L)   (faces)
//   ubar  = V^T ubar_g
// Kernels: tp_adj_volume_kernel (V u, forward traces, xbar, adjoint traces, volume part), tp_adj_face_kernel
// (reverse mode of the numerical flux; dual numbers through a boundary value), tp_adj_lift_kernel (face part and V^T).
// The reference has no adjoint; its linearisation is checked by complex step (test_support_solve_dg.c:83-110),
// which is what the tests compare this against.
#pragma once

#include "dgpu_tp.cuh"

namespace dgpu {

struct AdjArgs {
	const double* u;      // state (GLL coefficients) at which the Jacobian is taken
	const double* rbar;   // cotangent of R (GLL layout)
	double* ubar;         // result (GLL layout)
	double* atraces;      // [f][2][NV][NF]: E_lf xbar of each side
	double* wbar;         // [f][2][NV][NF]: (dF*/dW_side)^T S_f Fbar, in each side's own face-node order
};

// Reverse mode of euler_flux_ref: adds (dfr/dW)^T sbar to Wbar, sbar[j][eq] the cotangent of fr[j][eq].
template <int D>
__device__ __forceinline__ void euler_flux_ref_vjp(const double* W, const double* g, const double (*sbar)[D + 2],
                                                   double* Wbar)
{
	const double rho = W[0], E = W[D + 1];
	const double rho_inv = recip(rho);
	double u[D], U[D];
	double V2 = 0.0;
#pragma unroll
	for (int k = 0; k < D; ++k) {
		u[k] = rho_inv * W[1 + k];
		V2 += u[k] * u[k];
	}
	const double p = kGm1 * (E - 0.5 * rho * V2);
	const double Ep = E + p;
	double rhob = 0.0, Eb = 0.0, pb = 0.0;
	double mb[D], ub[D];
#pragma unroll
	for (int k = 0; k < D; ++k) {
		mb[k] = 0.0;
		ub[k] = 0.0;
	}
#pragma unroll
	for (int j = 0; j < D; ++j) {
		U[j] = 0.0;
#pragma unroll
		for (int i = 0; i < D; ++i)
			U[j] += g[j * D + i] * u[i];
		// fr_j[0] = rho U_j ; fr_j[1+m] = m_m U_j + p g_jm ; fr_j[D+1] = (E+p) U_j
		double Ub = sbar[j][0] * rho + sbar[j][D + 1] * Ep;
		rhob += sbar[j][0] * U[j];
#pragma unroll
		for (int m = 0; m < D; ++m) {
			Ub += sbar[j][1 + m] * W[1 + m];
			mb[m] += sbar[j][1 + m] * U[j];
			pb += sbar[j][1 + m] * g[j * D + m];
		}
		Eb += sbar[j][D + 1] * U[j];
		pb += sbar[j][D + 1] * U[j];
		// U_j = sum_i g_ji u_i
#pragma unroll
		for (int i = 0; i < D; ++i)
			ub[i] += Ub * g[j * D + i];
	}
	// p = GM1 (E - 0.5 rho V2)
	Eb += kGm1 * pb;
	rhob += -0.5 * kGm1 * V2 * pb;
	const double V2b = -0.5 * kGm1 * rho * pb;
	double rinvb = 0.0;
#pragma unroll
	for (int i = 0; i < D; ++i) {
		ub[i] += 2.0 * u[i] * V2b;          // V2 = sum u_i^2
		mb[i] += ub[i] * rho_inv;           // u_i = m_i rho_inv
		rinvb += ub[i] * W[1 + i];
	}
	rhob += -rinvb * rho_inv * rho_inv;   // rho_inv = 1 / rho
	Wbar[0] += rhob;
#pragma unroll
	for (int i = 0; i < D; ++i)
		Wbar[1 + i] += mb[i];
	Wbar[D + 1] += Eb;
}

// One side of the Lax-Friedrichs flux and its reverse: the quantities of euler_side_lf, then the cotangents of Vn, p, m.n
// and the wave speed carried back to the conserved state.
template <int D>
struct LfSide {
	double ri, mn, q, Vn, p, sa, sb, lam;

	__device__ __forceinline__ LfSide(const double* W, const double* n)
	{
		ri = recip(W[0]);
		double m2 = 0.0;
		mn = 0.0;
#pragma unroll
		for (int k = 0; k < D; ++k) {
			m2 += W[1 + k] * W[1 + k];
			mn += n[k] * W[1 + k];
		}
		q = m2 * ri;
		Vn = mn * ri;
		p = kGm1 * (W[D + 1] - 0.5 * q);
		sa = root(q * ri);
		sb = root(kGamma * p * ri);
		lam = sa + sb;
	}

	// f: half the flux's cotangent, maxV the wave speed of the face, sgn = 1 (left) or -1, lamb the cotangent of lam
	__device__ __forceinline__ void reverse(const double* W, const double* n, const double* f, double fn, double maxV,
	                                        double sgn, double lamb, double* Wb) const
	{
		double Vnb = f[D + 1] * (W[D + 1] + p), pb = fn + f[D + 1] * Vn;
#pragma unroll
		for (int k = 0; k < D; ++k)
			Vnb += f[1 + k] * W[1 + k];
		// the derivative of a root at 0 is taken as 0, as for the dual numbers
		const double ab = sa > 0.0 ? 0.5 * lamb * recip(sa) : 0.0, bb = sb > 0.0 ? 0.5 * kGamma * lamb * recip(sb) : 0.0;
		pb += bb * ri;
		const double qb = ab * ri - 0.5 * kGm1 * pb, mnb = f[0] + Vnb * ri, m2b = 2.0 * qb * ri;
		// 1/rho enters a = q/rho, b = gamma p/rho, Vn = m.n/rho and q = m^2/rho
		const double rb = ab * q + bb * p + Vnb * mn;
		const double wave = sgn * maxV;
		Wb[0] = wave * f[0] - ri * (rb * ri + qb * q);
#pragma unroll
		for (int k = 0; k < D; ++k)
			Wb[1 + k] = (wave + Vn) * f[1 + k] + mnb * n[k] + m2b * W[1 + k];
		Wb[D + 1] = (wave + Vn) * f[D + 1] + kGm1 * pb;
	}
};

// (dF*/dW_L)^T Fbar and (dF*/dW_R)^T Fbar of the Lax-Friedrichs flux (num_flux_lf_impl) by reverse mode.
template <int D>
__device__ __forceinline__ void num_flux_lf_vjp(const double* WL, const double* WR, const double* n, const double* Fbar,
                                                double* WbL, double* WbR)
{
	const LfSide<D> L(WL, n), R(WR, n);
	double f[D + 2], fn = 0.0, maxVb = 0.0;
#pragma unroll
	for (int k = 0; k < D + 2; ++k) {
		f[k] = 0.5 * Fbar[k];
		maxVb += f[k] * (WL[k] - WR[k]);
	}
#pragma unroll
	for (int k = 0; k < D; ++k)
		fn += f[1 + k] * n[k];
	const bool left = abs_less(R.lam, L.lam);
	const double maxV = left ? L.lam : R.lam;
	L.reverse(WL, n, f, fn, maxV, 1.0, left ? maxVb : 0.0, WbL);
	R.reverse(WR, n, f, fn, maxV, -1.0, left ? 0.0 : maxVb, WbR);
}

// One side of the Roe-Pike flux: velocity, pressure and enthalpy, and the way back to the conserved state.
template <int D>
struct RoeSide {
	double ri, u[D], V2, Vn, p, H;

	__device__ __forceinline__ RoeSide(const double* W, const double* n)
	{
		ri = recip(W[0]);
		V2 = Vn = 0.0;
#pragma unroll
		for (int k = 0; k < D; ++k) {
			u[k] = W[1 + k] * ri;
			V2 += u[k] * u[k];
			Vn += n[k] * u[k];
		}
		p = kGm1 * (W[D + 1] - 0.5 * W[0] * V2);
		H = (W[D + 1] + p) * ri;
	}

	// cotangents of rho, 1/rho, u, Vn, p, H and E; wave f the ones of the conserved state itself
	__device__ __forceinline__ void reverse(const double* W, const double* n, double rhob, double rib, double* ub,
	                                        double Vnb, double pb, double Hb, double Eb, double wave, const double* f,
	                                        double* Wb) const
	{
		const double Epb = Hb * ri, pt = pb + Epb, V2b = -kGm1 * pt * W[0];   // twice the cotangent of V2
		rib += Hb * (W[D + 1] + p);
#pragma unroll
		for (int k = 0; k < D; ++k) {
			const double b = ub[k] + Vnb * n[k] + V2b * u[k];
			rib += b * W[1 + k];
			Wb[1 + k] = b * ri + wave * f[1 + k];
		}
		Wb[0] = rhob - 0.5 * kGm1 * pt * V2 - rib * ri * ri + wave * f[0];
		Wb[D + 1] = Eb + Epb + kGm1 * pt + wave * f[D + 1];
	}
};

// The same for the Roe-Pike flux (num_flux_roe_impl, whose names this keeps; a trailing b marks a cotangent).
template <int D>
__device__ __forceinline__ void num_flux_roe_vjp(const double* WL, const double* WR, const double* n, const double* Fbar,
                                                 double* WbL, double* WbR)
{
	const RoeSide<D> L(WL, n), R(WR, n);
	const double r = root(WR[0] * L.ri), rP1_inv = recip(r + 1.0), rho = r * WL[0];
	double f[D + 2], u[D], Vn = 0.0, V2 = 0.0, fn = 0.0, fu = 0.0, fuL = 0.0, fuR = 0.0, fd = 0.0;
#pragma unroll
	for (int k = 0; k < D + 2; ++k) {
		f[k] = 0.5 * Fbar[k];
		fd += f[k] * (WR[k] - WL[k]);
	}
#pragma unroll
	for (int k = 0; k < D; ++k) {
		u[k] = (r * R.u[k] + L.u[k]) * rP1_inv;
		Vn += n[k] * u[k];
		V2 += u[k] * u[k];
		fn += f[1 + k] * n[k];
		fu += f[1 + k] * u[k];
		fuL += f[1 + k] * L.u[k];
		fuR += f[1 + k] * R.u[k];
	}
	const double H = (r * R.H + L.H) * rP1_inv, c = root(kGm1 * (H - 0.5 * V2)), c_inv = recip(c);
	const double dp = R.p - L.p, dVn = R.Vn - L.Vn, fE = f[D + 1];

	// wave speeds, with the branch each takes
	const double a1 = L.Vn - c, b1 = Vn - c, a5 = R.Vn + c, b5 = Vn + c;
	const bool side1 = abs_less(a1, b1), side5 = abs_less(b5, a5);
	const double s1 = (side1 ? a1 : b1) < 0.0 ? -1.0 : 1.0, s5 = (side5 ? a5 : b5) < 0.0 ? -1.0 : 1.0;
	const double l1 = s1 * (side1 ? a1 : b1), l5 = s5 * (side5 ? a5 : b5), l234 = fabs(Vn);
	const double lc1 = 0.5 * (l5 + l1) - l234, lc2 = 0.5 * (l5 - l1);
	const double rd = rho * dVn, dpc = dp * c_inv;
	const double A = lc2 * rd + lc1 * dpc, dis1 = A * c_inv, dis2 = lc1 * rd + lc2 * dpc;

	// back through the dissipation
	const double dis1b = -(f[0] + fu + fE * H), dis2b = -(fn + fE * Vn), Ab = dis1b * c_inv;
	const double lc1b = dis2b * rd + Ab * dpc, lc2b = Ab * rd + dis2b * dpc;
	const double rdb = Ab * lc2 + dis2b * lc1, dpcb = Ab * lc1 + dis2b * lc2;
	const double rhob = rdb * dVn, dVnb = rdb * rho, dpb = dpcb * c_inv;
	const double l1b = 0.5 * s1 * (lc1b - lc2b), l5b = 0.5 * s5 * (lc1b + lc2b), l234b = -fd - lc1b;
	double Vnb = -fE * dis2 + (Vn > 0.0 ? l234b : -l234b);
	double VnLb = fE * (WL[D + 1] + L.p) - dVnb, VnRb = fE * (WR[D + 1] + R.p) + dVnb;
	VnLb += side1 ? l1b : 0.0;
	VnRb += side5 ? l5b : 0.0;
	Vnb += (side1 ? 0.0 : l1b) + (side5 ? 0.0 : l5b);
	const double cb = l5b - l1b - (dis1b * A + dpcb * dp) * c_inv * c_inv;
	const double c2b = c > 0.0 ? 0.5 * cb * c_inv : 0.0;
	// Roe averages: d/dr of x = (r x_R + x_L) / (r + 1) is (x_R - x) / (r + 1)
	const double Hb = (kGm1 * c2b - fE * dis1) * rP1_inv;
	double rb = Hb * (R.H - H) + rhob * WL[0];
	double uLb[D], uRb[D];
#pragma unroll
	for (int k = 0; k < D; ++k) {
		const double ub = (Vnb * n[k] - kGm1 * c2b * u[k] - f[1 + k] * dis1) * rP1_inv;
		rb += ub * (R.u[k] - u[k]);
		uLb[k] = ub + f[1 + k] * WL[0] * L.Vn;
		uRb[k] = r * ub + f[1 + k] * WR[0] * R.Vn;
	}
	const double xb = r > 0.0 ? 0.5 * rb * recip(r) : 0.0;   // r = root(rho_R / rho_L)
	const double rvLb = f[0] + fuL, rvRb = f[0] + fuR;       // of rho Vn
	L.reverse(WL, n, rhob * r + rvLb * L.Vn, xb * WR[0], uLb, VnLb + rvLb * WL[0], fn + fE * L.Vn - dpb, Hb, fE * L.Vn,
	          l234, f, WbL);
	R.reverse(WR, n, xb * L.ri + rvRb * R.Vn, 0.0, uRb, VnRb + rvRb * WR[0], fn + fE * R.Vn + dpb, r * Hb, fE * R.Vn,
	          -l234, f, WbR);
}

// Both sides' cotangents of the numerical flux at one face node. Reverse mode costs about three fluxes; forward mode in the
// 2 NV directions of the two states, which it replaced, about 2 (1 + 2 NV).
template <int D, int FLUX>
__device__ __forceinline__ void num_flux_vjp(const double* WL, const double* WR, const double* n, const double* Fbar,
                                             double* WbL, double* WbR)
{
	if constexpr (FLUX == kRoePike)
		num_flux_roe_vjp<D>(WL, WR, n, Fbar, WbL, WbR);
	else
		num_flux_lf_vjp<D>(WL, WR, n, Fbar, WbL, WbR);
}

// (d/dW_L F*(W_L, W_b(W_L)))^T Fbar at a boundary face node, W_b the boundary value of its BC (the exterior state
// is data and carries no derivative): reverse mode through the flux, dual numbers through W_b.
template <int D, int NV, int FLUX>
__device__ __forceinline__ void num_flux_vjp_boundary(const TPParams& P, int b, int i, int NF, const double* WL,
                                                      const double* n, const double* Fbar, double* Wbar)
{
	Dual<1> L[NV], R[NV];
	double WR[NV], WbR[NV];
#pragma unroll
	for (int k = 0; k < NV; ++k)
		L[k] = Dual<1>(WL[k]);
	boundary_value<D, NV, kEuler, Dual<1>>(P, b, i, NF, L, n, R);
#pragma unroll
	for (int k = 0; k < NV; ++k)
		WR[k] = R[k].v;
	num_flux_vjp<D, FLUX>(WL, WR, n, Fbar, Wbar, WbR);
	// one direction at a time: all of them at once would set the registers of the interior faces too
#pragma unroll 1
	for (int dir = 0; dir < NV; ++dir) {
#pragma unroll
		for (int k = 0; k < NV; ++k)
			L[k].d[0] = k == dir ? 1.0 : 0.0;
		boundary_value<D, NV, kEuler, Dual<1>>(P, b, i, NF, L, n, R);
		double s = 0.0;
#pragma unroll
		for (int eq = 0; eq < NV; ++eq)
			s += WbR[eq] * R[eq].d[0];
#pragma unroll
		for (int k = 0; k < NV; ++k)
			if (k == dir)
				Wbar[k] += s;
	}
}

// ---------------------------------------------------------------------------------------------------------------
// Shared memory of tp_adj_volume_kernel per element (doubles) and its block exponents (ints): V u with its spreads, V^-T rbar,
// and the same two again as staged for the traces and the derivative.
template <int D, int Q, int NV>
struct AdjSmem {
	static constexpr int WORDS = 3 * NV * TPShape<D, Q>::N;
	static constexpr int EXP = 2 * (TPSmem<D, Q, NV>::AEXP + NV);
};

// The changes of basis, the traces of both fields and Dgl_j xbar contract in block fixed point (at q = 4: 240 products a
// node off the FP64 pipe, which keeps the flux's reverse mode). With the lift's, the adjoint of a HEX 12^3 p3 march of four
// steps went from 3.50 to 3.01 ms.
template <int D, int Q, int NV, int PDE>
__global__ void __launch_bounds__(TPShape<D, Q>::THREADS)
tp_adj_volume_kernel(const __grid_constant__ TPOps ops, const TPParams P, const AdjArgs A)
{
	using S = TPShape<D, Q>;
	constexpr int N = S::N, NF = S::NF, E = S::E;
	constexpr int AE = TPSmem<D, Q, NV>::AEXP, XE = AdjSmem<D, Q, NV>::EXP, PER_E = AdjSmem<D, Q, NV>::WORDS;
	extern __shared__ double smem[];
	TPOps* sops = reinterpret_cast<TPOps*>(smem);
	double* base = smem + sizeof(TPOps) / 8;
	int* sx = reinterpret_cast<int*>(base + E * PER_E);
	load_ops<kFixed<NV>>(sops, ops);
	const int tid = threadIdx.x, v0 = blockIdx.x * E, n_here = min(E, P.n_vol - v0);
	const int e = tid / N, node = tid % N, v = v0 + e;
	const bool active = e < n_here;
	for (int i = tid; i < E * XE; i += blockDim.x)
		sx[i] = 0;
	double W[NV], X[NV];
	if (active)
#pragma unroll
		for (int k = 0; k < NV; ++k) {
			W[k] = A.u[((size_t)v * NV + k) * N + node];
			X[k] = A.rbar[((size_t)v * NV + k) * N + node];
		}
	__syncthreads();
	double* su = base + e * PER_E;
	double* st = su + NV * N;
	double* sr = st + NV * N;
	tp_apply_fix<D, Q, NV, true>(W, su, st, sops->fB, sops->sB, sops->B, ops.fix, e, node, active, sx, XE);   // ug = V u
	tp_apply_fix<D, Q, NV, false>(X, sr, st, sops->fBinvT, sops->sBinvT, sops->BinvT, ops.fix, e, node, active, sx + AE, XE);
	if (active) {   // xbar = diag(1/(wJ)) V^-T rbar
		const double iw = P.inv_wJ[(size_t)v * N + node];
#pragma unroll
		for (int k = 0; k < NV; ++k)
			X[k] = mul(X[k], iw);
	}
	int eb[NV], ex[NV];
	const bool ok = tp_stage<N, NV, (NV > 1)>(W, ops.fix, e, node, active, su, sx + AE + NV, XE, eb);
	const bool okx = tp_stage<N, NV, false>(X, ops.fix, e, node, active, sr, sx + 2 * AE + NV, XE, ex);
	if (!active)
		return;

	// forward traces of ug and adjoint traces of xbar on the 2D local faces
	for (int it = node; it < 2 * D * NF; it += N) {
		const int lf = it / NF, t = it % NF;
		const int fs = P.vol_face[(size_t)v * 2 * D + lf];
		double* dst = P.traces + (size_t)fs * NV * NF + t;
		double* adst = A.atraces + (size_t)fs * NV * NF + t;
		double out[NV];
		tp_trace<D, Q, NV>(sops, su, eb, ok, lf, t, out);
#pragma unroll
		for (int k = 0; k < NV; ++k)
			dst[k * NF] = out[k];
		tp_trace<D, Q, NV>(sops, sr, ex, okx, lf, t, out);
#pragma unroll
		for (int k = 0; k < NV; ++k)
			adst[k * NF] = out[k];
	}
	double sb[D][NV];
	tp_gradient<D, Q, NV>(sops, sr, ex, okx, node, sb);   // Dgl_j xbar for each direction j
	double Wb[NV], g[D * D];
#pragma unroll
	for (int k = 0; k < NV; ++k)
		Wb[k] = 0.0;
#pragma unroll
	for (int c = 0; c < D * D; ++c)
		g[c] = P.gmet[((size_t)v * D * D + c) * N + node];
	if constexpr (PDE == kEuler) {
		euler_flux_ref_vjp<D>(W, g, sb, Wb);
	} else {
#pragma unroll
		for (int j = 0; j < D; ++j) {
			double gb = 0.0;
#pragma unroll
			for (int i = 0; i < D; ++i)
				gb += g[j * D + i] * P.b_adv[i];
			Wb[0] += gb * sb[j][0];
		}
	}
#pragma unroll
	for (int k = 0; k < NV; ++k)
		P.vol_gl[((size_t)v * NV + k) * N + node] = Wb[k];
}

// FP64-bound by the flux. Reverse mode took the adjoint of a HEX 12^3 p3 Lax-Friedrichs march of four steps from 4.76 to
// 3.50 ms. 128 registers: the largest count without spills that keeps four CTAs on an SM.
template <int D, int Q, int NV, int PDE, int FLUX>
__global__ void __launch_bounds__(128, 4)
tp_adj_face_kernel(const TPParams P, const AdjArgs A)
{
	using S = TPShape<D, Q>;
	constexpr int NF = S::NF;
	const int gid = blockIdx.x * blockDim.x + threadIdx.x;
	if (gid >= P.n_face * NF)
		return;
	const int f = gid / NF, i = gid % NF;
	const int b = P.bnd ? P.bnd[f] : -1;
	const double* tL = P.traces + (size_t)(2 * f) * NV * NF;
	const double* aL = A.atraces + (size_t)(2 * f) * NV * NF;
	const double* fg = P.fgeo + (size_t)f * (D + 1) * NF;
	double WL[NV], WR[NV], Fb[NV], n[D];
	const double sc = fg[D * NF + i];
#pragma unroll
	for (int k = 0; k < D; ++k)
		n[k] = fg[k * NF + i];
	double* wL = A.wbar + (size_t)(2 * f) * NV * NF;
	if (b >= 0) {
		// boundary face: R_L -= E_L^T S F*(W_L, W_b(W_L)) only, so Fbar = -S E_L xbar_L
#pragma unroll
		for (int k = 0; k < NV; ++k) {
			WL[k] = tL[k * NF + i];
			Fb[k] = -sc * aL[k * NF + i];
		}
		if constexpr (PDE == kEuler) {
			double WbL[NV];
			num_flux_vjp_boundary<D, NV, FLUX>(P, b, i, NF, WL, n, Fb, WbL);
#pragma unroll
			for (int k = 0; k < NV; ++k)
				wL[k * NF + i] = WbL[k];
		} else {
			double b_dot_n = 0.0;
#pragma unroll
			for (int k = 0; k < D; ++k)
				b_dot_n += P.b_adv[k] * n[k];
			// outflow (b.n > 0): the flux is b.n u_L on either branch of the upwind flux; inflow: the exterior
			wL[i] = b_dot_n > 0.0 ? b_dot_n * Fb[0] : 0.0;
		}
		return;
	}
	const int iR = P.nc ? P.nc[(size_t)f * NF + i] : i;
	const double* tR = P.traces + (size_t)(2 * f + 1) * NV * NF;
	const double* aR = A.atraces + (size_t)(2 * f + 1) * NV * NF;
#pragma unroll
	for (int k = 0; k < NV; ++k) {
		WL[k] = tL[k * NF + i];
		WR[k] = tR[k * NF + iR];
		// R_L -= E_L^T S F*, R_R += E_R^T S F* (right in its own node order): Fbar = S (E_R xbar_R - E_L xbar_L)
		Fb[k] = sc * (aR[k * NF + iR] - aL[k * NF + i]);
	}
	double* wR = A.wbar + (size_t)(2 * f + 1) * NV * NF;
	if constexpr (PDE == kEuler) {
		double WbL[NV], WbR[NV];
		num_flux_vjp<D, FLUX>(WL, WR, n, Fb, WbL, WbR);
#pragma unroll
		for (int k = 0; k < NV; ++k) {
			wL[k * NF + i] = WbL[k];
			wR[k * NF + iR] = WbR[k];
		}
	} else {
		double b_dot_n = 0.0;
#pragma unroll
		for (int k = 0; k < D; ++k)
			b_dot_n += P.b_adv[k] * n[k];
		const bool left = b_dot_n > kEps;   // numerical_flux_advection_T.c:69-72
		wL[i] = left ? b_dot_n * Fb[0] : 0.0;
		wR[iR] = left ? 0.0 : b_dot_n * Fb[0];
	}
}

// The lifting of the face cotangents and V^T in block fixed point, as in the residual's lift.
template <int D, int Q, int NV>
__global__ void __launch_bounds__(TPShape<D, Q>::THREADS)
tp_adj_lift_kernel(const __grid_constant__ TPOps ops, const TPParams P, const AdjArgs A)
{
	using S = TPShape<D, Q>;
	constexpr int N = S::N, NF = S::NF, E = S::E, PER_E = TPSmem<D, Q, NV>::LIFT;
	constexpr int NFT = TPSmem<D, Q, NV>::NFT, NR = (NFT + N - 1) / N;
	extern __shared__ double smem[];
	TPOps* sops = reinterpret_cast<TPOps*>(smem);
	double* base = smem + sizeof(TPOps) / 8;
	int* sx = reinterpret_cast<int*>(base + E * PER_E);   // 2 NV per element, of LEXP
	load_ops<kFixed<NV>>(sops, ops);
	const int tid = threadIdx.x, v0 = blockIdx.x * E, n_here = min(E, P.n_vol - v0);
	const int e = tid / N, node = tid % N, v = v0 + e;
	const bool active = e < n_here;
	double* sa = base + e * PER_E;
	double* sb = sa + NV * N;
	for (int i = tid; i < E * 2 * NV; i += blockDim.x)
		sx[i] = 0;
	double fv[NR][NV], ub[NV];
	if (active) {
#pragma unroll
		for (int k = 0; k < NV; ++k)
			ub[k] = P.vol_gl[((size_t)v * NV + k) * N + node];
#pragma unroll
		for (int r = 0; r < NR; ++r) {
			const int it = node + r * N;
			if (it >= NFT)
				break;
			const int lf = it / NF, t = it % NF;
			const double* src = A.wbar + (size_t)P.vol_face[(size_t)v * 2 * D + lf] * NV * NF;   // this side's own node order
#pragma unroll
			for (int k = 0; k < NV; ++k)
				fv[r][k] = src[k * NF + t];
		}
	}
	__syncthreads();
	tp_lift_sum<D, Q, NV>(sops, ops.fix, fv, ub, e, node, active, sa, sx, NV);
	tp_apply_fix<D, Q, NV, false>(ub, sa, sb, sops->fBT, sops->sBT, sops->BT, ops.fix, e, node, active, sx + E * NV, NV);
	if (active)   // ubar = V^T ubar_g
#pragma unroll
		for (int k = 0; k < NV; ++k)
			A.ubar[((size_t)v * NV + k) * N + node] = ub[k];
}

}  // namespace dgpu

namespace dgpu {

// Objective J = sum over the listed faces of the integral of pressure on side 0 (sum_i w_f J_f p(W_L)), and the
// cotangent of side 0's trace, w_f J_f dp/dW, written into wbar (whose other entries the caller zeroes).
template <int D, int NF, int NV>
__global__ void __launch_bounds__(256)
tp_objective_kernel(const TPParams P, const int* __restrict__ faces, int n_obj, double* contrib, double* wbar)
{
	if constexpr (NV != D + 2) {
		return;   // pressure is defined for the Euler equations only (dgpu_set_objective_faces refuses others)
	} else {
	const int gid = blockIdx.x * blockDim.x + threadIdx.x;
	if (gid >= n_obj * NF)
		return;
	const int f = faces[gid / NF], i = gid % NF;
	const double* tL = P.traces + (size_t)(2 * f) * NV * NF;
	const double sc = P.fgeo[((size_t)f * (D + 1) + D) * NF + i];
	const double rho = tL[i], E = tL[(D + 1) * NF + i];
	const double rho_inv = recip(rho);
	double V2 = 0.0, u[D];
#pragma unroll
	for (int k = 0; k < D; ++k) {
		u[k] = tL[(1 + k) * NF + i] * rho_inv;
		V2 += u[k] * u[k];
	}
	const double p = kGm1 * (E - 0.5 * rho * V2);
	contrib[gid] = sc * p;
	double* w = wbar + (size_t)(2 * f) * NV * NF;
	w[i] = sc * kGm1 * 0.5 * V2;                       // dp/drho
#pragma unroll
	for (int k = 0; k < D; ++k)
		w[(1 + k) * NF + i] = -sc * kGm1 * u[k];         // dp/dm_k
	w[(D + 1) * NF + i] = sc * kGm1;                   // dp/dE
	}
}

// out = a x + b y + c z (z may be null), elementwise over n doubles.
static __global__ void __launch_bounds__(256)
lincomb_kernel(size_t n, double a, const double* x, double b, const double* y, double c, const double* z,
               double* out)
{
	const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n)
		return;
	double s = a * x[i] + b * y[i];
	if (z)
		s += c * z[i];
	out[i] = s;
}

}  // namespace dgpu
