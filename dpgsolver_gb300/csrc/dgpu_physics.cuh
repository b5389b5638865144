// Flux physics for the explicit DG residual, FP64, as device inline functions.
//
// Each function states the reference routine it computes. The GB300 FP64 pipe (2 DFMA per cycle per SM) is the
// binding resource, so the numerical fluxes are written to need as few FP64 instructions as the same
// mathematics allows: each side's state is reduced once (one reciprocal of the density), the normal flux is
// formed from the normal velocity instead of contracting the full physical flux with the normal, and
// divisions by the same quantity are replaced by one reciprocal. These regroupings change rounding only.
#pragma once

#include <cuda_runtime.h>
#include <math.h>

#include <type_traits>

#include "dgpu_dual.cuh"

namespace dgpu {

using ::fabs;
using ::pow;

// 1/x, sqrt(x), a/b and the comparison of magnitudes of the flux routines' scalar type: doubles on the integer pipe
// (dgpu_fix.cuh), Dual in dgpu_dual.cuh.
__device__ __forceinline__ double recip(double x) { return fix_rcp(x); }
__device__ __forceinline__ double root(double x) { return fix_sqrt(x); }
__device__ __forceinline__ double quot(double a, double b) { return fix_div(a, b); }
template <typename A, typename B>
__device__ __forceinline__ auto quot(const A& a, const B& b)
{
	return a / b;
}

// The same where S: the argument is known to be a positive normal number with a normal result.
template <bool S, typename T>
__device__ __forceinline__ T recipx(const T& x)
{
	if constexpr (S && std::is_same<T, double>::value)
		return fix_rcp<false>(x);
	else
		return recip(x);
}
template <bool S, typename T>
__device__ __forceinline__ T rootx(const T& x)
{
	if constexpr (S && std::is_same<T, double>::value)
		return fix_sqrt<false>(x);
	else
		return root(x);
}

constexpr double kGamma = 1.4;          // definitions_physics.h:23
constexpr double kGm1 = 0.4;            // definitions_physics.h:24
constexpr double kEpsPhys = 1.0e-13;    // definitions_physics.h:30
constexpr double kEps = 1.0e-15;        // definitions_tol.h:23

enum Pde { kAdvection = 1, kEuler = 3, kNavierStokes = 4 };
enum Viscosity { kViscosityConstant = 101, kViscositySutherland = 102 };   // definitions_physics.h:34-36
enum NumFlux { kUpwind = 11, kRoePike = 31, kLaxFriedrichs = 32 };

// min_abs_real_T / max_abs_real_T (general/math_functions_T.c:222-236); T = double, or Dual for Jacobians.
template <typename T>
__device__ __forceinline__ T min_abs_real(const T& a, const T& b)
{
	T c = (fabs(a) < fabs(b) ? a : b);
	return (c < 0.0 ? -c : c);
}
template <typename T>
__device__ __forceinline__ T max_abs_real(const T& a, const T& b)
{
	T c = (fabs(a) > fabs(b) ? a : b);
	return (c < 0.0 ? -c : c);
}

// Products and sums with their rounding written out, so that every kernel a flux routine is inlined into (the launch
// forms of a batched mesh among them) rounds alike: mad is one fused operation, mul and add are never fused.
template <typename A, typename B, typename C>
__device__ __forceinline__ C mad(A a, B b, const C& c)
{
	return a * b + c;
}
__device__ __forceinline__ double mad(double a, double b, double c) { return __fma_rn(a, b, c); }
template <typename A, typename B>
__device__ __forceinline__ auto mul(A a, B b)
{
	return a * b;
}
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
// mul on the integer pipe (the same bits) where S: see fix_mul for what the factors must be.
template <bool S, typename A, typename B>
__device__ __forceinline__ auto mulx(A a, B b)
{
	if constexpr (S)
		return mul_fix(a, b);
	else
		return mul(a, b);
}
// The range in which mulx<true> may be used inside the flux routines: zero, or a magnitude of 2^-LO to 2^60, LO = 60 for
// densities, energies, viscosities and scalings, 150 for the components of vectors (momentum, normals, metric terms,
// gradients), which round-off leaves anywhere near zero. No product of a flux formed from such values leaves the normal
// range (the smallest, a velocity times a stress, stays above 2^-900).
template <int LO>
__device__ __forceinline__ bool mulx_range(double x)
{
	const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
	return h - ((1023u - LO) << 20) < ((60u + LO) << 20) || (h | (unsigned)__double2loint(x)) == 0u;
}
// A conserved state: density positive, every component in range.
template <int D, typename T>
__device__ __forceinline__ bool mulx_state(const T* W)
{
	bool ok = __double2hiint(value(W[0])) > 0 && mulx_range<60>(value(W[0])) && mulx_range<60>(value(W[D + 1]));
#pragma unroll
	for (int k = 0; k < D; ++k)
		ok = ok && mulx_range<150>(value(W[1 + k]));
	return ok;
}
template <int N>
__device__ __forceinline__ bool mulx_vector(const double* x)
{
	bool ok = true;
#pragma unroll
	for (int k = 0; k < N; ++k)
		ok = ok && mulx_range<150>(x[k]);
	return ok;
}
__device__ __forceinline__ bool positive(double x) { return __double2hiint(x) > 0 && __double2hiint(x) < 0x7ff00000; }

template <typename T>
__device__ __forceinline__ T add(const T& a, const T& b)
{
	return a + b;
}
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
template <typename T>
__device__ __forceinline__ T sub(const T& a, const T& b)
{
	return a - b;
}
__device__ __forceinline__ double sub(double a, double b) { return __dadd_rn(a, -b); }

__device__ __forceinline__ double min_abs_real(double a, double b) { return fabs(abs_less(a, b) ? a : b); }
__device__ __forceinline__ double max_abs_real(double a, double b) { return fabs(abs_less(b, a) ? a : b); }

// |a|, and the larger of two non-negative values (a NaN in a gives b).
template <typename T>
__device__ __forceinline__ T abs_real(const T& a)
{
	return a > 0.0 ? a : -a;
}
__device__ __forceinline__ double abs_real(double a) { return fabs(a); }
template <typename T>
__device__ __forceinline__ T larger(const T& a, const T& b)
{
	return a > b ? a : b;
}
__device__ __forceinline__ double larger(double a, double b) { return abs_less(b, a) ? a : b; }

// Contravariant volume flux at one cubature node for the Euler equations:
//   fr_j[eq] = sum_i g[j*D+i] f_i[eq]
// with f the physical flux of compute_Flux_T_euler / compute_Flux_euler_0 (flux_euler_T.c:71-143, 259-298)
// and g the metric terms (pre-multiplied by the cubature weight) of constructor_flux_ref_piece_T
// (compute_rlhs_T.c:71-110). The contraction is regrouped through the contravariant momentum
// M_j = sum_i g[j*D+i] m_i (the mass flux fr_j[0] itself) and velocity U_j = M_j / rho, and the pressure takes
// rho |u|^2 as |m|^2 / rho: the same sums with fewer FP64 operations.
// S: the lone products that mulx<S> takes off the FP64 pipe (the volume kernels' integer pipe is half full already).
template <int D, typename T = double, bool S = false>
__device__ __forceinline__ void euler_flux_ref(const T* W, const double* g, T (*fr)[D + 2])
{
	const T rho = W[0], E = W[D + 1];
	const T rho_inv = recipx<S>(rho);
	T m2 = mul(W[1], W[1]);
#pragma unroll
	for (int k = 1; k < D; ++k)
		m2 = mad(W[1 + k], W[1 + k], m2);
	const T p = mulx<S>(kGm1, mad(-0.5, mulx<S>(m2, rho_inv), E));
	const T Ep = add(E, p);
#pragma unroll
	for (int j = 0; j < D; ++j) {
		T M = mul(g[j * D], W[1]);
#pragma unroll
		for (int i = 1; i < D; ++i)
			M = mad(g[j * D + i], W[1 + i], M);
		const T U = mulx<S>(M, rho_inv);
		fr[j][0] = M;
#pragma unroll
		for (int m = 0; m < D; ++m)
			fr[j][1 + m] = mad(W[1 + m], U, mul(p, g[j * D + m]));
		fr[j][D + 1] = mulx<S>(Ep, U);
	}
}

// The FP64 form of the Roe-Pike flux, out of line and by value: it is rarely taken, and inlined beside the other form it
// would raise the registers of every face kernel (124 instead of 108).
template <int D>
struct FluxNode {
	double WL[D + 2], WR[D + 2], n[D], scale;
};
template <int D>
struct FluxValue {
	double F[D + 2];
};
template <int D>
__device__ __forceinline__ FluxNode<D> flux_node(const double* WL, const double* WR, const double* n, double scale)
{
	FluxNode<D> x;
#pragma unroll
	for (int k = 0; k < D + 2; ++k) {
		x.WL[k] = WL[k];
		x.WR[k] = WR[k];
	}
#pragma unroll
	for (int k = 0; k < D; ++k)
		x.n[k] = n[k];
	x.scale = scale;
	return x;
}

// One side of a face node for Lax-Friedrichs: m.n, the normal velocity Vn = m.n / rho, the pressure and the wave
// speed |V| + c, with rho |V|^2 formed as |m|^2 / rho (one reciprocal of the density, no velocity vector).
template <int D, typename T, bool S>
__device__ __forceinline__ void euler_side_lf(const T* W, const double* n, T& mn, T& Vn, T& p, T& lam)
{
	const T rho_inv = recipx<S>(W[0]);
	T m2 = mulx<S>(W[1], W[1]);
	mn = mulx<S>(n[0], W[1]);
#pragma unroll
	for (int k = 1; k < D; ++k) {
		m2 = mad(W[1 + k], W[1 + k], m2);
		mn = mad(n[k], W[1 + k], mn);
	}
	const T q = mulx<S>(m2, rho_inv);   // rho |V|^2
	Vn = mulx<S>(mn, rho_inv);
	p = mulx<S>(kGm1, mad(-0.5, q, W[D + 1]));
	lam = add(root(mulx<S>(q, rho_inv)), rootx<S>(mulx<S>(mulx<S>(kGamma, p), rho_inv)));   // p > 0: see below
}

// Lax-Friedrichs (compute_Numerical_Flux_T_euler_lax_friedrichs, numerical_flux_euler_T.c:60-327):
//   nF = 1/2 [ n.(F_L + F_R) + max(|V_L| + c_L, |V_R| + c_R) (W_L - W_R) ] x scale
// with n.F = (m.n, m Vn + p n, (E + p) Vn) of each side (compute_Flux_euler_0 contracted with n); the two sides'
// pressure terms share one product with n. scale (the face node's w J, or 1) is folded into the factor 1/2, which
// gives the same bits as scaling afterwards (the factor 1/2 is exact).
// Returns false when a pressure is not positive (S only: the products then meet NaN, which fix_mul does not take, and the
// speed of sound was formed without a check).
template <int D, typename T, bool S>
__device__ __forceinline__ bool num_flux_lf_impl(const T* WL, const T* WR, const double* n, T* nF, double scale)
{
	T mnL, VnL, pL, lamL, mnR, VnR, pR, lamR;
	euler_side_lf<D, T, S>(WL, n, mnL, VnL, pL, lamL);
	euler_side_lf<D, T, S>(WR, n, mnR, VnR, pR, lamR);
	if constexpr (S)
		if (!positive(value(pL)) || !positive(value(pR)))
			return false;
	const T maxV = larger(lamL, lamR);
	const double h = 0.5 * scale;
	const T pLR = add(pL, pR);
	nF[0] = mulx<S>(h, mad(maxV, sub(WL[0], WR[0]), add(mnL, mnR)));
#pragma unroll
	for (int k = 0; k < D; ++k)
		nF[1 + k] = mulx<S>(h, mad(maxV, sub(WL[1 + k], WR[1 + k]),
		                       mad(WL[1 + k], VnL, mad(WR[1 + k], VnR, mulx<S>(pLR, n[k])))));
	nF[D + 1] = mulx<S>(h, mad(maxV, sub(WL[D + 1], WR[D + 1]),
	                       mad(add(WL[D + 1], pL), VnL, mulx<S>(add(WR[D + 1], pR), VnR))));
	return true;
}

template <int D, typename T = double>
__device__ __forceinline__ void num_flux_lax_friedrichs(const T* WL, const T* WR, const double* n, T* nF,
                                                        double scale = 1.0)
{
	if (mulx_state<D>(WL) && mulx_state<D>(WR) && mulx_vector<D>(n) && mulx_range<60>(scale) &&
	    num_flux_lf_impl<D, T, true>(WL, WR, n, nF, scale))
		return;
	num_flux_lf_impl<D, T, false>(WL, WR, n, nF, scale);
}

// Roe-Pike with the entropy fix of Qu et al. 2015 (compute_Numerical_Flux_T_euler_roe_pike,
// numerical_flux_euler_T.c:470-778).
// scale (the face node's w J, or 1) is folded into the factor 1/2, which gives the same bits as scaling afterwards. Returns
// false when the squared speed of sound is not positive (S only).
template <int D, typename T, bool S>
__device__ __forceinline__ bool num_flux_roe_impl(const T* WL, const T* WR, const double* n, T* nF, double scale)
{
	const T rhoL = WL[0], rhoR = WR[0], EL = WL[D + 1], ER = WR[D + 1];
	const T rhoL_inv = recipx<S>(rhoL), rhoR_inv = recipx<S>(rhoR);
	T uL[D], uR[D], V2L, V2R, VnL, VnR;
#pragma unroll
	for (int k = 0; k < D; ++k) {
		uL[k] = mulx<S>(WL[1 + k], rhoL_inv);
		uR[k] = mulx<S>(WR[1 + k], rhoR_inv);
		V2L = k ? mad(uL[k], uL[k], V2L) : mulx<S>(uL[k], uL[k]);
		V2R = k ? mad(uR[k], uR[k], V2R) : mulx<S>(uR[k], uR[k]);
		VnL = k ? mad(n[k], uL[k], VnL) : mulx<S>(n[k], uL[k]);
		VnR = k ? mad(n[k], uR[k], VnR) : mulx<S>(n[k], uR[k]);
	}
	const T pL = mulx<S>(kGm1, mad(mulx<S>(-0.5, rhoL), V2L, EL)), HL = mulx<S>(add(EL, pL), rhoL_inv);
	const T pR = mulx<S>(kGm1, mad(mulx<S>(-0.5, rhoR), V2R, ER)), HR = mulx<S>(add(ER, pR), rhoR_inv);

	// Roe averages (divisions by r + 1 through one reciprocal)
	const T r = rootx<S>(mulx<S>(rhoR, rhoL_inv)), rP1_inv = recipx<S>(add(r, T(1.0))), rho = mulx<S>(r, rhoL);
	T u[D], Vn, V2;
#pragma unroll
	for (int k = 0; k < D; ++k) {
		u[k] = mulx<S>(mad(r, uR[k], uL[k]), rP1_inv);
		Vn = k ? mad(n[k], u[k], Vn) : mulx<S>(n[k], u[k]);
		V2 = k ? mad(u[k], u[k], V2) : mulx<S>(u[k], u[k]);
	}
	const T H = mulx<S>(mad(r, HR, HL), rP1_inv), c2 = mulx<S>(kGm1, mad(-0.5, V2, H)), c = rootx<S>(c2);   // c2 > 0, or returned below
	if constexpr (S)
		if (!positive(value(c2)))
			return false;
	const T c_inv = recipx<S>(c);
	const double h = 0.5 * scale;

	const T l1 = min_abs_real(sub(VnL, c), sub(Vn, c)), l5 = max_abs_real(add(VnR, c), add(Vn, c));
	const T l234 = abs_real(Vn);

	const T drho = sub(rhoR, rhoL), dE = sub(ER, EL), dp = sub(pR, pL), dVn = sub(VnR, VnL);
	const T lc1 = mad(0.5, add(l5, l1), -l234), lc2 = mulx<S>(0.5, sub(l5, l1));
	const T lc1_dp = mulx<S>(mulx<S>(lc1, dp), c_inv), lc2_dp = mulx<S>(mulx<S>(lc2, dp), c_inv);
	const T disInter1 = mulx<S>(mad(mulx<S>(lc2, rho), dVn, lc1_dp), c_inv);
	const T disInter2 = mad(mulx<S>(lc1, rho), dVn, lc2_dp);

	const T rhoVnL = mulx<S>(rhoL, VnL), rhoVnR = mulx<S>(rhoR, VnR), pLR = add(pL, pR);
	nF[0] = mulx<S>(h, sub(add(rhoVnL, rhoVnR), mad(l234, drho, disInter1)));
#pragma unroll
	for (int k = 0; k < D; ++k) {
		const T drhou = sub(WR[1 + k], WL[1 + k]);
		const T nFk = mad(rhoVnL, uL[k], mad(rhoVnR, uR[k], mulx<S>(n[k], pLR)));
		const T disk = mad(l234, drhou, mad(disInter1, u[k], mulx<S>(disInter2, n[k])));
		nF[1 + k] = mulx<S>(h, sub(nFk, disk));
	}
	nF[D + 1] = mulx<S>(h, sub(mad(VnL, add(EL, pL), mulx<S>(VnR, add(ER, pR))),
	                         mad(l234, dE, mad(disInter1, H, mulx<S>(disInter2, Vn)))));
	return true;
}

template <int D>
__device__ __noinline__ FluxValue<D> num_flux_roe_fp64(FluxNode<D> x)
{
	FluxValue<D> r;
	num_flux_roe_impl<D, double, false>(x.WL, x.WR, x.n, r.F, x.scale);
	return r;
}

template <int D, typename T = double>
__device__ __forceinline__ void num_flux_roe_pike(const T* WL, const T* WR, const double* n, T* nF, double scale = 1.0)
{
	if constexpr (std::is_same<T, double>::value) {
		if (!(mulx_state<D>(WL) && mulx_state<D>(WR) && mulx_vector<D>(n) && mulx_range<60>(scale) &&
		      num_flux_roe_impl<D, T, true>(WL, WR, n, nF, scale))) {
			const FluxValue<D> r = num_flux_roe_fp64<D>(flux_node<D>(WL, WR, n, scale));
#pragma unroll
			for (int k = 0; k < D + 2; ++k)
				nF[k] = r.F[k];
		}
	} else if (!(mulx_state<D>(WL) && mulx_state<D>(WR) && mulx_vector<D>(n) &&
	             num_flux_roe_impl<D, T, true>(WL, WR, n, nF, scale))) {
		num_flux_roe_impl<D, T, false>(WL, WR, n, nF, scale);
	}
}

// Upwind advection flux (compute_Numerical_Flux_T_advection_upwind, numerical_flux_advection_T.c:39-75).
template <int D>
__device__ __forceinline__ double num_flux_upwind(double uL, double uR, const double* n, const double* b)
{
	double b_dot_n = 0.0;
#pragma unroll
	for (int k = 0; k < D; ++k)
		b_dot_n += b[k] * n[k];
	return (b_dot_n > kEps ? b_dot_n * uL : b_dot_n * uR);
}

// ---- boundary values ----------------------------------------------------------------------------------------------
// BC codes after taking them modulo BC_STEP_SC (definitions_bc.h:33-64); set_function_pointers_num_flux_bc_advection
// and _euler (face_solver_T.c:203-275) select the boundary value by these.
constexpr int kBcStepSC = 10000;
enum BcCode {
	kBcRiemann = 101, kBcSlipWall = 102, kBcBackPressure = 103, kBcTotalTP = 104, kBcSupersonicIn = 105,
	kBcSupersonicOut = 106, kBcNoSlipAdiabatic = 111, kBcNoSlipDiabatic = 112, kBcNoSlipAllRotating = 113
};

// BC_Data (boundary_euler_T.c:44-49): the scalars the reference reads from the test case's input file.
struct BcData {
	double p_back;   // BC_BACKPRESSURE
	double t_total;  // BC_TOTAL_TP: total temperature, total pressure, specific gas constant
	double p_total;
	double r_s;
};

// True for the advection codes that take the upwind boundary value (inflow 1-3, outflow 11-13, upwind 41-46).
__host__ __device__ __forceinline__ bool bc_is_advection_upwind(int bc)
{
	return (bc >= 1 && bc <= 3) || (bc >= 11 && bc <= 13) || (bc >= 41 && bc <= 46);
}
__host__ __device__ __forceinline__ bool bc_is_euler(int bc)
{
	return bc >= kBcRiemann && bc <= kBcSupersonicOut;
}
// The boundary values the reference's Navier-Stokes takes (face_solver_T.c:277-300).
__host__ __device__ __forceinline__ bool bc_is_navier_stokes(int bc)
{
	return bc == kBcRiemann || bc == kBcSupersonicIn || bc == kBcSupersonicOut || bc == kBcNoSlipAdiabatic ||
	       bc == kBcNoSlipDiabatic || bc == kBcNoSlipAllRotating;
}

// Exterior state WR of an Euler boundary face node from the interior trace WL, the test case's solution at the node
// (ext, conserved: constructor_sol_bv) and the unit normal n (outward from the interior volume). bc is already
// reduced modulo kBcStepSC and is one of the four codes (the context validates them on creation).
//   kBcRiemann       constructor_Boundary_Value_T_euler_riemann (boundary_euler_T.c:99-180): the outgoing
//                    invariant Vn + 2c/(gamma-1) of the interior and the incoming one of the exterior give the
//                    normal velocity and speed of sound; entropy and tangential velocity come from the upwind side;
//                    supersonic faces take the upwind state whole;
//   kBcSlipWall      ..._euler_slipwall (:494-533): density and energy kept, momentum mirrored about the face;
//   kBcSupersonicIn  ..._euler_supersonic_inflow (:657-692): the exterior state;
//   kBcSupersonicOut ..._euler_supersonic_outflow (:705-745): the interior state;
//   kBcBackPressure  ..._euler_back_pressure (:772-866): the interior state where |V| >= c, else the interior
//                    velocity at pressure p_back and density gamma p_back / c^2;
//   kBcTotalTP       ..._euler_total_tp (:991-1120): the speed of sound from the interior's outgoing invariant and
//                    total enthalpy (the larger root of a quadratic), flow along the normal, temperature and
//                    pressure from the total values by the isentropic relations, density by the gas law.
template <int D, typename T>
__device__ __forceinline__ void euler_boundary_state(int bc, const T* WL, const double* ext, const double* n, T* WR,
                                                     const BcData& bd)
{
	constexpr int NV = D + 2;
	if (bc == kBcBackPressure || bc == kBcTotalTP) {
		const T rho_l = WL[0], rho_l_inv = recip(rho_l);
		T u_l[D], V2_l = 0.0, Vn_l = 0.0;
#pragma unroll
		for (int k = 0; k < D; ++k) {
			u_l[k] = WL[1 + k] * rho_l_inv;
			V2_l += u_l[k] * u_l[k];
			Vn_l += n[k] * u_l[k];
		}
		const T p_l = kGm1 * (WL[D + 1] - 0.5 * rho_l * V2_l);
		const T c2_l = kGamma * p_l * rho_l_inv;
		if (bc == kBcBackPressure) {
			if (!(root(V2_l) < root(c2_l))) {
#pragma unroll
				for (int k = 0; k < NV; ++k)
					WR[k] = WL[k];
			} else {
				const T rho_b = (kGamma * bd.p_back) / c2_l;
				WR[0] = rho_b;
#pragma unroll
				for (int k = 0; k < D; ++k)
					WR[1 + k] = u_l[k] * rho_b;
				WR[D + 1] = bd.p_back * (1.0 / kGm1) + 0.5 * rho_b * V2_l;
			}
			return;
		}
		const T H_l = (WL[D + 1] + p_l) * rho_l_inv;
		const T R_l = Vn_l + (2.0 / kGm1) * root(c2_l);
		constexpr double aQ = 1.0 + 2.0 / kGm1;
		const T bQ = -2.0 * R_l, cQ = 0.5 * kGm1 * (R_l * R_l - 2.0 * H_l);
		const T t1 = bQ * (-0.5 / aQ), t2 = root(bQ * bQ - 4.0 * aQ * cQ) * (0.5 / aQ);
		const T cM = t1 - t2, cP = t1 + t2;
		const T c = (cM > cP ? cM : cP);
		const T Vn = R_l - (2.0 / kGm1) * c;
		const T M = quot(Vn, c);
		const T Tb = quot(bd.t_total, 1.0 + 0.5 * kGm1 * M * M);
		const T iso = Tb * recip(bd.t_total);   // p / p_total is its 7/2 power (gamma = 7/5)
		const T p = bd.p_total * (iso * iso * iso * root(iso));
		const T rho = quot(p, bd.r_s * Tb);
		T V2 = 0.0;
		WR[0] = rho;
#pragma unroll
		for (int k = 0; k < D; ++k) {
			const T uk = Vn * n[k];
			V2 += uk * uk;
			WR[1 + k] = rho * uk;
		}
		WR[D + 1] = p * (1.0 / kGm1) + 0.5 * rho * V2;
		return;
	}
	if (bc == kBcSlipWall) {
		T rhoVn = 0.0;
#pragma unroll
		for (int k = 0; k < D; ++k)
			rhoVn += n[k] * WL[1 + k];
		WR[0] = WL[0];
#pragma unroll
		for (int k = 0; k < D; ++k)
			WR[1 + k] = WL[1 + k] - 2.0 * rhoVn * n[k];
		WR[D + 1] = WL[D + 1];
		return;
	}
	if (bc == kBcSupersonicIn) {
#pragma unroll
		for (int k = 0; k < NV; ++k)
			WR[k] = ext[k];
		return;
	}
	if (bc != kBcRiemann) {   // supersonic outflow
#pragma unroll
		for (int k = 0; k < NV; ++k)
			WR[k] = WL[k];
		return;
	}
	// Riemann: primitive variables of both sides
	const T rho_l = WL[0], rho_l_inv = recip(rho_l);
	T u_l[D], V2_l = 0.0, Vn_l = 0.0;
#pragma unroll
	for (int k = 0; k < D; ++k) {
		u_l[k] = WL[1 + k] * rho_l_inv;
		V2_l += u_l[k] * u_l[k];
		Vn_l += n[k] * u_l[k];
	}
	const T p_l = kGm1 * (WL[D + 1] - 0.5 * rho_l * V2_l);
	const double rho_r = ext[0];
	double u_r[D], V2_r = 0.0, Vn_r = 0.0;
#pragma unroll
	for (int k = 0; k < D; ++k) {
		u_r[k] = quot(ext[1 + k], rho_r);
		V2_r += u_r[k] * u_r[k];
		Vn_r += n[k] * u_r[k];
	}
	const double p_r = kGm1 * (ext[D + 1] - 0.5 * rho_r * V2_r);
	const T c_l = root(kGamma * p_l * rho_l_inv);
	const double c_r = root(quot(kGamma * p_r, rho_r));
	const T R_l = Vn_l + (2.0 / kGm1) * c_l;   // outgoing
	const T R_r = Vn_r - (2.0 / kGm1) * c_r;   // incoming
	const T Vn = 0.5 * (R_l + R_r), cc = 0.25 * kGm1 * (R_l - R_r);
	T rho, p, uvw[D];
	if (!(fabs(Vn) < fabs(cc))) {   // supersonic: the upwind side's state
		if (Vn < 0.0) {
			rho = rho_r;
			p = p_r;
#pragma unroll
			for (int k = 0; k < D; ++k)
				uvw[k] = u_r[k];
		} else {
			rho = rho_l;
			p = p_l;
#pragma unroll
			for (int k = 0; k < D; ++k)
				uvw[k] = u_l[k];
		}
	} else {                        // subsonic: entropy and tangential velocity from the upwind side
		// rho = (c^2 / (gamma s))^(1 / (gamma - 1)) with s = p / rho^gamma of the upwind side: for gamma = 7/5 that is
		// rho x^(5/2), x = c^2 rho / (gamma p) the ratio of the squared speeds of sound, which needs square roots only (a
		// pow is hundreds of FP64 operations, and the few warps at the boundary were half of a small mesh's face kernel).
		// The root of x is taken factor by factor: a negative pressure or density gives NaN, as its power does.
		const T c2g = (1.0 / kGamma) * cc * cc;
		if (Vn < 0.0) {
			const T t = quot(c2g, p_r), x = t * rho_r;
			rho = x * x * (root(t) * root(rho_r)) * rho_r;
#pragma unroll
			for (int k = 0; k < D; ++k)
				uvw[k] = Vn * n[k] + (u_r[k] - Vn_r * n[k]);
		} else {
			const T t = quot(c2g, p_l), x = t * rho_l;
			rho = x * x * (root(t) * root(rho_l)) * rho_l;
#pragma unroll
			for (int k = 0; k < D; ++k)
				uvw[k] = Vn * n[k] + (u_l[k] - Vn_l * n[k]);
		}
		p = c2g * rho;
	}
	T V2 = 0.0;
#pragma unroll
	for (int k = 0; k < D; ++k)
		V2 += uvw[k] * uvw[k];
	WR[0] = rho;
#pragma unroll
	for (int k = 0; k < D; ++k)
		WR[1 + k] = rho * uvw[k];
	WR[D + 1] = p * (1.0 / kGm1) + 0.5 * rho * V2;
}

// The boundary state out of line and by value (the exterior state in x.WR): few nodes take it, and its quotients and
// roots inlined beside a flux cost the interior nodes 4 % (Lax-Friedrichs face kernel at HEX 32^3 p3, which has no boundary:
// 127.7 us with it inlined before its quotients were rounded, 133.3 after, 122.4 out of line; the Roe-Pike residual of HEX 15^3 p4
// 311 us inlined, 302 out of line).
template <int D>
__device__ __noinline__ FluxValue<D> euler_boundary_call(int bc, FluxNode<D> x, BcData bd)
{
	FluxValue<D> r;
	euler_boundary_state<D, double>(bc, x.WL, x.WR, x.n, r.F, bd);
	return r;
}
template <int D, typename T>
__device__ __forceinline__ void euler_boundary(int bc, const T* WL, const double* ext, const double* n, T* WR, const BcData& bd)
{
	if constexpr (std::is_same<T, double>::value) {
		const FluxValue<D> r = euler_boundary_call<D>(bc, flux_node<D>(WL, ext, n, 0.0), bd);
#pragma unroll
		for (int k = 0; k < D + 2; ++k)
			WR[k] = r.F[k];
	} else {
		euler_boundary_state<D, T>(bc, WL, ext, n, WR, bd);
	}
}

// Exterior value of an advection boundary node (constructor_Boundary_Value_T_advection_upwind,
// boundary_advection_T.c:40-77): the exterior solution where b.n <= 0 (inflow), else the interior trace.
template <int D, typename T>
__device__ __forceinline__ T advection_boundary_value(const T& uL, double ext, const double* n, const double* b)
{
	double b_dot_n = 0.0;
#pragma unroll
	for (int k = 0; k < D; ++k)
		b_dot_n += b[k] * n[k];
	return b_dot_n <= 0.0 ? T(ext) : uL;
}

// ---- Navier-Stokes viscous flux -----------------------------------------------------------------------------------
// Viscous part of the Navier-Stokes flux at one node, subtracted from F[dir][eq] (the reference adds the negated
// viscous flux to the Euler flux: compute_Flux_12_T with compute_Flux_T_navier_stokes, flux_navier_stokes_T.c:175-284,
// 1005-1040). W: conserved state; G[dir][var]: its gradient. Velocity gradients (compute_duvw :708-720), stress
// tau = mu (grad u + grad u^T - 2/3 div u I) (compute_tau :776-799), scaled temperature gradient
// dTs = grad(E/rho) - 1/2 grad |u|^2 (compute_dTs :905-927), heat flux gamma/Pr mu dTs. mu: constant, or
// Sutherland's law mu = 0.08 mu_ref sqrt(T) / (1 + 112 / T), T = p / (rho r_s) (compute_mu_sutherland_T,
// solution_navier_stokes_T.c:246-256, solution_navier_stokes.h:31-32).
struct NsPhys {
	double mu, Pr, r_s;
	int viscosity;
	double wall_nf_E;   // BC_NOSLIP_DIABATIC: the wall's normal energy flux -mu Cp / Pr dTdn
};

// S: lone products on the integer pipe. The state and its gradient must then be in range (mulx_state, mulx_range).
template <int D, typename T, bool S = false>
__device__ __forceinline__ void ns_viscous_sub(const T* W, const T (*G)[D + 2], const NsPhys& ph, T (*F)[D + 2])
{
	const T rho = W[0], E = W[D + 1], rho_inv = recip(rho);
	T u[D], du[D][D];
#pragma unroll
	for (int k = 0; k < D; ++k)
		u[k] = mulx<S>(W[1 + k], rho_inv);
#pragma unroll
	for (int s = 0; s < D; ++s)
#pragma unroll
		for (int x = 0; x < D; ++x)
			du[s][x] = mulx<S>(rho_inv, mad(-G[x][0], u[s], G[x][1 + s]));
	T mu = ph.mu;
	if (ph.viscosity == kViscositySutherland) {
		T V2 = mul(u[0], u[0]);
#pragma unroll
		for (int k = 1; k < D; ++k)
			V2 = mad(u[k], u[k], V2);
		const T p = kGm1 * mad(mul(-0.5, rho), V2, E), Tt = p / (rho * ph.r_s);
		mu = 0.08 * ph.mu / (1.0 + 112.0 / Tt) * root(Tt);
	}
	T div = du[0][0];
#pragma unroll
	for (int k = 1; k < D; ++k)
		div = add(div, du[k][k]);
	T tau[D][D];
	const T mu2 = mul(mu, 2.0);
#pragma unroll
	for (int a = 0; a < D; ++a) {
		tau[a][a] = mul(mu2, mad(-1.0 / 3.0, div, du[a][a]));
#pragma unroll
		for (int b = 0; b < a; ++b)
			tau[a][b] = tau[b][a] = mul(mu, add(du[b][a], du[a][b]));
	}
	const T kappa = mul(kGamma / ph.Pr, mu), r2 = mulx<S>(rho_inv, rho_inv);
#pragma unroll
	for (int x = 0; x < D; ++x) {
		// dTs = grad(E / rho) - 1/2 grad |u|^2
		T dTs = mulx<S>(r2, mad(G[x][D + 1], rho, -mulx<S>(E, G[x][0])));
		T ut = mulx<S>(u[0], tau[x][0]);
#pragma unroll
		for (int k = 0; k < D; ++k) {
			dTs = mad(-u[k], du[k][x], dTs);
			if (k > 0)
				ut = mad(u[k], tau[x][k], ut);
		}
#pragma unroll
		for (int k = 0; k < D; ++k)
			F[x][1 + k] = sub(F[x][1 + k], tau[k][x]);
		F[x][D + 1] = sub(F[x][D + 1], mad(kappa, dTs, ut));
	}
}

// Both forms of ns_viscous_sub from zero: -F_v of a node. The FP64 form is out of line, by value: it is rarely taken.
template <int D>
struct NsNode {
	double W[D + 2], G[D][D + 2];
};
template <int D>
struct NsFlux {
	double F[D][D + 2];
};
template <int D>
__device__ __noinline__ NsFlux<D> ns_viscous_fp64(NsNode<D> x, NsPhys ph)
{
	NsFlux<D> r;
#pragma unroll
	for (int i = 0; i < D; ++i)
#pragma unroll
		for (int k = 0; k < D + 2; ++k)
			r.F[i][k] = 0.0;
	ns_viscous_sub<D, double>(x.W, x.G, ph, r.F);
	return r;
}
template <int D, typename T>
__device__ __forceinline__ void ns_viscous(const T* W, const T (*G)[D + 2], const NsPhys& ph, T (*F)[D + 2])
{
	if constexpr (std::is_same<T, double>::value) {
		// Sutherland's law gives NaN where the pressure is negative: it stays on the FP64 form
		if (!(mulx_state<D>(W) && mulx_vector<D * (D + 2)>(&G[0][0]) && ph.viscosity == kViscosityConstant &&
		      mulx_range<60>(ph.mu))) {
			NsNode<D> x;
#pragma unroll
			for (int k = 0; k < D + 2; ++k) {
				x.W[k] = W[k];
#pragma unroll
				for (int i = 0; i < D; ++i)
					x.G[i][k] = G[i][k];
			}
			const NsFlux<D> r = ns_viscous_fp64<D>(x, ph);
#pragma unroll
			for (int i = 0; i < D; ++i)
#pragma unroll
				for (int k = 0; k < D + 2; ++k)
					F[i][k] = r.F[i][k];
			return;
		}
	}
#pragma unroll
	for (int i = 0; i < D; ++i)
#pragma unroll
		for (int k = 0; k < D + 2; ++k)
			F[i][k] = T(0.0);
	ns_viscous_sub<D, T, std::is_same<T, double>::value>(W, G, ph, F);
}

// The contravariant Euler flux of a node, with mulx where its values allow.
template <int D>
__device__ __forceinline__ void euler_flux_node(const double* W, const double* g, double (*fr)[D + 2])
{
	if (mulx_state<D>(W) && mulx_vector<D * D>(g))
		euler_flux_ref<D, double, true>(W, g, fr);
	else
		euler_flux_ref<D>(W, g, fr);
}

}  // namespace dgpu
