// Dense-operator residual kernels for the non-tensor-product 3D volumes (TET, WEDGE, PYR) of a batched mesh.
//
// These volumes carry the caller's dense reference operators, as the reference applies its op_std operators with
// one small GEMM per volume (operator_T.c:96-156): s_vc = cv0_vs_vc s (constructor_sol_vc_interp,
// compute_volume_rlhs_T.c:277-285), the contravariant Euler flux at the cubature nodes, rhs = sum_j cv1_j^T
// (w fr_j) (compute_rhs_v_dg_like_T, compute_volume_rlhs_T.c:166-177), face traces cv0_vs_fc s at the face's
// canonical nodes, rhs -= cv0_vs_fc^T (w_f J_f F*) per face (compute_rhs_f_dg_like_T, compute_face_rlhs_T.c:
// 297-310) and M^-1 (scale_rhs_by_m_inv_std, solve_dg.c:265-272). Volumes are affine (constant J), so
// M^-1 = M_ref^-1 / J with M_ref = cv0^T diag(w) cv0 inverted once on the host. A group with a curved volume (J
// varying over the cubature nodes) keeps every volume's own M^-1 instead (dense_minv_kernel).
//
// One CTA handles E volumes of one group; every phase maps one output row of one volume (all variables) to one thread, or
// to up to eight consecutive lanes that share its terms when the CTA has threads to spare (fix_split_for), reading the
// operators through the L1 cache (they are shared by every CTA of the group) and the volume's state and fluxes from shared
// memory. The state stays in coefficient space between stages.
//
// The contractions run in block fixed point (dgpu_fix.cuh): as FP64 sums they were chains of 35 to 400 operations of 64
// cycles each, which bounded these kernels at every size. The blocks are one volume's values of one variable. A volume
// whose blocks leave the fixed-point range (Inf, NaN, huge values) takes FP64 loops in the same phases.
#pragma once

#include "dgpu_batched.cuh"

namespace dgpu {

struct DSmem {
	// doubles per element: state (NV n_vs), fluxes (D NV n_vc), for a factorised WEDGE the partial sums of the
	// sum-factorised contractions (factors of at most 32 terms, for fix_line's accumulators), and two sets of block exponents; the lift keeps the face terms, its rhs and the state
	static __host__ __device__ int vol(int nv, int n_vs, int n_vc) { return nv * n_vs + 3 * nv * n_vc + nv + 1; }
	static __host__ __device__ int prism_tmp(int nv, int n_tvs, int n_tvc, int n_lvs, int n_lvc)
	{
		return nv * (2 * n_lvs * n_tvc + n_lvc * n_tvs);
	}
	static __host__ __device__ int lift_faces(int nv, int n_lf, int nff_max) { return nv * n_lf * nff_max; }
	static __host__ __device__ int lift(int nv, int n_vs, int n_lf, int nff_max)
	{
		return 2 * nv * n_vs + 2 + lift_faces(nv, n_lf, nff_max) + nv + 1;
	}
};

// ---- blocks: len values of each of NV variables, contiguous per variable, at doubles `off` of an element ----
// Their largest exponents into the element's ints at double xo, from int `slot`; one warp per (element, variable).
template <int NV>
__device__ __forceinline__ void blk_max(double* smem, int PER_E, int n_here, int off, int len, int xo, int slot)
{
	const int lane = threadIdx.x & 31;
	for (int p = threadIdx.x >> 5; p < n_here * NV; p += blockDim.x >> 5) {
		const int e = p / NV, k = p % NV;
		const double* x = smem + e * PER_E + off + k * len;
		int m = 0;
		for (int i = lane; i < len; i += 32)
			m = max(m, fix_exponent(x[i]));
		m = __reduce_max_sync(0xffffffffu, m);
		if (lane == 0)
			reinterpret_cast<int*>(smem + e * PER_E + xo)[slot + k] = m;
	}
}

// Whether all of the element's blocks of the set are in range, as blk_pack left it.
template <int NV>
__device__ __forceinline__ bool blk_ok(const double* smem, int PER_E, int e, int xo, int slot)
{
	return reinterpret_cast<const int*>(smem + e * PER_E + xo)[2 * NV + (slot ? 1 : 0)] != 0;
}

// The values packed in place, for the elements in range (none unless fix: DGroup::fix), and the flags of blk_ok.
template <int NV>
__device__ __forceinline__ void blk_pack(double* smem, int PER_E, int n_here, bool fix, int off, int len, int xo, int slot)
{
	const int lane = threadIdx.x & 31;
	for (int p = threadIdx.x >> 5; p < n_here * NV; p += blockDim.x >> 5) {
		const int e = p / NV, k = p % NV;
		int* xe = reinterpret_cast<int*>(smem + e * PER_E + xo);
		bool ok = fix;
#pragma unroll
		for (int j = 0; j < NV; ++j)
			ok = ok && fix_in_range(xe[slot + j]);
		if (k == 0 && lane == 0)
			xe[2 * NV + (slot ? 1 : 0)] = ok;
		if (!ok)
			continue;
		const int eb = fix_block(xe[slot + k]);
		double* x = smem + e * PER_E + off + k * len;
		for (int i = lane; i < len; i += 32)
			reinterpret_cast<int2*>(x)[i] = fix_pack(x[i], eb);
	}
}

__device__ __forceinline__ FixW ldg_fix(const FixW* p)
{
	const int2 w = __ldg(reinterpret_cast<const int2*>(p));
	return FixW{w.x, w.y};
}

// acc[k] += sum_i op[i so] x[k len + i sx], i < n: sums of any length. Their operators are scaled to |W| < 2^61 and
// sum |W| <= 2^66 (a row of hundreds of terms scaled by its sum alone would keep too few bits of each entry); the low
// accumulator is folded into the high one every 16 products, exactly, which keeps it below 2^63, and leaves
// 0 <= m < 2^30.
// The terms are dealt to `split` lanes, of which this one is the part-th; fix_join adds the lanes' sums up (integers, so
// the result does not depend on the split).
template <int NV>
__device__ __forceinline__ void fix_dot(FixAcc* acc, const FixW* op, int so, const int2* x, int len, int sx, int n,
                                        int part = 0, int split = 1)
{
	for (int i0 = part; i0 < n; i0 += 16 * split) {
		const int i1 = min(n, i0 + 16 * split);
#pragma unroll 4
		for (int i = i0; i < i1; i += split) {
			const FixW w = ldg_fix(op + (long long)i * so);
#pragma unroll
			for (int k = 0; k < NV; ++k)
				fix_mac(acc[k], w, x[k * len + i * sx]);
		}
#pragma unroll
		for (int k = 0; k < NV; ++k) {
			acc[k].h += acc[k].m >> 30;
			acc[k].m &= (1ll << 30) - 1;
		}
	}
}

// Lanes of one output: split consecutive ones (a power of two). All lanes of the warp must call it.
template <int NV>
__device__ __forceinline__ void fix_join(FixAcc* acc, int split)
{
	for (int o = split >> 1; o > 0; o >>= 1)
#pragma unroll
		for (int k = 0; k < NV; ++k) {
			acc[k].h += __shfl_xor_sync(0xffffffffu, acc[k].h, o);
			acc[k].m += __shfl_xor_sync(0xffffffffu, acc[k].m, o);
		}
	if (split > 1)
#pragma unroll
		for (int k = 0; k < NV; ++k) {
			acc[k].h += acc[k].m >> 30;
			acc[k].m &= (1ll << 30) - 1;
		}
}

// Lanes per output for n outputs of `terms` products each, on a CTA of 256 threads: as many as the idle threads allow while
// a lane keeps 8 products.
__device__ __forceinline__ int fix_split_for(int n, int terms)
{
	int sp = 1;
	while (sp < 8 && n * sp * 2 <= 256 && terms >= 16 * sp)
		sp *= 2;
	return sp;
}

// The value of a folded sum (block eb, operator scale s).
__device__ __forceinline__ double fix_dot_value(const FixAcc& a, int eb, int s)
{
	const bool big = (unsigned long long)(a.h + (1ll << 58)) >> 59;   // |a.h| >= 2^58: its own unit is fine enough
	const long long r = big ? a.h : a.h * 8 + (a.m >> 27);
	return fix_to_double(r, fix_scale(eb, s) + (big ? 3 : 0));
}

// Traces of the CTA's volumes (state in shared memory at 0) at each face's canonical nodes.
template <int NV>
__device__ void dtraces(const BParams& P, const DGroup& G, int e0, int n_here, const double* smem, int PER_E, int xo)
{
	const int nvs = G.n_vs, nfm = G.nff_max, n = n_here * G.n_lf * nfm, sp = fix_split_for(n, nvs);
	for (int t0 = threadIdx.x & ~31; t0 < n * sp; t0 += blockDim.x) {   // whole warps: fix_join is a warp operation
		const int t = t0 + (threadIdx.x & 31), it = t / sp;
		const int i = it % nfm, el = it / nfm, lf = el % G.n_lf, e = min(el / G.n_lf, n_here - 1);
		const long long v = G.elem0 + e0 + e;
		const int4 fd = P.elf[v * kMaxLf + lf];
		const long long fb = P.fbase[fd.x];
		const int nff = (int)(P.fbase[fd.x + 1] - fb);
		const bool here = it < n && i < nff;
		const long long o = G.fop_off[(lf * G.n_ord + fd.w) * (kQMax + 1) + fd.z];
		const double* su = smem + e * PER_E;
		const bool ok = blk_ok<NV>(smem, PER_E, e, xo, 0);
		double W[NV];
		FixAcc acc[NV];
#pragma unroll
		for (int k = 0; k < NV; ++k)
			acc[k] = {0, 0};
		if (here && ok)
			fix_dot<NV>(acc, G.xfT + o + i, nff, reinterpret_cast<const int2*>(su), nvs, 1, nvs, t % sp, sp);
		fix_join<NV>(acc, sp);
		if (!here || t % sp)
			continue;
		if (ok) {
			const int* eb = reinterpret_cast<const int*>(su + xo);
#pragma unroll
			for (int k = 0; k < NV; ++k)
				W[k] = fix_dot_value(acc[k], fix_block(eb[k]), G.s_f);
		} else {
			const double* op = G.fops + o + (long long)i * nvs;
#pragma unroll 1
			for (int k = 0; k < NV; ++k) {
				double s = 0.0;
				for (int m = 0; m < nvs; ++m)
					s = fma(__ldg(op + m), su[k * nvs + m], s);
				W[k] = s;
			}
		}
		double* dst = P.traces + 2 * NV * fb + (long long)fd.y * NV * nff;
#pragma unroll
		for (int k = 0; k < NV; ++k)
			dst[k * nff + i] = W[k];
	}
}

// The w-weighted contravariant flux of W at cubature node r of an element, into its flux block [k][j][r] (doubles).
template <int D, int NV, int PDE>
__device__ __forceinline__ void dflux(const BParams& P, const DGroup& G, int elem, int r, const double* W, double* sf)
{
	const int nvc = G.n_vc;
	double g[D * D], fr[D][NV];
	const double* gm = P.gmet + G.gmet_off + (long long)elem * D * D * nvc;
#pragma unroll
	for (int c = 0; c < D * D; ++c)
		g[c] = gm[c * nvc + r];
	tp_flux<D, NV, PDE>(P.b_adv, W, g, fr);
#pragma unroll
	for (int j = 0; j < D; ++j)
#pragma unroll
		for (int k = 0; k < NV; ++k)
			sf[(k * D + j) * nvc + r] = fr[j][k];
}

// One output of a sum-factorised WEDGE pass as limbs at the pass's block exponent: sum |W| <= 2^62.
__device__ __forceinline__ int2 fix_line(const FixW* op, int so, const int2* x, int sx, int n)
{
	FixAcc a = {0, 0};
#pragma unroll 4
	for (int i = 0; i < n; ++i)
		fix_mac(a, ldg_fix(op + i * so), x[i * sx]);
	return fix_limbs(a.h * 4 + (a.m >> 28));
}

// Sum-factorised volume term of a WEDGE volume whose operators are Kronecker products of TRI and LINE factors
// (basis index c * n_tvs + t, node index rz * n_tvc + rt): s_vc in two passes (TRI, then LINE), the flux, then
// sum_j cv1_j^T (w fr_j) as LINE then TRI passes for x and y and TRI then LINE for z. Elements in range only.
template <int D, int NV, int PDE>
__device__ void dvol_prism_phases(const BParams& P, const DGroup& G, int e0, int n_here, double* smem, int PER_E, int xo)
{
	const int nvs = G.n_vs, nvc = G.n_vc, ntv = G.n_tvs, ntc = G.n_tvc, nlv = G.n_lvs, nlc = G.n_lvc;
	const int so = NV * nvs, to = so + D * NV * nvc;   // flux block, partial sums
	// 1a: v[k][c][rt] = sum_t T0[rt][t] s[k][c][t]
	for (int it = threadIdx.x; it < n_here * NV * nlv * ntc; it += blockDim.x) {
		const int e = it / (NV * nlv * ntc), rem = it % (NV * nlv * ntc);
		const int k = rem / (nlv * ntc), c = (rem / ntc) % nlv, rt = rem % ntc;
		const int2* su = reinterpret_cast<const int2*>(smem + e * PER_E) + k * nvs + c * ntv;
		if (blk_ok<NV>(smem, PER_E, e, xo, 0))
			reinterpret_cast<int2*>(smem + e * PER_E + to)[rem] = fix_line(G.xt0T + rt, ntc, su, 1, ntv);
	}
	__syncthreads();
	// 1b: W[k] at (rz, rt) = sum_c L0[rz][c] v[k][c][rt]; the flux there
	for (int it = threadIdx.x; it < n_here * nvc; it += blockDim.x) {
		const int e = it / nvc, r = it % nvc, rz = r / ntc, rt = r % ntc;
		if (!blk_ok<NV>(smem, PER_E, e, xo, 0))
			continue;
		const int2* v = reinterpret_cast<const int2*>(smem + e * PER_E + to) + rt;
		const int* eb = reinterpret_cast<const int*>(smem + e * PER_E + xo);
		double W[NV];
#pragma unroll
		for (int k = 0; k < NV; ++k) {
			FixAcc a = {0, 0};
			for (int c = 0; c < nlv; ++c)
				fix_mac(a, ldg_fix(G.xl0 + rz * nlv + c), v[(k * nlv + c) * ntc]);
			W[k] = fix_to_double(fix_sum(a), fix_scale(fix_block(eb[k]) + 62 - G.s_t0, G.s_l0));
		}
		dflux<D, NV, PDE>(P, G, e0 + e, r, W, smem + e * PER_E + so);
	}
	__syncthreads();
	blk_max<NV>(smem, PER_E, n_here, so, D * nvc, xo, NV);
	__syncthreads();
	blk_pack<NV>(smem, PER_E, n_here, G.fix, so, D * nvc, xo, NV);
	__syncthreads();
	// 2a: gx, gy[k][c][rt] = sum_rz L0[rz][c] f_x,y[k][rz][rt];  h[k][rz][t] = sum_rt T0[rt][t] f_z[k][rz][rt]
	const int gsz = NV * nlv * ntc;
	for (int it = threadIdx.x; it < n_here * gsz; it += blockDim.x) {
		const int e = it / gsz, rem = it % gsz;
		const int k = rem / (nlv * ntc), c = (rem / ntc) % nlv, rt = rem % ntc;
		if (!blk_ok<NV>(smem, PER_E, e, xo, NV))
			continue;
		const int2* f = reinterpret_cast<const int2*>(smem + e * PER_E + so) + k * D * nvc + rt;
		int2* tmp = reinterpret_cast<int2*>(smem + e * PER_E + to);
		tmp[rem] = fix_line(G.xl0 + c, nlv, f, ntc, nlc);
		tmp[gsz + rem] = fix_line(G.xl0 + c, nlv, f + nvc, ntc, nlc);
	}
	const int hsz = NV * nlc * ntv;
	for (int it = threadIdx.x; it < n_here * hsz; it += blockDim.x) {
		const int e = it / hsz, rem = it % hsz;
		const int k = rem / (nlc * ntv), rz = (rem / ntv) % nlc, t = rem % ntv;
		if (!blk_ok<NV>(smem, PER_E, e, xo, NV))
			continue;
		const int2* fz = reinterpret_cast<const int2*>(smem + e * PER_E + so) + (k * D + 2) * nvc + rz * ntc;
		reinterpret_cast<int2*>(smem + e * PER_E + to)[2 * gsz + rem] = fix_line(G.xt0 + t, ntv, fz, 1, ntc);
	}
	__syncthreads();
	// 2b: vol[k][c][t] = sum_rt (T1x[rt][t] gx[k][c][rt] + T1y[rt][t] gy[k][c][rt]) + sum_rz L1[rz][c] h[k][rz][t]
	for (int it = threadIdx.x; it < n_here * NV * nvs; it += blockDim.x) {
		const int e = it / (NV * nvs), rem = it % (NV * nvs), k = rem / nvs, c = (rem % nvs) / ntv, t = rem % ntv;
		if (!blk_ok<NV>(smem, PER_E, e, xo, NV) || !blk_ok<NV>(smem, PER_E, e, xo, 0))
			continue;
		const int2* tmp = reinterpret_cast<const int2*>(smem + e * PER_E + to);
		const int2* gx = tmp + (k * nlv + c) * ntc;
		FixAcc a = {0, 0};
		fix_dot<1>(&a, G.xt1 + t, ntv, gx, 0, 1, ntc);
		fix_dot<1>(&a, G.xt1 + (long long)ntc * ntv + t, ntv, gx + gsz, 0, 1, ntc);
		fix_dot<1>(&a, G.xl1 + c, nlv, tmp + 2 * gsz + k * nlc * ntv + t, 0, ntv, nlc);
		const int eb = fix_block(reinterpret_cast<const int*>(smem + e * PER_E + xo)[NV + k]);
		P.vol_gl[G.state_off + (long long)(e0 + e) * NV * nvs + rem] =
			fix_dot_value(a, eb + 62 - G.s_l0, G.s_t1);
	}
}

// The volume term of the elements that are out of range, in FP64 (dense operators; the state is read from memory and
// the fluxes go through the element's flux block).
template <int D, int NV, int PDE>
__device__ __noinline__ void dvol_fp64(const BParams& P, const DGroup& G, int e0, int n_here,
                                       const double* __restrict__ ublk, double* smem, int PER_E, int xo)
{
	const int nvs = G.n_vs, nvc = G.n_vc, so = NV * nvs;
	__syncthreads();
	for (int it = threadIdx.x; it < n_here * nvc; it += blockDim.x) {
		const int e = it / nvc, r = it % nvc;
		if (blk_ok<NV>(smem, PER_E, e, xo, 0) && blk_ok<NV>(smem, PER_E, e, xo, NV))
			continue;
		const double* row = G.cv0 + (long long)r * nvs;
		double W[NV];
#pragma unroll 1
		for (int k = 0; k < NV; ++k) {
			const double* su = ublk + ((long long)e * NV + k) * nvs;
			double s = 0.0;
			for (int m = 0; m < nvs; ++m)
				s = fma(__ldg(row + m), su[m], s);
			W[k] = s;
		}
		dflux<D, NV, PDE>(P, G, e0 + e, r, W, smem + e * PER_E + so);
	}
	__syncthreads();
	for (int it = threadIdx.x; it < n_here * NV * nvs; it += blockDim.x) {
		const int e = it / (NV * nvs), rem = it % (NV * nvs), k = rem / nvs, m = rem % nvs;
		if (blk_ok<NV>(smem, PER_E, e, xo, 0) && blk_ok<NV>(smem, PER_E, e, xo, NV))
			continue;
		const double* f = smem + e * PER_E + so + k * D * nvc;
		double acc = 0.0;
		for (int jr = 0; jr < D * nvc; ++jr)
			acc = fma(__ldg(G.cv1 + (long long)jr * nvs + m), f[jr], acc);
		P.vol_gl[G.state_off + (long long)(e0 + e) * NV * nvs + rem] = acc;
	}
}

// ---------------------------------------------------------------------------------------------------------------
// Volume term (coefficient space) + face traces at the canonical face nodes
// ---------------------------------------------------------------------------------------------------------------
template <int D, int NV, int PDE>
__device__ void dvol_body(const BParams& P, const DGroup& G, int e0, int E, const double* __restrict__ u,
                          double* smem)
{
	const int nvs = G.n_vs, nvc = G.n_vc;
	const int PER_E = G.vol_per_e, xo = PER_E - NV - 1, so = NV * nvs;
	const int n_here = min(E, G.n_vol - e0);
	const double* ublk = u + G.state_off + (long long)e0 * NV * nvs;
	for (int i = threadIdx.x; i < n_here * NV * nvs; i += blockDim.x) {
		const int e = i / (NV * nvs), r = i % (NV * nvs);
		smem[e * PER_E + r] = ublk[i];
	}
	__syncthreads();
	blk_max<NV>(smem, PER_E, n_here, 0, nvs, xo, 0);
	__syncthreads();
	blk_pack<NV>(smem, PER_E, n_here, G.fix, 0, nvs, xo, 0);
	__syncthreads();
	if (G.prism) {
		dvol_prism_phases<D, NV, PDE>(P, G, e0, n_here, smem, PER_E, xo);
	} else {
		// phase 1: state at the cubature nodes, contravariant flux, w-weighted (w is folded into the metrics)
		const int n1 = n_here * nvc, s1 = fix_split_for(n1, nvs);
		for (int t0 = threadIdx.x & ~31; t0 < n1 * s1; t0 += blockDim.x) {
			const int t = t0 + (threadIdx.x & 31), it = min(t / s1, n1 - 1), e = it / nvc, r = it % nvc;
			const bool ok = blk_ok<NV>(smem, PER_E, e, xo, 0);
			FixAcc acc[NV];
			double W[NV];
#pragma unroll
			for (int k = 0; k < NV; ++k)
				acc[k] = {0, 0};
			if (ok)
				fix_dot<NV>(acc, G.xcv0 + r, nvc, reinterpret_cast<const int2*>(smem + e * PER_E), nvs, 1, nvs, t % s1, s1);
			fix_join<NV>(acc, s1);
			if (!ok || t % s1 || t >= n1 * s1)
				continue;
			const int* eb = reinterpret_cast<const int*>(smem + e * PER_E + xo);
#pragma unroll
			for (int k = 0; k < NV; ++k)
				W[k] = fix_dot_value(acc[k], fix_block(eb[k]), G.s_cv0);
			dflux<D, NV, PDE>(P, G, e0 + e, r, W, smem + e * PER_E + so);
		}
		__syncthreads();
		blk_max<NV>(smem, PER_E, n_here, so, D * nvc, xo, NV);
		__syncthreads();
		blk_pack<NV>(smem, PER_E, n_here, G.fix, so, D * nvc, xo, NV);
		__syncthreads();
		// phase 2: rhs_vol[k][m] = sum_j sum_r cv1_j[r][m] sf[k][j][r]
		const int n2 = n_here * nvs, s2 = fix_split_for(n2, D * nvc);
		for (int t0 = threadIdx.x & ~31; t0 < n2 * s2; t0 += blockDim.x) {
			const int t = t0 + (threadIdx.x & 31), it = min(t / s2, n2 - 1), e = it / nvs, m = it % nvs;
			const bool ok = blk_ok<NV>(smem, PER_E, e, xo, NV);
			FixAcc acc[NV];
#pragma unroll
			for (int k = 0; k < NV; ++k)
				acc[k] = {0, 0};
			if (ok)
				fix_dot<NV>(acc, G.xcv1 + m, nvs, reinterpret_cast<const int2*>(smem + e * PER_E + so), D * nvc, 1, D * nvc,
				            t % s2, s2);
			fix_join<NV>(acc, s2);
			if (!ok || t % s2 || t >= n2 * s2)
				continue;
			const int* eb = reinterpret_cast<const int*>(smem + e * PER_E + xo) + NV;
			double* out = P.vol_gl + G.state_off + (long long)(e0 + e) * NV * nvs + m;
#pragma unroll
			for (int k = 0; k < NV; ++k)
				out[k * nvs] = fix_dot_value(acc[k], fix_block(eb[k]), G.s_cv1);
		}
	}
	dtraces<NV>(P, G, e0, n_here, smem, PER_E, xo);
	bool bad = false;
	for (int e = threadIdx.x; e < n_here; e += blockDim.x)
		bad = bad || !blk_ok<NV>(smem, PER_E, e, xo, 0) || !blk_ok<NV>(smem, PER_E, e, xo, NV);
	if (__syncthreads_or(bad)) {   // also: shared memory is reused by the next tile
		dvol_fp64<D, NV, PDE>(P, G, e0, n_here, ublk, smem, PER_E, xo);
		__syncthreads();
	}
}

// ---------------------------------------------------------------------------------------------------------------
// Lift of the face fluxes, M^-1, then the residual or the RK stage (coefficient space)
// ---------------------------------------------------------------------------------------------------------------
// enforce_positivity_highorder (solve.c:187-233) on the new states of the CTA's elements (kept at NV n_vs of
// each element's block): Bezier coefficients b = ccSB0 s per variable; one thread per element converts them to
// primitive variables, checks the average (error flag below EPS_PHYS) and minimum of the density, then of the
// pressure, and when a minimum is below EPS_PHYS blends every variable toward its average (correct_coef,
// :356-374) before the pressure check; corrected elements get s = ccBS0 b back in conserved variables. Elements
// that need no correction keep s (the reference's round trip is the identity up to rounding).
template <int NV>
__device__ void dense_positivity(const BParams& P, const DGroup& G, int e0, int n_here, const RkArgs& rk,
                                 double* smem, int PER_E)
{
	constexpr double kEpsPhys = 1e-13;   // definitions_tol.h EPS_PHYS
	constexpr int D = NV - 2;
	const int nvs = G.n_vs;
	__syncthreads();
	// FP32 pre-filter: per element the scales S_k = max |s_k| (into the free rhs half), then every Bezier node's
	// density and pressure lower bounds from FP32 coefficients and their rounding bound pos_err S_k; an element
	// whose bounds all clear the thresholds (which lie far above EPS_PHYS) needs no correction and is skipped
	// the state in FP32 once (after the NV scales in the free rhs half), so the n_vs^2 products run on FP32 only
	for (int it = threadIdx.x; it < n_here * NV * nvs; it += blockDim.x) {
		const int e = it / (NV * nvs), rem = it % (NV * nvs);
		reinterpret_cast<float*>(smem + e * PER_E + NV)[rem] = (float)smem[e * PER_E + NV * nvs + rem];
	}
	for (int p = threadIdx.x >> 5; p < n_here * NV; p += blockDim.x >> 5) {   // one warp per (volume, variable)
		const int e = p / NV, k = p % NV, lane = threadIdx.x & 31;
		const double* sv = smem + e * PER_E + NV * nvs + k * nvs;
		// the largest |s|'s high word, and the next one up: a bound of it within 2^-20 (NaN fails the tests below)
		int mx = 0;
		for (int a = lane; a < nvs; a += 32)
			mx = max(mx, __double2hiint(sv[a]) & 0x7fffffff);
		mx = __reduce_max_sync(0xffffffffu, mx);
		if (lane == 0) {
			smem[e * PER_E + k] = __hiloint2double(mx + 1, 0);
			if (k == 0)
				smem[e * PER_E + 2 * NV * nvs + 1] = 0.0;   // unsafe flag
		}
	}
	__syncthreads();
	for (int it = threadIdx.x; it < n_here * nvs; it += blockDim.x) {
		const int e = it / nvs, m = it % nvs;
		const float* sf = reinterpret_cast<const float*>(smem + e * PER_E + NV);
		const float* row = G.ccSB0f + (long long)m * nvs;
		float bk[NV];
#pragma unroll
		for (int k = 0; k < NV; ++k) {
			float acc = 0.f;
			for (int a = 0; a < nvs; ++a)
				acc += __ldg(row + a) * sf[k * nvs + a];
			bk[k] = acc;
		}
		const float err = G.pos_err;
		const float s_rho = (float)smem[e * PER_E];
		const float rho_lo = bk[0] - err * s_rho;
		bool safe = rho_lo > 1e-6f * s_rho + 1e-12f;
		if (safe) {
			float m2 = 0.f;
#pragma unroll
			for (int d = 0; d < D; ++d) {
				const float mk = fabsf(bk[1 + d]) + err * (float)smem[e * PER_E + 1 + d];
				m2 += mk * mk;
			}
			const float E_lo = bk[D + 1] - err * (float)smem[e * PER_E + D + 1];
			const float ke = 0.5f * m2 / rho_lo;
			const float p_lo = 0.4f * (E_lo - ke);
			safe = p_lo > 1e-5f * (fabsf(E_lo) + ke) + 1e-12f;   // NaN/Inf fail this test and go to the exact path
		}
		if (!safe)
			smem[e * PER_E + 2 * NV * nvs + 1] = 1.0;
	}
	__syncthreads();
	for (int it = threadIdx.x; it < n_here * NV * nvs; it += blockDim.x) {
		const int e = it / (NV * nvs), rem = it % (NV * nvs), k = rem / nvs, m = rem % nvs;
		if (smem[e * PER_E + 2 * NV * nvs + 1] == 0.0)
			continue;
		const double* sv = smem + e * PER_E + NV * nvs + k * nvs;
		const double* row = G.ccSB0 + (long long)m * nvs;
		double b = 0.0;
		for (int a = 0; a < nvs; ++a)
			b += __ldg(row + a) * sv[a];
		smem[e * PER_E + rem] = b;
	}
	__syncthreads();
	// conserved -> primitive (rho, u, p) at every Bezier node (convert_variables 'c' -> 'p'), node-parallel
	for (int it = threadIdx.x; it < n_here * nvs; it += blockDim.x) {
		const int e = it / nvs, m = it % nvs;
		if (smem[e * PER_E + 2 * NV * nvs + 1] == 0.0)
			continue;
		double* b = smem + e * PER_E;
		const double rho = b[m];
		double V2 = 0.0;
#pragma unroll
		for (int d = 0; d < D; ++d) {
			const double u = b[(1 + d) * nvs + m] / rho;
			b[(1 + d) * nvs + m] = u;
			V2 += u * u;
		}
		b[(D + 1) * nvs + m] = kGm1 * (b[(D + 1) * nvs + m] - 0.5 * rho * V2);
	}
	__syncthreads();
	// per element: the rhs half of its block now holds b, the other half s; the flag takes a spare scalar slot
	for (int e = threadIdx.x; e < n_here; e += blockDim.x) {
		double* b = smem + e * PER_E;
		bool corrected = false;
		if (smem[e * PER_E + 2 * NV * nvs + 1] == 0.0) {   // cleared by the pre-filter
			smem[e * PER_E + 2 * NV * nvs] = 0.0;
			continue;
		}
		for (int vr = 0; vr < NV; vr += NV - 1) {
			double avg = 0.0, mn = b[vr * nvs];
			for (int m = 0; m < nvs; ++m) {
				avg += b[vr * nvs + m];
				mn = fmin(mn, b[vr * nvs + m]);
			}
			avg /= nvs;
			if (!(avg >= kEpsPhys)) {
				atomicExch(P.err_flag, 1);
				break;
			}
			if (mn < kEpsPhys) {
				const double th = fmax(0.0, fmin(1.0, (avg - kEpsPhys) / (avg - mn)));
				for (int k = 0; k < NV; ++k) {
					double a = 0.0;
					for (int m = 0; m < nvs; ++m)
						a += b[k * nvs + m];
					a /= nvs;
					if ((k == 0 || k == NV - 1) && a < kEpsPhys)
						a = kEpsPhys;
					for (int m = 0; m < nvs; ++m)
						b[k * nvs + m] = th * b[k * nvs + m] + (1.0 - th) * a;
				}
				corrected = true;
			}
		}
		if (corrected)
			atomicAdd(P.n_corr, 1ull);
		smem[e * PER_E + 2 * NV * nvs] = corrected ? 1.0 : 0.0;
	}
	__syncthreads();
	// primitive -> conserved on the corrected elements, node-parallel
	for (int it = threadIdx.x; it < n_here * nvs; it += blockDim.x) {
		const int e = it / nvs, m = it % nvs;
		if (smem[e * PER_E + 2 * NV * nvs] == 0.0)
			continue;
		double* b = smem + e * PER_E;
		const double rho = b[m];
		double V2 = 0.0;
#pragma unroll
		for (int d = 0; d < D; ++d) {
			const double u = b[(1 + d) * nvs + m];
			V2 += u * u;
			b[(1 + d) * nvs + m] = rho * u;
		}
		b[(D + 1) * nvs + m] = b[(D + 1) * nvs + m] / kGm1 + 0.5 * rho * V2;
	}
	__syncthreads();
	for (int it = threadIdx.x; it < n_here * NV * nvs; it += blockDim.x) {
		const int e = it / (NV * nvs), rem = it % (NV * nvs), k = rem / nvs, m = rem % nvs;
		if (smem[e * PER_E + 2 * NV * nvs] == 0.0)
			continue;
		const double* bv = smem + e * PER_E + k * nvs;
		const double* row = G.ccBS0 + (long long)m * nvs;
		double s = 0.0;
		for (int a = 0; a < nvs; ++a)
			s += __ldg(row + a) * bv[a];
		rk.u[G.state_off + (long long)(e0 + e) * NV * nvs + rem] = s;
	}
}

template <int NV, int MODE>
__device__ void dlift_body(const BParams& P, const DGroup& G, int e0, int E, const RkArgs& rk, double* smem)
{
	const int nvs = G.n_vs, nfm = G.nff_max, nft = G.n_lf * nfm;
	const int PER_E = G.lift_per_e, fo = 2 * NV * nvs + 2, xo = PER_E - NV - 1;   // face terms, block exponents
	const int n_here = min(E, G.n_vol - e0);
	const int lane = threadIdx.x & 31;
	// phase 1: rhs = vol - sum_lf sgn cv0_fc^T nnf. The signed face terms of one variable (side 0: rhs -= ; side 1:
	// rhs -= (-nnf)) make a block; the volume term (with the source's cv0^T diag(w J) s), whose high modes are far larger
	// than a face term, is added in FP64.
	for (int p = threadIdx.x >> 5; p < n_here * NV; p += blockDim.x >> 5) {
		const int e = p / NV, k = p % NV;
		const long long v = G.elem0 + e0 + e, so = G.state_off + (long long)(e0 + e) * NV * nvs + k * nvs;
		double* x = smem + e * PER_E + fo + k * nft;
		double* r = smem + e * PER_E + k * nvs;
		int m = 0;
		for (int i = lane; i < nvs; i += 32)
			r[i] = P.source ? add(P.vol_gl[so + i], P.source[so + i]) : P.vol_gl[so + i];
		for (int it = lane; it < nft; it += 32) {
			const int lf = it / nfm, i = it % nfm;
			const int4 fd = P.elf[v * kMaxLf + lf];
			const long long fb = P.fbase[fd.x];
			const int nff = (int)(P.fbase[fd.x + 1] - fb);
			double t = 0.0;
			if (i < nff) {
				// side 1 reads the face flux (side 0's node order) at its own nodes through the inverse permutation
				t = P.nnf[NV * fb + (long long)k * nff + ((fd.y == 1 && P.nc_inv) ? P.nc_inv[fb + i] : i)];
				t = fd.y == 0 ? -t : t;
			}
			x[it] = t;
			m = max(m, fix_exponent(t));
		}
		m = __reduce_max_sync(0xffffffffu, m);
		if (lane == 0)
			reinterpret_cast<int*>(smem + e * PER_E + xo)[k] = m;
	}
	__syncthreads();
	blk_pack<NV>(smem, PER_E, n_here, G.fix, fo, nft, xo, 0);
	__syncthreads();
	const int n1 = n_here * nvs, s1 = fix_split_for(n1, nfm);
	for (int t0 = threadIdx.x & ~31; t0 < n1 * s1; t0 += blockDim.x) {   // whole warps: fix_join is a warp operation
		const int t = t0 + (threadIdx.x & 31), it = min(t / s1, n1 - 1), e = it / nvs, m = it % nvs;
		const long long v = G.elem0 + e0 + e;
		double* r = smem + e * PER_E + m;
		const bool ok = blk_ok<NV>(smem, PER_E, e, xo, 0);
		FixAcc acc[NV];
#pragma unroll
		for (int k = 0; k < NV; ++k)
			acc[k] = {0, 0};
		if (ok)
			for (int lf = 0; lf < G.n_lf; ++lf) {
				const int4 fd = P.elf[v * kMaxLf + lf];
				const int nff = (int)(P.fbase[fd.x + 1] - P.fbase[fd.x]);
				fix_dot<NV>(acc, G.xfL + G.fop_off[(lf * G.n_ord + fd.w) * (kQMax + 1) + fd.z] + m, nvs,
				            reinterpret_cast<const int2*>(smem + e * PER_E + fo) + lf * nfm, nft, 1, nff, t % s1, s1);
			}
		fix_join<NV>(acc, s1);
		if (t % s1 || t >= n1 * s1)
			continue;
		if (ok) {
			const int* eb = reinterpret_cast<const int*>(smem + e * PER_E + xo);
#pragma unroll
			for (int k = 0; k < NV; ++k)
				r[k * nvs] = add(r[k * nvs], fix_dot_value(acc[k], fix_block(eb[k]), G.s_f));
		} else {
#pragma unroll 1
			for (int k = 0; k < NV; ++k) {
				double acc = r[k * nvs];
				for (int lf = 0; lf < G.n_lf; ++lf) {
					const int4 fd = P.elf[v * kMaxLf + lf];
					const int nff = (int)(P.fbase[fd.x + 1] - P.fbase[fd.x]);
					const double* op = G.fops + G.fop_off[(lf * G.n_ord + fd.w) * (kQMax + 1) + fd.z] + m;
					const double* x = smem + e * PER_E + fo + k * nft + lf * nfm;
					for (int i = 0; i < nff; ++i)
						acc = fma(__ldg(op + (long long)i * nvs), x[i], acc);
				}
				r[k * nvs] = acc;
			}
		}
	}
	__syncthreads();
	// phase 2: R = M^-1 rhs, then the stage: 1/J alone for an orthonormal basis, a product with M_ref^-1 before it
	// otherwise (in fixed point, on the rhs packed in place), each volume's own M^-1 in a curved group
	const bool dense_m = !G.minv_vol && !G.minv_identity;
	if (dense_m) {
		blk_max<NV>(smem, PER_E, n_here, 0, nvs, xo, NV);
		__syncthreads();
		blk_pack<NV>(smem, PER_E, n_here, G.fix, 0, nvs, xo, NV);
		__syncthreads();
	}
	unsigned long long mx = 0ull;
	for (int it = threadIdx.x; it < n_here * NV * nvs; it += blockDim.x) {
		const int e = it / (NV * nvs), rem = it % (NV * nvs), k = rem / nvs, m = rem % nvs;
		const double* sr = smem + e * PER_E + k * nvs;
		double R;
		if (!dense_m || !blk_ok<NV>(smem, PER_E, e, xo, NV)) {
			if (G.minv_identity && !G.minv_vol) {
				R = sr[m];
			} else {
				const double* row = G.minv_vol ? G.minv_vol + ((long long)(e0 + e) * nvs + m) * nvs
				                               : G.minv + (long long)m * nvs;
				R = 0.0;
				for (int a = 0; a < nvs; ++a)
					R = fma(__ldg(row + a), sr[a], R);
			}
		} else {
			FixAcc acc = {0, 0};
			fix_dot<1>(&acc, G.xminv + m, nvs, reinterpret_cast<const int2*>(sr), 0, 1, nvs);
			R = fix_dot_value(acc, fix_block(reinterpret_cast<const int*>(smem + e * PER_E + xo)[NV + k]), G.s_minv);
		}
		if (!G.minv_vol)
			R = mul(R, G.inv_J[e0 + e]);
		const long long o = G.state_off + (long long)(e0 + e) * NV * nvs + rem;
		if (MODE == kModeRhs || rk.want_max) {
			const unsigned long long bits = abs_bits(R);
			mx = bits > mx ? bits : mx;
		}
		if constexpr (MODE == kModeRhs) {
			rk.rhs[o] = R;
		} else {
			const double s = rk.u[o];
			double sn;
			if (rk.stage == 0)
				rk.u0[o] = s;
			sn = rk_update(rk.stage, s, rk.stage == 0 ? s : rk.u0[o], rk.dt, R);
			rk.u[o] = sn;
			smem[e * PER_E + NV * nvs + rem] = sn;   // kept for the positivity check
		}
	}
	if constexpr (MODE != kModeRhs) {
		if (rk.positivity && G.ccSB0)
			dense_positivity<NV>(P, G, e0, n_here, rk, smem, PER_E);
	}
	if (MODE == kModeRhs || rk.want_max) {
#pragma unroll
		for (int off = 16; off > 0; off >>= 1) {
			const unsigned long long o = __shfl_xor_sync(0xffffffffu, mx, off);
			mx = o > mx ? o : mx;
		}
		if ((threadIdx.x & 31) == 0 && mx && P.max_bits)
			atomicMax(P.max_bits, mx);
	}
	__syncthreads();   // shared memory is reused by the next tile
}

// ---------------------------------------------------------------------------------------------------------------
// Kernels: one launch per dense group, and the bodies the fused kernels dispatch to
// ---------------------------------------------------------------------------------------------------------------

// Shared memory of dense_minv_kernel: the augmented matrix [M | I] (n_vs x 2 n_vs) and one column.
__host__ __device__ inline size_t dense_minv_smem(int nvs) { return (size_t)(2 * nvs * nvs + nvs) * sizeof(double); }

// M^-1 of one curved volume per CTA (set-up, once per context): M = cv0^T diag(w J) cv0 (constructor_mass_T,
// volume_solver_T.c:115-145) formed in shared memory, then inverted by Gauss-Jordan elimination. M is symmetric
// positive definite, so the pivots (Schur complements) are positive and no row exchange is needed.
// cv0: n_vc x n_vs; wJ: per volume n_vc values w_n J_n; minv: per volume n_vs x n_vs row-major.
static __global__ void __launch_bounds__(128) dense_minv_kernel(const double* __restrict__ cv0,
                                                         const double* __restrict__ wJ, int nvs, int nvc,
                                                         int n_vol, double* __restrict__ minv)
{
	extern __shared__ double sm[];
	const int v = blockIdx.x;
	if (v >= n_vol)
		return;
	const int w2 = 2 * nvs;
	double* A = sm;                // [M | I]
	double* col = sm + nvs * w2;   // column k before elimination step k
	const double* wj = wJ + (long long)v * nvc;
	for (int it = threadIdx.x; it < nvs * nvs; it += blockDim.x) {
		const int a = it / nvs, b = it % nvs;
		double s = 0.0;
		for (int r = 0; r < nvc; ++r)
			s += cv0[(long long)r * nvs + a] * wj[r] * cv0[(long long)r * nvs + b];
		A[a * w2 + b] = s;
		A[a * w2 + nvs + b] = (a == b) ? 1.0 : 0.0;
	}
	__syncthreads();
	for (int k = 0; k < nvs; ++k) {
		for (int i = threadIdx.x; i < nvs; i += blockDim.x)
			col[i] = A[i * w2 + k];
		__syncthreads();
		const double inv_p = 1.0 / col[k];
		for (int j = threadIdx.x; j < w2; j += blockDim.x)
			A[k * w2 + j] *= inv_p;
		__syncthreads();
		for (int it = threadIdx.x; it < nvs * w2; it += blockDim.x) {
			const int i = it / w2, j = it - i * w2;
			if (i != k)
				A[i * w2 + j] -= col[i] * A[k * w2 + j];
		}
		__syncthreads();
	}
	for (int it = threadIdx.x; it < nvs * nvs; it += blockDim.x) {
		const int a = it / nvs, b = it % nvs;
		minv[((long long)v * nvs + a) * nvs + b] = A[a * w2 + nvs + b];
	}
}

// Three CTAs per SM for both dense kernels (80 registers): they wait on chains of operator loads and integer products, at
// 14 to 19 % of the issue slots with two. Mixed types 18^3, 4 steps: 14.65 -> 13.07 ms; TRI/QUAD 96^2: 4.38 -> 4.34 ms.
template <int D, int NV, int PDE>
__global__ void __launch_bounds__(256, 3) dvol_group_kernel(const BParams P, int g, const double* __restrict__ u)
{
	extern __shared__ double smem[];
	const DGroup G = P.dgroups[g];
	if (blockIdx.x == 0 && threadIdx.x == 0 && P.max_bits && G.elem0 == 0)
		*P.max_bits = 0ull;
	dvol_body<D, NV, PDE>(P, G, blockIdx.x * G.E, G.E, u, smem);
}

template <int NV, int MODE>
__global__ void __launch_bounds__(256, 3) dlift_group_kernel(const BParams P, int g, const RkArgs rk)
{
	extern __shared__ double smem[];
	const DGroup G = P.dgroups[g];
	dlift_body<NV, MODE>(P, G, blockIdx.x * G.E, G.E, rk, smem);
}

// Fused persistent kernels: a CTA walks the tile list (grid-stride) and dispatches on the tile's group: a TP
// group's order (its operator set is reloaded into shared memory when the group changes) or a dense group.
// Each (group kind, q) body is called as a separate function (not inlined): the kernel then needs the registers
// of its largest body, not those of all bodies inlined into one switch.
template <int D, int Q, int NV, int PDE, bool GLL_IN>
__device__ __noinline__ void bvol_tile(const BParams& P, const BatchOps* sops, const BGroup& G, int e0, int E,
                                       const double* __restrict__ u, double* base)
{
	bvol_body<D, Q, NV, PDE, GLL_IN>(P, sops, G, e0, E, u, base);
}

template <int D, int NV, int PDE>
__device__ __noinline__ void dvol_tile(const BParams& P, const DGroup& G, int e0, int E, const double* __restrict__ u,
                                       double* base)
{
	dvol_body<D, NV, PDE>(P, G, e0, E, u, base);
}

template <int D, int Q, int NV, int MODE>
__device__ __noinline__ void blift_tile(const BParams& P, const BatchOps* sops, const BGroup& G, int e0, int E,
                                        const RkArgs& rk, double* base)
{
	blift_body<D, Q, NV, MODE>(P, sops, G, e0, E, rk, base);
}

template <int NV, int MODE>
__device__ __noinline__ void dlift_tile(const BParams& P, const DGroup& G, int e0, int E, const RkArgs& rk,
                                        double* base)
{
	dlift_body<NV, MODE>(P, G, e0, E, rk, base);
}

template <int D, int NV, int PDE, bool GLL_IN>
__global__ void __launch_bounds__(256, 2) bvol_fused_kernel(const BParams P, const BTile* tiles, int n_tiles,
                                                           const double* __restrict__ u)
{
	extern __shared__ double smem[];
	BatchOps* sops = reinterpret_cast<BatchOps*>(smem);
	double* base = smem + sizeof(BatchOps) / 8;
	if (blockIdx.x == 0 && threadIdx.x == 0 && P.max_bits)
		*P.max_bits = 0ull;
	int cur = -1;
	for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
		const BTile tl = tiles[t];
		if (tl.group >= P.n_groups) {
			const DGroup G = P.dgroups[tl.group - P.n_groups];
			dvol_tile<D, NV, PDE>(P, G, tl.e0, G.E_fused, u, base);
			continue;
		}
		if (tl.group != cur) {
			__syncthreads();
			load_batch_ops(sops, &P.ops[tl.group]);
			cur = tl.group;
			__syncthreads();
		}
		const BGroup G = P.groups[tl.group];
		const int E = (int)(blockDim.x / (D == 2 ? G.q * G.q : G.q * G.q * G.q));
		switch (G.q) {
		case 2: bvol_tile<D, 2, NV, PDE, GLL_IN>(P, sops, G, tl.e0, E, u, base); break;
		case 3: bvol_tile<D, 3, NV, PDE, GLL_IN>(P, sops, G, tl.e0, E, u, base); break;
		case 4: bvol_tile<D, 4, NV, PDE, GLL_IN>(P, sops, G, tl.e0, E, u, base); break;
		default: bvol_tile<D, 5, NV, PDE, GLL_IN>(P, sops, G, tl.e0, E, u, base); break;
		}
	}
}

// The RK stages that reduce no max |rhs| run the TP tiles without that path (as the per-group form does), capped at
// 4 CTAs per SM; the dense tiles take the want_max flag at run time.
template <int D, int NV, int MODE>
__global__ void __launch_bounds__(256, BLiftOccupancy<MODE>::value) blift_fused_kernel(const BParams P,
                                                                                     const BTile* tiles, int n_tiles,
                                                                                     const RkArgs rk)
{
	constexpr int DMODE = (MODE == kModeRkGlNoMax) ? kModeRkGl : MODE;
	extern __shared__ double smem[];
	BatchOps* sops = reinterpret_cast<BatchOps*>(smem);
	double* base = smem + sizeof(BatchOps) / 8;
	int cur = -1;
	for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
		const BTile tl = tiles[t];
		if (tl.group >= P.n_groups) {
			const DGroup G = P.dgroups[tl.group - P.n_groups];
			dlift_tile<NV, DMODE>(P, G, tl.e0, G.E_fused, rk, base);
			continue;
		}
		if (tl.group != cur) {
			__syncthreads();
			load_batch_ops(sops, &P.ops[tl.group]);
			cur = tl.group;
			__syncthreads();
		}
		const BGroup G = P.groups[tl.group];
		const int E = (int)(blockDim.x / (D == 2 ? G.q * G.q : G.q * G.q * G.q));
		switch (G.q) {
		case 2: blift_tile<D, 2, NV, MODE>(P, sops, G, tl.e0, E, rk, base); break;
		case 3: blift_tile<D, 3, NV, MODE>(P, sops, G, tl.e0, E, rk, base); break;
		case 4: blift_tile<D, 4, NV, MODE>(P, sops, G, tl.e0, E, rk, base); break;
		default: blift_tile<D, 5, NV, MODE>(P, sops, G, tl.e0, E, rk, base); break;
		}
	}
}

// ---------------------------------------------------------------------------------------------------------------
// Form 3: a whole stage in one cooperative persistent launch (volume tiles | face nodes | lift tiles)
// ---------------------------------------------------------------------------------------------------------------
// Barrier between the phases over every CTA of the grid. The launch is cooperative, so all CTAs are resident at
// once and the barrier completes; each wait is still bounded (limit_ns of the global timer, 2 s by default): a CTA
// that gives up sets *err = kErrBarrier and returns false, and the kernel then ends. bar[0] counts the arrivals of
// the current barrier and bar[1] its generation; the host zeroes both before each launch.
constexpr int kErrBarrier = 2;
constexpr unsigned long long kBarrierLimitNs = 2000000000ull;

__device__ __forceinline__ unsigned long long global_ns()
{
	unsigned long long t;
	asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
	return t;
}

__device__ __forceinline__ bool grid_barrier(unsigned* bar, int* err, unsigned long long limit_ns)
{
	__shared__ int ok;
	__syncthreads();   // the CTA's writes of this phase are issued
	if (threadIdx.x == 0) {
		ok = 1;
		volatile unsigned* gen = bar + 1;
		const unsigned g = *gen;   // cannot advance before this CTA arrives
		__threadfence();           // this CTA's writes are visible before its arrival
		if (atomicAdd(bar, 1u) == gridDim.x - 1) {
			atomicExch(bar, 0u);
			__threadfence();
			atomicAdd(bar + 1, 1u);
		} else {
			const unsigned long long t0 = global_ns();
			while (*gen == g) {
				if (global_ns() - t0 > limit_ns) {
					atomicExch(err, kErrBarrier);
					ok = 0;
					break;
				}
				__nanosleep(64);
			}
		}
		__threadfence();
	}
	__syncthreads();
	return ok != 0;
}

// The three phases of the fused form in one kernel: the volume tiles, every face node of the q_f-sorted list, the
// lift tiles; grid barriers in between. One occupancy serves all three phases: the shared memory of the largest
// tile (the q = 2 volume tile in 3D, 82 KB) already limits it to 2 CTAs per SM, so registers are capped there too
// (a 64-register cap would only add spills).
template <int D, int NV, int PDE, int FLUX, int MODE, bool GLL_IN>
__global__ void __launch_bounds__(256, 2)
bstage_kernel(const BParams P, const BTile* __restrict__ tiles, int n_tiles, const double* __restrict__ u,
              const int* __restrict__ node_face, long long n_nodes, const RkArgs rk, unsigned* bar,
              unsigned long long limit_ns)
{
	constexpr int DMODE = (MODE == kModeRkGlNoMax) ? kModeRkGl : MODE;
	extern __shared__ double smem[];
	BatchOps* sops = reinterpret_cast<BatchOps*>(smem);
	double* base = smem + sizeof(BatchOps) / 8;
	if (blockIdx.x == 0 && threadIdx.x == 0 && P.max_bits)
		*P.max_bits = 0ull;
	int cur = -1;
	for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
		const BTile tl = tiles[t];
		if (tl.group >= P.n_groups) {
			const DGroup G = P.dgroups[tl.group - P.n_groups];
			dvol_tile<D, NV, PDE>(P, G, tl.e0, G.E_fused, u, base);
			continue;
		}
		if (tl.group != cur) {
			__syncthreads();
			load_batch_ops(sops, &P.ops[tl.group]);
			cur = tl.group;
			__syncthreads();
		}
		const BGroup G = P.groups[tl.group];
		const int E = (int)(blockDim.x / (D == 2 ? G.q * G.q : G.q * G.q * G.q));
		switch (G.q) {
		case 2: bvol_tile<D, 2, NV, PDE, GLL_IN>(P, sops, G, tl.e0, E, u, base); break;
		case 3: bvol_tile<D, 3, NV, PDE, GLL_IN>(P, sops, G, tl.e0, E, u, base); break;
		case 4: bvol_tile<D, 4, NV, PDE, GLL_IN>(P, sops, G, tl.e0, E, u, base); break;
		default: bvol_tile<D, 5, NV, PDE, GLL_IN>(P, sops, G, tl.e0, E, u, base); break;
		}
	}
	if (!grid_barrier(bar, P.err_flag, limit_ns))
		return;
	for (long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x; gid < n_nodes;
	     gid += (long long)gridDim.x * blockDim.x) {
		const int f = node_face[gid];
		const long long fb = P.fbase[f];
		bface_node_rt<D, NV, PDE, FLUX>(P, f, (int)(gid - fb), (int)(P.fbase[f + 1] - fb));
	}
	if (!grid_barrier(bar, P.err_flag, limit_ns))
		return;
	for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
		const BTile tl = tiles[t];
		if (tl.group >= P.n_groups) {
			const DGroup G = P.dgroups[tl.group - P.n_groups];
			dlift_tile<NV, DMODE>(P, G, tl.e0, G.E_fused, rk, base);
			continue;
		}
		if (tl.group != cur) {
			__syncthreads();
			load_batch_ops(sops, &P.ops[tl.group]);
			cur = tl.group;
			__syncthreads();
		}
		const BGroup G = P.groups[tl.group];
		const int E = (int)(blockDim.x / (D == 2 ? G.q * G.q : G.q * G.q * G.q));
		switch (G.q) {
		case 2: blift_tile<D, 2, NV, MODE>(P, sops, G, tl.e0, E, rk, base); break;
		case 3: blift_tile<D, 3, NV, MODE>(P, sops, G, tl.e0, E, rk, base); break;
		case 4: blift_tile<D, 4, NV, MODE>(P, sops, G, tl.e0, E, rk, base); break;
		default: blift_tile<D, 5, NV, MODE>(P, sops, G, tl.e0, E, rk, base); break;
		}
	}
}

// Face numerical flux at every node of the faces in [node_lo, node_hi) of the q_f-sorted face node list.
template <int D, int NV, int PDE, int FLUX>
__global__ void __launch_bounds__(256) bface_nodes_kernel(const BParams P, const int* __restrict__ node_face,
                                                           long long node_lo, long long node_hi)
{
	for (long long gid = node_lo + (long long)blockIdx.x * blockDim.x + threadIdx.x; gid < node_hi;
	     gid += (long long)gridDim.x * blockDim.x) {
		const int f = node_face[gid];
		const long long fb = P.fbase[f];
		bface_node_rt<D, NV, PDE, FLUX>(P, f, (int)(gid - fb), (int)(P.fbase[f + 1] - fb));
	}
}

}  // namespace dgpu
