// Block fixed-point contractions: FP64-accurate short dot products on the integer pipe.
//
// Why. The FP64 pipe of GB300 retires one warp instruction per scheduler every 64 cycles (measured: DFMA 62, DADD and
// DMUL 74 cycles at 1.92 GHz, conversions between double and integer or float 62, double to float 29), while a 32 x 32
// -> 64 bit multiply-add (IMAD.WIDE) takes 2, an integer add 1, a shift or a logic operation 2. An operator entry times
// a value as three wide multiply-adds is therefore ten times cheaper than one DFMA, as long as the operands' conversion
// is shared by several products. The contractions of the residual (1D derivative, interpolation, traces, lifting)
// are such products with constant operators.
//
// Representation. The values that enter one sum share a block exponent eb, the largest biased exponent among them
// (taken over one element and one variable, so that an element's result does not depend on its neighbours in the
// launch). A value v is held as the integer X = v 2^(1082 - eb), |X| < 2^60, rounded to a multiple of 4 and kept as
// two limbs, X = h 2^32 + 4 l with l balanced (|l| <= 2^29). An operator entry w is W = w 2^s = h 2^32 + 4 l likewise.
// sum X W then needs h h, h l and l h products only:
//   sum X W / 2^64 = a.h + a.m / 2^30,   a.h = sum hX hW,   a.m = sum (hW lX + lW hX).
// s is chosen on the host so that sum |W| <= 2^63 over every sum an operator enters (and |W| < 2^62), which bounds
// a.h by 2^59 and, for at most 32 terms, a.m by 2^62: neither accumulator can overflow.
//
// Accuracy. fix_pack truncates in its shift and then rounds to a multiple of 4: a value is held to less than 3 units, at most
// 3 2^-59 of its block's largest magnitude (exactly, where it lies at most 2^5 below it). An operator entry is rounded to 2 units of
// its own. The dropped l l products are at most 2^62 each, against a sum of up to 2^60 sum |W|: with the operators' rounding,
// 6 terms of 2^-62 of max |v| sum |w| at worst (2^-55.4 for the 15 terms of a derivative at p = 4), and typically, since both
// l are balanced and have no bias, a few 2^-60. FP64 arithmetic rounds every partial sum to 2^-53. The result is rounded
// once to FP64, to nearest.
//
// States. What lies far below its block's largest value keeps less than FP64's relative precision. Where that would be felt,
// an element stays in FP64 arithmetic: a state whose densities or energies spread over more than kFixSpread binary orders
// (fix_spread; the fluxes divide by the density), which holds both to FP64's own bound on every line of nodes. Its momenta
// are then at most sqrt(2 rho E), so 2^5 times sqrt(2 rho E) of any node (positive pressure), and held to the bound of
// that, the scale at which every numerical flux adds them to density differences times the wave speed. The advected scalar has
// no such coupling, nor has the tangent along a unit direction: both contract in FP64 (kFixed, tp_jvp_volume_kernel).
// Directions and cotangents of whole meshes lose nothing that the changes of basis at both ends, which mix the values of an
// element, would have kept.
//
// Operators outside fix_usable (not finite, beyond 2^24 or below 2^-24, basis functions of different scales) have no such form.
//
// Range. Infinities, NaN, magnitudes of 2^824 and above and non-zero blocks below 2^-823 do not enter: fix_in_range
// tells, and the caller keeps its FP64 loop for such an element, which propagates them as before. (A block of zeros and
// denormals enters as zeros.)
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace dgpu {

struct FixW {
	int l, h;
};

struct FixAcc {
	long long h, m;
};

constexpr int kFixMin = 200, kFixMax = 1846;   // biased block exponents that enter

__device__ __forceinline__ int fix_exponent(double x)
{
	return (__double2hiint(x) >> 20) & 0x7ff;
}
constexpr int kFixSpread = 4;

// Reduced by elem_max beside the exponents: the smallest exponent, as 2047 minus it.
__device__ __forceinline__ int fix_low(double x) { return 2047 - fix_exponent(x); }
__device__ __forceinline__ bool fix_spread(int eb, int low) { return eb - (2047 - low) <= kFixSpread; }
__device__ __forceinline__ bool fix_in_range(int eb)
{
	return eb == 0 || (unsigned)(eb - kFixMin) <= (unsigned)(kFixMax - kFixMin);
}
__device__ __forceinline__ int fix_block(int eb) { return eb < kFixMin ? kFixMin : eb; }

// Limbs of an integer: l from the low word taken as signed, h with the carry that makes up for it.
__device__ __forceinline__ int2 fix_split(long long X)
{
	return make_int2((int)X >> 2, (int)((X + 0x80000000ll) >> 32));
}

// x as limbs (.x = l, .y = h) at block exponent eb >= its own exponent.
__device__ __forceinline__ int2 fix_pack(double x, int eb)
{
	const int hi = __double2hiint(x), lo = __double2loint(x);
	const unsigned mh = (hi & 0x000fffff) | 0x00100000;
	unsigned long long m = ((unsigned long long)__funnelshift_l(lo, mh, 7) << 32) | ((unsigned)lo << 7);
	asm("shr.u64 %0, %0, %1;" : "+l"(m) : "r"(eb - ((hi >> 20) & 0x7ff)));   // clamps: 0 beyond 63
	const long long s = hi >> 31;
	const long long X = (long long)(m ^ (unsigned long long)s) + (2 - s);    // sign, and half of the last kept unit
	return fix_split(X);
}

__device__ __forceinline__ void fix_mac(FixAcc& a, const FixW w, const int2 x)
{
	a.h += (long long)w.h * x.y;
	a.m += (long long)w.h * x.x;
	a.m += (long long)w.l * x.y;
}

// sum X W / 2^61: |result| <= 2^62.
__device__ __forceinline__ long long fix_sum(const FixAcc& a) { return a.h * 8 + (a.m >> 27); }

// Exponent that makes fix_sum a value: v = fix_sum 2^fix_scale for a block eb and an operator scaled by 2^s.
__device__ __forceinline__ int fix_scale(int eb, int s) { return 61 - s + eb - 1082; }

// r 2^e rounded to nearest, by integer operations (a conversion on the FP64 pipe costs twice as much); the result must
// be a normal number, |r| < 2^63.
__device__ __forceinline__ double fix_to_double(long long r, int e)
{
	const int sg = (int)(r >> 63);
	unsigned long long u = ((unsigned long long)r ^ (long long)sg) - (long long)sg;
	const int n = __clzll((long long)u);
	u <<= (n - 1) & 63;                                   // leading bit at 62 (r = 0: u stays 0)
	const unsigned long long q = (u + 0x200) >> 10;       // 53 bits, or 2^53 after a carry
	int hi = (int)(q >> 32) + ((1085 - n + e) << 20);     // the leading bit adds one to the exponent field
	hi = (hi & 0x7fffffff) | (sg & 0x80000000);
	return u ? __hiloint2double(hi, (int)q) : 0.0;
}

// Limbs of an integer value |X| < 2^60 (a contraction's result that enters the next one).
__device__ __forceinline__ int2 fix_limbs(long long X)
{
	return fix_split(X + 2);
}

// Per-element maxima of K non-negative integers over the threads of each element (N consecutive threads per element,
// e = threadIdx.x / N), into sx[e * stride + k]. sx must be zero before (a barrier in between), and the caller
// synchronises before reading. All threads of the CTA must call it.
template <int N, int K>
__device__ __forceinline__ void elem_max(const int (&x)[K], int e, bool active, int* sx, int stride)
{
	const int lane = threadIdx.x & 31;
	if constexpr (N == 4 || N == 8 || N == 16) {   // elements aligned inside a warp
#pragma unroll
		for (int k = 0; k < K; ++k) {
			int r = x[k];
#pragma unroll
			for (int o = N / 2; o > 0; o >>= 1)
				r = max(r, __shfl_xor_sync(0xffffffffu, r, o));
			if (active && lane % N == 0)
				sx[e * stride + k] = r;
		}
	} else if constexpr (N < 32) {   // up to five elements in a warp: segmented maxima towards each one's first lane
		const int node = threadIdx.x - e * N;
#pragma unroll
		for (int k = 0; k < K; ++k) {
			int r = x[k];
#pragma unroll
			for (int o = 1; o < N; o *= 2) {
				const int t = __shfl_down_sync(0xffffffffu, r, o);
				if (node + o < N && lane + o < 32)
					r = max(r, t);
			}
			if (active && (node == 0 || lane == 0))
				atomicMax(sx + e * stride + k, r);
		}
	} else {
		const int w0 = (threadIdx.x & ~31);
		const int e0 = w0 / N, e1 = (N % 32 == 0) ? e0 : (w0 + 31) / N;
		for (int s = e0; s <= e1; ++s)
#pragma unroll
			for (int k = 0; k < K; ++k) {
				const int r = __reduce_max_sync(0xffffffffu, (active && e == s) ? x[k] : 0);
				if (lane == 0 && r > 0)
					atomicMax(sx + s * stride + k, r);
			}
	}
}

// One 1D pass along `dir` of limb blocks: out[var][node] = sum_m M[a(node)][m] in[var][a -> m], rescaled to limbs.
// sum |W| <= 2^62 for these operators, so |out| < 2^60 at a block exponent raised by 62 - s.
template <int D, int Q, int NV>
__device__ __forceinline__ void fix_pass(const int2* __restrict__ in, int2* __restrict__ out, const FixW (*M)[5], int dir,
                                         int node)
{
	constexpr int N = (D == 2 ? Q * Q : Q * Q * Q);
	const int stride = (dir == 0 ? 1 : (dir == 1 ? Q : Q * Q));
	const int a = (dir == 0 ? node % Q : (dir == 1 ? (node / Q) % Q : node / (Q * Q)));
	const int base = node - a * stride;
	FixW w[Q];
#pragma unroll
	for (int m = 0; m < Q; ++m)
		w[m] = M[a][m];
#pragma unroll
	for (int v = 0; v < NV; ++v) {
		FixAcc s = {0, 0};
#pragma unroll
		for (int m = 0; m < Q; ++m)
			fix_mac(s, w[m], in[v * N + base + m * stride]);
		out[v * N + node] = fix_limbs(s.h * 4 + (s.m >> 28));
	}
}

// ---------------------------------------------------------------------------------------------------------------
// Reciprocal, quotient, square root and magnitude comparison of doubles on the integer pipe
// ---------------------------------------------------------------------------------------------------------------
// 1/x, sqrt(x) and a/b in FP64 arithmetic take 8 to 10 operations of 64 cycles; a comparison takes one. Newton's iteration
// (Newton-Raphson for 1/x, the binomial series of sqrt(s0^2 + r) for the root) on integers, started from the FP32
// approximations of the special function unit, needs about 50 to 70 cycles. It gives 63 bits that are at most 0.5 above and 2.4
// below the value (over 2^30 arguments, with seeds up to two units off). One in 256 lies so near to the middle of two
// doubles that this does not tell which way to round: those go by the remainder, which is exact in 64 bits. Every bit is
// then the one of the FP64 operation. (No quotient, reciprocal or root of 53-bit numbers that is not one itself lies in the
// middle.) The remainder for all of them cost 7 % of the Lax-Friedrichs face kernel, this 1 %. Zeros, denormals, Inf, NaN, negative roots and results that would be denormal take the FP64 operation.

// 2^63 / d for a mantissa d in [1, 2), given by the low 20 bits of hi and lo. The seed y is in
// [1/2, 1] for every leading mantissa (rcp.approx is within one unit, and no 1/f rounds below 1/2).
__device__ __forceinline__ unsigned long long fix_rcp63(int hi, int lo)
{
	const float f = __int_as_float((__funnelshift_l(lo, hi, 3) & 0x007fffff) | 0x3f800000);   // [1, 2)
	float y;
	asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(f));
	const unsigned M = (min(__float_as_uint(y), 0x3f7fffffu) & 0x007fffff) | 0x00800000;      // y 2^24
	const unsigned dh = (hi & 0x000fffff) | 0x00100000;                                        // 1.m 2^52
	// e = d y - 1 in units of 2^-76, exactly: |e| < 2^54, so the low 64 bits suffice
	const long long e = (long long)((unsigned long long)(unsigned)lo * M + ((unsigned long long)(dh * M) << 32));
	const int eh = (int)(e >> 32);
	// y (1 - e + e^2) in units of 2^-63
	const long long t = (long long)eh * (int)M + (long long)(((unsigned long long)(unsigned)e * M) >> 32);
	const unsigned sq = (unsigned)(((long long)eh * eh) >> 17);
	return ((unsigned long long)M << 39) + ~(t >> 5) + __umulhi(sq, M);   // ~: the next one below
}
// Whether a value of 63 bits is that near to the middle of two of 53, which adding 513 makes a multiple of 2^10.
__device__ __forceinline__ bool fix_middle(unsigned long long R) { return (((unsigned)R + 515) & 1023) < 4; }
__device__ __forceinline__ unsigned long long fix_mantissa(int hi, int lo)
{
	return ((unsigned long long)((hi & 0x000fffff) | 0x00100000) << 32) | (unsigned)lo;
}

// ANY: false where the caller knows that argument and result are normal numbers (a root's argument positive).
template <bool ANY = true>
__device__ __forceinline__ double fix_rcp(double x)
{
	const int hi = __double2hiint(x), lo = __double2loint(x);
	const int ex = (hi >> 20) & 0x7ff;
	const unsigned long long R = fix_rcp63(hi, lo);
	unsigned long long q = (R + 513) >> 10;   // 53 bits, leading bit 52 (or 2^53)
	const bool normal = !ANY || (unsigned)(ex - 1) < 2044u;   // not 0, denormal, Inf, NaN; and so is the result
	if (fix_middle(R) || !normal) {                   // one branch for both
		if (!normal)
			return 1.0 / x;
		const unsigned long long d = fix_mantissa(hi, lo);
		q = (R - 16) >> 10;                           // the integer below
		const unsigned long long rem = 0ull - d * q;  // 2^105 - d q
		q += 2 * rem > d;
	}
	const int rh = (int)(q >> 32) + ((2044 - ex) << 20);
	return __hiloint2double(rh | (hi & 0x80000000), (int)q);
}

__device__ __forceinline__ double fix_div(double a, double b)
{
	const int ha = __double2hiint(a), hb = __double2hiint(b);
	const int ea = (ha >> 20) & 0x7ff, eb = (hb >> 20) & 0x7ff;
	unsigned long long A = fix_mantissa(ha, __double2loint(a));
	const unsigned long long d = fix_mantissa(hb, __double2loint(b));
	const int s = A < d, ex = ea - eb + 1022 - s;   // exponent of the result, less the leading bit's one
	if ((unsigned)(ea - 1) >= 2046u || (unsigned)(eb - 1) >= 2046u || (unsigned)ex >= 2045u)
		return a / b;
	A <<= s;
	// q = A 2^52 / d, 53 bits: taken 3/16 to 21/16 low from 2^63 / d, then by the remainder
	unsigned long long q = (__umul64hi(A << 5, fix_rcp63(hb, __double2loint(b))) - 4) >> 4;
	const unsigned long long rem = (A << 52) - q * d;
	q += 2 * rem > d;
	return __hiloint2double(((int)(q >> 32) + (ex << 20)) | ((ha ^ hb) & 0x80000000), (int)q);
}

template <bool ANY = true>
__device__ __forceinline__ double fix_sqrt(double x)
{
	const int hi = __double2hiint(x), lo = __double2loint(x);
	const int ex = hi >> 20;   // negative for a negative argument
	const bool normal = !ANY || (unsigned)(ex - 1) < 2046u;
	const int t = (ex + 1) & 1;   // x = f 4^k, f = 1.m 2^t in [1, 4)
	const float f = __int_as_float((__funnelshift_l(lo, hi, 3) & 0x007fffff) | (0x3f800000 + (t << 23)));
	float y;
	asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(f));
	const unsigned M = (min(__float_as_uint(y), 0x3f7fffffu) & 0x007fffff) | 0x00800000;      // y 2^24, y in [1/2, 1]
	const unsigned long long X = fix_mantissa(hi, lo) << (8 + t);                                // f 2^60
	const unsigned S0 = (unsigned)(((unsigned long long)(unsigned)(X >> 32) * M) >> 22);         // s0 = f y, 2^30
	const long long r = (long long)(X - (unsigned long long)S0 * S0);                           // f - s0^2, 2^60
	const int d = (int)(((1ll << 54) - (long long)((unsigned long long)S0 * M)) >> 4);           // 1 - s0 y, 2^50
	// u = r y / 2 in units of 2^-62, then sqrt(f) = s0 + u + u (d - u y / 2) + ...
	const long long u = (long long)(((unsigned long long)(unsigned)r * M) >> 23) + (((r >> 32) * (int)M) << 9);
	const int U = (int)(u >> 12);                                                               // 2^50
	const int z = d - (int)(((long long)U * (int)M) >> 25);
	const long long v = ((long long)U * z) >> 38;
	const unsigned long long V = ((unsigned long long)S0 << 32) + u + v;                         // sqrt(f) 2^62
	unsigned long long q = (V + 513) >> 10;
	if (fix_middle(V) || !normal) {
		if (!normal)
			return ::sqrt(x);
		q = (V - 16) >> 10;                                                                     // the integer below
		const unsigned long long rem = ((unsigned long long)((unsigned)lo << (20 + t)) << 32) - q * q;   // f 2^104 - q^2
		q += rem > q;                                                                          // f 2^104 > (q + 1/2)^2
	}
	const int rh = (int)(q >> 32) + ((((ex - 1023 - t) >> 1) + 1022) << 20);
	return __hiloint2double(rh, (int)q);
}

// |a| < |b|, false when either is NaN.
__device__ __forceinline__ bool abs_less(double a, double b)
{
	const unsigned long long ua = (unsigned long long)__double_as_longlong(a) & 0x7fffffffffffffffull;
	const unsigned long long ub = (unsigned long long)__double_as_longlong(b) & 0x7fffffffffffffffull;
	return ua < ub && ub <= 0x7ff0000000000000ull;
}

// a b rounded to nearest even, bit for bit __dmul_rn, for factors that are zero or normal and a product that is zero
// or normal (the caller knows their magnitudes). About 35 integer instructions, the time of one DMUL, but on a pipe that
// the pointwise fluxes leave idle: they run their lone products here and their sums and fused products on the FP64 pipe.
__device__ __forceinline__ double fix_mul(double a, double b)
{
	const int ha = __double2hiint(a), hb = __double2hiint(b);
	const unsigned la = __double2loint(a), lb = __double2loint(b);
	const unsigned mah = (ha & 0x000fffff) | 0x00100000, bh = (hb & 0x000fffff) | 0x00100000;
	// (a's mantissa 2^11) x (b's mantissa): 116 or 117 bits, the 53 or 52 leading ones above bit 64
	const unsigned ah = __funnelshift_l(la, mah, 11), al = la << 11;
	const unsigned long long t0 = (unsigned long long)al * lb;
	const unsigned long long t1 = (unsigned long long)ah * lb + (t0 >> 32);
	const unsigned long long t2 = (unsigned long long)al * bh + (unsigned)t1;
	unsigned long long hi = (unsigned long long)ah * bh + (t1 >> 32) + (t2 >> 32);
	unsigned long long lo = (t2 << 32) | (unsigned)t0;
	int ex = (ha & 0x7ff00000) + (hb & 0x7ff00000) - (1023 << 20);
	if (!(hi >> 52)) {
		hi = hi * 2 + (lo >> 63);
		lo *= 2;
		ex -= 1 << 20;
	}
	const bool up = (lo >> 63) && ((lo << 1) || (hi & 1));
	hi += up;                                    // the leading bit (and a carry) adds to the exponent field
	int rh = (int)(hi >> 32) + ex;
	unsigned rl = (unsigned)hi;
	if (!((ha & 0x7fffffff) && (hb & 0x7fffffff)))
		rh = rl = 0;
	return __hiloint2double(rh | ((ha ^ hb) & 0x80000000), rl);
}

// a b with the bits of __dmul_rn for any factors: fix_mul when they are zero or normal and the product stays normal, the FP64
// operation otherwise.
__device__ __forceinline__ double mul_int(double a, double b)
{
	const int ea = (__double2hiint(a) >> 20) & 0x7ff, eb = (__double2hiint(b) >> 20) & 0x7ff;
	if ((unsigned)(ea - 1) < 2046u && (unsigned)(eb - 1) < 2046u && (unsigned)(ea + eb - 1025) < 2042u)
		return fix_mul(a, b);
	return __dmul_rn(a, b);
}

}  // namespace dgpu
