// The arithmetic of csrc/dgpu_fix.cuh on arrays, for the tests: op 0 fix_rcp(a), 1 fix_sqrt(a), 2 fix_div(a, b),
// 3 fix_mul(a, b), 4 mul_int(a, b).
#include "dgpu_fix.cuh"

__global__ void probe_kernel(int op, const double* a, const double* b, double* out, long long n)
{
	for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
		out[i] = op == 0 ? dgpu::fix_rcp(a[i]) : op == 1 ? dgpu::fix_sqrt(a[i]) : op == 2 ? dgpu::fix_div(a[i], b[i])
		       : op == 3 ? dgpu::fix_mul(a[i], b[i]) : dgpu::mul_int(a[i], b[i]);
}

extern "C" int fix_probe(int op, const double* a, const double* b, double* out, long long n)
{
	double *d[3] = {nullptr, nullptr, nullptr};
	const size_t bytes = (size_t)n * sizeof(double);
	cudaError_t e = cudaSuccess;
	for (int k = 0; k < 3 && e == cudaSuccess; ++k)
		e = cudaMalloc((void**)&d[k], bytes);
	if (e == cudaSuccess)
		e = cudaMemcpy(d[0], a, bytes, cudaMemcpyHostToDevice);
	if (e == cudaSuccess)
		e = cudaMemcpy(d[1], b, bytes, cudaMemcpyHostToDevice);
	if (e == cudaSuccess) {
		probe_kernel<<<1024, 256>>>(op, d[0], d[1], d[2], n);
		e = cudaMemcpy(out, d[2], bytes, cudaMemcpyDeviceToHost);
	}
	for (double* p : d)
		cudaFree(p);
	return (int)e;
}

// The volume term's contractions of the uniform kernels on given states and fluxes at the cubature nodes.
#include "dgpu_host_ops.h"

namespace dgpu {

template <int D, int Q, int NV>
__global__ void __launch_bounds__(TPShape<D, Q>::THREADS)
probe_volume_kernel(const __grid_constant__ TPOps ops, int n, const double* W, const double* F, double* traces, double* vol,
                    int* fixed)
{
	using S = TPShape<D, Q>;
	constexpr int N = S::N, NF = S::NF, VOL = TPSmem<D, Q, NV>::VOL, XE = TPSmem<D, Q, NV>::EXP;
	extern __shared__ double smem[];
	TPOps* sops = reinterpret_cast<TPOps*>(smem);
	double* base = smem + sizeof(TPOps) / 8;
	int* sx = reinterpret_cast<int*>(base + S::E * VOL);
	load_ops(sops, ops);
	const int e = threadIdx.x / N, node = threadIdx.x % N, v = blockIdx.x * S::E + e;
	const bool active = e < S::E && v < n;
	for (int i = threadIdx.x; i < S::E * XE; i += blockDim.x)
		sx[i] = 0;
	double w[NV], f[D][NV];
	if (active)
		for (int k = 0; k < NV; ++k) {
			w[k] = W[((size_t)v * NV + k) * N + node];
			for (int j = 0; j < D; ++j)
				f[j][k] = F[(((size_t)v * D + j) * NV + k) * N + node];
		}
	__syncthreads();
	double *su = base + (active ? e : 0) * VOL, *sf = su + 2 * NV * N;
	int eb[2 * NV];
	const bool ok = tp_stage_volume<D, Q, NV>(w, f, ops.fix, e, node, active, su, sf, sx, XE, eb);
	if (!active)
		return;
	double out[NV];
	if (node == 0)
		fixed[v] = ok;
	tp_derivative<D, Q, NV>(sops, sf, eb, ok, node, out);
	for (int k = 0; k < NV; ++k)
		vol[((size_t)v * NV + k) * N + node] = out[k];
	for (int it = node; it < 2 * D * NF; it += N) {
		tp_trace<D, Q, NV>(sops, su, eb, ok, it / NF, it % NF, out);
		for (int k = 0; k < NV; ++k)
			traces[(((size_t)v * 2 * D + it / NF) * NV + k) * NF + it % NF] = out[k];
	}
}

template <int D, int Q>
cudaError_t probe_volume(const TPOps& ops, int n, double** d, int* fixed)
{
	using S = TPShape<D, Q>;
	constexpr int NV = D + 2;
	const int smem = sizeof(TPOps) + S::E * (TPSmem<D, Q, NV>::VOL * 8 + TPSmem<D, Q, NV>::EXP * 4);
	const cudaError_t e = cudaFuncSetAttribute(probe_volume_kernel<D, Q, NV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
	                                           smem);
	if (e != cudaSuccess)
		return e;
	probe_volume_kernel<D, Q, NV><<<(n + S::E - 1) / S::E, S::THREADS, smem>>>(ops, n, d[0], d[1], d[2], d[3], fixed);
	return cudaGetLastError();
}

}  // namespace dgpu

// W: n x NV x N, F: n x D x NV x N (NV = D + 2); traces: n x 2D x NV x NF, vol: n x NV x N, fixed: n; lb: 2 x 5 and
// Dgl: 5 x 5, the FP64 operators the kernels take. cv0, cv1 (q x q), cv0f (2 x q): a 1D operator set, its other arrays
// are not read.
extern "C" int fix_probe_volume(int d, int p, const double* cv0, const double* cv1, const double* cv0f, int n, const double* W,
                                const double* F, double* traces, double* vol, int* fixed, double* lb, double* Dgl)
{
	dgpu_tp_operators o;
	memset(&o, 0, sizeof o);
	o.p = p;
	o.cv0_vs_vc = cv0;
	o.cv1_vs_vc = cv1;
	o.cv0_vs_fc = cv0f;
	dgpu::TPOps ops;
	if (!dgpu::derive_tp_ops(&o, d, &ops))
		return -1;
	memcpy(lb, ops.lb, sizeof ops.lb);
	memcpy(Dgl, ops.Dgl, sizeof ops.Dgl);
	const int q = p + 1, NF = d == 2 ? q : q * q, N = NF * q, NV = d + 2;
	const size_t len[4] = {(size_t)n * NV * N, (size_t)n * d * NV * N, (size_t)n * 2 * d * NV * NF, (size_t)n * NV * N};
	double* dev[4] = {nullptr, nullptr, nullptr, nullptr};
	int* dfix = nullptr;
	cudaError_t e = cudaMalloc((void**)&dfix, n * sizeof(int));
	for (int k = 0; k < 4 && e == cudaSuccess; ++k)
		e = cudaMalloc((void**)&dev[k], len[k] * sizeof(double));
	if (e == cudaSuccess)
		e = cudaMemcpy(dev[0], W, len[0] * sizeof(double), cudaMemcpyHostToDevice);
	if (e == cudaSuccess)
		e = cudaMemcpy(dev[1], F, len[1] * sizeof(double), cudaMemcpyHostToDevice);
	if (e == cudaSuccess)
		switch (10 * d + q) {
		case 23: e = dgpu::probe_volume<2, 3>(ops, n, dev, dfix); break;
		case 25: e = dgpu::probe_volume<2, 5>(ops, n, dev, dfix); break;
		case 32: e = dgpu::probe_volume<3, 2>(ops, n, dev, dfix); break;
		case 34: e = dgpu::probe_volume<3, 4>(ops, n, dev, dfix); break;
		default: e = cudaErrorInvalidValue;
		}
	if (e == cudaSuccess)
		e = cudaMemcpy(traces, dev[2], len[2] * sizeof(double), cudaMemcpyDeviceToHost);
	if (e == cudaSuccess)
		e = cudaMemcpy(vol, dev[3], len[3] * sizeof(double), cudaMemcpyDeviceToHost);
	if (e == cudaSuccess)
		e = cudaMemcpy(fixed, dfix, n * sizeof(int), cudaMemcpyDeviceToHost);
	for (double* x : dev)
		cudaFree(x);
	cudaFree(dfix);
	return (int)e;
}
