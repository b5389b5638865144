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
