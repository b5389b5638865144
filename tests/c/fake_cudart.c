/* A stand-in for the CUDA runtime on host memory, to run the library's host code without a GPU: allocations are malloc,
 * copies are memcpy, kernels are not executed. fake_fail_at(n) makes the n-th of the following calls that can fail return
 * cudaErrorMemoryAllocation; fake_calls() counts them. */
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

static long fail_at = 0, calls = 0;

void fake_fail_at(long n) { fail_at = n, calls = 0; }
long fake_calls(void) { return calls; }

static cudaError_t call(void) { return ++calls == fail_at ? cudaErrorMemoryAllocation : cudaSuccess; }
static int handle;

#define OK_STUB(name, args) \
	cudaError_t name args { return call(); }

#undef cudaGetDeviceProperties
cudaError_t cudaMalloc(void** p, size_t n)
{
	cudaError_t e = call();
	*p = e ? NULL : calloc(n ? n : 1, 1);
	return e;
}
cudaError_t cudaFree(void* p)
{
	free(p);
	return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k)
{
	(void)k;
	cudaError_t e = call();
	if (!e)
		memcpy(d, s, n);
	return e;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st)
{
	(void)st;
	return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemset(void* d, int v, size_t n)
{
	cudaError_t e = call();
	if (!e)
		memset(d, v, n);
	return e;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st)
{
	(void)st;
	return cudaMemset(d, v, n);
}
cudaError_t cudaGetDevice(int* d)
{
	*d = 0;
	return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n)
{
	*n = 1;
	return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(struct cudaDeviceProp* p, int d)
{
	(void)d;
	memset(p, 0, sizeof *p);
	p->major = 10, p->minor = 3, p->multiProcessorCount = 152, p->sharedMemPerBlockOptin = 232448;
	return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d)
{
	(void)d;
	*v = a == cudaDevAttrComputeCapabilityMajor ? 10 : a == cudaDevAttrComputeCapabilityMinor ? 3
	   : a == cudaDevAttrMultiProcessorCount ? 152 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 1;
	return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* f, int b, size_t s)
{
	(void)f, (void)b, (void)s;
	*n = 2;
	return call();
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int b, size_t s, unsigned g)
{
	(void)g;
	return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, f, b, s);
}
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes* a, const void* f)
{
	(void)f;
	memset(a, 0, sizeof *a);
	return call();
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f)
{
	(void)f;
	*s = (cudaStream_t)&handle;
	return call();
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned f)
{
	(void)f;
	*e = (cudaEvent_t)&handle;
	return call();
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b)
{
	(void)a, (void)b;
	*ms = 1.0f;
	return call();
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s)
{
	*p = (void*)s;
	return call();
}
const char* cudaGetErrorName(cudaError_t e) { return e ? "cudaErrorMemoryAllocation" : "cudaSuccess"; }
const char* cudaGetErrorString(cudaError_t e) { return e ? "out of memory" : "no error"; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes* a, const void* p)
{
	memset(a, 0, sizeof *a);
	(void)p;
	return cudaSuccess;
}
#pragma GCC diagnostic ignored "-Wunused-parameter"
OK_STUB(cudaEventDestroy, (cudaEvent_t e))
OK_STUB(cudaEventRecord, (cudaEvent_t e, cudaStream_t s))
OK_STUB(cudaEventSynchronize, (cudaEvent_t e))
OK_STUB(cudaFuncSetAttribute, (const void* f, enum cudaFuncAttribute a, int v))
OK_STUB(cudaGraphDestroy, (cudaGraph_t g))
OK_STUB(cudaGraphExecDestroy, (cudaGraphExec_t g))
OK_STUB(cudaGraphInstantiate, (cudaGraphExec_t * g, cudaGraph_t h, unsigned long long f))
OK_STUB(cudaGraphLaunch, (cudaGraphExec_t g, cudaStream_t s))
OK_STUB(cudaLaunchCooperativeKernel, (const void* f, dim3 g, dim3 b, void** a, size_t s, cudaStream_t st))
OK_STUB(cudaStreamBeginCapture, (cudaStream_t s, enum cudaStreamCaptureMode m))
OK_STUB(cudaStreamDestroy, (cudaStream_t s))
OK_STUB(cudaStreamEndCapture, (cudaStream_t s, cudaGraph_t* g))
OK_STUB(cudaStreamSynchronize, (cudaStream_t s))
OK_STUB(cudaStreamWaitEvent, (cudaStream_t s, cudaEvent_t e, unsigned f))

/* what the compiler's launch stubs call */
OK_STUB(__cudaLaunchKernel, (void* k, dim3 g, dim3 b, void** a, size_t s, cudaStream_t st))
cudaError_t __cudaGetKernel(void** k, const void* f) { return *k = (void*)f, cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, void* st) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st) { return cudaSuccess; }
void** __cudaRegisterFatBinary(void* f) { return (void**)&handle; }
void __cudaRegisterFatBinaryEnd(void** h) {}
void __cudaUnregisterFatBinary(void** h) {}
void __cudaRegisterFunction(void** h, const char* f, char* d, const char* n, int t, void* a, void* b, void* c, void* e, int* w) {}
void __cudaRegisterVar(void** h, char* v, char* d, const char* n, int e, size_t s, int c, int g) {}
