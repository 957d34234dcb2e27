// The device's inverse of a direction component (csrc/trace_core.hpp), value by value.
#include <cuda_runtime.h>

#include "trace_core.hpp"

__global__ void kInverse(const float* in, float* out, int n)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) {
		out[i] = rgl::safeInv(in[i]);
	}
}

// host_out: the host's; device_out: the device's. Returns a CUDA status.
extern "C" int inverses(const float* in, float* host_out, float* device_out, int n)
{
	for (int i = 0; i < n; ++i) {
		host_out[i] = rgl::safeInv(in[i]);
	}
	float *dIn = nullptr, *dOut = nullptr;
	const size_t bytes = sizeof(float) * (size_t) n;
	cudaError_t e = cudaMalloc(&dIn, bytes);
	if (e == cudaSuccess) {
		e = cudaMalloc(&dOut, bytes);
	}
	if (e == cudaSuccess) {
		e = cudaMemcpy(dIn, in, bytes, cudaMemcpyHostToDevice);
	}
	if (e == cudaSuccess) {
		kInverse<<<(n + 255) / 256, 256>>>(dIn, dOut, n);
		e = cudaMemcpy(device_out, dOut, bytes, cudaMemcpyDeviceToHost);
	}
	cudaFree(dIn);
	cudaFree(dOut);
	return (int) e;
}
