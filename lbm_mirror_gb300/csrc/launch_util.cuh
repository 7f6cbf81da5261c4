// Host helpers of kernel launches.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

namespace kel {
namespace gb {

// A launch that may start while the one before it on the stream drains
// (overlap; the kernel waits for it with grid_dependency_wait).
template <class Kernel, class P>
static cudaError_t launch_overlapped(Kernel kern, dim3 grid, int block, int smem, cudaStream_t st, bool overlap, const P &p) {
	cudaLaunchAttribute at;
	at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
	at.val.programmaticStreamSerializationAllowed = 1;
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = grid;
	cfg.blockDim = dim3(block);
	cfg.dynamicSmemBytes = smem;
	cfg.stream = st;
	cfg.attrs = &at;
	cfg.numAttrs = overlap ? 1 : 0;
	const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p);
	if (e != cudaSuccess) cudaGetLastError(); // reported here, not by the next call too
	return e;
}

// Lets a kernel use `bytes` of dynamic shared memory; the attribute is set to
// the device's whole opt-in size once per kernel and device (`done`: bit per
// device), so that no later call with a smaller footprint lowers it under
// another thread.
template <class Kernel>
static cudaError_t allow_smem(Kernel kern, int bytes, std::atomic<uint64_t> &done) {
	if (bytes <= 48 * 1024) return cudaSuccess;
	int dev = 0, optin = 0;
	cudaError_t e = cudaGetDevice(&dev);
	if (e != cudaSuccess) return e;
	const uint64_t bit = dev < 64 ? (uint64_t)1 << dev : 0;
	if (bit && (done.load() & bit)) return cudaSuccess;
	if ((e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return e;
	if (bytes > optin) return cudaErrorInvalidConfiguration;
	if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, optin)) != cudaSuccess) return e;
	done.fetch_or(bit);
	return cudaSuccess;
}

} // namespace gb
} // namespace kel
