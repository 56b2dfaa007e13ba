// A stand-in for the CUDA runtime, driver entry points and NVRTC, for tests of the host runtime without a
// GPU. "Device" memory is host memory; kernels do nothing but call `on_launch`. Copies to the device are
// pending until something orders them: work on the same stream, or a wait for it. A cudaMemcpy from pageable
// memory may return once the data is staged, so its copy is pending on the default stream, which
// non-blocking streams do not wait for.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <nvrtc.h>

#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <string>
#include <vector>

namespace fake {

struct copy
{
	cudaStream_t s;
	void* dst;
	std::vector<char> data;
};
inline std::vector<copy> pending;
inline std::map<void*, size_t> device, pinned; // live allocations
inline std::function<void(const std::string& kernel, cudaStream_t, void** args, unsigned block, size_t smem)> on_launch;
inline std::function<bool(size_t bytes)> fail_malloc; // true: this cudaMalloc fails
inline bool fail_register = false;					  // host memory cannot be pinned
inline std::string fail_function;					  // this kernel cannot be found
inline cudaError_t last = cudaSuccess;

inline size_t held(const std::map<void*, size_t>& m)
{
	size_t n = 0;
	for (const auto& x : m)
		n += x.second;
	return n;
}
inline void run_copies(cudaStream_t s)
{
	for (size_t i = 0; i < pending.size();)
	{
		if (pending[i].s != s)
		{
			i++;
			continue;
		}
		std::memcpy(pending[i].dst, pending[i].data.data(), pending[i].data.size());
		pending.erase(pending.begin() + (std::ptrdiff_t)i);
	}
}
inline void enqueue(cudaStream_t s, void* dst, const void* src, size_t n, cudaMemcpyKind kind)
{
	if (kind == cudaMemcpyHostToDevice)
	{
		const char* p = static_cast<const char*>(src);
		pending.push_back({ s, dst, std::vector<char>(p, p + n) });
		return;
	}
	run_copies(s);
	std::memcpy(dst, src, n);
}

inline CUresult module_load(CUmodule* m, const void*)
{
	*m = reinterpret_cast<CUmodule>(new int);
	return CUDA_SUCCESS;
}
inline CUresult module_unload(CUmodule m)
{
	delete reinterpret_cast<int*>(m);
	return CUDA_SUCCESS;
}
inline CUresult get_function(CUfunction* f, CUmodule, const char* name)
{
	if (fail_function == name)
		return CUDA_ERROR_OUT_OF_MEMORY;
	static std::map<std::string, std::string> names;
	*f = reinterpret_cast<CUfunction>(&names.emplace(name, name).first->second);
	return CUDA_SUCCESS;
}
inline CUresult launch(CUfunction f, unsigned, unsigned, unsigned, unsigned block, unsigned, unsigned, unsigned smem,
					   CUstream s, void** args, void**)
{
	if (!f)
		return CUDA_ERROR_INVALID_HANDLE;
	run_copies((cudaStream_t)s);
	if (on_launch)
		on_launch(*reinterpret_cast<std::string*>(f), (cudaStream_t)s, args, block, smem);
	return CUDA_SUCCESS;
}
inline CUresult set_attribute(CUfunction, CUfunction_attribute, int) { return CUDA_SUCCESS; }
inline CUresult error_string(CUresult, const char** s)
{
	*s = "error";
	return CUDA_SUCCESS;
}
inline CUresult occupancy(int* n, CUfunction, int, size_t)
{
	*n = 1;
	return CUDA_SUCCESS;
}

} // namespace fake

extern "C" {
cudaError_t CUDARTAPI cudaMalloc(void** p, size_t n)
{
	if (fake::fail_malloc && fake::fail_malloc(n))
		return fake::last = cudaErrorMemoryAllocation;
	*p = std::calloc(n, 1);
	fake::device[*p] = n;
	return cudaSuccess;
}
cudaError_t CUDARTAPI cudaFree(void* p)
{
	fake::device.erase(p);
	std::free(p);
	return cudaSuccess;
}
cudaError_t CUDARTAPI cudaHostAlloc(void** p, size_t n, unsigned)
{
	*p = std::malloc(n);
	fake::pinned[*p] = n;
	return cudaSuccess;
}
cudaError_t CUDARTAPI cudaHostRegister(void* p, size_t n, unsigned)
{
	if (fake::fail_register)
		return fake::last = cudaErrorMemoryAllocation;
	fake::pinned[p] = n;
	return cudaSuccess;
}
cudaError_t CUDARTAPI cudaHostUnregister(void* p)
{
	fake::pinned.erase(p);
	return cudaSuccess;
}
cudaError_t CUDARTAPI cudaFreeHost(void* p)
{
	fake::pinned.erase(p);
	std::free(p);
	return cudaSuccess;
}
cudaError_t CUDARTAPI cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k)
{
	fake::enqueue(nullptr, d, s, n, k);
	return cudaSuccess;
}
cudaError_t CUDARTAPI cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st)
{
	fake::enqueue(st, d, s, n, k);
	return cudaSuccess;
}
cudaError_t CUDARTAPI cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st)
{
	fake::run_copies(st);
	std::memset(d, v, n);
	return cudaSuccess;
}
cudaError_t CUDARTAPI cudaStreamSynchronize(cudaStream_t s)
{
	fake::run_copies(s);
	return cudaSuccess;
}
cudaError_t CUDARTAPI cudaStreamCreateWithFlags(cudaStream_t* s, unsigned)
{
	static size_t next = 1000;
	*s = reinterpret_cast<cudaStream_t>(next++);
	return cudaSuccess;
}
cudaError_t CUDARTAPI cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventCreate(cudaEvent_t* e)
{
	*e = reinterpret_cast<cudaEvent_t>(new int);
	return cudaSuccess;
}
cudaError_t CUDARTAPI cudaEventDestroy(cudaEvent_t e)
{
	delete reinterpret_cast<int*>(e);
	return cudaSuccess;
}
cudaError_t CUDARTAPI cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t)
{
	*ms = 0.f;
	return cudaSuccess;
}
cudaError_t CUDARTAPI cudaGetDevice(int* d)
{
	*d = 0;
	return cudaSuccess;
}
cudaError_t CUDARTAPI cudaSetDevice(int) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaGetDeviceCount(int* n)
{
	*n = 1;
	return cudaSuccess;
}
#undef cudaGetDeviceProperties
cudaError_t CUDARTAPI cudaGetDeviceProperties_v2(cudaDeviceProp* p, int)
{
	std::memset(p, 0, sizeof *p);
	p->multiProcessorCount = 148;
	p->major = 10;
	return cudaSuccess;
}
const char* CUDARTAPI cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t CUDARTAPI cudaGetLastError() { return std::exchange(fake::last, cudaSuccess); }
cudaError_t CUDARTAPI cudaLibraryLoadData(cudaLibrary_t*, const void*, cudaJitOption*, void**, unsigned, cudaLibraryOption*,
										  void**, unsigned)
{
	return cudaErrorNotSupported;
}
cudaError_t CUDARTAPI cudaLibraryGetKernel(cudaKernel_t*, cudaLibrary_t, const char*) { return cudaErrorNotSupported; }
cudaError_t CUDARTAPI cudaLibraryUnload(cudaLibrary_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaGetDriverEntryPointByVersion(const char* name, void** f, unsigned, unsigned long long,
													   cudaDriverEntryPointQueryResult* q)
{
	const std::map<std::string, void*> all = {
		{ "cuModuleLoadData", (void*)fake::module_load },	 { "cuModuleUnload", (void*)fake::module_unload },
		{ "cuModuleGetFunction", (void*)fake::get_function }, { "cuLaunchKernel", (void*)fake::launch },
		{ "cuFuncSetAttribute", (void*)fake::set_attribute }, { "cuGetErrorString", (void*)fake::error_string },
		{ "cuOccupancyMaxActiveBlocksPerMultiprocessor", (void*)fake::occupancy },
	};
	*f = all.at(name);
	*q = cudaDriverEntryPointSuccess;
	return cudaSuccess;
}
nvrtcResult nvrtcCreateProgram(nvrtcProgram* p, const char*, const char*, int, const char* const*, const char* const*)
{
	*p = nullptr;
	return NVRTC_SUCCESS;
}
nvrtcResult nvrtcCompileProgram(nvrtcProgram, int, const char* const*) { return NVRTC_SUCCESS; }
nvrtcResult nvrtcDestroyProgram(nvrtcProgram*) { return NVRTC_SUCCESS; }
nvrtcResult nvrtcGetCUBINSize(nvrtcProgram, size_t* n)
{
	*n = 1;
	return NVRTC_SUCCESS;
}
nvrtcResult nvrtcGetCUBIN(nvrtcProgram, char* c)
{
	*c = 0;
	return NVRTC_SUCCESS;
}
nvrtcResult nvrtcGetProgramLogSize(nvrtcProgram, size_t* n)
{
	*n = 0;
	return NVRTC_SUCCESS;
}
nvrtcResult nvrtcGetProgramLog(nvrtcProgram, char*) { return NVRTC_SUCCESS; }
const char* nvrtcGetErrorString(nvrtcResult) { return "error"; }
}
