// Host runtime: NVRTC compilation, module loading through the CUDA driver API (resolved at
// run time with cudaGetDriverEntryPointByVersion, so the library loads on hosts without a GPU
// driver), and the run drivers.
#include "runtime.h"
#include "sparse_bins.h"

#include <curand_kernel.h>
#include <nvrtc.h>

#include <algorithm>
#include <array>
#include <chrono>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <mutex>
#include <numeric>
#include <sstream>
#include <thread>

#include <sys/mman.h>

#include "kernels/params.cuh"

namespace mb {

namespace {

#include "engine_src.inc" // mb_params_source, mb_engine_source (embedded kernels/*.cuh)

struct driver_api
{
	CUresult (*ModuleLoadData)(CUmodule*, const void*) = nullptr;
	CUresult (*ModuleUnload)(CUmodule) = nullptr;
	CUresult (*ModuleGetFunction)(CUfunction*, CUmodule, const char*) = nullptr;
	CUresult (*LaunchKernel)(CUfunction, unsigned, unsigned, unsigned, unsigned, unsigned, unsigned, unsigned, CUstream,
							 void**, void**) = nullptr;
	CUresult (*FuncSetAttribute)(CUfunction, CUfunction_attribute, int) = nullptr;
	CUresult (*GetErrorString)(CUresult, const char**) = nullptr;
	CUresult (*OccupancyMaxActiveBlocksPerMultiprocessor)(int*, CUfunction, int, size_t) = nullptr;
};

template <typename F>
void resolve(const char* name, F& fn)
{
	void* p = nullptr;
	cudaDriverEntryPointQueryResult q;
	cudaError_t e = cudaGetDriverEntryPointByVersion(name, &p, 12000, cudaEnableDefault, &q);
	if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !p)
		throw engine_error(MB_ERR_CUDA, std::string("cannot resolve CUDA driver entry point ") + name);
	fn = reinterpret_cast<F>(p);
}

const driver_api& drv()
{
	static driver_api api;
	static std::once_flag once;
	static std::string failure;
	std::call_once(once, [] {
		try
		{
			resolve("cuModuleLoadData", api.ModuleLoadData);
			resolve("cuModuleUnload", api.ModuleUnload);
			resolve("cuModuleGetFunction", api.ModuleGetFunction);
			resolve("cuLaunchKernel", api.LaunchKernel);
			resolve("cuFuncSetAttribute", api.FuncSetAttribute);
			resolve("cuGetErrorString", api.GetErrorString);
			resolve("cuOccupancyMaxActiveBlocksPerMultiprocessor", api.OccupancyMaxActiveBlocksPerMultiprocessor);
		}
		catch (const std::exception& e)
		{
			failure = e.what();
		}
	});
	if (!failure.empty())
		throw engine_error(MB_ERR_CUDA, failure);
	return api;
}

void cu_throw(CUresult r, const char* what)
{
	if (r == CUDA_SUCCESS)
		return;
	const char* s = nullptr;
	if (drv().GetErrorString)
		drv().GetErrorString(r, &s);
	throw engine_error(MB_ERR_CUDA, std::string(what) + ": " + (s ? s : "CUDA driver error") + " (" +
										std::to_string((int)r) + ")");
}

std::string cuda_include_dir()
{
	if (const char* e = std::getenv("MABOSS_CUDA_INCLUDE"))
		return e;
#ifdef MB_CUDA_INCLUDE
	return MB_CUDA_INCLUDE;
#else
	return "/usr/local/cuda/include";
#endif
}

int parse_constexpr(const std::string& src, const std::string& name, int fallback)
{
	const std::string key = "constexpr int " + name + " = ";
	auto p = src.find(key);
	if (p == std::string::npos)
		return fallback;
	return std::atoi(src.c_str() + p + key.size());
}

// XORWOW's step as 160 x 160 bit matrices over GF(2) (bit 32 k + b: bit b of state word k), squared up to
// whole subsequences of 2^67 steps: for digit position k and digit d the matrix of d 4^k subsequences,
// in the order mb_initialize_random reads ([k][d - 1][word of row + 5 row group][lane]). Takes 5 ms, once
// per process.
struct bit_matrix
{
	std::vector<std::array<unsigned long long, 3>> row = std::vector<std::array<unsigned long long, 3>>(160);
	bit_matrix operator*(const bit_matrix& o) const
	{
		bit_matrix r;
		for (int j = 0; j < 160; j++)
		{
			std::array<unsigned long long, 3> acc{};
			for (int q = 0; q < 3; q++)
				for (unsigned long long m = row[j][q]; m; m &= m - 1)
				{
					const auto& x = o.row[64 * q + __builtin_ctzll(m)];
					acc[0] ^= x[0], acc[1] ^= x[1], acc[2] ^= x[2];
				}
			r.row[j] = acc;
		}
		return r;
	}
};

const std::vector<unsigned>& xorwow_jump_table()
{
	static const std::vector<unsigned> table = [] {
		bit_matrix a;
		auto flip = [&](int to, int from) { a.row[to][from / 64] ^= 1ull << (from % 64); };
		for (int b = 0; b < 32; b++)
		{
			for (int k = 0; k < 4; k++) // x <- y <- z <- w <- v
				flip(32 * k + b, 32 * (k + 1) + b);
			// v <- v ^ (v << 4) ^ t ^ (t << 1) with t = x ^ (x >> 2)
			flip(128 + b, 128 + b);
			if (b >= 4)
				flip(128 + b, 128 + b - 4);
			for (int s = 0; s < 2; s++)
				if (b >= s)
				{
					flip(128 + b, b - s);
					if (b - s + 2 < 32)
						flip(128 + b, b - s + 2);
				}
		}
		for (int i = 0; i < 67; i++)
			a = a * a;
		std::vector<unsigned> t((size_t)32 * 3 * 25 * 32);
		for (int k = 0; k < 32; k++)
		{
			const bit_matrix a2 = a * a, a3 = a2 * a;
			const bit_matrix* digit[3] = { &a, &a2, &a3 };
			for (int d = 0; d < 3; d++)
				for (int e = 0; e < 25; e++)
					for (int lane = 0; lane < 32; lane++)
					{
						const int word = e % 5, group = e / 5;
						t[((size_t)(3 * k + d) * 25 + e) * 32 + lane] =
							(unsigned)(digit[d]->row[32 * group + lane][word / 2] >> (32 * (word % 2)));
					}
			a = a2 * a2;
		}
		return t;
	}();
	return table;
}

std::mutex cache_mu;
std::map<size_t, std::vector<char>>& cubin_cache()
{
	static std::map<size_t, std::vector<char>> c;
	return c;
}

template <typename T>
T* ptr(const dbuf& b)
{
	return b.as<T>();
}

unsigned next_pow2(unsigned long long v)
{
	unsigned p = 1;
	while (p < v && p < (1u << 30))
		p <<= 1;
	return p;
}

} // namespace

void cuda_throw(cudaError_t e, const char* what)
{
	if (e == cudaSuccess)
		return;
	cudaGetLastError();
	int code = (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) ? MB_ERR_NO_DEVICE
			   : (e == cudaErrorMemoryAllocation)							 ? MB_ERR_LIMIT
																			 : MB_ERR_CUDA;
	throw engine_error(code, std::string(what) + ": " + cudaGetErrorString(e));
}

dbuf::~dbuf()
{
	if (p)
		cudaFree(p);
}

namespace {
// returned blocks of host_stage, the longest unused first (never destroyed: the driver may be gone at
// process exit)
struct stage_pool
{
	std::mutex mu;
	std::vector<host_stage::block> blocks;
	size_t kept = 0;
	static constexpr size_t most = 64ull << 20;
};
stage_pool& stages()
{
	static stage_pool* pool = new stage_pool;
	return *pool;
}

constexpr size_t huge_page = 2ull << 20;

// Pinned memory, null where that fails. From 2 MB on it is mapped as huge pages and registered: 16 MB take 2
// ms and 64 MB 8 ms, where cudaHostAlloc (4 KB pages) takes 9 and 24 ms, and a copy into new pageable memory
// 7 and 29 ms. Below, cudaHostAlloc.
host_stage::block pinned_block(size_t bytes)
{
	host_stage::block b;
	b.size = bytes;
	if (bytes < huge_page)
	{
		if (cudaHostAlloc(&b.p, bytes, cudaHostAllocPortable) != cudaSuccess)
			b.p = nullptr;
	}
	else
	{
		b.mapped = bytes + huge_page; // room for the alignment
		void* base = mmap(nullptr, b.mapped, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
		if (base != MAP_FAILED)
		{
			b.base = base;
			b.p = reinterpret_cast<void*>((reinterpret_cast<uintptr_t>(base) + huge_page - 1) / huge_page * huge_page);
			madvise(b.p, bytes, MADV_HUGEPAGE);
			madvise(b.p, bytes, MADV_DONTFORK); // (a child that writes must not move the pages that are registered)
			if (cudaHostRegister(b.p, bytes, cudaHostRegisterPortable) != cudaSuccess)
			{
				munmap(base, b.mapped);
				b.p = nullptr;
			}
		}
	}
	if (!b.p)
		(void)cudaGetLastError();
	return b;
}

void free_block(const host_stage::block& b) noexcept
{
	if (b.mapped)
	{
		cudaHostUnregister(b.p);
		munmap(b.base, b.mapped);
	}
	else
		cudaFreeHost(b.p);
}
} // namespace

void host_stage::reserve(size_t bytes)
{
	if (bytes <= b.size)
		return;
	release();
	// powers of two below 2 MB, above whole huge pages with an eighth to spare (the next run's lists differ a little)
	size_t want = 4096;
	if (bytes > huge_page / 2)
		want = (bytes + bytes / 8 + huge_page - 1) / huge_page * huge_page;
	else
		while (want < bytes)
			want <<= 1;
	stage_pool& pool = stages();
	{
		// the smallest block that holds them, of at most four times the size or 8 MB
		std::lock_guard<std::mutex> lk(pool.mu);
		size_t best = pool.blocks.size();
		for (size_t i = 0; i < pool.blocks.size(); i++)
			if (pool.blocks[i].size >= bytes && pool.blocks[i].size <= std::max(4 * want, 4 * huge_page) &&
				(best == pool.blocks.size() || pool.blocks[i].size <= pool.blocks[best].size))
				best = i;
		if (best < pool.blocks.size())
		{
			b = pool.blocks[best];
			pool.blocks.erase(pool.blocks.begin() + (std::ptrdiff_t)best);
			pool.kept -= b.size;
			return;
		}
	}
	b = pinned_block(want);
	if (!b.p)
	{
		b = block();
		b.p = std::malloc(want);
		if (!b.p)
			throw engine_error(MB_ERR_LIMIT, "out of host memory for the result's copies");
		b.size = want;
		b.pinned = false;
	}
}

void host_stage::warm()
{
	static std::once_flag once;
	std::call_once(once, [] {
		host_stage s;
		s.reserve(2 * huge_page - 2 * huge_page / 8);
	});
}

void host_stage::release() noexcept
{
	if (!b.p)
		return;
	std::vector<block> freed;
	if (!b.pinned)
		std::free(b.p);
	else
	{
		stage_pool& pool = stages();
		bool keep = b.size <= stage_pool::most;
		{
			std::lock_guard<std::mutex> lk(pool.mu);
			try
			{
				if (keep)
				{
					freed.reserve(pool.blocks.size());
					pool.blocks.push_back(b);
					pool.kept += b.size;
				}
			}
			catch (...)
			{
				keep = false;
			}
			while (pool.kept > stage_pool::most) // (the block just returned is the last, and fits alone)
			{
				freed.push_back(pool.blocks.front());
				pool.kept -= pool.blocks.front().size;
				pool.blocks.erase(pool.blocks.begin());
			}
		}
		if (!keep)
			free_block(b);
		for (const block& x : freed)
			free_block(x);
	}
	b = block();
}

void dbuf::alloc(size_t n)
{
	if (p)
		cudaFree(p);
	p = nullptr;
	bytes = 0;
	if (n == 0)
		return;
	cudaError_t e = cudaMalloc(&p, n);
	if (e == cudaErrorMemoryAllocation && kept_buffers::give_back())
	{
		(void)cudaGetLastError();
		e = cudaMalloc(&p, n);
	}
	if (e != cudaSuccess)
		p = nullptr;
	cuda_throw(e, "cudaMalloc");
	bytes = n;
}

namespace {
// the kept buffers of the process, the longest unused first (never destroyed: objects may outlive it)
struct kept_list
{
	std::mutex mu;
	std::vector<kept_buffers*> all;
};
kept_list& kept()
{
	static kept_list* list = new kept_list;
	return *list;
}
} // namespace

kept_buffers::kept_buffers()
{
	std::lock_guard<std::mutex> lk(kept().mu);
	kept().all.push_back(this);
}

void kept_buffers::forget()
{
	std::lock_guard<std::mutex> lk(kept().mu);
	std::vector<kept_buffers*>& all = kept().all;
	all.erase(std::find(all.begin(), all.end(), this));
}

// (with the list's mutex held, and the device current)
bool kept_buffers::trim(int device, size_t most)
{
	size_t total = 0;
	bool freed = false;
	for (const kept_buffers* b : kept().all)
		total += b->device == device && b->users == 0 ? b->held() : 0;
	for (kept_buffers* b : kept().all)
		if (total > most && b->device == device && b->users == 0 && b->held() > 0)
		{
			total -= b->held();
			b->drop();
			freed = true;
		}
	return freed;
}

bool kept_buffers::give_back()
{
	int device = 0;
	if (cudaGetDevice(&device) != cudaSuccess)
		return false;
	std::lock_guard<std::mutex> lk(kept().mu);
	return trim(device, 0);
}

kept_use::kept_use(kept_buffers& buffers, int device, size_t most_bytes) : b(buffers), most(most_bytes)
{
	std::lock_guard<std::mutex> lk(kept().mu);
	b.device = device;
	b.users++;
	std::vector<kept_buffers*>& all = kept().all;
	const auto it = std::find(all.begin(), all.end(), &b);
	std::rotate(it, it + 1, all.end());
}

kept_use::~kept_use()
{
	std::lock_guard<std::mutex> lk(kept().mu);
	if (--b.users > 0)
		return;
	if (b.held() > most)
		b.drop();
	kept_buffers::trim(b.device, kept_buffers::max_idle);
}

context::context(int dev) : device(dev)
{
	int count = 0;
	MB_CUDA(cudaGetDeviceCount(&count));
	if (dev < 0 || dev >= count)
		throw engine_error(MB_ERR_NO_DEVICE, "CUDA device " + std::to_string(dev) + " not present");
	MB_CUDA(cudaSetDevice(dev));
	MB_CUDA(cudaFree(nullptr)); // make the primary context current
	cudaDeviceProp prop;
	MB_CUDA(cudaGetDeviceProperties(&prop, dev));
	sm_count = prop.multiProcessorCount;
	cc_major = prop.major;
	cc_minor = prop.minor;
	if (cc_major != 10)
		throw engine_error(MB_ERR_NO_DEVICE, std::string("this engine is built for sm_100a (B200); device is ") +
												 prop.name + " sm_" + std::to_string(cc_major) + std::to_string(cc_minor));
	MB_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
	host_stage::warm(); // 1 ms here, where making the first context takes 700 and more, for the first calls
}

context::~context()
{
	if (stream)
	{
		cudaSetDevice(device);
		cudaStreamDestroy(stream);
	}
}

module::~module()
{
	cudaSetDevice(ctx->device);
	last_runner.reset();
	for (cudaEvent_t e : { run0, run1 })
		if (e)
			cudaEventDestroy(e);
	for (int f = 0; f < FAMILY_COUNT; f++)
		if (mods[f])
			drv().ModuleUnload(mods[f]);
	if (batch_lib)
		cudaLibraryUnload(batch_lib);
}

std::vector<char> compile_cubin(const std::string& generated_code, std::string& log, int family)
{
	static const char* defines[FAMILY_COUNT] = { "#define MB_FAMILY_EXACT 1\n", "#define MB_FAMILY_FAST 1\n",
												 "#define MB_FAMILY_EPOCH 1\n",
												 "#define MB_FAMILY_EPOCH 1\n#define MB_EPOCH_DENSE 1\n",
												 "#define MB_FAMILY_BATCH 1\n" };
	if (family < 0 || family >= FAMILY_COUNT)
		throw engine_error(MB_ERR_INVALID, "bad kernel family");
	if (family == FAMILY_BATCH && generated_code.find("#define MBG_INCREMENTAL 1") == std::string::npos)
		throw engine_error(MB_ERR_INVALID, "the batched kernels need a model whose rates all have the @logic form");
	const std::string source = generated_code + "\n// ---- engine: kernel parameter blocks\n" + mb_params_source +
							   "\n// ---- engine: kernels\n" + defines[family] + mb_engine_source +
							   (family == FAMILY_BATCH ? std::string("\n// ---- engine: batched kernels\n") +
															 mb_batched_source
													   : std::string());
	const int N = parse_constexpr(generated_code, "state_size", -1);
	const int W = parse_constexpr(generated_code, "state_words", -1);
	if (N <= 0 || W != (N + 31) / 32)
		throw engine_error(MB_ERR_COMPILE, "generated code does not define state_size/state_words");
	const std::string inc = "-I" + cuda_include_dir();
	const char* opts[] = { "-arch=sm_100a", "-std=c++17", "-lineinfo", "-DNDEBUG", "--device-int128", inc.c_str() };
	const size_t key = std::hash<std::string>()(source + inc);
	{
		std::lock_guard<std::mutex> lk(cache_mu);
		auto it = cubin_cache().find(key);
		if (it != cubin_cache().end())
			return it->second;
	}
	nvrtcProgram prog;
	if (nvrtcCreateProgram(&prog, source.c_str(), "maboss_b200_model.cu", 0, nullptr, nullptr) != NVRTC_SUCCESS)
		throw engine_error(MB_ERR_COMPILE, "nvrtcCreateProgram failed");
	nvrtcResult r = nvrtcCompileProgram(prog, (int)(sizeof opts / sizeof opts[0]), opts);
	size_t log_size = 0;
	nvrtcGetProgramLogSize(prog, &log_size);
	log.assign(log_size, '\0');
	if (log_size)
		nvrtcGetProgramLog(prog, &log[0]);
	if (r != NVRTC_SUCCESS)
	{
		nvrtcDestroyProgram(&prog);
		throw engine_error(MB_ERR_COMPILE, std::string("NVRTC compilation failed: ") + nvrtcGetErrorString(r) + "\n" + log);
	}
	size_t n = 0;
	nvrtcGetCUBINSize(prog, &n);
	std::vector<char> cubin(n);
	nvrtcGetCUBIN(prog, cubin.data());
	nvrtcDestroyProgram(&prog);
	std::lock_guard<std::mutex> lk(cache_mu);
	cubin_cache()[key] = cubin;
	return cubin;
}

std::unique_ptr<module> compile_module(context& ctx, const std::string& generated_code)
{
	MB_CUDA(cudaSetDevice(ctx.device));
	auto m = std::make_unique<module>();
	m->ctx = &ctx;
	m->state_size = parse_constexpr(generated_code, "state_size", -1);
	m->state_words = parse_constexpr(generated_code, "state_words", -1);
	m->noninternal_count = parse_constexpr(generated_code, "mbg_noninternal_count", -1);
	m->incremental = generated_code.find("#define MBG_INCREMENTAL 1") != std::string::npos ||
					 generated_code.find("#define MBG_INCREMENTAL_MANY 1") != std::string::npos;
	m->integer_rates = generated_code.find("#define MBG_INTEGER_RATES 1") != std::string::npos;
	m->dense_epochs = generated_code.find("#define MBG_EPOCH_DENSE 1") != std::string::npos;
	m->gate_words = parse_constexpr(generated_code, "mbg_gate_words", 0);
	m->table_threads = parse_constexpr(generated_code, "mbg_table_threads", 0);
	m->table_bytes = (size_t)parse_constexpr(generated_code, "mbg_table_bytes", 0);
	m->source = generated_code;
	// the fast family is compiled now so that errors in the generated code surface here
	m->ensure(FAMILY_FAST);
	return m;
}

std::unique_ptr<module> compile_batch_module(context& ctx, const std::string& generated_code)
{
	auto m = std::make_unique<module>();
	m->ctx = &ctx;
	m->state_size = parse_constexpr(generated_code, "state_size", -1);
	m->state_words = parse_constexpr(generated_code, "state_words", -1);
	m->noninternal_count = parse_constexpr(generated_code, "mbg_noninternal_count", -1);
	m->incremental = generated_code.find("#define MBG_INCREMENTAL 1") != std::string::npos;
	m->integer_rates = generated_code.find("#define MBG_INTEGER_RATES 1") != std::string::npos;
	m->gate_words = parse_constexpr(generated_code, "mbg_gate_words", 0);
	m->source = generated_code;
	return m;
}

namespace {
std::mutex family_mu;
}

void module::ensure(int family)
{
	std::lock_guard<std::mutex> lk(family_mu);
	if (loaded[family])
		return;
	MB_CUDA(cudaSetDevice(ctx->device));
	if (!mods[family])
	{
		auto t0 = std::chrono::steady_clock::now();
		std::string lg;
		std::vector<char> cubin = compile_cubin(source, lg, family);
		compile_seconds += std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
		if (!lg.empty())
			log += lg;
		if (family == FAMILY_BATCH)
		{
			cudaKernel_t kf = nullptr, kg = nullptr;
			if (!batch_lib)
				MB_CUDA(cudaLibraryLoadData(&batch_lib, cubin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0));
			MB_CUDA(cudaLibraryGetKernel(&kf, batch_lib, "mb_batched_fast_static"));
			MB_CUDA(cudaLibraryGetKernel(&kg, batch_lib, "mb_batched_grad_static"));
			batched_fast_static = reinterpret_cast<const void*>(kf);
			batched_grad_static = reinterpret_cast<const void*>(kg);
			loaded[family] = true;
			return;
		}
		CUmodule cm = nullptr;
		cu_throw(drv().ModuleLoadData(&cm, cubin.data()), "cuModuleLoadData");
		mods[family] = cm;
	}
	// a call that fails below leaves the family not loaded: the next one goes on with the module that is there
	// (init_random and init_state mark their groups, so they are set last)
	auto get = [&](CUfunction& f, const char* name) {
		cu_throw(drv().ModuleGetFunction(&f, mods[family], name), name);
	};
	if (family == FAMILY_EXACT)
		get(fused_exact, "mb_fused_exact");
	if (family == FAMILY_FAST)
		get(fused_fast, "mb_fused_fast");
	if (family == FAMILY_EPOCH)
		get(sim_epoch, "mb_simulate_epoch");
	if (family == FAMILY_EPOCH_DENSE)
		get(sim_epoch_dense, "mb_simulate_epoch");
	if (family != FAMILY_FAST && !init_random)
	{
		if (!ctx->xorwow_jump.p)
		{
			const std::vector<unsigned>& t = xorwow_jump_table();
			dbuf b(t.size() * sizeof(unsigned));
			// on the context's stream and waited for: cudaMemcpy may return before a copy from pageable memory has
			// reached the device, and neither that stream (non-blocking) nor a caller's waits for the default one
			MB_CUDA(cudaMemcpyAsync(b.p, t.data(), b.bytes, cudaMemcpyHostToDevice, ctx->stream));
			MB_CUDA(cudaStreamSynchronize(ctx->stream));
			ctx->xorwow_jump = std::move(b);
		}
		get(init_random, "mb_initialize_random");
	}
	if (!init_state)
	{
		get(window_epoch, "mb_window_epoch");
		get(final_epoch, "mb_final_epoch");
		get(fixed_epoch, "mb_fixed_epoch");
		get(compact_count, "mb_compact_count");
		get(compact_scan, "mb_compact_scan");
		get(compact_scatter, "mb_compact_scatter");
		get(fixed_extract, "mb_fixed_extract");
		get(bins_extract, "mb_bins_extract");
		get(init_state, "mb_initialize_initial_state");
	}
	loaded[family] = true;
}

void module::ensure_any()
{
	if (!init_state)
		ensure(FAMILY_FAST);
}

void launch(CUfunction f, unsigned grid, unsigned block, size_t smem, cudaStream_t s, void** args)
{
	if (grid == 0)
		return;
	if (smem > 48 * 1024)
		cu_throw(drv().FuncSetAttribute(f, CU_FUNC_ATTRIBUTE_MAX_DYNAMIC_SHARED_SIZE_BYTES, (int)smem),
				 "cuFuncSetAttribute");
	cu_throw(drv().LaunchKernel(f, grid, 1, 1, block, 1, 1, (unsigned)smem, (CUstream)s, args, nullptr),
			 "cuLaunchKernel");
}

int occupancy_blocks(CUfunction f, int block, size_t smem)
{
	int n = 0;
	// the occupancy calculator counts dynamic shared memory above 48 KB only after the opt-in
	if (smem > 48 * 1024)
		cu_throw(drv().FuncSetAttribute(f, CU_FUNC_ATTRIBUTE_MAX_DYNAMIC_SHARED_SIZE_BYTES, (int)smem),
				 "cuFuncSetAttribute");
	cu_throw(drv().OccupancyMaxActiveBlocksPerMultiprocessor(&n, f, block, smem), "cuOccupancyMaxActiveBlocks");
	return std::max(n, 1);
}

run_config config_from_layout(const model_layout& L, int mode)
{
	run_config c;
	c.mode = mode;
	c.sample_count = L.sample_count;
	c.seed = L.seed;
	c.max_time = L.max_time;
	c.time_tick = L.time_tick;
	c.discrete_time = L.discrete_time;
	c.istate = L.istate;
	c.noninternal_nodes = L.noninternal_nodes;
	return c;
}

int occupancy_exponent(long long n_traj, float tick, bool discrete)
{
	// per-bin sums are bounded by n * tick (continuous); discrete bins are plain counts
	if (discrete)
		return 0;
	const double bound = std::max(1.0, (double)std::max(1LL, n_traj) * (double)std::max(tick, 1e-30f));
	return std::clamp((int)std::floor(61.0 - std::log2(bound)), 0, 100);
}

int entropy_exponent(long long n_traj, float tick, bool discrete)
{
	// h <= log2(20) < 8 per slice
	const double per = discrete ? 8.0 : 8.0 * (double)std::max(tick, 1e-30f);
	const double bound = std::max(1.0, (double)std::max(1LL, n_traj) * per);
	return std::clamp((int)std::floor(61.0 - std::log2(bound)), 0, 100);
}

double result::window_prob(int w, unsigned bin) const
{
	if (compact)
	{
		// the window's entries are sorted by state
		const auto a = sp_idx.begin() + (std::ptrdiff_t)sp_begin[w], e = sp_idx.begin() + (std::ptrdiff_t)sp_begin[w + 1];
		const auto it = std::lower_bound(a, e, (unsigned __int128)bin);
		return (it != e && *it == (unsigned __int128)bin) ? sparse_prob((size_t)(it - sp_idx.begin())) : 0.0;
	}
	const size_t i = (size_t)w * n_bins + bin;
	if (discrete_time)
		return (double)win_cnt[i] / (double)n_traj;
	return ((double)win_occ[i] / fx) / ((double)n_traj * (double)time_tick);
}

double result::sparse_prob(size_t i) const
{
	if (discrete_time)
		return (double)sp_val[i] / (double)n_traj;
	return ((double)sp_val[i] / fx) / ((double)n_traj * (double)time_tick);
}

double result::window_th(int w) const
{
	double v = ((double)win_h[w] / fx_h) / (double)n_traj;
	return discrete_time ? v : v / (double)time_tick;
}

// ---------------------------------------------------------------- statistics state

void stats_state::init(module& m, float tick, float tmax, bool discrete, const std::vector<int>& noninternal,
					   long long n, int fixed_capacity_log2, cudaStream_t s, unsigned secs, long long scale_traj,
					   int bin_capacity_log2)
{
	mod = &m;
	if (secs == 0 || (secs & ~7u))
		throw engine_error(MB_ERR_INVALID, "statistics sections must be a non-empty subset of MB_STATS_ALL");
	sections = secs;
	m.ensure_any();
	const int k = (int)noninternal.size();
	if ((secs & 3u) && m.noninternal_count >= 0 && m.noninternal_count != k)
		throw engine_error(MB_ERR_INVALID, "the module was generated for " + std::to_string(m.noninternal_count) +
											   " non-internal nodes, the statistics got " + std::to_string(k));
	if (k > 112)
		throw engine_error(MB_ERR_LIMIT, "more than 112 non-internal nodes (" + std::to_string(k) + ")");
	wide = k > 20 && (secs & 3u);
	for (int i : noninternal)
		if (i < 0 || i >= m.state_size)
			throw engine_error(MB_ERR_INVALID, "non-internal node index out of range");
	if (!(secs & 1u))
		tick = tmax = 1.f; // no windows: one placeholder window
	if (!(tick > 0.f) || !(tmax > 0.f))
		throw engine_error(MB_ERR_INVALID, "max_time and time_tick must be positive");
	const float q = tmax / tick;
	const double T = std::ceil((double)q);
	if (T > (double)(1 << 24))
		throw engine_error(MB_ERR_LIMIT, "too many windows (max_time / time_tick)");
	n_windows = (int)T;
	if (wide && n_windows > 65533)
		throw engine_error(MB_ERR_LIMIT, "sparse window bins support at most 65533 windows");
	n_bins = wide ? 0u : 1u << std::min(k, 20);
	discrete_time = discrete;
	time_tick = tick;
	max_time = tmax;
	noninternal_nodes = noninternal;
	const long long n_scale = scale_traj > 0 ? scale_traj : n;
	fx = std::ldexp(1.0, occupancy_exponent(n_scale, tick, discrete));
	fx_h = std::ldexp(1.0, entropy_exponent(n_scale, tick, discrete));
	h_in_smem = n_windows * sizeof(long long) <= 48 * 1024 ? 1 : 0;

	const size_t cells = (size_t)n_windows * n_bins;
	if (wide)
	{
		// one table for the window bins and (at window T) the final states; automatic size: four
		// slots per trajectory and window (a chaotic network makes ~1.5 distinct bins per trajectory
		// and window and shares almost none across trajectories), 2^16 to 2^28 slots
		const long long want = std::min<long long>(std::max(n, 1LL) * (n_windows + 1), 1LL << 26);
		bin_cap = bin_capacity_log2 > 0 ? (1u << std::min(bin_capacity_log2, 30))
										: std::max(1u << 16, (unsigned)std::min<unsigned long long>(next_pow2(4 * want), 1ull << 28));
		bin_keys.alloc((size_t)bin_cap * sizeof(mb_key128));
		bin_vals.alloc((size_t)bin_cap * sizeof(long long));
	}
	fp_cap = 0;
	if (sections & 4u)
	{
		fp_cap = fixed_capacity_log2 > 0
					 ? (1u << std::min(fixed_capacity_log2, 28))
					 : next_pow2((unsigned long long)std::max(1024LL, std::min(std::max(n, 0LL), 1LL << 22) * 2));
		fp_states.alloc((size_t)fp_cap * m.state_words * sizeof(unsigned));
	}
	// the counts of trajectories at a fixed point are behind the occupancy sums
	has_tail = (sections & 1u) && !wide && !discrete && cells <= tail_max_cells;
	const std::pair<dview*, size_t> parts[] = {
		{ &counters, 64 },
		{ &h, (sections & 1u) ? n_windows * sizeof(long long) : 0 },
		{ &fin, (sections & 2u) && !wide ? n_bins * sizeof(unsigned) : 0 },
		{ &cnt, (sections & 1u) && !wide && discrete ? cells * sizeof(unsigned) : 0 },
		{ &occ, (sections & 1u) && !wide && !discrete
					? cells * (sizeof(long long) + (has_tail ? sizeof(unsigned) : 0))
					: 0 },
		{ &fp_keys, (size_t)fp_cap * sizeof(mb_key128) },
		{ &fp_counts, (size_t)fp_cap * sizeof(unsigned) },
	};
	size_t total = 0;
	for (const auto& part : parts)
		total += (part.second + 255) / 256 * 256;
	arena.alloc(total);
	size_t at = 0;
	for (const auto& part : parts)
	{
		part.first->bytes = part.second;
		part.first->p = part.second ? static_cast<char*>(arena.p) + at : nullptr;
		at += (part.second + 255) / 256 * 256;
	}
	zero(s);

	p = mb_stats_params{};
	p.n_windows = n_windows;
	p.n_bins = n_bins;
	p.win_tick = tick;
	p.h_in_smem = h_in_smem;
	p.fx = fx;
	p.fx_h = fx_h;
	p.win_occ = occ.as<long long>();
	p.win_cnt = cnt.as<unsigned>();
	p.win_h = h.as<long long>();
	p.final_cnt = fin.as<unsigned>();
	p.fp_keys = fp_keys.as<mb_key128>();
	p.fp_counts = fp_counts.as<unsigned>();
	p.fp_states = fp_states.as<unsigned>();
	p.fp_mask = fp_cap ? fp_cap - 1 : 0;
	p.bin_keys = bin_keys.as<mb_key128>();
	p.bin_vals = bin_vals.as<long long>();
	p.bin_mask = bin_cap ? bin_cap - 1 : 0;
	p.fp_overflow = fp_overflow_ctr();
	p.bin_overflow = bin_overflow_ctr();
	p.tail = has_tail ? reinterpret_cast<unsigned*>(occ.as<long long>() + cells) : nullptr;
}

void stats_state::zero(cudaStream_t s)
{
	for (dbuf* b : { &arena, &bin_keys, &bin_vals })
		if (b->p)
			MB_CUDA(cudaMemsetAsync(b->p, 0, b->bytes, s));
	extracted = false;
}

void stats_state::set_istate(const std::vector<float>& is, cudaStream_t s)
{
	if ((int)is.size() != mod->state_size)
		throw engine_error(MB_ERR_INVALID, "initial probabilities must have one entry per node");
	if (istate.bytes != is.size() * sizeof(float))
		istate.alloc(is.size() * sizeof(float));
	MB_CUDA(cudaMemcpyAsync(istate.p, is.data(), istate.bytes, cudaMemcpyHostToDevice, s));
}

void stats_state::window_batch(cudaStream_t s, int n, int stride, int traj_len, const unsigned* traj_states,
							   const float* traj_times, const float* traj_h)
{
	if (!(sections & 1u))
		throw engine_error(MB_ERR_INVALID, "these statistics were created without the window section");
	if (n <= 0)
		return;
	mb_stats_params sp = p;
	void* a[] = { &n, &stride, &traj_len, &traj_states, &traj_times, &traj_h, &sp };
	launch(mod->window_epoch, (n + 255) / 256, 256, h_smem(), s, a);
}

void stats_state::final_batch(cudaStream_t s, int n, int stride, const unsigned* last_states,
							  const unsigned char* statuses)
{
	if (!(sections & 2u))
		throw engine_error(MB_ERR_INVALID, "these statistics were created without the final-state section");
	if (n <= 0)
		return;
	mb_stats_params sp = p;
	void* a[] = { &n, &stride, &last_states, &statuses, &sp };
	launch(mod->final_epoch, (n + 255) / 256, 256, 0, s, a);
}

void stats_state::fixed_batch(cudaStream_t s, int n, int stride, const unsigned* last_states,
							  const unsigned char* statuses)
{
	if (!(sections & 4u))
		throw engine_error(MB_ERR_INVALID, "these statistics were created without the fixed-point section");
	if (n <= 0)
		return;
	mb_stats_params sp = p;
	void* a[] = { &n, &stride, &last_states, &statuses, &sp };
	launch(mod->fixed_epoch, (n + 255) / 256, 256, 0, s, a);
}

std::unique_ptr<result> stats_state::finalize(long long n, cudaStream_t s)
{
	auto rp = std::make_unique<result>();
	result& r = *rp;
	const module& m = *mod;
	r.state_size = m.state_size;
	r.state_words = m.state_words;
	r.n_windows = n_windows;
	r.n_bins = n_bins;
	r.n_traj = n;
	r.discrete_time = discrete_time;
	r.time_tick = time_tick;
	r.max_time = max_time;
	r.noninternal_nodes = noninternal_nodes;
	r.fx = fx;
	r.fx_h = fx_h;
	r.sections = sections;
	r.wide = wide;
	kept_use use(scratch, m.ctx->device, sort_scratch::most);
	const size_t cells = (size_t)n_windows * n_bins;
	// compact the occupied fixed-point slots on the device; the same launch adds the window sums of the
	// trajectories that were counted at their fixed point (and clears the counts)
	if (extracted)
	{
		MB_CUDA(cudaMemsetAsync(extract_ctr(), 0, sizeof(unsigned), s));
		MB_CUDA(cudaMemsetAsync(bin_extract_ctr(), 0, sizeof(unsigned), s));
	}
	extracted = true;
	// compaction buffers, allocated with the first result and kept for the next runs
	if (fp_cap && out_counts.bytes != (size_t)fp_cap * sizeof(unsigned))
	{
		out_counts.alloc((size_t)fp_cap * sizeof(unsigned));
		out_states.alloc((size_t)fp_cap * m.state_words * sizeof(unsigned));
	}
	if (fp_cap || p.tail)
	{
		unsigned cap = fp_cap, tail_blocks = p.tail ? (n_bins + MB_TAIL_COLS - 1) / MB_TAIL_COLS : 0u;
		mb_stats_params sp = p;
		mb_key128* keys = p.fp_keys;
		unsigned* counts = p.fp_counts;
		unsigned* states = p.fp_states;
		unsigned* out_n = extract_ctr();
		unsigned* os = out_states.as<unsigned>();
		unsigned* oc = out_counts.as<unsigned>();
		void* args[] = { &sp, &tail_blocks, &cap, &keys, &counts, &states, &out_n, &os, &oc };
		constexpr unsigned threads = 32 * MB_TAIL_COLS;
		mb::launch(m.fixed_extract, tail_blocks + (cap + threads - 1) / threads, threads, 0, s, args);
	}
	if (wide)
	{
		// compact the occupied bins on the device, then sort them (and merge any key that two
		// concurrent first insertions stored twice) on the host
		if (out_bin_keys.bytes != (size_t)bin_cap * sizeof(mb_key128))
		{
			out_bin_keys.alloc((size_t)bin_cap * sizeof(mb_key128));
			out_bin_vals.alloc((size_t)bin_cap * sizeof(long long));
		}
		unsigned cap = bin_cap;
		mb_key128* keys = p.bin_keys;
		long long* vals = p.bin_vals;
		unsigned* out_n = bin_extract_ctr();
		mb_key128* ok = out_bin_keys.as<mb_key128>();
		long long* ov = out_bin_vals.as<long long>();
		void* args[] = { &cap, &keys, &vals, &out_n, &ok, &ov };
		launch(m.bins_extract, (cap + 255) / 256, 256, 0, s, args);
		unsigned nb = 0, ovf = 0;
		MB_CUDA(cudaMemcpyAsync(&nb, bin_extract_ctr(), sizeof nb, cudaMemcpyDeviceToHost, s));
		MB_CUDA(cudaMemcpyAsync(&ovf, bin_overflow_ctr(), sizeof ovf, cudaMemcpyDeviceToHost, s));
		MB_CUDA(cudaStreamSynchronize(s));
		// sorted on the device, copied into pinned memory, decoded by host threads
		stage.reserve((size_t)nb * (sizeof(mb_key128) + sizeof(long long)));
		const size_t at_vals = (size_t)nb * sizeof(mb_key128);
		if (nb)
		{
			sort_bins(ok, ov, nb, scratch, s);
			MB_CUDA(cudaMemcpyAsync(stage.as<void>(), scratch.out_keys.p, nb * sizeof(mb_key128), cudaMemcpyDeviceToHost, s));
			MB_CUDA(cudaMemcpyAsync(stage.as<void>(at_vals), scratch.out_vals.p, nb * sizeof(long long), cudaMemcpyDeviceToHost, s));
			MB_CUDA(cudaStreamSynchronize(s));
		}
		decode_sorted_bins(stage.as<uint64_t>(), stage.as<long long>(at_vals), nb, n_windows, (int)std::thread::hardware_concurrency(),
						   r.sp_w, r.sp_idx, r.sp_val, r.sp_begin, r.fin_idx, r.fin_cnt);
		r.bin_overflow = ovf;
	}
	// a large dense histogram: only its non-zero cells (selected on the device in cell order), when
	// they are at most a quarter of it
	if ((sections & 1u) && !wide && cells >= compact_min_cells)
	{
		const long long nz = compact_cells(discrete_time ? nullptr : occ.as<long long>(),
										   discrete_time ? cnt.as<unsigned>() : nullptr, cells, cells / 4, cell_idx,
										   cell_vals, m.ctx->sm_count, scratch, s);
		if (nz >= 0)
		{
			stage.reserve((size_t)nz * (sizeof(unsigned long long) + sizeof(long long)));
			const size_t at_vals = (size_t)nz * sizeof(unsigned long long);
			if (nz)
			{
				MB_CUDA(cudaMemcpyAsync(stage.as<void>(), cell_idx.p, (size_t)nz * sizeof(unsigned long long),
										cudaMemcpyDeviceToHost, s));
				MB_CUDA(cudaMemcpyAsync(stage.as<void>(at_vals), cell_vals.p, (size_t)nz * sizeof(long long),
										cudaMemcpyDeviceToHost, s));
				MB_CUDA(cudaStreamSynchronize(s));
			}
			const unsigned long long* idx = stage.as<unsigned long long>();
			const long long* vals = stage.as<long long>(at_vals);
			r.sp_w.resize((size_t)nz);
			r.sp_idx.resize((size_t)nz);
			r.sp_val.resize((size_t)nz);
			parallel_ranges((size_t)nz, (int)std::thread::hardware_concurrency(), [&](size_t a, size_t e) {
				for (size_t i = a; i < e; i++)
				{
					r.sp_w[i] = (int)(idx[i] / n_bins);
					r.sp_idx[i] = (unsigned __int128)(idx[i] % n_bins);
					r.sp_val[i] = vals[i];
				}
			});
			if (stage.bytes() > max_kept_stage)
				stage.release();
			r.sp_begin.assign((size_t)n_windows + 1, 0);
			for (int w = 0; w <= n_windows; w++)
				r.sp_begin[w] = (size_t)(std::lower_bound(r.sp_w.begin(), r.sp_w.end(), w) - r.sp_w.begin());
			r.compact = true;
		}
	}
	// counters, entropy sums, final states and a window histogram of at most 32 MB in one copy, with the first
	// fixed points; a larger histogram straight into the result
	const dview& win = discrete_time ? cnt : occ;
	const size_t win_bytes = cells * (discrete_time ? sizeof(unsigned) : sizeof(long long));
	const bool has_win = (sections & 1u) && !wide && !r.compact, win_staged = has_win && win_bytes <= (32u << 20);
	auto offset = [&](const dview& v) { return (size_t)(static_cast<char*>(v.p) - static_cast<char*>(arena.p)); };
	size_t front = 64;
	if (h.p)
		front = offset(h) + h.bytes;
	if (fin.p)
		front = offset(fin) + fin.bytes;
	if (win_staged)
		front = offset(win) + win_bytes;
	front = (front + 255) / 256 * 256;
	const int W = m.state_words;
	const unsigned first = std::min(fp_cap, 256u); // fixed points copied before their number is known
	stage.reserve(front + (size_t)first * (W + 1) * sizeof(unsigned));
	const size_t at_counts = front, at_states = front + first * sizeof(unsigned);
	MB_CUDA(cudaMemcpyAsync(stage.as<void>(), arena.p, std::min(front, arena.bytes), cudaMemcpyDeviceToHost, s));
	if (first)
	{
		MB_CUDA(cudaMemcpyAsync(stage.as<void>(at_counts), out_counts.p, first * sizeof(unsigned), cudaMemcpyDeviceToHost, s));
		MB_CUDA(cudaMemcpyAsync(stage.as<void>(at_states), out_states.p, (size_t)first * W * sizeof(unsigned),
								cudaMemcpyDeviceToHost, s));
	}
	if (has_win && !win_staged)
	{
		if (discrete_time)
			r.win_cnt.resize(cells);
		else
			r.win_occ.resize(cells);
		void* to = discrete_time ? static_cast<void*>(r.win_cnt.data()) : static_cast<void*>(r.win_occ.data());
		MB_CUDA(cudaMemcpyAsync(to, win.p, win_bytes, cudaMemcpyDeviceToHost, s));
	}
	MB_CUDA(cudaStreamSynchronize(s));
	const unsigned* ctr = stage.as<unsigned>();
	std::memcpy(&r.transitions, stage.as<char>(sizeof(unsigned long long)), sizeof r.transitions);
	r.fixed_overflow = ctr[4];
	r.rate_errors = ctr[6];
	const unsigned nfp = ctr[5];
	if (h.p)
		r.win_h.assign(stage.as<long long>(offset(h)), stage.as<long long>(offset(h)) + n_windows);
	if (fin.p)
		r.final_cnt.assign(stage.as<unsigned>(offset(fin)), stage.as<unsigned>(offset(fin)) + n_bins);
	if (win_staged && discrete_time)
		r.win_cnt.assign(stage.as<unsigned>(offset(cnt)), stage.as<unsigned>(offset(cnt)) + cells);
	else if (win_staged)
		r.win_occ.assign(stage.as<long long>(offset(occ)), stage.as<long long>(offset(occ)) + cells);
	std::vector<unsigned> st((size_t)nfp * W), cn(nfp);
	if (nfp > first)
	{
		stage.reserve((size_t)nfp * (W + 1) * sizeof(unsigned));
		MB_CUDA(cudaMemcpyAsync(stage.as<void>(), out_counts.p, nfp * sizeof(unsigned), cudaMemcpyDeviceToHost, s));
		MB_CUDA(cudaMemcpyAsync(stage.as<unsigned>() + nfp, out_states.p, st.size() * sizeof(unsigned), cudaMemcpyDeviceToHost, s));
		MB_CUDA(cudaStreamSynchronize(s));
		std::copy_n(stage.as<unsigned>(), nfp, cn.begin());
		std::copy_n(stage.as<unsigned>() + nfp, st.size(), st.begin());
	}
	else
	{
		std::copy_n(stage.as<unsigned>(at_counts), nfp, cn.begin());
		std::copy_n(stage.as<unsigned>(at_states), st.size(), st.begin());
	}
	set_fixed_sorted(r, st, cn);
	return rp;
}

void set_fixed_sorted(result& r, const std::vector<unsigned>& st, const std::vector<unsigned>& cn)
{
	const int W = r.state_words;
	const size_t nfp = cn.size();
	std::vector<size_t> order(nfp);
	std::iota(order.begin(), order.end(), size_t(0));
	std::sort(order.begin(), order.end(), [&](size_t a, size_t b) {
		for (int w = W - 1; w >= 0; w--)
		{
			const unsigned x = st[a * W + w], y = st[b * W + w];
			if (x != y)
				return x < y;
		}
		return false;
	});
	r.fixed_states.resize(nfp * W);
	r.fixed_counts.resize(nfp);
	for (size_t i = 0; i < nfp; i++)
	{
		std::copy(st.begin() + order[i] * W, st.begin() + (order[i] + 1) * W, r.fixed_states.begin() + i * W);
		r.fixed_counts[i] = cn[order[i]];
	}
}

std::unique_ptr<result> merge_results(const std::vector<const result*>& parts)
{
	if (parts.empty())
		throw engine_error(MB_ERR_INVALID, "merge: no results");
	const result& a = *parts[0];
	auto out = std::make_unique<result>();
	result& r = *out;
	r.state_size = a.state_size;
	r.state_words = a.state_words;
	r.n_windows = a.n_windows;
	r.n_bins = a.n_bins;
	r.discrete_time = a.discrete_time;
	r.time_tick = a.time_tick;
	r.max_time = a.max_time;
	r.noninternal_nodes = a.noninternal_nodes;
	r.fx = a.fx;
	r.fx_h = a.fx_h;
	r.sections = a.sections;
	r.win_occ.assign(a.win_occ.size(), 0);
	r.win_cnt.assign(a.win_cnt.size(), 0);
	r.win_h.assign(a.win_h.size(), 0);
	r.final_cnt.assign(a.final_cnt.size(), 0);
	r.wide = a.wide;
	r.compact = a.compact;
	r.bin_overflow = 0;
	std::map<std::vector<unsigned>, unsigned long long> fixed;
	std::map<std::pair<int, unsigned __int128>, long long> bins;
	std::map<unsigned __int128, unsigned long long> finals;
	for (const result* p : parts)
	{
		const result& b = *p;
		if (b.wide != a.wide || b.compact != a.compact)
			throw engine_error(MB_ERR_INVALID, "merge: the results are not shards of the same run");
		for (size_t i = 0; i < b.sp_w.size(); i++)
			bins[{ b.sp_w[i], b.sp_idx[i] }] += b.sp_val[i];
		for (size_t i = 0; i < b.fin_idx.size(); i++)
			finals[b.fin_idx[i]] += b.fin_cnt[i];
		r.bin_overflow += b.bin_overflow;
		if (b.state_size != a.state_size || b.n_windows != a.n_windows || b.n_bins != a.n_bins ||
			b.discrete_time != a.discrete_time || b.time_tick != a.time_tick || b.max_time != a.max_time ||
			b.noninternal_nodes != a.noninternal_nodes || b.sections != a.sections)
			throw engine_error(MB_ERR_INVALID, "merge: the results are not shards of the same run");
		if (b.fx != a.fx || b.fx_h != a.fx_h)
			throw engine_error(MB_ERR_INVALID, "merge: different fixed-point scales (run every shard with the same "
											   "stats_trajectories)");
		r.n_traj += b.n_traj;
		for (size_t i = 0; i < r.win_occ.size(); i++)
			r.win_occ[i] += b.win_occ[i];
		for (size_t i = 0; i < r.win_cnt.size(); i++)
			r.win_cnt[i] += b.win_cnt[i];
		for (size_t i = 0; i < r.win_h.size(); i++)
			r.win_h[i] += b.win_h[i];
		for (size_t i = 0; i < r.final_cnt.size(); i++)
			r.final_cnt[i] += b.final_cnt[i];
		for (size_t j = 0; j < b.fixed_counts.size(); j++)
			fixed[std::vector<unsigned>(b.fixed_states.begin() + j * b.state_words,
										b.fixed_states.begin() + (j + 1) * b.state_words)] += b.fixed_counts[j];
		r.fixed_overflow += b.fixed_overflow;
		r.rate_errors += b.rate_errors;
		r.transitions += b.transitions;
		r.kernel_ms = std::max(r.kernel_ms, b.kernel_ms);
		r.total_ms = std::max(r.total_ms, b.total_ms);
		r.epochs = std::max(r.epochs, b.epochs);
	}
	std::vector<unsigned> st, cn;
	for (auto& [state, count] : fixed)
	{
		st.insert(st.end(), state.begin(), state.end());
		cn.push_back((unsigned)count);
	}
	set_fixed_sorted(r, st, cn);
	if (r.wide || r.compact)
	{
		for (auto& [key, v] : bins)
		{
			r.sp_w.push_back(key.first);
			r.sp_idx.push_back(key.second);
			r.sp_val.push_back(v);
		}
		for (auto& [idx, c] : finals)
		{
			r.fin_idx.push_back(idx);
			r.fin_cnt.push_back((unsigned)c);
		}
		r.sp_begin.assign(r.n_windows + 1, 0);
		for (int w = 0, e = 0; w <= r.n_windows; w++)
		{
			while (e < (int)r.sp_w.size() && r.sp_w[e] < w)
				e++;
			r.sp_begin[w] = e;
		}
	}
	return out;
}

// ---------------------------------------------------------------- run drivers

namespace {

// Enqueues the fused kernel (and, in exact mode with `rng`, the parallel XORWOW initialisation);
// returns the number of kernels launched.
unsigned launch_fused(module& m, const run_config& c, stats_state& st, long long n, cudaStream_t s, void* rng,
					  unsigned* init_states)
{
	if (n == 0)
		return 0;
	mb_fused_params P{};
	P.st = st.p;
	P.istate = st.istate.as<float>();
	P.seed = c.seed;
	P.first_traj = c.first_traj;
	P.n_traj = (unsigned)n;
	P.traj_len = c.mode == MB_MODE_FUSED_EXACT ? c.traj_len : 0;
	P.next_traj = st.next_traj();
	P.transitions = st.transitions();
	P.errors = st.error_ctr();
	m.ensure(c.mode == MB_MODE_FUSED_EXACT ? FAMILY_EXACT : FAMILY_FAST);
	CUfunction f = c.mode == MB_MODE_FUSED_EXACT ? m.fused_exact : m.fused_fast;
	unsigned launches = 0;
	if (c.mode == MB_MODE_FUSED_EXACT && rng)
	{
		int cnt = (int)n, per = init_random_per(n);
		unsigned long long seed = c.seed, first = c.first_traj;
		unsigned* jump = m.ctx->xorwow_jump.as<unsigned>();
		void* a[] = { &cnt, &seed, &first, &rng, &per, &jump, &P.istate, &init_states, &cnt };
		launch(m.init_random, init_random_blocks(n, per), 256, 0, s, a);
		P.rands = rng;
		P.init_states = init_states;
		launches++;
	}
	int block = c.block;
	size_t smem = st.h_smem();
	// discrete counts in shared memory: histograms of at most 16 KB, so that the occupancy stays (lockstep kernels)
	P.st.cnt_in_smem = m.gate_words && (c.mode == MB_MODE_FUSED_EXACT || m.fast_incremental()) && st.discrete_time &&
					   !st.wide && (size_t)st.n_windows * st.n_bins <= 4096;
	if (P.st.cnt_in_smem)
		smem += (size_t)st.n_windows * st.n_bins * sizeof(unsigned);
	const bool dense = !(c.mode == MB_MODE_FUSED_EXACT ? m.incremental : m.fast_incremental());
	if (dense && block == 256 && c.blocks_per_sm <= 0)
	{
		// (no smaller shape asked for) a kernel of more than 128 registers has one block of 256 threads on an SM: smaller
		// ones leave fewer registers unused
		int most = occupancy_blocks(f, 256, smem) * 256;
		for (int b : { 192, 128 })
			if (most < 512 && occupancy_blocks(f, b, smem) * b > most)
				most = occupancy_blocks(f, b, smem) * b, block = b;
	}
	if (!dense)
	{
		// per thread in shared memory: state words, unstable masks and word rate sums; or per warp its array
		constexpr size_t max_smem = 227 * 1024;
		block = std::min(block, 128);
		if (m.table_threads && c.blocks_per_sm <= 0 && c.block > 128)
		{
			// (no shape of at most 128 threads asked for) one block an SM with all that fits; in a small run only
			// the warps that it needs on each SM
			const long long lanes = lanes_per_warp(n, m.ctx->sm_count), warps = (n + lanes - 1) / lanes;
			block = (int)std::min<long long>(m.table_threads, 32 * ((warps + m.ctx->sm_count - 1) / m.ctx->sm_count));
		}
		while (block > 32 && m.fused_smem(block) + smem > max_smem)
			block -= 32;
		if (m.fused_smem(block) + smem > max_smem)
			throw engine_error(MB_ERR_LIMIT, "model too large for the incremental kernel's shared memory");
		smem += m.fused_smem(block);
	}
	// an explicit block count per SM also fixes the shared-memory carve-out to what those blocks need
	// (+1 KB reserved per block), leaving the rest of the SM's 256 KB of L1/shared memory to L1
	// for the model tables; by default the driver picks the carve-out of the highest occupancy
	int carve = -1;
	if (c.blocks_per_sm > 0)
		carve = std::min(100, (int)((c.blocks_per_sm * (smem + 1024) * 100 + 228 * 1024 - 1) / (228 * 1024)));
	cu_throw(drv().FuncSetAttribute(f, CU_FUNC_ATTRIBUTE_PREFERRED_SHARED_MEMORY_CARVEOUT, carve),
			 "cuFuncSetAttribute");
	const int per_sm = c.blocks_per_sm > 0 ? c.blocks_per_sm : occupancy_blocks(f, block, smem);
	P.lanes = dense && m.state_words > max_spread_words ? 32 : lanes_per_warp(n, m.ctx->sm_count);
	const long long per_block = (long long)(block / 32) * P.lanes, needed = (n + per_block - 1) / per_block;
	const unsigned grid = (unsigned)std::max(1LL, std::min<long long>(needed, (long long)per_sm * m.ctx->sm_count));
	void* args[] = { &P };
	launch(f, grid, block, smem, s, args);
	return launches + 1;
}

// Buffered epochs (simulation_runner.cu:54-180): simulate -> stats -> partition -> refill.
} // namespace

void simulate_epoch(module& m, bool dense, cudaStream_t s, int n, int stride, int L, unsigned* last_states,
					float* last_times, void* rands, unsigned* traj_states, float* traj_times, float* traj_h,
					unsigned char* statuses, unsigned long long* transitions)
{
	if (n <= 0)
		return;
	void* a[] = { &n, &stride, &L, &last_states, &last_times, &rands, &traj_states, &traj_times, &traj_h, &statuses,
				  &transitions };
	if (dense)
	{
		m.ensure(FAMILY_EPOCH_DENSE);
		launch(m.sim_epoch_dense, (n + 255) / 256, 256, 0, s, a);
		return;
	}
	m.ensure(FAMILY_EPOCH);
	if (!m.incremental || m.dense_epochs)
	{
		launch(m.sim_epoch, (n + 255) / 256, 256, 0, s, a);
		return;
	}
	// per thread in shared memory: state words, unstable masks, word-end running sums; or per warp its array
	constexpr size_t max_smem = 227 * 1024;
	int block = 128;
	auto bytes = [&](int b) { return m.fused_smem(b) - m.table_bytes; }; // (its tables are in global memory)
	while (block > 32 && bytes(block) > max_smem)
		block -= 32;
	const size_t smem = bytes(block);
	if (smem > max_smem)
		throw engine_error(MB_ERR_LIMIT, "model too large for the incremental epoch kernel's shared memory");
	launch(m.sim_epoch, (n + block - 1) / block, block, smem, s, a);
}

size_t partition_scratch_bytes(int n)
{
	const size_t nb = (size_t)(std::max(n, 1) + 1023) / 1024;
	return (2 * nb + 1) * sizeof(unsigned);
}

void partition(module& m, cudaStream_t s, int n, int stride, const unsigned char* statuses, const unsigned* states,
			   const float* times, const void* rands, unsigned* out_states, float* out_times, void* out_rands,
			   void* scratch, unsigned* kept, bool rejected_rands)
{
	if (n < 0 || stride < n)
		throw engine_error(MB_ERR_INVALID, "partition: need 0 <= n <= stride");
	if (n > (1 << 30))
		throw engine_error(MB_ERR_LIMIT, "partition: batch larger than 2^30 trajectories");
	m.ensure_any();
	if (n == 0)
	{
		MB_CUDA(cudaMemsetAsync(kept, 0, sizeof(unsigned), s));
		return;
	}
	int nb = (n + 1023) / 1024;
	unsigned* bcp = static_cast<unsigned*>(scratch);
	unsigned* bop = bcp + nb;
	void* a1[] = { &n, &statuses, &bcp };
	launch(m.compact_count, nb, 1024, 0, s, a1);
	void* a2[] = { &nb, &bcp, &bop };
	launch(m.compact_scan, 1, 1024, 0, s, a2);
	int rej = rejected_rands ? 1 : 0;
	void* a3[] = { &n, &stride, &statuses, &bop, &states, &times, &rands, &out_states, &out_times, &out_rands, &rej };
	launch(m.compact_scatter, nb, 1024, 0, s, a3);
	MB_CUDA(cudaMemcpyAsync(kept, bop + nb, sizeof(unsigned), cudaMemcpyDeviceToDevice, s));
}

namespace {

void run_epochs(module& m, const run_config& c, stats_state& st, epoch_buffers& E, long long n, cudaStream_t s,
				int& epochs, unsigned& launches)
{
	const int W = m.state_words;
	const int L = std::max(2, c.traj_len);
	if (n <= 0)
		return;
	m.ensure(c.mode == MB_MODE_EPOCH_DENSE ? FAMILY_EPOCH_DENSE : FAMILY_EPOCH);
	const long long Bll = std::min<long long>(std::max(1, c.batch_limit), n);
	const int B = (int)Bll;
	if (E.batch != B) // (a runner's L and W do not change)
	{
		E.drop();
		for (int k = 0; k < 2; k++)
		{
			E.states[k].alloc((size_t)W * B * 4);
			E.times[k].alloc((size_t)B * 4);
			E.rands[k].alloc((size_t)B * sizeof(curandState));
		}
		E.traj_states.alloc((size_t)L * W * B * 4);
		E.traj_times.alloc((size_t)L * B * 4);
		E.traj_h.alloc((size_t)L * B * 4);
		E.statuses.alloc((size_t)B);
		E.scratch.alloc(256 + partition_scratch_bytes(B));
		E.batch = B;
	}
	dbuf &st0 = E.states[0], &st1 = E.states[1], &t0 = E.times[0], &t1 = E.times[1], &r0 = E.rands[0], &r1 = E.rands[1];
	dbuf &ts = E.traj_states, &tt = E.traj_times, &th = E.traj_h, &stat = E.statuses, &scratch = E.scratch;
	unsigned long long* trans = st.transitions();
	float* istate = st.istate.as<float>();

	// fresh_rng: new random streams (trajectory id `first` + i); else the refilled slots continue the
	// random states that the partition left there (the reference's refill, simulation_runner.cu:150-153)
	auto init = [&](int cnt, int offset, unsigned long long first, dbuf& sbuf, dbuf& tbuf, dbuf& rbuf,
					bool fresh_rng) {
		unsigned long long seed = c.seed;
		void* rptr = rbuf.as<char>() + (size_t)offset * sizeof(curandState);
		int per = init_random_per(cnt);
		unsigned* jump = m.ctx->xorwow_jump.as<unsigned>();
		unsigned* no_states = nullptr;
		void* a1[] = { &cnt, &seed, &first, &rptr, &per, &jump, &istate, &no_states, &cnt };
		if (fresh_rng)
		{
			launch(m.init_random, init_random_blocks(cnt, per), 256, 0, s, a1);
			launches++;
		}
		int stride = B;
		unsigned* sp = sbuf.as<unsigned>() + offset;
		float* tp = tbuf.as<float>() + offset;
		void* a2[] = { &cnt, &stride, &istate, &sp, &tp, &rptr };
		launch(m.init_state, (cnt + 255) / 256, 256, 0, s, a2);
		launches++;
	};

	init(B, 0, c.first_traj, st0, t0, r0, true);
	long long next_id = B;
	int in_batch = B;
	dbuf *cs = &st0, *ct = &t0, *cr = &r0, *ns = &st1, *nt = &t1, *nr = &r1;
	while (in_batch > 0)
	{
		int stride = B;
		int len = L;
		unsigned* ls = cs->as<unsigned>();
		float* lt = ct->as<float>();
		void* rr = cr->p;
		unsigned* tsp = ts.as<unsigned>();
		float* ttp = tt.as<float>();
		float* thp = th.as<float>();
		unsigned char* stp = stat.as<unsigned char>();
		simulate_epoch(m, c.mode == MB_MODE_EPOCH_DENSE, s, in_batch, stride, len, ls, lt, rr, tsp, ttp, thp, stp,
					   trans);
		launches += 7; // simulate, three statistics, three partition kernels
		// statistics plugins in the order of main.cpp:65-74
		st.final_batch(s, in_batch, stride, ls, stp);
		st.fixed_batch(s, in_batch, stride, ls, stp);
		st.window_batch(s, in_batch, stride, len, tsp, ttp, thp);
		// partition CONTINUE trajectories to the front of the other buffer set
		unsigned* kept_dev = scratch.as<unsigned>();
		partition(m, s, in_batch, stride, stp, ls, lt, rr, ns->as<unsigned>(), nt->as<float>(), nr->p,
				  scratch.as<char>() + 256, kept_dev, c.refill_reuse_rng);
		unsigned kept = 0;
		MB_CUDA(cudaMemcpyAsync(&kept, kept_dev, sizeof kept, cudaMemcpyDeviceToHost, s));
		MB_CUDA(cudaStreamSynchronize(s));
		std::swap(cs, ns);
		std::swap(ct, nt);
		std::swap(cr, nr);
		const int add = (int)std::max(0LL, std::min<long long>(B - (long long)kept, n - next_id));
		if (add > 0)
		{
			init(add, (int)kept, c.first_traj + next_id, *cs, *ct, *cr, !c.refill_reuse_rng);
			next_id += add;
		}
		in_batch = (int)kept + add;
		epochs++;
	}
}

} // namespace

runner::runner(module& m, const run_config& c) : mod(&m), cfg(c)
{
	MB_CUDA(cudaSetDevice(m.ctx->device));
	if (c.sample_count < 0)
		throw engine_error(MB_ERR_INVALID, "negative sample_count");
	if (c.block <= 0 || c.block > 256 || (c.block % 32) != 0)
		throw engine_error(MB_ERR_INVALID, "block size must be a multiple of 32 in [32, 256]");
	if (c.mode != MB_MODE_EPOCH && c.mode != MB_MODE_EPOCH_DENSE && c.mode != MB_MODE_FUSED_EXACT &&
		c.mode != MB_MODE_FUSED_FAST)
		throw engine_error(MB_ERR_INVALID, "unknown run mode");
	cudaStream_t s = m.ctx->stream;
	if (c.stats_trajectories < 0 || (c.stats_trajectories > 0 && c.stats_trajectories < c.sample_count))
		throw engine_error(MB_ERR_INVALID, "stats_trajectories must be 0 or at least sample_count");
	st.init(m, c.time_tick, c.max_time, c.discrete_time, c.noninternal_nodes, c.sample_count, c.fixed_capacity_log2, s,
			7u, c.stats_trajectories, c.bin_capacity_log2);
	st.set_istate(c.istate, s);
	if (c.mode == MB_MODE_FUSED_EXACT && c.sample_count > 0)
	{
		rng_chunk = std::min(c.sample_count, max_rng_states);
		if (m.incremental)
			rng_chunk = std::max(1LL, std::min(rng_chunk, max_init_bytes / (4 * m.state_words)));
		for (bool done = false; !done;)
			try
			{
				rng.alloc((size_t)rng_chunk * sizeof(curandState));
				if (m.incremental)
					init_states.alloc((size_t)4 * m.state_words * rng_chunk);
				done = true;
			}
			catch (const engine_error& e)
			{
				// less memory, more launches
				if (e.code != MB_ERR_LIMIT || rng_chunk <= 1 << 16)
					throw;
				rng.alloc(0);
				rng_chunk = (rng_chunk + 1) / 2;
			}
	}
	MB_CUDA(cudaEventCreate(&ev0));
	MB_CUDA(cudaEventCreate(&ev1));
	MB_CUDA(cudaStreamSynchronize(s));
}

runner::~runner()
{
	cudaSetDevice(mod->ctx->device);
	for (cudaEvent_t e : { ev0, ev1 })
		if (e)
			cudaEventDestroy(e);
}

unsigned runner::kernel_launches() const { return launches; }

void runner::launch(cudaStream_t s)
{
	MB_CUDA(cudaSetDevice(mod->ctx->device));
	st.set_istate(cfg.istate, s); // the run's input, uploaded by every launch
	st.zero(s);
	MB_CUDA(cudaEventRecord(ev0, s));
	epochs = 0;
	launches = 0;
	if (cfg.mode == MB_MODE_EPOCH || cfg.mode == MB_MODE_EPOCH_DENSE)
	{
		kept_use use(epoch, mod->ctx->device, epoch_buffers::most); // (the last epoch is waited for)
		run_epochs(*mod, cfg, st, epoch, cfg.sample_count, s, epochs, launches);
	}
	else
	{
		if (cfg.sample_count > 0xffffffffLL)
			throw engine_error(MB_ERR_LIMIT, "sample_count above 2^32 - 1");
		run_config c = cfg;
		const long long chunk = rng_chunk > 0 ? rng_chunk : std::max(1LL, cfg.sample_count);
		for (long long done = 0; done < cfg.sample_count; done += chunk)
		{
			if (done)
				MB_CUDA(cudaMemsetAsync(st.next_traj(), 0, sizeof(unsigned long long), s));
			c.first_traj = cfg.first_traj + (unsigned long long)done;
			launches += launch_fused(*mod, c, st, std::min(chunk, cfg.sample_count - done), s, rng.p, init_states.as<unsigned>());
		}
		epochs = 1;
	}
	MB_CUDA(cudaEventRecord(ev1, s));
}

std::unique_ptr<result> runner::collect(cudaStream_t s)
{
	MB_CUDA(cudaSetDevice(mod->ctx->device));
	auto r = st.finalize(cfg.sample_count, s);
	MB_CUDA(cudaEventSynchronize(ev1));
	MB_CUDA(cudaEventElapsedTime(&r->kernel_ms, ev0, ev1));
	r->epochs = epochs;
	return r;
}

std::vector<tuned_shape> autotune(module& m, const run_config& c)
{
	if (c.mode != MB_MODE_FUSED_EXACT && c.mode != MB_MODE_FUSED_FAST)
		throw engine_error(MB_ERR_INVALID, "the autotuner covers the fused modes");
	m.ensure(c.mode == MB_MODE_FUSED_EXACT ? FAMILY_EXACT : FAMILY_FAST);
	CUfunction f = c.mode == MB_MODE_FUSED_EXACT ? m.fused_exact : m.fused_fast;
	// candidate shapes: the incremental kernels take at most 128 threads and 12 bytes of shared memory
	// per state word and thread; the dense kernels any multiple of 32 up to 256
	std::vector<std::pair<int, int>> cands;
	const bool incr = c.mode == MB_MODE_FUSED_EXACT ? m.incremental : m.fast_incremental();
	if (incr && m.table_threads)
		cands.push_back({ 256, 0 }); // the kernel's own shape (mbg_table_threads, one block an SM)
	const std::vector<int> blocks = incr ? std::vector<int>{ 128, 96, 64 } : std::vector<int>{ 256, 128 };
	for (int block : blocks)
	{
		size_t smem = incr ? m.fused_smem(block) : 0;
		if (smem > 227 * 1024)
			continue;
		MB_CUDA(cudaSetDevice(m.ctx->device));
		cu_throw(drv().FuncSetAttribute(f, CU_FUNC_ATTRIBUTE_PREFERRED_SHARED_MEMORY_CARVEOUT, -1), "cuFuncSetAttribute");
		const int per_sm = occupancy_blocks(f, block, smem + (size_t)std::ceil(std::max(1.0, (double)c.max_time /
																							   std::max(c.time_tick, 1e-30f))) *
																  8);
		cands.push_back({ block, per_sm });
		if (per_sm >= 2)
			cands.push_back({ block, per_sm - 1 });
	}
	if (cands.empty())
		throw engine_error(MB_ERR_LIMIT, "model too large for the incremental kernel's shared memory");
	// a slice of the run: four times what the largest candidate keeps resident, at most the run itself
	long long resident = 0;
	for (auto& cd : cands)
		resident = std::max(resident, (long long)(cd.second ? cd.first * cd.second : m.table_threads) * m.ctx->sm_count);
	run_config probe = c;
	probe.sample_count = std::max(1LL, std::min(c.sample_count, 4 * resident));
	probe.stats_trajectories = 0;
	std::vector<tuned_shape> out;
	for (size_t i = 0; i < cands.size(); i++)
	{
		probe.block = cands[i].first;
		probe.blocks_per_sm = cands[i].second;
		runner rn(m, probe);
		for (int rep = 0; rep < (i == 0 ? 2 : 1); rep++) // the first probe also warms the module up
		{
			rn.launch(m.ctx->stream);
			auto r = rn.collect(m.ctx->stream);
			if (rep == (i == 0 ? 1 : 0))
				out.push_back({ cands[i].first, cands[i].second,
								r->kernel_ms > 0 ? (double)r->transitions / (r->kernel_ms * 1e-3) : 0.0 });
		}
	}
	std::stable_sort(out.begin(), out.end(),
					 [](const tuned_shape& a, const tuned_shape& b) { return a.transitions_per_s > b.transitions_per_s; });
	return out;
}

bool same_run(const run_config& a, const run_config& b)
{
	return a.mode == b.mode && a.sample_count == b.sample_count && a.seed == b.seed && a.first_traj == b.first_traj &&
		   a.max_time == b.max_time && a.time_tick == b.time_tick && a.discrete_time == b.discrete_time &&
		   a.istate == b.istate && a.noninternal_nodes == b.noninternal_nodes && a.traj_len == b.traj_len &&
		   a.batch_limit == b.batch_limit && a.block == b.block && a.blocks_per_sm == b.blocks_per_sm &&
		   a.fixed_capacity_log2 == b.fixed_capacity_log2 && a.stats_trajectories == b.stats_trajectories &&
		   a.bin_capacity_log2 == b.bin_capacity_log2 && a.refill_reuse_rng == b.refill_reuse_rng;
}

std::unique_ptr<result> run(module& m, const run_config& c)
{
	// the module keeps the runner (device buffers) of its last run and reuses it for the same config
	std::lock_guard<std::mutex> lk(m.run_mu);
	cudaStream_t s = m.ctx->stream;
	MB_CUDA(cudaSetDevice(m.ctx->device));
	if (!m.run0)
		MB_CUDA(cudaEventCreate(&m.run0));
	if (!m.run1)
		MB_CUDA(cudaEventCreate(&m.run1));
	MB_CUDA(cudaEventRecord(m.run0, s));
	if (!m.last_runner || !same_run(m.last_runner->cfg, c))
	{
		m.last_runner.reset();
		m.last_runner = std::make_unique<runner>(m, c);
	}
	runner& rn = *m.last_runner;
	rn.launch(s);
	std::unique_ptr<result> r = rn.collect(s);
	MB_CUDA(cudaEventRecord(m.run1, s));
	MB_CUDA(cudaEventSynchronize(m.run1));
	MB_CUDA(cudaEventElapsedTime(&r->total_ms, m.run0, m.run1));
	return r;
}

} // namespace mb
