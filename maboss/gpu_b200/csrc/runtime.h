// Host runtime of the B200 trajectory engine: device context, NVRTC-compiled model modules,
// run drivers (fused persistent kernel and buffered epochs) and host-side results.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "codegen.h"
#include "maboss_b200.h"
#include "sparse_bins.h"
#include "kernels/params.cuh"

namespace mb {

// Status codes (MB_OK, MB_ERR_*) and run modes (MB_MODE_*) come from the C ABI header.

struct engine_error : std::runtime_error
{
	int code;
	engine_error(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

void cuda_throw(cudaError_t e, const char* what);
#define MB_CUDA(x) ::mb::cuda_throw((x), #x)

// Lanes of each warp that take trajectories in a run of n. A warp's lanes run their own trajectories, so
// a step of 32 of them costs two to three times the instructions of a step of one, and a run too small
// for two warps on each scheduler waits on latencies: it is spread over 8 warps an SM with fewer lanes
// each. Kernel time before -> after (with 12 warps an SM), us: 32-node example model, exact mode, 1e3
// trajectories 1255 -> 411 (408), 1e4 1360 -> 645 (630); 50 nodes fast 1e3 687 -> 363 (365), 1e4 734 ->
// 617 (652), 3e4 799 -> 729 (768); 87-node example model fast 3e4 4804 -> 4585 (4969: slower).
inline int lanes_per_warp(long long n, int sm_count)
{
	const long long warps = 8LL * sm_count, lanes = (n + warps - 1) / warps;
	return lanes < 1 ? 1 : lanes > 32 ? 32 : (int)lanes;
}

// The dense kernels of larger networks are not spread: a step is the code of every node, more than an SM's instruction
// caches hold, which all SMs then fetch at once. Fast mode, 1e3 trajectories, in full warps -> spread, ms: 120 nodes
// 0.87 -> 0.55, 200 nodes 3.0 -> 2.5, 400 nodes 41 -> 48 and (another network) 19 -> 40.
constexpr int max_spread_words = 8;

// mb_initialize_random: consecutive trajectories per warp and the grid for n trajectories. One per warp until
// the chip has 32 warps an SM to hide the latency of the jumps to each warp's first trajectory, then as
// many as keep that number of warps, up to 128 (the jumps are then a twentieth of the work).
inline int init_random_per(long long n)
{
	const long long warps = 148LL * 32, per = (n + warps - 1) / warps;
	return per < 1 ? 1 : per > 128 ? 128 : (int)per;
}
inline unsigned init_random_blocks(long long n, int per)
{
	const long long block = (long long)per * (MB_INIT_THREADS / 32);
	return (unsigned)((n + block - 1) / block);
}

// Device memory owned by the runtime.
struct dbuf
{
	void* p = nullptr;
	size_t bytes = 0;
	dbuf() = default;
	explicit dbuf(size_t n) { alloc(n); }
	dbuf(const dbuf&) = delete;
	dbuf& operator=(const dbuf&) = delete;
	dbuf(dbuf&& o) noexcept : p(o.p), bytes(o.bytes) { o.p = nullptr, o.bytes = 0; }
	dbuf& operator=(dbuf&& o) noexcept
	{
		std::swap(p, o.p);
		std::swap(bytes, o.bytes);
		return *this;
	}
	~dbuf();
	void alloc(size_t n);
	template <typename T>
	T* as() const
	{
		return static_cast<T*>(p);
	}
};

// A part of a dbuf.
struct dview
{
	void* p = nullptr;
	size_t bytes = 0;
	template <typename T>
	T* as() const
	{
		return static_cast<T*>(p);
	}
};

// Pinned host memory for the copies of a result. Allocating it takes long (0.13 ms a MB from 2 MB on, 1 to 3 ms
// for the first MB), so a run's statistics keep theirs, and it comes from and goes back to a pool of the
// process: at most 64 MB, the longest unused freed first. Any thread may borrow and return. Where pinning
// fails, plain memory.
class host_stage
{
public:
	struct block
	{
		void* p = nullptr;
		size_t size = 0;
		bool pinned = true;
		void* base = nullptr; // of the mapping that p lies in (huge pages), and its bytes
		size_t mapped = 0;
	};
	host_stage() = default;
	~host_stage() { release(); }
	host_stage(const host_stage&) = delete;
	host_stage& operator=(const host_stage&) = delete;
	void reserve(size_t bytes); // (what it held is lost)
	void release() noexcept;	// gives the memory back
	static void warm();			// 4 MB for the pool, once in the process
	size_t bytes() const { return b.size; }
	template <typename T>
	T* as(size_t offset = 0) const
	{
		return reinterpret_cast<T*>(static_cast<char*>(b.p) + offset);
	}

private:
	block b;
};

// Device buffers that an object keeps between its calls only to spare the next call their allocation. While a call
// uses them (kept_use) they are its own. The others are given back, by any thread, when an allocation on their
// device fails; and together they hold at most max_idle bytes of a device, the longest unused going first.
class kept_buffers
{
public:
	kept_buffers();
	kept_buffers(const kept_buffers&) = delete;
	kept_buffers& operator=(const kept_buffers&) = delete;
	virtual ~kept_buffers() = default;
	virtual size_t held() const = 0;
	virtual void drop() = 0;
	// frees what is not in use on the current device; false: nothing was there
	static bool give_back();
	static constexpr size_t max_idle = 4ull << 30;

protected:
	void forget(); // (the first thing a destructor does)

private:
	friend class kept_use;
	static bool trim(int device, size_t most);
	int device = 0, users = 0;
};

// The scope of a call that uses kept buffers (whose work on the device has been waited for at its end). Above `most`
// bytes they are freed at its end.
class kept_use
{
public:
	kept_use(kept_buffers& b, int device, size_t most);
	~kept_use();
	kept_use(const kept_use&) = delete;
	kept_use& operator=(const kept_use&) = delete;

private:
	kept_buffers& b;
	size_t most;
};

// Device scratch of sort_bins and compact_cells, kept between runs.
struct sort_scratch : kept_buffers
{
	dbuf lo, lo_sorted, hi, hi_sorted, pos, pos_a, pos_b, tmp, counters, out_keys, out_vals;
	static constexpr size_t most = 1ull << 30;
	~sort_scratch() override { forget(); }
	static void reserve(dbuf& b, size_t bytes)
	{
		if (b.bytes < bytes)
			b.alloc(bytes + bytes / 4);
	}
	size_t held() const override
	{
		size_t total = 0;
		for (const dbuf* b : { &lo, &lo_sorted, &hi, &hi_sorted, &pos, &pos_a, &pos_b, &tmp, &counters, &out_keys, &out_vals })
			total += b->bytes;
		return total;
	}
	void drop() override
	{
		for (dbuf* b : { &lo, &lo_sorted, &hi, &hi_sorted, &pos, &pos_a, &pos_b, &tmp, &counters, &out_keys, &out_vals })
			b->alloc(0);
	}
};

struct context
{
	int device = 0;
	int sm_count = 0;
	int cc_major = 0, cc_minor = 0;
	cudaStream_t stream = nullptr; // owned, non-blocking
	dbuf xorwow_jump; // jump matrices of mb_initialize_random, uploaded with the first module that has it
	explicit context(int device);
	~context();
};

// Kernel families, compiled (NVRTC) and loaded on first use: the generated per-node code is
// inlined only into the kernels of the family that needs it.
enum kernel_family : int
{
	FAMILY_EXACT = 0, // mb_fused_exact
	FAMILY_FAST = 1,  // mb_fused_fast (incremental or dense)
	FAMILY_EPOCH = 2, // mb_simulate_epoch (incremental for @logic-form models, else dense)
	FAMILY_EPOCH_DENSE = 3, // mb_simulate_epoch with every node's rate function evaluated per step
	FAMILY_BATCH = 4, // mb_batched_fast_static / mb_batched_grad_static: the batched kernels for this network
	FAMILY_COUNT = 5
};

// Kernel handles resolved from NVRTC-compiled modules.
struct module
{
	context* ctx = nullptr;
	CUmodule mods[FAMILY_COUNT] = { nullptr, nullptr, nullptr, nullptr, nullptr };
	bool loaded[FAMILY_COUNT] = { false, false, false, false, false }; // with every handle and table its kernels need
	// FAMILY_BATCH is loaded as a runtime-API library: its kernels are cudaKernel_t handles, which the
	// batch engine's runtime-API launches, occupancy queries and graph nodes take like its own kernels
	cudaLibrary_t batch_lib = nullptr;
	const void* batched_fast_static = nullptr;
	const void* batched_grad_static = nullptr;
	int state_size = 0, state_words = 0;
	int noninternal_count = -1; // from the generated code (mbg_noninternal_count), -1 if absent
	bool incremental = false;	// @logic-form model: exact and epoch modes use the incremental kernels (generated MBG_INCREMENTAL)
	bool integer_rates = false; // fast mode's incremental kernel too (generated MBG_INTEGER_RATES), else its dense kernel
	bool dense_epochs = false; // epoch mode's dense kernel all the same (generated MBG_EPOCH_DENSE)
	bool fast_incremental() const { return incremental && integer_rates; }
	// words of a warp's array in the lockstep kernels (generated MBG_GATES), 0: the incremental kernels
	int gate_words = 0;
	// threads of a block of the fused incremental kernels with their tables in shared memory and the tables'
	// bytes (generated MBG_TABLE_THREADS), 0: tables in global memory
	int table_threads = 0;
	size_t table_bytes = 0;
	// dynamic shared memory of a block of a fused incremental kernel, without the entropy sums
	size_t fused_smem(int block) const
	{
		return gate_words ? (size_t)4 * gate_words * (block / 32) : table_bytes + (size_t)12 * state_words * block;
	}
	bool has_layout = false; // compiled from a model (full layout known)
	model_layout layout;
	std::string source; // generated model source that was compiled with the engine
	std::mutex run_mu;	// whole runs (run()) of this module are serialised
	std::unique_ptr<struct runner> last_runner; // buffers of the last run(), reused for the same config
	cudaEvent_t run0 = nullptr, run1 = nullptr; // around a whole run()
	std::string log;	// NVRTC log

	CUfunction fused_exact = nullptr, fused_fast = nullptr;
	CUfunction init_random = nullptr, init_state = nullptr, sim_epoch = nullptr, sim_epoch_dense = nullptr;
	CUfunction window_epoch = nullptr, final_epoch = nullptr, fixed_epoch = nullptr;
	CUfunction compact_count = nullptr, compact_scan = nullptr, compact_scatter = nullptr, fixed_extract = nullptr;
	CUfunction bins_extract = nullptr;

	void ensure(int family);		// compile + load a family if needed (thread-safe)
	void ensure_any();				// at least one family (the shared statistics kernels)
	double compile_seconds = 0;		// NVRTC time spent so far
	~module();
};

// Compile generated model code together with the engine kernels (NVRTC, -arch=sm_100a).
std::unique_ptr<module> compile_module(context& ctx, const std::string& generated_code);
// A module whose kernel families are all compiled on first use (compile_module compiles the fast
// family at once); the batch engine uses it for FAMILY_BATCH only.
std::unique_ptr<module> compile_batch_module(context& ctx, const std::string& generated_code);
// NVRTC compilation only (no device needed): returns the cubin, throws on failure.
std::vector<char> compile_cubin(const std::string& generated_code, std::string& log, int family = FAMILY_FAST);

void launch(CUfunction f, unsigned grid, unsigned block, size_t smem, cudaStream_t s, void** args);

// One epoch of the buffered simulation (mb_simulate_epoch) over n trajectories of a batch of capacity
// `stride`; `dense` selects the reference's per-step evaluation of every rate function.
void simulate_epoch(module& m, bool dense, cudaStream_t s, int n, int stride, int L, unsigned* last_states,
					float* last_times, void* rands, unsigned* traj_states, float* traj_times, float* traj_h,
					unsigned char* statuses, unsigned long long* transitions);

// The non-zero cells of a dense window histogram (`occ` int64 or `cnt` u32, whichever is not null), in
// increasing cell order (window, then state): their cell indices into idx_out (u64) and values into
// val_out (int64), both grown as needed. Returns the number of cells, or -1 without writing them
// when there are more than max_entries (the dense copy is then cheaper).
long long compact_cells(const long long* occ, const unsigned* cnt, unsigned long long cells,
						unsigned long long max_entries, dbuf& idx_out, dbuf& val_out, int sm_count,
						sort_scratch& scratch, cudaStream_t s);

// Sorts n sparse-bin records by their 128-bit keys (window, then non-internal index) on the device (sort.cu).
// Asynchronous; the sorted bins are in scratch.out_keys and scratch.out_vals.
void sort_bins(const mb_key128* keys, const long long* vals, unsigned n, sort_scratch& scratch, cudaStream_t s);

// Stable partition of the CONTINUE trajectories of an epoch batch into another buffer set
// (last_states SoA [word * stride + i], last_times, random states); the number kept is written to
// the device word *kept. `scratch` holds partition_scratch_bytes(n) bytes. With rejected_rands the
// random states of the other trajectories fill out_rands[kept, n), last first.
size_t partition_scratch_bytes(int n);
void partition(module& m, cudaStream_t s, int n, int stride, const unsigned char* statuses, const unsigned* states,
			   const float* times, const void* rands, unsigned* out_states, float* out_times, void* out_rands,
			   void* scratch, unsigned* kept, bool rejected_rands = false);
int occupancy_blocks(CUfunction f, int block, size_t smem);

struct run_config
{
	int mode = MB_MODE_FUSED_EXACT;
	long long sample_count = 0;
	unsigned long long seed = 0;
	unsigned long long first_traj = 0; // RNG subsequence of trajectory 0
	float max_time = 0, time_tick = 0; // exact host floats for window statistics
	bool discrete_time = false;
	std::vector<float> istate;
	std::vector<int> noninternal_nodes;
	int traj_len = 100;				 // trajectory_len_limit (simulation_runner.cu:51)
	int batch_limit = 1000000;		 // trajectory_batch_limit (simulation_runner.cu:50)
	int block = 256;
	int blocks_per_sm = 0;			 // 0 = occupancy calculator
	int fixed_capacity_log2 = 0;	 // 0 = automatic
	long long stats_trajectories = 0; // trajectory count the fixed-point scales are chosen for (0 = sample_count)
	int bin_capacity_log2 = 0;		  // sparse bins (more than 20 non-internal nodes): table size, 0 = automatic
	bool refill_reuse_rng = false;	  // epoch modes: refilled slots continue the finished trajectories' random states
};

run_config config_from_layout(const model_layout& L, int mode);

// Dense window histograms of at least this many cells (T x 2^k; 134 MB of int64 sums) are returned as
// their non-zero cells only, when those are at most a quarter of the cells.
constexpr unsigned long long compact_min_cells = 1ull << 24;

// Dense continuous histograms of at most this many cells keep a count of the trajectories at a fixed
// point beside each cell (mb_record_fixed): 16 MB at most, cleared and scanned once a run in 20 us. Above
// it each window of such a trajectory is added on its own, and no second large array is kept.
constexpr unsigned long long tail_max_cells = 1ull << 22;

struct result
{
	int state_size = 0, state_words = 0, n_windows = 0;
	unsigned n_bins = 0;
	long long n_traj = 0;
	bool discrete_time = false;
	float time_tick = 0, max_time = 0;
	std::vector<int> noninternal_nodes;
	double fx = 1, fx_h = 1; // fixed-point scales of win_occ / win_h
	std::vector<long long> win_occ;
	std::vector<unsigned> win_cnt;
	std::vector<long long> win_h;
	std::vector<unsigned> final_cnt;
	std::vector<uint32_t> fixed_states; // n_fixed * state_words, sorted like the reference's std::map
	std::vector<unsigned> fixed_counts;
	unsigned fixed_overflow = 0;
	unsigned rate_errors = 0; // trajectories stopped on a non-finite total rate
	unsigned sections = 7;	  // statistics present: 1 windows, 2 final states, 4 fixed points
	// more than 20 non-internal nodes: sparse window bins (sorted by window, then index; sp_begin[w]
	// is the first entry of window w) and sparse final states (sorted by index); n_bins is 0
	bool wide = false;
	// at most 20 non-internal nodes but a large histogram (compact_min_cells or more cells): only its
	// non-zero cells, in the same sparse form (sp_*), selected on the device; final states dense
	bool compact = false;
	bulk_vector<int> sp_w;
	bulk_vector<unsigned __int128> sp_idx;
	bulk_vector<long long> sp_val; // occupancy in fixed point (continuous) or count (discrete)
	std::vector<size_t> sp_begin;  // [n_windows + 1]
	std::vector<unsigned __int128> fin_idx;
	std::vector<unsigned> fin_cnt;
	unsigned bin_overflow = 0; // bin additions that found no slot in the table (lost)
	double sparse_prob(size_t i) const; // probability of window entry i
	unsigned long long transitions = 0;
	float kernel_ms = 0; // device time of the simulation kernels
	float total_ms = 0;	 // device time of the whole run (setup + kernels + result copies)
	int epochs = 0;

	double window_prob(int w, unsigned bin) const; // window_average_small.cpp:126-140 (fp64)
	bool sparse_windows() const { return wide || compact; }
	double window_th(int w) const;				   // TH column (window_average_small.cpp:222-223)
};

// Fixed points stored in the order of std::map<static_state_t> (state.h:43-49: compared from the
// highest word down), from `counts.size()` records of r.state_words words.
void set_fixed_sorted(result& r, const std::vector<unsigned>& states, const std::vector<unsigned>& counts);
// The statistics of the union of disjoint trajectory sets (shards of one run): integer sums of the
// accumulators and the union of the fixed points. The parts must share the model's dimensions, the
// windows and the fixed-point scales (runs with the same stats_trajectories).
std::unique_ptr<result> merge_results(const std::vector<const result*>& parts);

// Fixed-point exponents (shared with the oracle so that both convert slices identically).
int occupancy_exponent(long long n_traj, float tick, bool discrete);
int entropy_exponent(long long n_traj, float tick, bool discrete);

// Device accumulators of the three built-in statistics plugins (window averages, final
// states, fixed points) for one run.
struct stats_state
{
	module* mod = nullptr;
	// one buffer for all accumulators that a launch clears (one clear), in the order counters, h, fin, occ or
	// cnt, fp_keys, fp_counts: the part that a result copies back is at its front (one copy)
	dbuf arena;
	dview occ, cnt, h, fin, fp_keys, fp_counts, counters;
	dbuf fp_states, istate;
	bool extracted = false; // the extraction counters are not cleared since the last finalize
	dbuf out_counts, out_states; // compacted fixed points (finalize)
	dbuf bin_keys, bin_vals, out_bin_keys, out_bin_vals; // sparse bins (more than 20 non-internal nodes)
	dbuf cell_idx, cell_vals; // non-zero cells of a large dense histogram (compact results), kept across runs
	sort_scratch scratch;
	// a result's copies, one after the other, kept across runs (the sorted sparse bins whatever their size; the cells of
	// a compact histogram up to max_kept_stage bytes)
	host_stage stage;
	static constexpr size_t max_kept_stage = 1ull << 30;
	unsigned bin_cap = 0;
	bool wide = false;
	bool has_tail = false; // occ is followed by the counts of mb_record_fixed (u32 per cell)
	unsigned fp_cap = 0;
	int n_windows = 0;
	unsigned n_bins = 0;
	bool discrete_time = false;
	float time_tick = 0, max_time = 0;
	double fx = 1, fx_h = 1;
	int h_in_smem = 0;
	std::vector<int> noninternal_nodes;
	unsigned sections = 7; // MB_STATS_WINDOWS | MB_STATS_FINAL | MB_STATS_FIXED
	mb_stats_params p{};   // device pointers + scales passed to the statistics kernels

	void init(module& m, float time_tick, float max_time, bool discrete, const std::vector<int>& noninternal,
			  long long n_traj, int fixed_capacity_log2, cudaStream_t s, unsigned sections = 7,
			  long long scale_traj = 0, // trajectories the fixed-point scales are chosen for (0 = n_traj)
			  int bin_capacity_log2 = 0);
	void zero(cudaStream_t s); // clear every accumulator (asynchronous)
	void set_istate(const std::vector<float>& istate, cudaStream_t s);
	size_t h_smem() const { return h_in_smem ? (size_t)n_windows * sizeof(long long) : 0; }
	void window_batch(cudaStream_t s, int n, int stride, int traj_len, const unsigned* traj_states,
					  const float* traj_times, const float* traj_h);
	void final_batch(cudaStream_t s, int n, int stride, const unsigned* last_states, const unsigned char* statuses);
	void fixed_batch(cudaStream_t s, int n, int stride, const unsigned* last_states, const unsigned char* statuses);
	// counters (u64 view): [0] work counter, [1] transitions, [2] low: fixed-table overflow,
	// high: extracted fixed points, [3] low: trajectories stopped on a non-finite total rate
	unsigned long long* next_traj() const { return counters.as<unsigned long long>(); }
	unsigned long long* transitions() const { return counters.as<unsigned long long>() + 1; }
	unsigned* fp_overflow_ctr() const { return counters.as<unsigned>() + 4; }
	unsigned* extract_ctr() const { return counters.as<unsigned>() + 5; }
	unsigned* error_ctr() const { return counters.as<unsigned>() + 6; }
	unsigned* bin_overflow_ctr() const { return counters.as<unsigned>() + 7; }
	unsigned* bin_extract_ctr() const { return counters.as<unsigned>() + 8; }
	// copy everything back (synchronises the stream)
	std::unique_ptr<result> finalize(long long n_traj, cudaStream_t s);
};

// Device buffers of the epoch modes' batch (states, times, random states twice, trajectory slots). Kept for the next
// launch where they take at most 4 GB: allocating and freeing the 0.2 GB of 1e5 trajectories of the 87-node
// example model took 9 to 20 ms a run.
struct epoch_buffers : kept_buffers
{
	dbuf states[2], times[2], rands[2], traj_states, traj_times, traj_h, statuses, scratch;
	int batch = 0;
	static constexpr size_t most = 4ull << 30;
	~epoch_buffers() override { forget(); }
	size_t held() const override
	{
		size_t total = traj_states.bytes + traj_times.bytes + traj_h.bytes + statuses.bytes + scratch.bytes;
		for (int k = 0; k < 2; k++)
			total += states[k].bytes + times[k].bytes + rands[k].bytes;
		return total;
	}
	void drop() override
	{
		batch = 0;
		for (dbuf* b : { states, times, rands })
			for (int k = 0; k < 2; k++)
				b[k].alloc(0);
		for (dbuf* b : { &traj_states, &traj_times, &traj_h, &statuses, &scratch })
			b->alloc(0);
	}
};

// A run whose device buffers are allocated once: launch() zeroes the accumulators and enqueues the
// simulation on a stream without synchronising (fused modes), collect() copies the results back.
struct runner
{
	module* mod = nullptr;
	run_config cfg;
	stats_state st;
	cudaEvent_t ev0 = nullptr, ev1 = nullptr;
	int epochs = 0;
	unsigned launches = 0; // engine kernels enqueued by the last launch()
	// exact mode: XORWOW states and (incremental kernels) initial states of the trajectories of a launch. A run of
	// more is several launches: the kernels start every trajectory from these, as curand_init in them, for
	// the runs without, took 96 registers and a stack frame
	dbuf rng, init_states;
	long long rng_chunk = 0; // trajectories of a launch
	static constexpr long long max_rng_states = 1LL << 24;
	static constexpr long long max_init_bytes = 1LL << 30;
	epoch_buffers epoch;
	runner(module& m, const run_config& c);
	~runner();
	void launch(cudaStream_t s);
	std::unique_ptr<result> collect(cudaStream_t s);
	unsigned kernel_launches() const; // engine kernels enqueued by the last launch()
};

// Run a whole simulation with the built-in statistics.
std::unique_ptr<result> run(module& m, const run_config& cfg);

// Launch-shape autotuner of the fused kernels: times candidate (threads per block, resident blocks per
// SM) pairs on a slice of the run's own trajectories and returns them fastest first.
struct tuned_shape
{
	int block = 0, blocks_per_sm = 0;
	double transitions_per_s = 0;
};
std::vector<tuned_shape> autotune(module& m, const run_config& cfg);

} // namespace mb
