// The host runtime on a stand-in for CUDA (fake_cuda.h): one check per name, exit status 0 when it holds.
#include "fake_cuda.h"
#include "model.h"
#include "runtime.h"

#include <cstdio>

namespace mb {
// (sort.cu's, which these checks do not reach)
long long compact_cells(const long long*, const unsigned*, unsigned long long, unsigned long long, dbuf&, dbuf&, int,
						sort_scratch&, cudaStream_t)
{
	return -1;
}
void sort_bins(const mb_key128*, const long long*, unsigned, sort_scratch&, cudaStream_t) {}
} // namespace mb

namespace {

int failures = 0;
#define CHECK(x) \
	do \
	{ \
		if (!(x)) \
		{ \
			std::printf("%s:%d: %s\n", __FILE__, __LINE__, #x); \
			failures++; \
		} \
	} while (0)

template <class F>
bool throws(F f)
{
	try
	{
		f();
		return false;
	}
	catch (const mb::engine_error&)
	{
		return true;
	}
}

struct program
{
	mb::context ctx{ 0 };
	mb::model_t model;
	std::unique_ptr<mb::module> m;
	program()
	{
		mb::parse_bnd(model, "node A { logic = B; rate_up = @logic ? 1 : 0; rate_down = @logic ? 0 : 1; }\n"
							 "node B { logic = !A; rate_up = @logic ? 2 : 0; rate_down = @logic ? 0 : 1; }\n", "bnd");
		mb::parse_cfg(model, "max_time = 4; time_tick = 1; sample_count = 100;\n", "cfg");
		m = mb::compile_module(ctx, mb::generate_code(model));
		m->layout = mb::analyze_model(model);
		m->has_layout = true;
	}
	mb::run_config config(int mode, long long n) const
	{
		mb::run_config c = mb::config_from_layout(m->layout, mode);
		c.sample_count = n;
		return c;
	}
};

// The jump matrices are on the device when the first kernel that reads them starts, whichever stream it is on.
void jump_table_is_there_before_the_first_launch()
{
	for (int own = 0; own < 2; own++)
	{
		program p;
		cudaStream_t s = p.ctx.stream;
		if (!own)
			cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
		int seen = 0;
		fake::on_launch = [&](const std::string& kernel, cudaStream_t, void** args, unsigned, size_t) {
			if (kernel != "mb_initialize_random")
				return;
			seen++;
			const unsigned* table = *static_cast<unsigned**>(args[5]);
			CHECK(table != nullptr);
			bool filled = false;
			for (int i = 0; table && i < 32 * 3 * 25 * 32; i++)
				filled |= table[i] != 0;
			CHECK(filled);
		};
		mb::runner r(*p.m, p.config(MB_MODE_FUSED_EXACT, 100));
		r.launch(s);
		CHECK(seen == 1);
		fake::on_launch = nullptr;
	}
}

// A family that could not be loaded whole is not taken for loaded: the next call loads the rest.
void family_loads_after_a_failure()
{
	{
		program p;
		bool fail = true;
		fake::fail_malloc = [&](size_t) { return fail; };
		CHECK(throws([&] { p.m->ensure(mb::FAMILY_EXACT); }));
		fail = false;
		p.m->ensure(mb::FAMILY_EXACT);
		CHECK(p.m->fused_exact && p.m->init_random && p.ctx.xorwow_jump.p);
		fake::fail_malloc = nullptr;
	}
	for (const char* name : { "mb_simulate_epoch", "mb_initialize_random" })
	{
		program p;
		fake::fail_function = name;
		CHECK(throws([&] { p.m->ensure(mb::FAMILY_EPOCH); }));
		fake::fail_function.clear();
		p.m->ensure(mb::FAMILY_EPOCH);
		CHECK(p.m->sim_epoch && p.m->init_random);
	}
}

// Staging memory: hardly more than was asked for, reused for requests of about its size, at most 64 MB of it kept
// when nobody holds any, and plain memory where pinning fails.
void staging_memory_is_bounded()
{
	const size_t mb = 1 << 20;
	for (size_t bytes : { (size_t)1, 5000 * (size_t)1, mb + 1, 3 * mb, 65 * mb, 130 * mb })
	{
		mb::host_stage s;
		s.reserve(bytes);
		CHECK(s.bytes() >= bytes && s.bytes() <= std::max(2 * mb, bytes) * 5 / 4 + 2 * mb);
		std::memset(s.as<char>(), 1, bytes);
		CHECK(reinterpret_cast<uintptr_t>(s.as<char>()) % 16 == 0);
	}
	CHECK(fake::held(fake::pinned) <= 64 * mb);
	{
		mb::host_stage a;
		a.reserve(20 * mb);
		const void* was = a.as<void>();
		a.release();
		mb::host_stage b;
		b.reserve(21 * mb);
		CHECK(b.as<void>() == was);
		mb::host_stage c;
		c.reserve(100000); // (not the large one)
		CHECK(c.bytes() < 4 * mb);
	}
	{
		std::vector<mb::host_stage> many(12);
		for (mb::host_stage& x : many)
			x.reserve(20 * mb);
	}
	CHECK(fake::held(fake::pinned) <= 64 * mb);
	fake::fail_register = true;
	mb::host_stage plain;
	plain.reserve(500 * mb);
	std::memset(plain.as<char>(), 1, 500 * mb);
	CHECK(fake::held(fake::pinned) <= 64 * mb);
	fake::fail_register = false;
}

// Buffers kept between the runs of several modules: at most 4 GB in all, given back when another allocation fails,
// and not while a run uses them.
void kept_buffers_are_given_back()
{
	program a, b, c;
	std::vector<std::unique_ptr<mb::runner>> runners;
	const mb::run_config batch = a.config(MB_MODE_EPOCH, 1000000); // 1.3 GB of buffers
	for (program* p : { &a, &b, &c })
		for (int k = 0; k < 2; k++)
		{
			runners.push_back(std::make_unique<mb::runner>(*p->m, batch));
			runners.back()->launch(p->ctx.stream);
		}
	size_t kept = 0;
	for (const auto& r : runners)
		kept += r->epoch.held();
	CHECK(kept > 2500u << 20);
	CHECK(kept <= mb::kept_buffers::max_idle);
	CHECK(runners.back()->epoch.held() > 0 && runners.front()->epoch.held() == 0); // (the longest unused went first)

	// a device that is full but for 100 MB: the next run's buffers come from those that wait
	const size_t limit = fake::held(fake::device) + (100 << 20);
	fake::fail_malloc = [&](size_t n) { return fake::held(fake::device) + n > limit; };
	mb::runner more(*a.m, batch);
	more.launch(a.ctx.stream);
	CHECK(more.epoch.held() > 1u << 30);
	CHECK(fake::held(fake::device) <= limit);
	// no room at all: the run that fails does not take its own buffers away from under itself, and leaves none
	const size_t full = fake::held(fake::device);
	fake::fail_malloc = [&](size_t n) { return n > 1 << 20 && fake::held(fake::device) + n > full / 8; };
	CHECK(throws([&] { runners[0]->launch(a.ctx.stream); }));
	fake::fail_malloc = nullptr;
	runners[0]->launch(a.ctx.stream);
	CHECK(runners[0]->epoch.held() > 1u << 30);
}

// Exact runs whose random and initial states do not fit take more launches, which cover every trajectory once.
void exact_run_in_more_launches_where_memory_is_short()
{
	program p;
	long long next = 0, launches = 0;
	fake::on_launch = [&](const std::string& kernel, cudaStream_t, void** args, unsigned, size_t) {
		if (kernel != "mb_initialize_random")
			return;
		CHECK(*static_cast<unsigned long long*>(args[2]) == (unsigned long long)next);
		next += *static_cast<int*>(args[0]);
		launches++;
	};
	p.m->ensure(mb::FAMILY_EXACT);
	fake::fail_malloc = [&](size_t n) { return n > 20u << 20; };
	mb::run_config c = p.config(MB_MODE_FUSED_EXACT, 1000001);
	c.fixed_capacity_log2 = 10;
	mb::runner r(*p.m, c);
	r.launch(p.ctx.stream);
	CHECK(next == 1000001 && launches > 1);
	fake::fail_malloc = nullptr;
	fake::on_launch = nullptr;
}

} // namespace

int main(int argc, char** argv)
{
	const std::map<std::string, void (*)()> checks = {
		{ "jump_table_is_there_before_the_first_launch", jump_table_is_there_before_the_first_launch },
		{ "family_loads_after_a_failure", family_loads_after_a_failure },
		{ "staging_memory_is_bounded", staging_memory_is_bounded },
		{ "kept_buffers_are_given_back", kept_buffers_are_given_back },
		{ "exact_run_in_more_launches_where_memory_is_short", exact_run_in_more_launches_where_memory_is_short },
	};
	for (int i = 1; i < argc; i++)
		checks.at(argv[i])();
	return failures != 0;
}
