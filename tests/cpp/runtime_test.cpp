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

} // namespace

int main(int argc, char** argv)
{
	const std::map<std::string, void (*)()> checks = {
		{ "jump_table_is_there_before_the_first_launch", jump_table_is_there_before_the_first_launch },
		{ "family_loads_after_a_failure", family_loads_after_a_failure },
	};
	for (int i = 1; i < argc; i++)
		checks.at(argv[i])();
	return failures != 0;
}
