// Gate networks of the lockstep kernels (gates.h).
#include "gates.h"

#include <algorithm>

namespace mb {

namespace {

// A Boolean expression in negation normal form: negations only at literals; AND and OR flattened.
struct bexpr
{
	enum kind_t
	{
		LIT,
		CONST,
		AND,
		OR,
		XOR
	} kind = CONST;
	int node = -1;	  // LIT
	bool neg = false; // LIT: negated, CONST: the value
	std::vector<bexpr> ch;
};

struct unsupported
{
};

bexpr negated(bexpr e)
{
	switch (e.kind)
	{
		case bexpr::LIT:
		case bexpr::CONST: e.neg = !e.neg; break;
		case bexpr::AND:
		case bexpr::OR:
			e.kind = e.kind == bexpr::AND ? bexpr::OR : bexpr::AND;
			for (bexpr& c : e.ch)
				c = negated(std::move(c));
			break;
		case bexpr::XOR: e.ch[0] = negated(std::move(e.ch[0])); break;
	}
	return e;
}

bexpr parse(const model_t& m, const expr& e, const std::string& current, int depth = 0)
{
	using K = expr::kind_t;
	if (depth > 4096)
		throw unsupported();
	bexpr r;
	switch (e.kind)
	{
		case K::literal:
			if (e.value != 0.f && e.value != 1.f)
				throw unsupported();
			r.neg = e.value != 0.f;
			return r;
		case K::identifier:
			r.kind = bexpr::LIT;
			r.node = m.node_index(e.name);
			if (r.node < 0)
				throw unsupported();
			return r;
		case K::alias: return parse(m, m.nodes[m.node_index(current)].get_attr(e.name.substr(1)), current, depth + 1);
		case K::paren: return parse(m, *e.a, current, depth + 1);
		case K::unary:
			if (e.op != op_t::NOT)
				throw unsupported();
			return negated(parse(m, *e.a, current, depth + 1));
		case K::binary:
		{
			if (e.op != op_t::AND && e.op != op_t::OR && e.op != op_t::XOR)
				throw unsupported();
			bexpr a = parse(m, *e.a, current, depth + 1), b = parse(m, *e.b, current, depth + 1);
			if (e.op == op_t::XOR)
			{
				if (a.kind == bexpr::CONST)
					return a.neg ? negated(std::move(b)) : b;
				if (b.kind == bexpr::CONST)
					return b.neg ? negated(std::move(a)) : a;
				r.kind = bexpr::XOR;
				r.ch.push_back(std::move(a));
				r.ch.push_back(std::move(b));
				return r;
			}
			r.kind = e.op == op_t::AND ? bexpr::AND : bexpr::OR;
			for (bexpr* x : { &a, &b })
			{
				if (x->kind == bexpr::CONST)
				{
					if (x->neg == (r.kind == bexpr::OR)) // 1 in an OR, 0 in an AND
						return *x;
					continue;
				}
				if (x->kind == r.kind)
					for (bexpr& c : x->ch)
						r.ch.push_back(std::move(c));
				else
					r.ch.push_back(std::move(*x));
			}
			if (r.ch.empty())
			{
				bexpr c; // 0 | 0 or 1 & 1
				c.neg = r.kind == bexpr::AND;
				return c;
			}
			if (r.ch.size() == 1)
				return bexpr(r.ch[0]);
			return r;
		}
		default: throw unsupported();
	}
}

struct builder
{
	int zero, one; // words of the constants
	struct item
	{
		gate g;
		int level; // 0: reads nodes only
	};
	std::vector<item> temps; // word index -1 - t in a gate's inputs
	int level_of(int word) const { return word < 0 ? temps[-1 - word].level + 1 : 0; }

	int word(const bexpr& e)
	{
		if (e.kind == bexpr::LIT)
			return 2 * e.node + (e.neg ? 1 : 0);
		if (e.kind == bexpr::CONST)
			return e.neg ? one : zero;
		const gate g = make(e);
		if (temps.size() >= 4096)
			throw unsupported();
		int level = 0;
		for (int i : g.in)
			level = std::max(level, level_of(i));
		temps.push_back({ g, level });
		return -(int)temps.size();
	}
	gate make(const bexpr& e)
	{
		switch (e.kind)
		{
			case bexpr::AND:
			{
				std::vector<bexpr> ch;
				for (const bexpr& c : e.ch)
					ch.push_back(negated(c));
				gate g = make_or(std::move(ch));
				g.invert = !g.invert;
				return g;
			}
			case bexpr::OR: return make_or(e.ch);
			case bexpr::XOR:
				return { { word(e.ch[0]), word(negated(e.ch[1])), word(negated(e.ch[0])), word(e.ch[1]) }, true, false };
			default: return { { word(e), one, zero, zero }, true, false };
		}
	}
	static bool is_pair(const bexpr& e)
	{
		return e.kind == bexpr::AND && e.ch.size() == 2 && e.ch[0].kind == bexpr::LIT && e.ch[1].kind == bexpr::LIT;
	}
	gate make_or(std::vector<bexpr> ch)
	{
		std::vector<bexpr> pairs, singles;
		for (bexpr& c : ch)
			(is_pair(c) ? pairs : singles).push_back(std::move(c));
		for (;;)
		{
			const size_t P = pairs.size(), S = singles.size();
			if (P == 0 && S <= 4)
			{
				// not (all negated)
				gate g = { { one, one, one, one }, false, true };
				for (size_t i = 0; i < S; i++)
					g.in[i] = word(negated(singles[i]));
				return g;
			}
			if (P + S <= 2 && S <= 1)
			{
				gate g = { { zero, zero, zero, zero }, true, false };
				int at = 0;
				for (const bexpr& p : pairs)
				{
					g.in[at++] = word(p.ch[0]);
					g.in[at++] = word(p.ch[1]);
				}
				if (S)
				{
					g.in[at++] = word(singles[0]);
					g.in[at++] = one;
				}
				return g;
			}
			// one more level: an OR of up to four singles, or of two pairs, becomes a single
			bexpr part;
			part.kind = bexpr::OR;
			std::vector<bexpr>& from = S >= 2 ? singles : pairs;
			const size_t take = S >= 2 ? std::min<size_t>(4, S) : 2;
			for (size_t i = 0; i < take; i++)
				part.ch.push_back(std::move(from[from.size() - take + i]));
			from.resize(from.size() - take);
			singles.insert(singles.begin(), std::move(part));
		}
	}
};

// ---- factored forms from truth tables
//
// Logics of example models are written as sums of many products (153 literals for 10 inputs) of a function
// that a dozen literals express. The table of the function (32 patterns a word; input t of `in` at bit t) is
// split recursively: by a literal that is a factor or a term of it, else by a literal x as f = x g | h or
// f = (x | g) & h, where g and h are only bounded from below and above, so that they lose inputs.

typedef std::vector<unsigned> table;

struct factoring
{
	std::vector<int> in; // nodes
	static unsigned low(int t)
	{
		static const unsigned masks[5] = { 0xaaaaaaaau, 0xccccccccu, 0xf0f0f0f0u, 0xff00ff00u, 0xffff0000u };
		return masks[t];
	}
	// f with input t fixed to v
	static table cofactor(const table& f, int t, bool v)
	{
		table r(f.size());
		for (size_t w = 0; w < f.size(); w++)
		{
			if (t >= 5)
			{
				const size_t bit = (size_t)1 << (t - 5);
				r[w] = f[v ? w | bit : w & ~bit];
				continue;
			}
			const unsigned x = v ? f[w] & low(t) : f[w] & ~low(t);
			r[w] = v ? x | x >> (1 << t) : x | x << (1 << t);
		}
		return r;
	}
	template <class F>
	static table map(const table& a, const table& b, F f)
	{
		table r(a.size());
		for (size_t w = 0; w < a.size(); w++)
			r[w] = f(a[w], b[w]);
		return r;
	}
	static table both(const table& a, const table& b) { return map(a, b, [](unsigned x, unsigned y) { return x & y; }); }
	static table either(const table& a, const table& b) { return map(a, b, [](unsigned x, unsigned y) { return x | y; }); }
	static table except(const table& a, const table& b) { return map(a, b, [](unsigned x, unsigned y) { return x & ~y; }); }
	static bool all(const table& a, unsigned v)
	{
		return std::all_of(a.begin(), a.end(), [&](unsigned x) { return x == v; });
	}
	static bool within(const table& a, const table& b) { return all(except(a, b), 0u); }
	table of(const bexpr& e) const
	{
		const size_t words = (size_t)1 << (in.size() > 5 ? in.size() - 5 : 0);
		table r(words, e.kind == bexpr::AND ? ~0u : 0u);
		switch (e.kind)
		{
			case bexpr::CONST: return table(words, e.neg ? ~0u : 0u);
			case bexpr::LIT:
			{
				const int t = (int)(std::find(in.begin(), in.end(), e.node) - in.begin());
				for (size_t w = 0; w < words; w++)
					r[w] = (t < 5 ? low(t) : (w >> (t - 5)) & 1 ? ~0u : 0u) ^ (e.neg ? ~0u : 0u);
				return r;
			}
			default:
				for (const bexpr& c : e.ch)
				{
					const table x = of(c);
					for (size_t w = 0; w < words; w++)
						r[w] = e.kind == bexpr::AND ? r[w] & x[w] : e.kind == bexpr::OR ? r[w] | x[w] : r[w] ^ x[w];
				}
				return r;
		}
	}
	bexpr literal(int t, bool neg) const
	{
		bexpr e;
		e.kind = bexpr::LIT;
		e.node = in[t];
		e.neg = neg;
		return e;
	}
	static bexpr join(bexpr::kind_t kind, bexpr a, bexpr b)
	{
		bexpr r;
		r.kind = kind;
		for (bexpr* x : { &a, &b })
		{
			if (x->kind == bexpr::CONST)
			{
				if (x->neg == (kind == bexpr::OR))
					return *x;
				continue;
			}
			if (x->kind == kind)
				r.ch.insert(r.ch.end(), x->ch.begin(), x->ch.end());
			else
				r.ch.push_back(*x);
		}
		if (r.ch.empty())
		{
			bexpr c;
			c.neg = kind == bexpr::AND;
			return c;
		}
		if (r.ch.size() == 1)
			return bexpr(r.ch[0]);
		return r;
	}
	// drops the inputs that a function between the bounds can do without
	static void reduce(table& lo, table& hi, std::vector<int>& vars)
	{
		for (size_t i = 0; i < vars.size();)
		{
			const table l = either(cofactor(lo, vars[i], false), cofactor(lo, vars[i], true));
			const table h = both(cofactor(hi, vars[i], false), cofactor(hi, vars[i], true));
			if (!within(l, h))
			{
				i++;
				continue;
			}
			lo = l;
			hi = h;
			vars.erase(vars.begin() + (std::ptrdiff_t)i);
		}
	}
	static size_t support(table lo, table hi, std::vector<int> vars)
	{
		reduce(lo, hi, vars);
		return vars.size();
	}
	// an expression of a function between lo and hi
	bexpr make(table lo, table hi, std::vector<int> vars) const
	{
		bexpr e;
		if (all(lo, 0u))
			return e; // 0
		if (all(hi, ~0u))
		{
			e.neg = true;
			return e;
		}
		reduce(lo, hi, vars);
		size_t best = ~(size_t)0;
		int at = -1, form = 0;
		for (int t : vars)
		{
			const table l[2] = { cofactor(lo, t, false), cofactor(lo, t, true) };
			const table h[2] = { cofactor(hi, t, false), cofactor(hi, t, true) };
			for (int v = 0; v < 2; v++) // the literal is true where the input is v
			{
				if (all(l[1 - v], 0u))
					return join(bexpr::AND, literal(t, v == 0), make(l[v], h[v], vars));
				if (all(h[v], ~0u))
					return join(bexpr::OR, literal(t, v == 0), make(l[1 - v], h[1 - v], vars));
			}
			for (int v = 0; v < 2; v++)
			{
				const table hh = both(h[0], h[1]), ll = either(l[0], l[1]);
				if (within(l[1 - v], hh))
				{
					const size_t c = support(l[1 - v], hh, vars) + support(except(l[v], hh), h[v], vars);
					if (c < best)
						best = c, at = t, form = v;
				}
				if (within(ll, h[v]))
				{
					const size_t c = support(ll, h[v], vars) + support(l[1 - v], either(h[1 - v], map(ll, ll, [](unsigned x, unsigned) { return ~x; })), vars);
					if (c < best)
						best = c, at = t, form = 2 + v;
				}
			}
		}
		if (at < 0) // x g | !x h
		{
			const int t = vars[0];
			const bexpr g = make(cofactor(lo, t, true), cofactor(hi, t, true), vars);
			const bexpr h = make(cofactor(lo, t, false), cofactor(hi, t, false), vars);
			return join(bexpr::OR, join(bexpr::AND, literal(t, false), g), join(bexpr::AND, literal(t, true), h));
		}
		const int v = form & 1;
		const table l[2] = { cofactor(lo, at, false), cofactor(lo, at, true) };
		const table h[2] = { cofactor(hi, at, false), cofactor(hi, at, true) };
		if (form < 2) // x g | rest
		{
			const bexpr rest = make(l[1 - v], both(h[0], h[1]), vars);
			const bexpr g = make(except(l[v], of(rest)), h[v], vars);
			return join(bexpr::OR, join(bexpr::AND, literal(at, v == 0), g), rest);
		}
		// (x | g) & rest
		const bexpr rest = make(either(l[0], l[1]), h[v], vars);
		const table not_rest = map(of(rest), l[0], [](unsigned x, unsigned) { return ~x; });
		const bexpr g = make(l[1 - v], either(h[1 - v], not_rest), vars);
		return join(bexpr::AND, join(bexpr::OR, literal(at, v == 0), g), rest);
	}
};

void inputs_of(const bexpr& e, std::vector<int>& in)
{
	if (e.kind == bexpr::LIT && std::find(in.begin(), in.end(), e.node) == in.end())
		in.push_back(e.node);
	for (const bexpr& c : e.ch)
		inputs_of(c, in);
}

size_t literals_of(const bexpr& e)
{
	size_t n = e.kind == bexpr::LIT ? 1 : 0;
	for (const bexpr& c : e.ch)
		n += literals_of(c);
	return n;
}

// Intermediate gates of an expression and their levels.
std::pair<size_t, int> cost_of(const bexpr& e)
{
	builder b{ 1 << 20, (1 << 20) + 1, {} };
	b.make(e);
	int levels = 0;
	for (const builder::item& t : b.temps)
		levels = std::max(levels, t.level + 1);
	return { b.temps.size(), levels };
}

// The logic as written, or its factored form where that takes fewer gates.
bexpr shorter(bexpr e)
{
	factoring f;
	inputs_of(e, f.in);
	if (f.in.size() < 2 || f.in.size() > 10 || literals_of(e) <= 4)
		return e;
	const std::pair<size_t, int> cost = cost_of(e);
	if (cost.first <= 1)
		return e;
	const table t = f.of(e);
	std::vector<int> vars(f.in.size());
	for (size_t i = 0; i < vars.size(); i++)
		vars[i] = (int)i;
	bexpr g = f.make(t, t, vars);
	return cost_of(g) < cost ? g : e;
}

} // namespace

gate_network build_gates(const model_t& m)
{
	gate_network net;
	const int N = (int)m.nodes.size(), W = (N + 31) / 32;
	if (N == 0 || W > gate_max_words)
		return net;
	builder b;
	b.zero = 64 * W;
	b.one = 64 * W + 1;
	std::vector<gate> finals((size_t)32 * W, gate{ { b.zero, b.zero, b.zero, b.zero }, true, false });
	try
	{
		for (int i = 0; i < N; i++)
			finals[i] = b.make(shorter(parse(m, m.nodes[i].get_attr("logic"), m.nodes[i].name)));
	}
	catch (const unsupported&)
	{
		return net;
	}
	// intermediate gates by level, each level in rounds of 32
	std::vector<int> order(b.temps.size()), slot(b.temps.size());
	for (size_t t = 0; t < order.size(); t++)
		order[t] = (int)t;
	std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return b.temps[x].level < b.temps[y].level; });
	int at = 0, level = 0;
	for (int t : order)
	{
		if (b.temps[t].level != level)
			at = (at + 31) / 32 * 32;
		level = b.temps[t].level;
		slot[t] = at++;
	}
	net.rounds = (at + 31) / 32;
	net.gates.assign((size_t)32 * net.rounds, gate{ { b.zero, b.zero, b.zero, b.zero }, true, false });
	const int base = 64 * W + 2;
	auto resolved = [&](gate g) {
		for (int& i : g.in)
			if (i < 0)
				i = base + slot[-1 - i];
		return g;
	};
	for (size_t t = 0; t < b.temps.size(); t++)
		net.gates[slot[t]] = resolved(b.temps[t].g);
	for (const gate& g : finals)
		net.gates.push_back(resolved(g));
	net.words = base + 32 * std::max(1, net.rounds);
	net.ok = net.words < 8192 && 22 * (net.rounds + W) + 20 * W <= gate_max_cost;
	return net;
}

} // namespace mb
