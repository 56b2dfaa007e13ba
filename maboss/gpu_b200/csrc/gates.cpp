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
			finals[i] = b.make(parse(m, m.nodes[i].get_attr("logic"), m.nodes[i].name));
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
	// instructions of a step of 32 trajectories, about: 22 a round of gates, 20 a transposed word. Above,
	// re-evaluating the flipped node's dependents alone is cheaper
	net.ok = net.words < 8192 && 22 * (net.rounds + W) + 20 * W <= gate_max_cost;
	return net;
}

} // namespace mb
