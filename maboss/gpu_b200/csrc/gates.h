// The logic of a network as levels of gates for the lockstep kernels (kernels/engine.cuh): a warp
// evaluates every node's logic for its 32 trajectories at once, one bit a trajectory.
#pragma once

#include <vector>

#include "model.h"

namespace mb {

// out = ((a & b) op (c & d)) ^ invert with op = or / and. Inputs are words of the warp's array: node i is
// word 2 i, its negation 2 i + 1 (32 ceil(N / 32) nodes), then the constants 0 and 1, then the
// intermediate gates in order.
struct gate
{
	int in[4];
	bool is_or, invert;
};

struct gate_network
{
	bool ok = false; // every logic is made of nodes, 0, 1, NOT, AND, OR, XOR, and the network is small enough
	int rounds = 0;	 // rounds of 32 intermediate gates; a round reads nodes and earlier rounds only
	int words = 0;	 // words of the warp's array
	std::vector<gate> gates; // 32 rounds intermediate ones, then one per node (padded to whole words)
};

constexpr int gate_max_words = 8;	 // networks of at most 256 nodes
constexpr int gate_max_cost = 1000;

gate_network build_gates(const model_t& m);

} // namespace mb
