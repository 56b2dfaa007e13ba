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
// Instructions of a step of 32 trajectories, about: 22 a round of gates, 20 a transposed word. Networks up to it are
// faster than with the dependents of each flip alone, by (fast mode 2e5 to 3e5 trajectories | exact 1e5 | epoch
// 2e4): 16 nodes, 36 rounds 2.4x | 2.0 | 8.2, 32 nodes, 36 rounds 2.3 | 2.1 | 5.9, 64 nodes, 30 rounds 2.9 | 2.3 |
// 4.0, 128 nodes, 14 rounds 2.3 | 2.1 | 3.7, 250 nodes, 24 rounds 1.95 | 1.7 | 3.3, and least with few rounds on many
// nodes: 250 nodes, 6 rounds 1.13 | 1.2 | 2.4. Above it nothing was measured.
constexpr int gate_max_cost = 1000;

gate_network build_gates(const model_t& m);

} // namespace mb
