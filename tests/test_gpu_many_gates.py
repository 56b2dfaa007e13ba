"""Lockstep kernels with more than 8 rounds of gates, and batches of networks of more than two state words with a
gradient."""
import re

import numpy as np
import pytest

import maboss.gpu_b200 as mb
from oracle.oracle import OracleModel
from test_gpu_batch_edges import _many_parameters

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ins,rounds", [(16, 12, 20), (90, 8, 9), (250, 6, 12)])
@pytest.mark.parametrize("mode", ["exact", "fast", "epoch"])
def test_many_rounds_of_gates_match_the_oracle(gpu, n, ins, rounds, mode):
    rng = np.random.default_rng(n)
    names = [f"L{i}" for i in range(n)]
    bnd, cfg = "", "max_time = 3; time_tick = 0.3; sample_count = 1000;\n"
    for i in range(n):
        pool = [names[j] for j in rng.choice(n, ins, replace=False)]

        def logic(lits):
            if len(lits) == 1:
                return ("!" if rng.random() < 0.4 else "") + lits[0]
            cut = len(lits) // 2
            return f"({logic(lits[:cut])} {rng.choice(['&', '|', '^'], p=[0.45, 0.45, 0.1])} {logic(lits[cut:])})"

        up, down = rng.uniform(0.2, 3.0, 2)
        # (more literals than inputs in the networks whose functions are not factored)
        lits = [pool[j] for j in rng.integers(0, ins, 60)] if ins > 10 else pool
        bnd += f"node {names[i]} {{ logic = {logic(lits)}; rate_up = @logic ? {up:.6g} : 0; rate_down = @logic ? 0 : {down:.6g}; }}\n"
        cfg += f"L{i}.is_internal = 1;\n" if i >= 5 else ""
    m = mb.Model(bnd, cfg)
    found = re.search(r"mbg_gate_rounds = (\d+)", m.generate_code())
    assert found and int(found.group(1)) >= rounds
    res = gpu.compile(m).run(mode=mode, sample_count=900, seed=3, traj_len=20)
    ref = OracleModel(bnd, cfg).run(n=900, mode=1 if mode == "fast" else 0, seed=3, traj_len=20)
    assert res.transitions == ref["transitions"]
    assert np.array_equal(res.final_counts, ref["final"])
    assert np.all(np.abs(res.window_probs - ref["probs"]) <= 1e-5 + 1e-4 * ref["probs"])


@pytest.mark.parametrize("nodes", [65, 96, 200])
def test_gradients_of_networks_of_several_words(gpu, nodes):
    m = mb.Model(*_many_parameters(nodes, 12, 1, seed=nodes))
    names = sorted(m.variables)[::7]
    theta = {k: m.variable(k) for k in names}
    out = []
    for spec in (True, False):
        b = mb.Batch(gpu)
        b.set_specialize(spec)
        net = b.add_model(m)
        vs = [b.add_variant(net, 700, theta, grad_params=names), b.add_variant(net, 300, {k: 1.2 * x for k, x in theta.items()},
                                                                            grad_params=names, first_traj=50)]
        cot = np.random.default_rng(2).normal(size=(12, 16))
        b.run_gradient(5, {v: cot for v in vs})
        out.append([(b.result(v).raw()["occ"], b.result(v).transitions, b.gradient(v)) for v in vs])
    for (occ, steps, g), (occ2, steps2, g2) in zip(*out):
        assert steps == steps2 and np.array_equal(occ, occ2)
        # (f64 atomic sums, whose order changes from launch to launch)
        assert np.allclose(g, g2, rtol=1e-11, atol=1e-11 * np.abs(g2).max())
