"""Batches at the edges of what they take."""
import numpy as np
import pytest

import maboss.gpu_b200 as mb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("discrete", [0, 1])
@pytest.mark.parametrize("spec", [True, False], ids=["specialised", "generic"])
def test_no_transitions_in_no_time(gpu, spec, discrete):
    """max_time = 0: no step has a length, so none counts, at a fixed point neither; every trajectory ends in the
    state that it starts in."""
    bnd = ("node A { logic = A & B; rate_up = @logic ? 1 : 0; rate_down = @logic ? 0 : 1; }\n"
           "node B { logic = A & B; rate_up = @logic ? 1 : 0; rate_down = @logic ? 0 : 1; }\n")
    cfg = f"A.istate = 0.5; B.istate = 0.5; max_time = 0; time_tick = 1; discrete_time = {discrete}; sample_count = 1000;\n"
    b = mb.Batch(gpu)
    b.set_specialize(spec)
    v = b.add_variant(b.add_model(mb.Model(bnd, cfg)), 1000)
    b.run(1)
    r = b.result(v)
    assert r.transitions == 0
    assert r.final_counts.sum() == 1000 and np.all(r.final_counts > 150)
    assert sum(c for _, c in r.fixed) == r.final_counts[0] + r.final_counts[3]


def _many_parameters(nodes, windows, sums, seed=0):
    """A network whose rates are sums of `sums` variables each."""
    rng = np.random.default_rng(seed)
    bnd, cfg = "", f"max_time = {windows}; time_tick = 1; sample_count = 100;\n"
    for i in range(nodes):
        rates = []
        for d in "ud":
            names = [f"${d}{i}_{k}" for k in range(sums)]
            cfg += "".join(f"{x} = {rng.uniform(0.1, 0.4):.6g};\n" for x in names)
            rates.append("(" + " + ".join(names) + ")")
        a, b = rng.choice(nodes, 2, replace=False)
        bnd += (f"node N{i} {{ logic = N{a} {rng.choice(['&', '|'])} !N{b}; rate_up = @logic ? {rates[0]} : 0; "
                f"rate_down = @logic ? 0 : {rates[1]}; }}\n")
        cfg += f"N{i}.istate = 0.5;\n" + (f"N{i}.is_internal = 1;\n" if i >= 4 else "")
    return bnd, cfg


@pytest.mark.parametrize("nodes,windows,sums,parameters,autotune",
                         [(20, 1000, 6, 220, False), (250, 500, 1, 440, True)])
def test_gradient_of_as_many_parameters_as_the_general_kernel_takes(gpu, nodes, windows, sums, parameters, autotune):
    """The lockstep kernel's arrays and entropy sums take more shared memory than the general kernel's rows here."""
    model = mb.Model(*_many_parameters(nodes, windows, sums))
    names = sorted(model.variables)[:parameters]
    theta = {k: model.variable(k) for k in names}
    grads, results = [], []
    for spec in (True, False):
        b = mb.Batch(gpu)
        b.set_options(use_graph=False, autotune=autotune)
        b.set_specialize(spec)
        v = b.add_variant(b.add_model(model), 600, theta, grad_params=names)
        cot = np.random.default_rng(1).normal(size=(windows, 16))
        b.run_gradient(3, {v: cot})
        grads.append(b.gradient(v))
        results.append(b.result(v))
    assert results[0].transitions == results[1].transitions
    assert np.array_equal(results[0].raw()["occ"], results[1].raw()["occ"])
    # (f64 atomic sums, whose order changes from launch to launch)
    assert np.allclose(grads[0], grads[1], rtol=1e-11, atol=1e-11 * np.abs(grads[1]).max())
