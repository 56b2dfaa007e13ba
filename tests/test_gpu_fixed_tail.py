"""Window sums of trajectories that stay at a fixed point until max_time: they are counted once and spread
over the remaining windows by a scan (dense continuous histograms), or added window by window
(histograms above 2^22 cells). Against the CPU oracle, which adds every window, with the tolerance of
the parity tests (1e-5 + 1e-4 p: logf and with it the times differ in the last place)."""
import numpy as np
import pytest

import maboss.gpu_b200 as mb
from oracle.oracle import OracleModel

pytestmark = pytest.mark.gpu


def decay(n_out, max_time, tick, extra=0, discrete=0):
    """Nodes that switch off once and stay off: some trajectories begin at the fixed point."""
    n = n_out + extra
    bnd = "".join(f"node D{i} {{ logic = D{i} & !D{i}; rate_up = @logic ? 1 : 0; rate_down = @logic ? 0 : {1 + i % 3}; }}\n"
                  for i in range(n))
    cfg = "".join(f"D{i}.istate = 0.4;\n" for i in range(n))
    cfg += "".join(f"D{i}.is_internal = 1;\n" for i in range(n_out, n))
    cfg += f"max_time = {max_time}; time_tick = {tick}; discrete_time = {discrete}; sample_count = 1000;\n"
    return bnd, cfg


# windows: 1, 31, 32, 33 (one scan step and its edges), a ragged last window, several steps; columns: 1
# to 2 blocks of the scan; the last one is above 2^22 cells (no scan)
@pytest.mark.parametrize("n_out,max_time,tick", [(1, 1, 1), (3, 31, 1), (3, 6.4, 0.2), (4, 33, 1), (4, 6.3, 0.4),
                                                 (2, 100, 0.5), (16, 33, 0.5)])
@pytest.mark.parametrize("mode", ["exact", "fast", "epoch"])
def test_fixed_tail_windows_match_oracle(gpu, n_out, max_time, tick, mode):
    bnd, cfg = decay(n_out, max_time, tick, extra=2)
    n = 1500
    mod = gpu.compile(mb.Model(bnd, cfg))
    res = mod.run(mode=mode, sample_count=n, seed=3)
    ref = OracleModel(bnd, cfg).run(n=n, mode=1 if mode == "fast" else 0, seed=3)
    p, q = res.window_probs, ref["probs"]
    assert np.all(np.abs(p - q) <= 1e-5 + 1e-4 * q), np.abs(p - q).max()
    assert res.transitions == ref["transitions"]
    assert [c for _, c in res.fixed] == list(ref["fixed_counts"])
    # the counts are cleared behind: launches that are not collected do not add up
    runner = mod.runner(mode=mode, sample_count=n, seed=3)
    runner.launch()
    runner.launch()
    assert np.array_equal(runner.result().raw()["occ"], res.raw()["occ"])
    assert np.array_equal(mod.run(mode=mode, sample_count=n, seed=3).raw()["occ"], res.raw()["occ"])


def test_fixed_tail_windows_of_a_batch(gpu):
    bnd, cfg = decay(4, 6.3, 0.4)
    model = mb.Model(bnd, cfg)
    b = mb.Batch(gpu)
    nets = [b.add_model(model), b.add_model(mb.Model(*decay(2, 33, 1)))]
    vs = [b.add_variant(nets[0], 700), b.add_variant(nets[1], 900), b.add_variant(nets[0], 1100, first_traj=5)]
    for _ in range(2):
        b.run(seed=3)
    mod = gpu.compile(model)
    for v, kw in ((vs[0], dict(sample_count=700)), (vs[2], dict(sample_count=1100, first_traj=5))):
        assert np.array_equal(b.result(v).raw()["occ"], mod.run(mode="fast", seed=3, **kw).raw()["occ"])
