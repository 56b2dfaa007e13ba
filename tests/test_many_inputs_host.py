"""Models with logics of 13 to 16 inputs keep the dense kernels where the incremental ones have no room, and in epoch
mode where they are faster."""
import numpy as np
import pytest

import maboss.gpu_b200 as mb
from oracle.oracle import OracleModel
from test_many_inputs import model


@pytest.mark.parametrize("nodes,windows,incremental", [(16000, 300, True), (18000, 3000, False), (19200, 256, True),
                                                        (19200, 257, False)])
def test_incremental_only_where_a_warp_fits(nodes, windows, incremental):
    """32 threads' rows (12 bytes a state word and thread) and the entropy sums (8 bytes a window, in shared memory up
    to 48 KB) have 227 KB; the dense kernels, which such models had before, need no rows."""
    rng = np.random.default_rng(0)
    bnd = "".join(f"node N{i} {{ logic = N{(i + 1) % nodes}; rate_up = @logic ? 1 : 0; rate_down = @logic ? 0 : 1; }}\n"
                  for i in range(nodes - 1))
    wide = " & ".join(f"N{j}" for j in rng.choice(nodes, 13, replace=False))
    bnd += f"node N{nodes - 1} {{ logic = {wide}; rate_up = @logic ? 1 : 0; rate_down = @logic ? 0 : 1; }}\n"
    cfg = "".join(f"N{i}.is_internal = 1;\n" for i in range(4, nodes))
    code = mb.Model(bnd, cfg + f"max_time = {windows}; time_tick = 1; sample_count = 10;\n").generate_code()
    assert ("#define MBG_INCREMENTAL_MANY 1" in code) == incremental


@pytest.mark.parametrize("inputs,compare,nodes,dense", [(14, True, 40, True), (13, True, 160, True), (13, True, 161, False),
                                                        (13, False, 40, False), (12, True, 40, False)])
def test_epochs_are_dense_in_small_networks_without_gates(inputs, compare, nodes, dense):
    code = mb.Model(*model(inputs, compare, n=nodes)).generate_code()
    assert ("#define MBG_EPOCH_DENSE 1" in code) == dense
    assert ("#define MBG_GATES 1" in code) == (not compare)


@pytest.mark.gpu
@pytest.mark.parametrize("nodes", [40, 160, 161])
def test_epochs_match_the_oracle_on_both_sides(gpu, nodes):
    bnd, cfg = model(13, True, n=nodes)
    ref = OracleModel(bnd, cfg).run(n=700, mode=0, seed=4)
    for mode in ("epoch", "epoch_dense"):
        res = gpu.compile(mb.Model(bnd, cfg)).run(mode=mode, sample_count=700, seed=4, batch_limit=300)
        assert res.transitions == ref["transitions"]
        assert np.array_equal(res.final_counts, ref["final"])
        assert np.all(np.abs(res.window_probs - ref["probs"]) <= 1e-5 + 1e-4 * ref["probs"])
