"""Models with logics of 13 to 16 inputs keep the dense kernels where the incremental ones have no room."""
import numpy as np
import pytest

import maboss.gpu_b200 as mb


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
