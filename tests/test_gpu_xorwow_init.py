"""XORWOW states by matrix jumps and the initial states drawn with them: exact mode against the oracle (which
calls curand_init) at the edges of the warps' shares of trajectories and for high trajectory numbers."""
import numpy as np
import pytest

import maboss.gpu_b200 as mb
from maboss.gpu_b200 import synth
from oracle.oracle import OracleModel

pytestmark = pytest.mark.gpu


# one trajectory per warp, a part of a warp's lanes, 2 to 9 per warp with a short last one, and 40 per warp
# (two rounds of 32 lanes, the second one of 8)
@pytest.mark.parametrize("n,first", [(1, 0), (31, 3), (4737, 0), (40_001, (1 << 40) + 7), (5_000, (1 << 63) + 5),
                                     (186_000, 2)])
def test_exact_mode_streams_match_oracle(gpu, n, first):
    bnd, cfg = synth.c1()
    res = gpu.compile(mb.Model(bnd, cfg)).run(mode="exact", sample_count=n, seed=11, first_traj=first)
    ref = OracleModel(bnd, cfg).run(n=n, mode=0, seed=11, first=first)
    assert res.transitions == ref["transitions"]
    assert np.array_equal(res.final_counts, ref["final"])


def test_initial_states_of_several_words(gpu):
    bnd, cfg = synth.c3(n=70, n_out=5, max_time=3.0)
    for mode in ("exact", "epoch"):
        res = gpu.compile(mb.Model(bnd, cfg)).run(mode=mode, sample_count=5_003, seed=4)
        ref = OracleModel(bnd, cfg).run(n=5_003, mode=0, seed=4)
        assert res.transitions == ref["transitions"] and np.array_equal(res.final_counts, ref["final"])


def test_runs_of_several_launches(gpu):
    """More trajectories than the random states that are kept (2^24): several launches, the same sums as two runs."""
    mod = gpu.compile(mb.Model(*synth.c1()))
    n, first = (1 << 24) + 1000, 1 << 24
    whole = mod.run(mode="exact", sample_count=n, seed=2)
    parts = [mod.run(mode="exact", sample_count=k, seed=2, first_traj=f, stats_trajectories=n)
             for k, f in ((first, 0), (1000, first))]
    merged = mb.merge_results(parts)
    assert whole.transitions == merged.transitions
    assert np.array_equal(whole.final_counts, merged.final_counts)
    assert np.array_equal(whole.raw()["occ"], merged.raw()["occ"])
