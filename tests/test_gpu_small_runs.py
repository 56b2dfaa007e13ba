"""Small runs are spread over more warps with fewer lanes each (8 warps an SM): the results at the edges of that
rule (one lane, one to two, 31 to 32, more than resident) equal the oracle's."""
import numpy as np
import pytest

import maboss.gpu_b200 as mb
from maboss.gpu_b200 import synth
from oracle.oracle import OracleModel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["exact", "fast"])
@pytest.mark.parametrize("k", [0, 1, 1.0009, 2, 31, 31.5, 32.001])
def test_small_runs_match_oracle(gpu, mode, k):
    n = max(1, int(round(k * 8 * gpu.sm_count)))
    bnd, cfg = synth.c1()
    model = mb.Model(bnd, cfg)
    res = gpu.compile(model).run(mode=mode, sample_count=n, seed=5)
    ref = OracleModel(bnd, cfg).run(n=n, mode=1 if mode == "fast" else 0, seed=5)
    assert res.transitions == ref["transitions"]
    assert np.array_equal(res.final_counts, ref["final"])
    assert np.all(np.abs(res.window_probs - ref["probs"]) <= 1e-5 + 1e-4 * ref["probs"])
    if mode == "fast":
        b = mb.Batch(gpu)
        v = b.add_variant(b.add_model(model), n)
        b.run(seed=5)
        assert np.array_equal(b.result(v).raw()["occ"], res.raw()["occ"])
