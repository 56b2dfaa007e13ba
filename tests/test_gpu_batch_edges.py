"""Batches at the edges of what they take."""
import numpy as np
import pytest

import maboss.gpu_b200 as mb
from maboss.gpu_b200 import synth

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
