"""Exact mode above 256 nodes (tables in shared memory, sums in chunks of four nodes): the total rates, and with
them every flip and waiting time, must stay the reference's sequential fp32 sums, whatever the rates:
against the oracle, which adds every node."""
import numpy as np
import pytest

import maboss.gpu_b200 as mb
from oracle.oracle import OracleModel

pytestmark = pytest.mark.gpu


def model(n, kind, seed=0):
    rng = np.random.default_rng(seed)
    bnd = ""
    for i in range(n):
        a, b = rng.choice(n, 2, replace=False)
        logic = f"{'!' if rng.random() < 0.5 else ''}T{a} {rng.choice(['&', '|'])} {'!' if rng.random() < 0.5 else ''}T{b}"
        if kind == "dyadic":  # few bits: half-way cases in most binades
            up, down = (rng.integers(1, 64, 2) / 2.0 ** rng.integers(0, 6, 2)).tolist()
        elif kind == "fine":  # many bits, the lowest ones at the binades' half steps
            up, down = (1 + rng.integers(0, 2**16, 2) / 2.0**16).tolist()
        elif kind == "equal":
            up = down = 0.3
        elif kind == "wide":
            up, down = (10.0 ** rng.uniform(-3, 3, 2)).tolist()
        else:
            up, down = rng.uniform(0.1, 10.0, 2).tolist()
        bnd += f"node T{i} {{ logic = {logic}; rate_up = @logic ? {up:.6g} : 0; rate_down = @logic ? 0 : {down:.6g}; }}\n"
    cfg = "".join(f"T{i}.is_internal = 1;\n" for i in range(4, n))
    return bnd, cfg + f"max_time = {0.3 if kind == 'wide' else 2}; time_tick = 0.25; sample_count = 1000;\n"


@pytest.mark.parametrize("n", [257, 320, 1000])
@pytest.mark.parametrize("kind", ["dyadic", "fine", "equal", "wide", "uniform"])
def test_exact_sums_match_oracle(gpu, n, kind):
    bnd, cfg = model(n, kind, seed=n)
    assert "MBG_GATES" not in mb.Model(bnd, cfg).generate_code()
    samples = 20_000 // n
    ref = OracleModel(bnd, cfg).run(n=samples, mode=0, seed=6, traj_len=9)
    mod = gpu.compile(mb.Model(bnd, cfg))
    for mode in ("exact", "epoch"):
        res = mod.run(mode=mode, sample_count=samples, seed=6, traj_len=9)
        assert res.transitions == ref["transitions"]
        assert np.array_equal(res.final_counts, ref["final"])
        assert np.all(np.abs(res.window_probs - ref["probs"]) <= 1e-5 + 1e-4 * ref["probs"])
