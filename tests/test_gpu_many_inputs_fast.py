"""Fast mode of models with logics of 13 to 17 inputs, which run the dense kernel: the same distributions as the
oracle's fast mode (its trajectories draw other numbers)."""
import numpy as np
import pytest

import maboss.gpu_b200 as mb
from conftest import assert_statistically_equal
from oracle.oracle import OracleModel
from test_many_inputs import model


def _means(values):
    values = np.asarray(values, np.float64)
    return values.mean(0), values.std(0, ddof=1) / np.sqrt(len(values))


@pytest.mark.gpu
@pytest.mark.parametrize("inputs,compare", [(13, False), (14, True), (16, False), (17, False)])
def test_distributions_match_the_oracle(gpu, inputs, compare):
    bnd, cfg = model(inputs, compare)
    n, seeds = 2000, range(10, 22)
    module, oracle = gpu.compile(mb.Model(bnd, cfg)), OracleModel(bnd, cfg)
    runs = [module.run(mode="fast", sample_count=n, seed=s) for s in seeds]
    refs = [oracle.run(n=n, mode=1, seed=s + 100) for s in seeds]
    total = n * len(seeds)
    assert_statistically_equal(np.mean([r.window_probs for r in runs], 0), total, np.mean([r["probs"] for r in refs], 0), total)
    assert_statistically_equal(np.sum([r.final_counts for r in runs], 0) / total, total,
                               np.sum([r["final"] for r in refs], 0) / total, total)
    # 12 means each: within 6 standard errors of their difference (17 values and a two-sided t of about 22 degrees of
    # freedom: about 1e-4 in all)
    for a, b in (([[r.transitions / n] for r in runs], [[r["transitions"] / n] for r in refs]),
                 ([r.window_entropy for r in runs], [r["th"] for r in refs])):
        (ma, sa), (mb_, sb) = _means(a), _means(b)
        assert np.all(np.abs(ma - mb_) <= 6 * np.hypot(sa, sb)), (ma, mb_)
