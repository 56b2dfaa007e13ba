"""Logics of 13 to 16 inputs: exact and epoch modes run incrementally on truth tables with a second
extension record, fast mode keeps the dense kernel; 17 inputs stay dense everywhere."""
import ctypes as C
import subprocess

import numpy as np
import pytest

import maboss.gpu_b200 as mb
from oracle.oracle import OracleModel
from test_codegen_host import PRELUDE

WRAPPER = r"""
extern "C" int host_logic(int i, const uint32_t* s)
{
    const int r = mbg_inc_self[i];
    const uint4 rec = mbg_inc_crec[r], ext = mbg_inc_cext[r];
    const uint2 ext2 = mbg_inc_cext2[r];
    const int m = (rec.x >> 16) & 31;
    const unsigned ins[8] = { rec.z, rec.w, ext.x, ext.y, ext.z, ext.w, ext2.x, ext2.y };
    unsigned p = 0;
    for (int t = 0; t < m; t++)
    {
        const unsigned node = (ins[t >> 1] >> ((t & 1) * 16)) & 0xffffu;
        p |= ((s[node >> 5] >> (node & 31)) & 1u) << t;
    }
    const unsigned w = m <= 5 ? rec.y : mbg_inc_tt[rec.y + (p >> 5)];
    return (w >> (p & 31)) & 1u;
}
extern "C" int host_bit_rate_is_zero(int i, const uint32_t* s)
{
    float r[64];
    compute_transition_rates(r, s);
    return r[i] == 0.f;
}
"""


def model(inputs, compare=False, n=40, seed=1):
    """A network with two nodes of `inputs` inputs (with `compare`, one written with a comparison, which
    is evaluated pattern by pattern), the others of one to three."""
    rng = np.random.default_rng(seed)
    names = [f"M{i}" for i in range(n)]
    bnd = ""
    for i in range(n):
        k = inputs if i in (5, n - 1) else int(rng.integers(1, 4))
        lits = [("!" if rng.random() < 0.4 else "") + names[j] for j in rng.choice(n, k, replace=False)]
        expr = lits[0]
        for x in lits[1:]:
            expr = f"({expr} {rng.choice(['&', '|', '^'] if i in (5, n - 1) else ['&', '|'])} {x})"
        if compare and i == 5:
            expr = "(" + " + ".join(x.lstrip("!") for x in lits) + f") >= {inputs // 2}"
        up, down = rng.uniform(0.2, 4.0, 2)
        bnd += (f"node {names[i]} {{ logic = {expr}; rate_up = @logic ? {up:.6g} : 0; "
                f"rate_down = @logic ? 0 : {down:.6g}; }}\n")
    cfg = "".join(f"{names[i]}.is_internal = 1;\n" for i in range(6, n))
    return bnd, cfg + "max_time = 8; time_tick = 0.5; sample_count = 1000;\n"


@pytest.mark.parametrize("inputs,compare", [(13, False), (14, True), (16, False)])
def test_tables_encode_the_logic(tmp_path, inputs, compare):
    code = mb.Model(*model(inputs, compare)).generate_code()
    assert "#define MBG_INCREMENTAL_MANY 1" in code and "#define MBG_INTEGER_RATES" not in code
    (tmp_path / "m.cpp").write_text(PRELUDE + code + WRAPPER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-o", str(tmp_path / "m.so"),
                    str(tmp_path / "m.cpp")], check=True, timeout=300)
    L = C.CDLL(str(tmp_path / "m.so"))
    rng = np.random.default_rng(0)
    for _ in range(400):
        s = rng.integers(0, 2**32, 2, dtype=np.uint32) & np.array([0xFFFFFFFF, 0xFF], np.uint32)
        for i in (5, 7, 39):
            on = bool((s[i >> 5] >> np.uint32(i & 31)) & 1)
            # a node is stable (rate 0) exactly when its bit equals its logic
            assert bool(L.host_logic(i, s.ctypes.data_as(C.c_void_p))) == (
                on == bool(L.host_bit_rate_is_zero(i, s.ctypes.data_as(C.c_void_p))))


def test_17_inputs_stay_dense():
    assert "MBG_INCREMENTAL" not in mb.Model(*model(17)).generate_code()


@pytest.mark.gpu
@pytest.mark.parametrize("inputs,compare", [(13, False), (14, True), (16, False), (17, False)])
@pytest.mark.parametrize("mode", ["exact", "epoch", "fast"])
def test_many_inputs_match_oracle(gpu, inputs, compare, mode):
    bnd, cfg = model(inputs, compare)
    res = gpu.compile(mb.Model(bnd, cfg)).run(mode=mode, sample_count=1200, seed=2)
    ref = OracleModel(bnd, cfg).run(n=1200, mode=1 if mode == "fast" else 0, seed=2)
    if mode != "fast":  # (the dense fast kernel has no restatement that draws the same numbers)
        assert res.transitions == ref["transitions"]
        assert np.array_equal(res.final_counts, ref["final"])
        assert np.all(np.abs(res.window_probs - ref["probs"]) <= 1e-5 + 1e-4 * ref["probs"])
    else:
        assert abs(res.window_probs.sum() - ref["probs"].sum()) <= 1e-3 * ref["probs"].sum()


@pytest.mark.gpu
def test_batches_refuse_many_inputs(gpu):
    b = mb.Batch(gpu)
    with pytest.raises(mb.EngineError):
        b.add_model(mb.Model(*model(13)))
