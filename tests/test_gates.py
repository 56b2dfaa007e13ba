"""Lockstep kernels (networks of at most 256 nodes): the gate tables encode every node's logic, and the kernels
equal the oracle at the edges of the state words, for one to three and for many rate values."""
import ctypes as C
import subprocess

import numpy as np
import pytest

import maboss.gpu_b200 as mb
from oracle.oracle import OracleModel
from conftest import model_text
from test_codegen_host import PRELUDE

WRAPPER = r"""
// every node's logic for 32 states at once: st[i] has node i's bit of each of them
extern "C" void host_gates(const uint32_t* st, uint32_t* logic)
{
    uint32_t ns[mbg_gate_words] = { 0 };
    for (int i = 0; i < 32 * state_words; i++)
    {
        ns[2 * i] = i < state_size ? st[i] : 0u;
        ns[2 * i + 1] = ~ns[2 * i];
    }
    ns[64 * state_words + 1] = ~0u;
    for (int g = 0; g < 32 * (mbg_gate_rounds + state_words); g++)
    {
        const uint2 d = mbg_gates[g];
        const uint32_t x = ns[(d.x & 0x7fffu) / 4] & ns[((d.x >> 16) & 0x7fffu) / 4];
        const uint32_t y = ns[(d.y & 0x7fffu) / 4] & ns[((d.y >> 16) & 0x7fffu) / 4];
        const uint32_t r = ((d.x >> 31) ? x | y : x & y) ^ ((d.y >> 31) ? ~0u : 0u);
        const int i = g - 32 * mbg_gate_rounds;
        if (i < 0)
            ns[64 * state_words + 2 + g] = r;
        else if (i < state_size)
            logic[i] = r;
    }
}
extern "C" void host_rates(float* r, const uint32_t* s) { compute_transition_rates(r, s); }
extern "C" int host_classes()
{
#ifdef MBG_RATE_CLASSES
    return MBG_RATE_CLASSES;
#else
    return 0;
#endif
}
"""


def model(n, values=None, seed=0, discrete=0, depth=3):
    """n nodes with random logic (AND, OR, XOR, NOT, the constants) and rates from `values` (default: random)."""
    rng = np.random.default_rng(seed)
    names = [f"L{i}" for i in range(n)]

    def logic(d):
        if d == 0 or rng.random() < 0.25:
            x = names[rng.integers(n)] if rng.random() < 0.97 else str(rng.integers(2))
            return f"!{x}" if rng.random() < 0.3 else x
        op = rng.choice(["&", "|", "^"], p=[0.45, 0.45, 0.1])
        e = f"({logic(d - 1)} {op} {logic(d - 1)})"
        return f"!{e}" if rng.random() < 0.2 else e

    bnd = ""
    for name in names:
        up, down = rng.choice(values, 2) if values else rng.uniform(0.2, 3.0, 2)
        bnd += f"node {name} {{ logic = {logic(depth)}; rate_up = @logic ? {up:.6g} : 0; rate_down = @logic ? 0 : {down:.6g}; }}\n"
    cfg = "".join(f"{x}.is_internal = 1;\n" for x in names[5:])
    return bnd, cfg + f"max_time = 4; time_tick = 0.3; discrete_time = {discrete}; sample_count = 1000;\n"


@pytest.mark.parametrize("name", ["cellcycle", "sizek", "metastasis", "Montagud2022_Prostate_Cancer"])
def test_gates_encode_the_logic_of_example_models(tmp_path, name):
    """(logics of up to 236 literals, whose gates come from a factored form)"""
    m = mb.Model(*model_text(name))
    L = _gate_library(tmp_path, m.generate_code())
    _check_gates(L, m.num_nodes, False)


@pytest.mark.parametrize("n,values", [(1, [1.0]), (31, None), (32, [1.0, 10.0]), (33, [0.5, 0.0]), (64, None),
                                      (97, [1.0, 2.0, 4.0]), (200, None)])
def test_gates_encode_the_logic(tmp_path, n, values):
    L = _gate_library(tmp_path, mb.Model(*model(n, values)).generate_code())
    assert L.host_classes() == (0 if values is None else len([v for v in values if v > 0]) if n > 1 else 1)
    _check_gates(L, n, values is None)


@pytest.mark.parametrize("seed", range(4))
def test_gates_of_long_logics(tmp_path, seed):
    """Random trees of up to 32 literals of 12 nodes (factored where that is shorter), XOR and constants among them."""
    L = _gate_library(tmp_path, mb.Model(*model(12, seed=seed, depth=5)).generate_code())
    _check_gates(L, 12, True)


def _gate_library(tmp_path, code):
    assert "#define MBG_GATES 1" in code
    (tmp_path / "m.cpp").write_text(PRELUDE + code + WRAPPER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-o", str(tmp_path / "m.so"),
                    str(tmp_path / "m.cpp")], check=True, timeout=300)
    return C.CDLL(str(tmp_path / "m.so"))


def _check_gates(L, n, positive):
    rng = np.random.default_rng(1)
    for _ in range(8):
        bits = rng.random((n, 32)) < 0.5
        st = (bits.astype(np.uint64) << np.arange(32, dtype=np.uint64)).sum(1).astype(np.uint32)
        out = np.zeros(n, np.uint32)
        L.host_gates(st.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p))
        for t in range(32):
            words = np.zeros((n + 31) // 32, np.uint32)
            for i in range(n):
                words[i >> 5] |= np.uint32(int(bits[i, t]) << (i & 31))
            r = np.zeros(n, np.float32)
            L.host_rates(r.ctypes.data_as(C.c_void_p), words.ctypes.data_as(C.c_void_p))
            unstable = ((out >> np.uint32(t)) & 1).astype(bool) != bits[:, t]
            assert not (r[~unstable] != 0).any()
            if positive:  # (a listed rate may be 0)
                assert (r[unstable] != 0).all()


def test_no_gates_above_256_nodes():
    assert "MBG_GATES" in mb.Model(*model(256, depth=1)).generate_code()
    assert "MBG_GATES" not in mb.Model(*model(257, depth=1)).generate_code()


@pytest.mark.gpu
@pytest.mark.parametrize("n,values,discrete", [(1, [1.0], 0), (31, None, 0), (32, [1.0, 10.0], 1), (33, [0.5, 0.0], 0),
                                               (64, None, 1), (65, [3.0], 0), (97, [1.0, 2.0, 4.0], 0), (200, None, 0)])
@pytest.mark.parametrize("mode", ["exact", "fast", "epoch"])
def test_lockstep_kernels_match_oracle(gpu, n, values, discrete, mode):
    bnd, cfg = model(n, values, seed=n, discrete=discrete)
    res = gpu.compile(mb.Model(bnd, cfg)).run(mode=mode, sample_count=1300, seed=9, traj_len=7)
    raw = res.raw()
    ref = OracleModel(bnd, cfg).run(n=1300, mode=1 if mode == "fast" else 0, seed=9, traj_len=7,
                                    occ_exp=raw["occ_exp"], ent_exp=raw["ent_exp"])
    assert res.transitions == ref["transitions"]
    assert np.array_equal(res.final_counts, ref["final"])
    assert [c for _, c in res.fixed] == list(ref["fixed_counts"])
    if discrete:
        assert np.array_equal(raw["cnt"], ref["cnt"])
    else:
        assert np.all(np.abs(res.window_probs - ref["probs"]) <= 1e-5 + 1e-4 * ref["probs"])
    assert np.all(np.abs(res.window_entropy - ref["th"]) <= 1e-6 + 1e-4 * np.abs(ref["th"]))
