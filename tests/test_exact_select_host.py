"""The choice of the node that flips in the incremental and lockstep exact kernels, compiled for the host from the
kernels' source: for every r in [0, total] it is the reference's prefix count (simulation.cu:9-21), r = 0 (a
total rate so small that its product with a uniform number underflows) included."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from test_codegen_host import PRELUDE

ENGINE = os.path.join(ROOT, "maboss", "gpu_b200", "csrc", "kernels", "engine.cuh")

HOST = r"""
inline int __ffs(uint32_t x) { return __builtin_ffs((int)x); }
inline float __uint_as_float(uint32_t x) { float f; __builtin_memcpy(&f, &x, 4); return f; }
constexpr int state_words = WORDS;
constexpr int MB_LW = WORDS;
static float mbg_inc_rate[64 * WORDS];
struct view
{
    uint32_t s[WORDS], u[WORDS], q[WORDS];
    uint32_t S(int w) const { return s[w]; }
    uint32_t U(int w) const { return u[w]; }
    uint32_t Q(int w) const { return q[w]; }
};
inline float mb_rate(const view&, int w, int b, unsigned on) { return mbg_inc_rate[2 * (32 * w + b) + on]; }
"""

CALLS = r"""
extern "C" void host_select(const float* rates, const uint32_t* s, const uint32_t* u, float r, int* out)
{
    __builtin_memcpy(mbg_inc_rate, rates, sizeof mbg_inc_rate);
    view v;
    mb_lock k;
    float q[WORDS], run = 0.f;
    for (int w = 0; w < WORDS; w++)
    {
        for (int b = 0; b < 32; b++)
            if ((u[w] >> b) & 1u)
                run += rates[2 * (32 * w + b) + ((s[w] >> b) & 1u)];
        v.s[w] = k.s[w] = s[w];
        v.u[w] = k.u[w] = u[w];
        q[w] = run;
        __builtin_memcpy(&v.q[w], &run, 4);
    }
    out[0] = mb_exact_select(v, r);
    out[1] = mb_lock_exact_select(k, q, r);
}
"""


def _function(text, start):
    a = text.index(start)
    return text[a:text.index("\n}", a) + 2] + (";" if start.startswith("struct") else "") + "\n"


@pytest.mark.parametrize("words", [1, 3, 8])
def test_select_is_the_prefix_count(tmp_path, words):
    text = open(ENGINE).read()
    parts = [_function(text, x) for x in ("struct mb_lock\n", "template <class V>\n__device__ __forceinline__ int mb_exact_select",
                                          "__device__ __forceinline__ int mb_lock_exact_select")]
    src = PRELUDE + f"#define WORDS {words}\n" + HOST + "".join(parts) + CALLS
    (tmp_path / "s.cpp").write_text(src)
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-shared", "-fPIC", "-o", str(tmp_path / "s.so"), str(tmp_path / "s.cpp")],
                   check=True, timeout=300)
    lib = C.CDLL(str(tmp_path / "s.so"))
    rng = np.random.default_rng(words)
    out = np.zeros(2, np.int32)
    for trial in range(600):
        scale = [1.0, 1e-44, 3.0][trial % 3]
        rates = (rng.uniform(0.1, 4.0, (32 * words, 2)) * scale).astype(np.float32)
        rates[rng.random(rates.shape) < 0.1] = 0.0
        state = rng.integers(0, 2**32, words, dtype=np.uint32)
        unstable = rng.integers(0, 2**32, words, dtype=np.uint32) & rng.integers(0, 2**32, words, dtype=np.uint32)
        unstable[rng.random(words) < 0.4] = 0  # empty words, the first one among them
        sums, run = np.zeros(32 * words, np.float32), np.float32(0)
        for i in range(32 * words):
            if (unstable[i >> 5] >> np.uint32(i & 31)) & 1:
                run = np.float32(run + rates[i, (state[i >> 5] >> np.uint32(i & 31)) & 1])
            sums[i] = run
        if run == 0:
            continue
        for r in (np.float32(0), np.float32(run), np.float32(rng.random()) * run, np.float32(1e-45), sums[sums > 0][0]):
            r = min(np.float32(r), run)
            lib.host_select(rates.ctypes.data_as(C.c_void_p), state.ctypes.data_as(C.c_void_p),
                            unstable.ctypes.data_as(C.c_void_p), C.c_float(float(r)), out.ctypes.data_as(C.c_void_p))
            assert list(out) == [int((sums < r).sum())] * 2, (trial, float(r))
