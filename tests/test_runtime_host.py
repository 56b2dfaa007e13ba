"""The host runtime without a GPU: order of uploads, loading after a failure, bounds of what is kept, on the stand-in
for CUDA of tests/cpp/fake_cuda.h."""
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "maboss", "gpu_b200", "csrc")


@pytest.fixture(scope="module")
def runtime_test(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("runtime") / "runtime_test")
    objects = [os.path.join(CSRC, "_build", f"{n}.o")
               for n in ("model", "codegen", "gates", "runtime", "output", "sparse_bins")]
    subprocess.run(["g++", "-O1", "-std=c++17", "-I/usr/local/cuda/include", "-I" + os.path.join(ROOT, "include"), "-I" + CSRC,
                    os.path.join(ROOT, "tests", "cpp", "runtime_test.cpp"), *objects, "-lpthread", "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("check", ["jump_table_is_there_before_the_first_launch", "family_loads_after_a_failure",
                                   "staging_memory_is_bounded", "kept_buffers_are_given_back",
                                   "exact_run_in_more_launches_where_memory_is_short"])
def test_runtime(runtime_test, check):
    p = subprocess.run([runtime_test, check], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0, p.stdout + p.stderr
