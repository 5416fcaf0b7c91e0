"""The work list of the FP64 kernel for small batches on the CPU:
tests/cxx/small_items_check.cu is compiled against the library's internal
header, linked against libfrpa.so and run without a GPU.  Also the autotuner's
candidates for plans that this kernel may serve."""
import os
import shutil
import subprocess
import types

import numpy as np
import pytest

from fast_rpa_eval_b200 import _lib, autotune

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
LIB_DIR = os.path.join(ROOT, "fast_rpa_eval_b200", "lib")


@pytest.mark.skipif(not os.path.exists(NVCC), reason="nvcc not available")
@pytest.mark.skipif(not os.path.exists(os.path.join(LIB_DIR, "libfrpa.so")), reason="libfrpa.so not built")
def test_small_batch_work_lists(tmp_path):
    exe = str(tmp_path / "small_items_check")
    build = [NVCC, "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "include"),
             "-I" + os.path.join(ROOT, "fast_rpa_eval_b200", "csrc"),
             os.path.join(ROOT, "tests", "cxx", "small_items_check.cu"), "-o", exe,
             "-L" + LIB_DIR, "-lfrpa", "-Xlinker", "-rpath=" + LIB_DIR]
    subprocess.run(build, check=True, capture_output=True, timeout=300)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr


def test_autotune_candidates_are_different_launches():
    small = types.SimpleNamespace(n_compute_c_batches=np.array([40, 120, 0], np.int32))
    large = types.SimpleNamespace(n_compute_c_batches=np.array([40, 121], np.int32))
    c = autotune.candidates(small, _lib.RHO1_FP64)
    assert [x for x in c if x["fp64_small"] == 2] == [{"fp64_small": 2}]
    assert [{k: v for k, v in x.items() if k != "fp64_small"} for x in c if x["fp64_small"] == 1] == autotune.FP64_SPACE
    for mode in (_lib.RHO1_FP64, _lib.RHO1_SPLIT_BF16, _lib.RHO1_SPLIT_I8):
        assert autotune.candidates(large, mode) == autotune.space(mode)
    assert autotune.candidates(small, _lib.RHO1_SPLIT_BF16) == autotune.space(_lib.RHO1_SPLIT_BF16)
