"""Which plan a convolution of the tensor-core kernel takes, and what is remembered of a measurement: the planner's host code
compiled with its CUDA calls replaced (`conv_plans.cu`). Needs nvcc, no GPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path_factory.mktemp("plans") / "conv_plans")
    # the kernels are not run: the compiler need not optimise them
    r = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=compute_100a", "-Xcicc", "-O0", "-std=c++17", "-I",
                        os.path.join(HERE, "..", "rembrandt_b200", "csrc"), os.path.join(HERE, "conv_plans.cu"), "-o", exe],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    return exe


@pytest.mark.parametrize("scenario", ["remembered_flat_does_not_fit", "paddings_are_measured_apart", "sub_tiles_of_other_modes",
                                      "deterministic_keeps_one_order", "pairs_win_by_a_margin", "flat_tiles_within_the_cap",
                                      "addends_are_aligned", "strided_outputs_are_aligned", "row_plans_win_by_a_margin",
                                      "row_plans_are_remembered"])
def test_plans(program, scenario):
    r = subprocess.run([program, scenario], capture_output=True, text=True, timeout=60,
                       env={k: v for k, v in os.environ.items() if not k.startswith("RB_GEMM_")})
    assert r.returncode == 0, r.stdout + r.stderr
