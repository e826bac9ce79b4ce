"""Error paths of the trajectory analysis' host code on the CPU: csrc/analysis.cu linked with a CUDA runtime
made of host memory whose calls fail one at a time (tests/native/analysis_errors.cpp)."""
import os
import shutil
import subprocess

import pytest

from conftest import REPO


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    nvcc = shutil.which(os.environ.get("NVCC", "nvcc"))
    if not nvcc:
        pytest.skip("nvcc not available")
    d = tmp_path_factory.mktemp("analysis_errors")
    exe = str(d / "analysis_errors")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O1", "-std=c++17", "-cudart", "none",
                    "--expt-relaxed-constexpr", "-I", os.path.join(REPO, "include"),
                    "-I", os.path.join(REPO, "capsid-souffle_gb300", "csrc"),
                    os.path.join(REPO, "capsid-souffle_gb300", "csrc", "analysis.cu"),
                    os.path.join(REPO, "tests", "native", "analysis_errors.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("what", ["drains", "grows"])
def test_failing_calls_and_allocations(checker, what):
    r = subprocess.run([checker, what], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
