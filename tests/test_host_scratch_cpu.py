"""The library's device buffers against a fake of the CUDA runtime (host_scratch.cu):
what a captured graph addresses stays where it is, and a failed allocation leaves
nothing behind that a later call takes for valid."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("nvcc not found")
    exe = str(tmp_path_factory.mktemp("host") / "host_scratch")
    subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                    "-diag-suppress", "177", "-cudart", "none", os.path.join(HERE, "host_scratch.cu"),
                    os.path.join(HERE, "..", "deepcharacters_b200", "csrc", "hc_common.cu"), "-o", exe],
                   check=True)
    return exe


@pytest.mark.parametrize("check", ["uv_held", "uv_recorded", "uv_no_memory", "fan_entries", "resident",
                                   "spare_held", "spare_no_memory", "failed_allocation"])
def test_host_buffers(program, check):
    r = subprocess.run([program, check], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
