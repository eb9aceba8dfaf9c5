"""The tensor-core kernels' bounded waits: a wait that runs out is reported whichever warp gave up."""
import os
import subprocess

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu


def test_a_wait_that_runs_out_in_the_last_warp_is_reported(tmp_path):
    exe = str(tmp_path / "wait_status_check")
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17",
                    "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "leviathan_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "wait_status_check.cu"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=60).stdout.split()
    assert out == ["0", "8"]   # LEV_DEV_TIMEOUT
