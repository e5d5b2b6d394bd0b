"""Host-only check of the choice between the DSSIM map pass's tiles and strips
(tests/ds_form_check.cu) against the times of both forms on a B200.  Builds the
harness with nvcc (host code only runs) and links the library for the planner's
host helpers."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "turbo-metrics_b200")
CUDA = "/usr/local/cuda"


@pytest.mark.skipif(shutil.which("nvcc") is None and not os.path.exists(os.path.join(CUDA, "bin", "nvcc")),
                    reason="nvcc not available")
def test_dssim_form_is_the_faster_one(tmb, tmp_path):
    nvcc = os.path.join(CUDA, "bin", "nvcc") if os.path.exists(os.path.join(CUDA, "bin", "nvcc")) else "nvcc"
    exe = str(tmp_path / "ds_form_check")
    subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a",
                    os.path.join(ROOT, "tests", "ds_form_check.cu"), "-o", exe, "-L" + PKG, "-lssim2b200",
                    "-L" + os.path.join(CUDA, "lib64"), "-lcudart", "-Xlinker", "-rpath=" + PKG],
                   check=True, capture_output=True)
    env = dict(os.environ)
    env["LD_LIBRARY_PATH"] = PKG + os.pathsep + os.path.join(CUDA, "lib64") + os.pathsep + env.get("LD_LIBRARY_PATH", "")
    out = subprocess.run([exe], capture_output=True, text=True, env=env, timeout=120)
    assert out.returncode == 0 and out.stdout.strip().endswith("OK fails=0"), out.stdout + out.stderr
