"""The constant tables of the rate kernels, checked on the host
(rates_tables_check.cu includes the library's own rates.cu; nothing runs on a
GPU)."""
import os
import shutil
import subprocess

import pytest

from test_sparse_plan import ROOT, cuda_home


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    cuda = cuda_home()
    nvcc = shutil.which("nvcc") or (cuda and os.path.join(cuda, "bin", "nvcc"))
    if not nvcc or not os.path.exists(nvcc):
        pytest.skip("nvcc is missing")
    exe = str(tmp_path_factory.mktemp("rates_tables") / "check")
    src = os.path.join(ROOT, "tests", "rates_tables", "rates_tables_check.cu")
    # the library's own architecture; the device code is only compiled along
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O1", "-std=c++17", "-cudart", "shared",
                        f"-I{ROOT}/include", "-o", exe, src, "-lpthread"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return exe


@pytest.mark.parametrize("what", ["align", "threads"])
def test_tables(check, what):
    r = subprocess.run([check, what], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
