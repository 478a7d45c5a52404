"""The rounds of the block integrator's leaf-column elimination against a
row-by-row elimination, bit for bit, on the host (gather_check.cpp includes the
library's own pdr_net.cpp)."""
import os
import shutil
import subprocess

import pytest

from test_sparse_plan import ROOT, cuda_home


def test_gather_rounds(tmp_path):
    cuda = cuda_home()
    if shutil.which("g++") is None or cuda is None:
        pytest.skip("g++ or the CUDA headers are missing")
    exe = str(tmp_path / "gather_check")
    src = os.path.join(ROOT, "tests", "sparse_plan", "gather_check.cpp")
    libdir = os.path.join(cuda, "lib64") if os.path.exists(os.path.join(cuda, "lib64")) else os.path.join(cuda, "lib")
    # no contraction: a product and a sum fuse where the program says so
    r = subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", f"-I{cuda}/include", f"-I{ROOT}/include",
                        "-o", exe, src, f"-L{libdir}", "-lcudart", f"-Wl,-rpath,{libdir}"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe, os.path.join(ROOT, "data"), "reduced", "mynetwork", "full"], capture_output=True,
                       text=True, timeout=300)
    print(r.stdout)
    assert r.returncode == 0, r.stdout + r.stderr
