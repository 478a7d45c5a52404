"""The FP64 elementary functions of the kernels (fp64_fast.cuh), compiled for the
host and checked there (fp64_check.cpp)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DIR = os.path.join(ROOT, "tests", "fp64_check")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ is missing")
    exe = str(tmp_path_factory.mktemp("fp64") / "fp64_check")
    # a product and a sum fuse where the code says so, and nowhere else
    r = subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=gnu++17", f"-I{DIR}", "-o", exe,
                        os.path.join(DIR, "fp64_check.cpp"), "-lquadmath"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return exe


@pytest.mark.parametrize("what", ["rounding", "tables", "functions"])
def test_functions(check, what):
    r = subprocess.run([check, what], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
