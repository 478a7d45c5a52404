"""The warp integrator's packed term tables, replayed on the host against the
stoichiometry (packed_check.cpp includes the library's own pdr_net.cpp): the
reduced network, and made-up ones of 32 ODE species at the ends of the packed
fields."""
import os
import random
import shutil
import subprocess

import pytest

from test_sparse_plan import ROOT, cuda_home

DATA = os.path.join(ROOT, "data")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    cuda = cuda_home()
    if shutil.which("g++") is None or cuda is None:
        pytest.skip("g++ or the CUDA headers are missing")
    exe = str(tmp_path_factory.mktemp("packed") / "packed_check")
    src = os.path.join(ROOT, "tests", "table_check", "packed_check.cpp")
    libdir = os.path.join(cuda, "lib64") if os.path.exists(os.path.join(cuda, "lib64")) else os.path.join(cuda, "lib")
    r = subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", f"-I{cuda}/include", f"-I{ROOT}/include", "-o",
                        exe, src, f"-L{libdir}", "-lcudart", f"-Wl,-rpath,{libdir}"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return exe


# 20 neutral species, 12 cations
NAMES = [f"N{i}" for i in range(20)] + [f"I{i}+" for i in range(12)]


def write_network(tmp_path, reactions):
    """reactions: lists of (reactants, products)."""
    sp, rt = str(tmp_path / "species.d"), str(tmp_path / "rates.d")
    with open(sp, "w") as f:
        for i, s in enumerate(NAMES + ["e-"]):
            f.write(f"{i + 1},{s},0.0,1.0\n")
    with open(rt, "w") as f:
        for i, (a, b) in enumerate(reactions):
            a, b = (list(a) + [""] * 3)[:3], (list(b) + [""] * 4)[:4]
            f.write(f"{i + 1},{','.join(a)},{','.join(b)},1.0E-10,0.0,0.0,L,10,41000,A,\n")
    return sp, rt


def run(check, sp, rt, layout, want):
    r = subprocess.run([check, sp, rt, layout, want], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


def test_reduced_network(check):
    run(check, *(f"{DATA}/{f}_reduced.d" for f in ("species", "rates", "layout")), "warp")


def many(n, seed):
    """n distinct reactions among all species (the same reactants and products
    side by side would make a duplicate group), electron reactions among them."""
    rng = random.Random(seed)
    out = []
    while len(out) < n:
        a = [rng.choice(NAMES), rng.choice(NAMES + ["e-"]) if rng.random() < 0.8 else "CRP"]
        out.append((a, rng.sample(NAMES, rng.randint(1, 4))))
    return out


# 9,600 reactions: more than 8,191 rate constants, and the mixed form's arrays of one
# warp (16 bytes a reaction) still fit a block's 227 KB
@pytest.mark.parametrize("nreac,want", [(2000, "warp"), (8300, "warp"), (9600, "warp"), (16500, "block"),
                                        (33000, "block")])
def test_size_of_the_network(check, tmp_path, nreac, want):
    run(check, *write_network(tmp_path, many(nreac, nreac)), "-", want)


def test_electron_alone_in_its_reactions(check, tmp_path):
    """No pair of the electron and few enough pairs that they all fit beside the
    x_e sum (129 free lanes): a one-body electron reaction still reads x_e."""
    pairs = [(NAMES[i], NAMES[j]) for i in range(16) for j in range(i, 16)]
    for npair in (1, 129, 130):
        reac = [(p, [NAMES[20 + k % 12]]) for k, p in enumerate(pairs[:npair])] + [(("e-", "FREEZE"), ["N3", "N19"])]
        out = run(check, *write_network(tmp_path, reac), "-", "warp")
        assert "pair rounds 6" in out
