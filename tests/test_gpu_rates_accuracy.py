"""Rounding errors of the photo and thermal rates against extended precision.

The library's exp and pow evaluated the reference's expressions with errors of
1.58e-16 rms (photo-rates, 12 rays, host evaluation of both networks, nearly all
of it the rounding of gamma A_V) and 6.8e-16 (thermal, the rounding of gamma/T).
The kernel's own exponentials have to do no worse: a photo-rate's rounding that
remains is that of 2^(j/1024), of the series, of the field's product and of the
sum, 1.43e-16 in a host evaluation, and a thermal one's 6e-17.  A single thermal
rate carries the rounding of T/300, |beta| 2^-53, and those of the table's row
times alpha, of the last sum and of the remainder, 4 2^-53 with room."""
import csv

import numpy as np
import pytest

import pdrgpu as G
import workloads as W

pytestmark = pytest.mark.gpu
L = np.longdouble


def rows(name):
    with open(f"{G.DATA}/rates_{name}.d") as f:
        out = [[x.strip() for x in r] for r in csv.reader(f) if any(x.strip() for x in r)]
    # members of a duplicate group are left out: only one of them has a rate
    dup = [i for i in range(1, len(out)) if out[i][1:8] == out[i - 1][1:8]]
    dup = set(dup) | {i - 1 for i in dup}
    return [(i, r) for i, r in enumerate(out) if i not in dup]


def errors(rate, i, ref):
    got = rate[:, i].astype(L)
    m = (ref > L(1e-90)) & (ref < L(0.9))
    return ((got - ref)[m] / ref[m]).astype(float)


@pytest.mark.parametrize("name,cfg", [("reduced", "C1"), ("full", "C2")])
def test_errors(cuda, name, cfg):
    import torch
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=cuda, dtype=torch.float64)  # noqa: E731
    w = W.chemistry(cfg, ncell=400, seed=81)
    ph = G.phys(w.zeta, w.omega, w.grain_radius, w.metallicity, w.g2d, w.v_turb_kms)
    rate, st = G.reaction_rates(G.Network(name), ph, t(w.T), t(w.Td), t(w.rad_surface), t(w.AV), t(w.column5))
    rate = rate.cpu().numpy()
    assert int(st.abs().sum()) == 0
    T, AV, rad = w.T.astype(L), w.AV.astype(L), w.rad_surface.astype(L)
    with open(f"{G.DATA}/species_{name}.d") as f:
        species = {ln.split(",")[1].strip() for ln in f if ln.strip()}
    num = lambda s: L(float(s)) if s else L(0)  # noqa: E731
    photo, thermal = [], []
    for i, r in rows(name):
        a, b, g = num(r[8]), num(r[9]), num(r[10])
        if r[2] == "PHOTON" and r[1] not in ("H2", "HD", "CO", "C"):
            photo.append(errors(rate, i, (a * rad * np.exp(-g * AV) / 2).sum(axis=1)))
        elif r[2] in species:
            if r[1] == r[2] == "H" or r[3] or g < -200 or "PAH" in r[1] + r[2]:
                continue
            e = errors(rate, i, a * (T / 300) ** b * np.exp(-g / T))
            assert e.size == 0 or np.abs(e).max() <= (abs(float(b)) + 4) * 2.0 ** -53, i
            thermal.append(e)
    photo, thermal = np.concatenate(photo), np.concatenate(thermal)
    rms = lambda e: np.sqrt((e ** 2).mean())  # noqa: E731
    print(name, "photo", len(photo), rms(photo), np.abs(photo).max(), "thermal", len(thermal), rms(thermal), np.abs(thermal).max())
    assert len(photo) > 5000 and len(thermal) > 20000
    assert rms(photo) < 1.55e-16 and np.abs(photo).max() < 1.3e-15
    assert rms(thermal) < 1.0e-16
