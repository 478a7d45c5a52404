"""Level populations at the edges of the batched kernels: batch remainders, one
ray and many, and optical depths at and beyond the guards of the escape
probability, against the oracle.

Tolerances as in test_gpu_levpop.py: 1e-6 for populations above 1e-6 of the
coolant density and for the cooling; the exponentials and divisions carry at
most about an ulp."""
import numpy as np
import pytest

import oracle as O
import pdrgpu as G
import workloads as W

pytestmark = pytest.mark.gpu


def both(cuda, key, ncell, nrays, precision, special=False, pseudo1d=False):
    import torch
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=cuda, dtype=torch.float64)  # noqa: E731
    oc = O.Coolant(key)
    lp = W.levpop(ncell=ncell, seed=71)
    tau = W.levpop_tau(ncell, oc.nlin, seed=72, nrays=nrays)
    if special:
        tau[:, :, :9] = [-10.0, -5.0, -1.0, -1.0e-9, 0.0, 1.0e-8, 700.0, 1.0e5, 1.0e50]
    dens = lp["n_H"] * W.COOLANT_X[key]
    spop = np.array([oc.lte(T, d) for T, d in zip(lp["T"], dens)])
    args = (lp["n_H"], lp["T"], lp["Td"], lp["partner5"], dens, spop, tau)
    ref = oc.levpop(*args, pseudo1d=int(pseudo1d))
    got = G.level_populations(G.Coolant(key), *[t(a) for a in args], pseudo1d=pseudo1d, precision=precision, want_line=True)
    return dens, ref, [g.cpu().numpy() for g in got]


def check(dens, ref, got):
    pop_r, cool_r, line_r, _ = ref
    pop, cool, line, status = got
    assert ((status == 0) | (status == 2)).all()
    m = pop_r > 1e-6 * dens[:, None]
    assert (np.abs(pop - pop_r)[m] / pop_r[m]).max() < 1e-6
    m = np.abs(cool_r) > 1e-40
    assert (np.abs(cool - cool_r)[m] / np.abs(cool_r)[m]).max() < 1e-6
    big = np.abs(line_r) > 1e-6 * np.abs(line_r).reshape(len(dens), -1).max(axis=1)[:, None, None]
    assert (np.abs(line - line_r)[big] / np.abs(line_r[big])).max() < 1e-6
    assert np.array_equal(line != 0, line_r != 0)


@pytest.mark.parametrize("key", ["CII", "CO"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("ncell,nrays", [(1, 12), (33, 1), (70, 48)])
def test_batches_and_rays(cuda, key, precision, ncell, nrays):
    check(*both(cuda, key, ncell, nrays, precision))


@pytest.mark.parametrize("key", ["OI", "CO"])
def test_optical_depth_guards(cuda, key):
    check(*both(cuda, key, 40, 12, "fp64", special=True))


def test_batch_independence(cuda):
    """A cell's result does not depend on the batch it is in (C+, past one block's batch on every SM)."""
    n = 6000
    _, _, small = both(cuda, "CII", 64, 12, "fp64")
    import torch
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=cuda, dtype=torch.float64)  # noqa: E731
    oc = O.Coolant("CII")
    lp = W.levpop(ncell=64, seed=71)
    tau = W.levpop_tau(64, oc.nlin, seed=72)
    dens = lp["n_H"] * W.COOLANT_X["CII"]
    spop = np.array([oc.lte(T, d) for T, d in zip(lp["T"], dens)])
    rep = lambda a: t(np.concatenate([a] * (n // 64 + 1))[:n])  # noqa: E731
    got = G.level_populations(G.Coolant("CII"), *[rep(a) for a in (lp["n_H"], lp["T"], lp["Td"], lp["partner5"], dens, spop, tau)])
    assert np.array_equal(got[0].cpu().numpy(), np.concatenate([small[0]] * (n // 64 + 1))[:n])
