"""Reaction rates at the edges of the batched kernel: batch remainders, the ends
of the fast path's ranges, and cells beyond them (which the general path
evaluates), against the oracle.

Tolerance 1e-12 relative, as for the rates everywhere: the kernel's
exponentials and powers carry at most about 2 ulp, and the oracle's rounding of
gamma/T is worth up to 230 ulp at the 1e-99 cut-off."""
import numpy as np
import pytest

import oracle as O
import pdrgpu as G
import workloads as W

pytestmark = pytest.mark.gpu


def run(cuda, name, w, zeta=None):
    import torch
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=cuda, dtype=torch.float64)  # noqa: E731
    ph = G.phys(w.zeta, w.omega, w.grain_radius, w.metallicity, w.g2d, w.v_turb_kms)
    rate, st = G.reaction_rates(G.Network(name), ph, t(w.T), t(w.Td), t(w.rad_surface), t(w.AV), t(w.column5))
    return rate.cpu().numpy(), st.cpu().numpy()


def oracle(name, w):
    net = O.Network(name)
    return net.rates(O.phys(w.zeta, w.omega, w.grain_radius, w.metallicity, w.g2d, w.v_turb_kms), w.T, w.Td,
                     w.rad_surface, w.AV, w.column5)[0]


def close(got, ref):
    assert np.array_equal(got > 0, ref > 0)
    m = ref > 0
    assert (np.abs(got - ref)[m] / ref[m]).max() < 1e-12


@pytest.mark.parametrize("name,cfg", [("reduced", "C1"), ("full", "C2"), ("mynetwork", "C1")])
@pytest.mark.parametrize("ncell", [1, 33, 913])
def test_batches(cuda, name, cfg, ncell):
    w = W.chemistry(cfg, ncell=ncell, seed=61)
    rate, st = run(cuda, name, w)
    assert (st == 0).all()
    close(rate, oracle(name, w))


def test_ranges_and_general_path(cuda):
    w = W.chemistry("C1", ncell=40, seed=62)
    # ends of the fast path's temperature range, and beyond them
    w.T[:6] = [1.0e-2, 1.0e8, 5.0e-3, 2.0e8, 2.7, 300.0]
    # the shielding functions' branches: empty columns, both ends of the CO grid, knots of the splines
    w.column5[6] = 0.0
    w.column5[7, :, 0], w.column5[7, :, 2] = 1.0e24, 1.0e20
    w.column5[8, :, 0], w.column5[8, :, 2] = 1.0e20 - 1.0, 1.0e15 - 1.0
    w.column5[9, :, 0] = np.geomspace(1.0e9, 1.0e22, 12)
    w.column5[10, 3, 2] = 1.0e31            # beyond the fast path
    w.column5[11, 5, 3] = 1.0e-40           # beyond the fast path
    # extinction: none, the scattering's one-exponential limit from both sides, opaque
    w.AV[12] = 0.0
    w.AV[13] = np.linspace(0.2, 0.5, 12)
    w.AV[14] = np.geomspace(30.0, 1.0e5, 12)
    w.rad_surface[15] = 0.0
    w.rad_surface[16, ::2] = 0.0
    rate, st = run(cuda, "reduced", w)
    assert (st == 0).all()
    close(rate, oracle("reduced", w))


def test_negative_rate_status(cuda):
    """A negative field gives negative photo-rates: reported as the lowest reaction number, stored as 0."""
    w = W.chemistry("C1", ncell=5, seed=63)
    w.rad_surface[2] = -1.0
    rate, st = run(cuda, "reduced", w)
    net = O.Network("reduced")
    photo = [i + 1 for i, ln in enumerate(open(G.DATA + "/rates_reduced.d")) if ln.split(",")[2] == "PHOTON"]
    assert st.tolist() == [0, 0, -min(photo), 0, 0] and net.nreac == rate.shape[1]
    assert (rate[2, np.array(photo) - 1] == 0).all()
