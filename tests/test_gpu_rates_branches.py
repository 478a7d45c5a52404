"""Reaction rates at the values where the reference changes its expression: the
scattering function's one- and five-exponential forms (they differ by 3.8e-4 at
tau = 1) and its exponents of 100, the H2 self-shielding's Doppler cores, and
gamma < -200 below a reaction's temperature range.  The fast path has to take the
reference's side of each, to the last bit.

Tolerance 1e-12 relative, as for the rates everywhere; a value on the wrong side
is 3e-8 to 1 off."""
import os

import numpy as np
import pytest

import oracle as O
import pdrgpu as G
import workloads as W

pytestmark = pytest.mark.gpu


def dev(a, d):
    import torch
    return torch.as_tensor(np.ascontiguousarray(a), device=d, dtype=torch.float64)


def compare(cuda, w, name="reduced", **kw):
    ph = (w.zeta, w.omega, w.grain_radius, w.metallicity, w.g2d, w.v_turb_kms)
    rate, st = G.reaction_rates(G.Network(name, **kw), G.phys(*ph), dev(w.T, cuda), dev(w.Td, cuda),
                                dev(w.rad_surface, cuda), dev(w.AV, cuda), dev(w.column5, cuda))
    rate, st = rate.cpu().numpy(), st.cpu().numpy()
    ref = O.Network(name, **kw).rates(O.phys(*ph), w.T, w.Td, w.rad_surface, w.AV, w.column5)[0]
    assert (st == 0).all()
    assert np.array_equal(rate > 0, ref > 0)
    m = ref > 0
    assert (np.abs(rate - ref)[m] / ref[m]).max() < 1e-12
    return ref


def around(x, ulps=12):
    """x, its neighbours, and values up to 2e-7 of it away."""
    out = [x]
    for _ in range(ulps):
        out = [np.nextafter(out[0], -np.inf), *out, np.nextafter(out[-1], np.inf)]
    for rel in (1e-12, 1e-10, 1e-9, 5e-9, 1.2e-8, 3e-8, 1e-7, 2e-7):
        out += [x * (1 - rel), x * (1 + rel)]
    return np.array(out)


def cells(n):
    w = W.chemistry("C1", ncell=n, seed=71)
    w.column5[:, :, 0] = 1.0e15
    w.column5[:, :, 2] = 1.0e13
    return w


K = np.array([0.7514, 0.8490, 1.013, 1.282, 2.005, 5.832])


@pytest.mark.parametrize("tau", [1.0, *(100.0 / K[1:])])
def test_scattering_at_1000(cuda, tau):
    # tau(1000 A)/tau(V) is a knot of the extinction curve, 4.65
    av = around(tau * 1.086 / 4.65)
    w = cells(len(av))
    w.AV[:] = av[:, None]
    thin = (av / 1.086) * 4.65 < 1.0
    assert tau != 1.0 or (thin.any() and not thin.all())
    compare(cuda, w)


def test_scattering_at_the_mean_wavelength_of_co(cuda):
    L = O.lib()
    import ctypes as C
    L.orc_xlambda.restype = L.orc_lbar.restype = C.c_double
    L.orc_xlambda.argtypes, L.orc_lbar.argtypes = [C.c_double, C.c_int], [C.c_double, C.c_double]
    for nco, nh2 in ((1.0e13, 1.0e15), (1.0e16, 1.0e21), (3.0e17, 2.0e20)):
        x = L.orc_xlambda(L.orc_lbar(nco, nh2), 0)
        for tau in (1.0, 100.0 / K[1], 100.0 / K[2]):
            # the wavelength's own rounding moves tau by an ulp or so: no closer than 1e-12
            av = around(tau * 1.086 / x, ulps=0)[1:]
            w = cells(len(av))
            w.column5[:, :, 0], w.column5[:, :, 2] = nh2, nco
            w.AV[:] = av[:, None]
            compare(cuda, w)


@pytest.mark.parametrize("taud", [2.0, 10.0, 100.0])
def test_h2_doppler_core(cuda, taud):
    dopw = 1.0e5 / (1000.0 * 1.0e-8)
    nh2 = around(taud * dopw / (0.5 * 1.497358985e-2 * 1.0e-2))
    w = cells(len(nh2))
    w.column5[:, :, 0] = nh2[:, None]
    compare(cuda, w)


def test_gamma_of_minus_200(cuda, tmp_path):
    """Zero below RTMIN for gamma < -200, however close to it."""
    gammas = [-200.0, np.nextafter(-200.0, -300), -200.000001, -200.00001, -200.1, np.nextafter(-200.0, 0), -199.999999]
    # behind the reduced network's reactions, each gamma without and with a power of T
    with open(os.path.join(G.DATA, "species_reduced.d")) as f, open(os.path.join(tmp_path, "species_edge.d"), "w") as g:
        g.write(f.read())
    with open(os.path.join(G.DATA, "rates_reduced.d")) as f, open(os.path.join(tmp_path, "rates_edge.d"), "w") as g:
        lines = f.read().rstrip("\n").split("\n")
        n0 = len(lines)
        for i, gam in enumerate(gammas):
            for a, b, beta in (("C", "Mg", 0.0), ("O", "Mg", 0.5)):
                p = "H" if i % 2 else "H2"   # neighbours differ, so that they are no duplicate group
                lines.append(f"{len(lines) + 1},{a},{b},,{a},{p},,,1.0E-18,{beta},{float(gam)!r},L,50,41000,A,")
        g.write("\n".join(lines) + "\n")
    w = W.chemistry("C1", ncell=3, seed=72)
    w.T[:] = [20.0, 49.999, 50.0]
    ref = compare(cuda, w, name="edge", data_dir=str(tmp_path))
    below = np.repeat(np.array(gammas) < -200.0, 2)
    assert (ref[:2, n0:] == 0).all(axis=0).tolist() == below.tolist() and (ref[2] > 0)[n0:].all()
