"""Every heating term by itself against the oracle, in the range of the fast
elementary functions, at its ends and beyond them (where the library's are
taken).

Tolerance 1e-13 of the term, or of the larger of the parts it is the difference
of: a term is a product or quotient of at most some 20 factors, each rounded to
2^-53, with powers to 1.4 2^-52 whose arguments (T, delta) carry up to 4 roundings
themselves; 60 2^-53 is 7e-15.  The PAH term's exponent beta carries four more,
times ln delta (at most 150 here): 5e-14.  The Newton iteration for the grain charge stops at
a change of 1e-2, so it may take one step more only where that change is met to
the last bits."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
import pdrgpu as G
import workloads as W

pytestmark = pytest.mark.gpu
NAMES = ["photoelectric", "PAH", "Weingartner", "C ionisation", "H2 formation", "H2 photodissociation", "FUV pumping",
         "cosmic rays", "turbulence", "chemical", "gas-grain"]


def dev(a, d):
    import torch
    return torch.as_tensor(np.ascontiguousarray(a), device=d, dtype=torch.float64)


def parts(n, T, xe, uv):
    """Magnitudes of the two parts of the photoelectric and the PAH heating."""
    R4 = lambda x: np.float64(np.float32(x))  # noqa: E731
    hab, EV, KB = 1.68 * uv, 1.60217646e-12, 1.38065040e-16
    xk, xd = KB * T / (13.6 * EV), 6.0 / 13.6
    gam = 2.9e-4 * 0.1 * np.sqrt(T) * hab / (xe * n)
    delta, x = xk - xd + gam, 0.5
    for _ in range(100):
        new = x - (x ** 3 + delta * x * x - gam) / (3 * x * x + delta * 2 * x)
        done, x = abs(new - x) < 1e-2, new
        if done:
            break
    pe = 2.7e-25 * 1.8 * n * 0.1 * hab * max(abs((1 - x) ** 2 / x), abs(xk * (x * x - 1) / (x * x)))
    d = hab * np.sqrt(T) / (xe * n)
    eps = 4.87e-2 / (1 + 4e-3 * d ** R4(0.73)) + 3.65e-2 * (T / 1e4) ** R4(0.7) / (1 + 2e-4 * d)
    return pe, 1.30e-24 * eps * hab * n


@pytest.mark.parametrize("name,network", [("reduced", 0), ("full", 1)])
def test_terms(cuda, name, network):
    n = 96
    w = W.chemistry("C1", ncell=n, seed=101)
    onet = O.Network(name)
    rng = np.random.Generator(np.random.PCG64(102))
    ab = 10.0 ** rng.uniform(-12, -1, (n, onet.nspec))
    uv = 10.0 ** rng.uniform(-2, 3, n)
    w.T[:] = 10.0 ** rng.uniform(0.0, 5.0, n)
    # the ends of the fast range, and beyond: T 1 to 1e6, dust 0 to 1e6, field and x_e n 1e-30 to 1e30
    w.T[:8] = [1.0, np.nextafter(1.0, 0), 0.5, 1.0e6, np.nextafter(1.0e6, 1e7), 3.0e6, 2.7, 1.0e4]
    w.Td[8:12] = [0.0, 1.0e6, 2.0e6, 1.0e-3]
    uv[12:16] = [1.0e-30, 1.0e-31, 1.0e-3, 1.0e6]
    e = onet.species.index("e-")
    ab[16:20, e] = [1.0e-30 / w.n_H[16], 1.0e-31 / w.n_H[17], 1.0e-20, 0.9]
    ph = O.phys(w.zeta, w.omega, w.grain_radius, w.metallicity, w.g2d, w.v_turb_kms)
    rates, _ = onet.rates(ph, np.clip(w.T, 10.0, 1e4), w.Td + 10.0, w.rad_surface, w.AV, w.column5)
    _, nr, _ = onet.rates_cell(ph, w.T[20], w.Td[20], w.rad_surface[20], w.AV[20], w.column5[20].ravel())
    nr = np.ascontiguousarray(nr, dtype=np.int32)
    ref = np.zeros((n, 12))
    for c in range(n):
        out = np.zeros(12)
        O.lib().orc_heating(onet.p, network, C.byref(ph), w.n_H[c], w.T[c], w.Td[c], uv[c],
                            O._ptr(np.ascontiguousarray(ab[c])), O._ptr(np.ascontiguousarray(rates[c])),
                            O._ptr(nr, O._ip), O._ptr(out))
        ref[c] = out
    got = G.heating(G.Network(name), network, G.phys(w.zeta, w.omega, w.grain_radius, w.metallicity, w.g2d, w.v_turb_kms),
                    dev(w.n_H, cuda), dev(w.T, cuda), dev(w.Td, cuda), dev(uv, cuda), dev(ab, cuda),
                    dev(rates, cuda)).cpu().numpy()
    scale = np.abs(ref)
    for c in range(n):
        with np.errstate(all="ignore"):
            pe, pah = parts(w.n_H[c], w.T[c], ab[c, e], uv[c])
        scale[c, 0], scale[c, 1] = max(scale[c, 0], pe), max(scale[c, 1], pah)
    scale[:, 11] = scale[:, [1, 3, 4, 5, 6, 7, 8, 9, 10]].max(axis=1)
    assert np.array_equal(np.isfinite(got), np.isfinite(ref)) and np.isfinite(ref).all()
    for k, term in enumerate(NAMES + ["total"]):
        err = np.abs(got[:, k] - ref[:, k]) / np.where(scale[:, k] > 0, scale[:, k], 1.0)
        assert err.max() < 1e-13, (term, int(err.argmax()), err.max())
