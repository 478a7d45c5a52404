"""Rates that the fast path leaves to the general one as a whole: more rays than a
block's shared memory holds, an albedo or a Doppler width outside the fast path's
ranges.  Tolerance 1e-12 relative, as for the rates everywhere."""
import numpy as np
import pytest

import oracle as O
import pdrgpu as G
import workloads as W

pytestmark = pytest.mark.gpu


def dev(a, d):
    import torch
    return torch.as_tensor(np.ascontiguousarray(a), device=d, dtype=torch.float64)


def compare(cuda, name, w, **kw):
    k = dict(zeta=w.zeta, omega=w.omega, rad=w.grain_radius, z=w.metallicity, g2d=w.g2d, v=w.v_turb_kms)
    k.update(kw)
    ph = tuple(k.values())
    rate, st = G.reaction_rates(G.Network(name), G.phys(*ph), dev(w.T, cuda), dev(w.Td, cuda), dev(w.rad_surface, cuda),
                                dev(w.AV, cuda), dev(w.column5, cuda))
    rate, st = rate.cpu().numpy(), st.cpu().numpy()
    ref = O.Network(name).rates(O.phys(*ph), w.T, w.Td, w.rad_surface, w.AV, w.column5)[0]
    assert (st == 0).all() and np.isfinite(ref).all()
    assert np.array_equal(rate > 0, ref > 0)
    m = ref > 0
    assert (np.abs(rate - ref)[m] / ref[m]).max() < 1e-12


@pytest.mark.parametrize("nrays", [1, 3, 48, 512, 513, 768])
def test_rays(cuda, nrays):
    w = W.chemistry("C1", ncell=7, seed=111)
    pick = np.arange(nrays) % 12
    shift = (1.0 + 0.01 * (np.arange(nrays) // 12))
    w.AV = w.AV[:, pick] * shift
    w.column5 = w.column5[:, pick] * shift[:, None]
    w.rad_surface = w.rad_surface[:, pick] * 12.0 / nrays
    compare(cuda, "reduced", w)


@pytest.mark.parametrize("name", ["reduced", "full"])
@pytest.mark.parametrize("kw", [{"omega": 1.0 - 1.0e-7}, {"omega": 1.0 - 2.0e-6}, {"omega": -2.0e6}, {"v": 0.5e-10}, {"v": 1.0e16}],
                         ids=str)
def test_physics(cuda, name, kw):
    compare(cuda, name, W.chemistry("C2" if name == "full" else "C1", ncell=9, seed=112), **kw)
