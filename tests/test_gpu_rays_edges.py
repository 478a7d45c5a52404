"""The ray kernels at their edges, bit for bit against the oracle: rays longer
than a chunk of eight points, rays without points, populations that are zero or
so small that the reciprocal's residual step would underflow, and a bad grid
index on one ray of a block."""
import numpy as np
import pytest

import oracle as O
import pdrgpu as G
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("key", ["CII", "CI", "CO"])
@pytest.mark.parametrize("n,points,step", [(3, 1, 0.05), (4, 8, 0.02), (5, 29, 0.01)])
def test_optical_depths(cuda, key, n, points, step):
    import torch
    r = W.rays(n, points, step_pc=step)
    oc = O.Coolant(key)
    rng = np.random.Generator(np.random.PCG64(78))
    dens = r["rho"] * W.COOLANT_X[key]
    T = rng.uniform(10.0, 300.0, r["ngrid"])
    pop = np.array([oc.lte(t, d) for t, d in zip(T, dens)]) * rng.uniform(0.5, 1.5, (r["ngrid"], oc.nlev))
    pop[0] = 0.0
    pop[1] *= 1.0e-290
    pop[2, 1:] = 0.0
    ref = oc.optical_depths(r, pop, T[:r["ncell"]], 1.0e5)
    rays, keep = G.device_rays(r, cuda)
    t = lambda a: torch.as_tensor(a, device=cuda)  # noqa: E731
    out = G.optical_depths(G.Coolant(key), rays, t(pop), t(T[:r["ncell"]]), 1.0e5).cpu().numpy()
    assert np.array_equal(out, ref)
    # one bad index: NaN on that ray's lines, every other ray unchanged
    bad = int(np.argmax(r["epray"]))
    gp = keep["gridpoint"]
    gp[int(r["offset"][bad]) + int(r["epray"][bad])] = r["ngrid"]
    out = G.optical_depths(G.Coolant(key), rays, t(pop), t(T[:r["ncell"]]), 1.0e5).cpu().numpy()
    c, j = bad // 12, bad % 12
    assert np.isnan(out[c, :, j]).all()
    mask = np.ones(ref.shape, bool)
    mask[c, :, j] = False
    assert np.array_equal(out[mask], ref[mask])


@pytest.mark.parametrize("n,points", [(3, 1), (5, 20)])
def test_uvfield_and_columns(cuda, n, points):
    import torch
    r = W.rays(n, points, step_pc=0.02, nspec=9)
    gvec = (10.0, 0.0, 0.0)
    col, av, rad, uv = O.uvfield(r, field=0, G=gvec, metallicity=1.0)
    rays, keep = G.device_rays(r, cuda)
    rho, ab = torch.as_tensor(r["rho"], device=cuda), torch.as_tensor(r["abundance"], device=cuda)
    gcol, gav, grad, guv = G.uvfield(rays, rho, 0, gvec, r["vectors"])
    assert np.array_equal(gcol.cpu().numpy(), col) and np.array_equal(gav.cpu().numpy(), av)
    assert np.array_equal(grad.cpu().numpy(), rad)
    assert np.allclose(guv.cpu().numpy(), uv, rtol=1e-14, atol=0)
    assert np.array_equal(G.column_densities(rays, rho, ab, [0, 8]).cpu().numpy(), O.columns(r, [0, 8]))


def test_more_rays_than_a_block(cuda):
    """300 rays per cell: the field in rounds of a block's threads."""
    import torch
    n, nr = 3, 300
    rng = np.random.Generator(np.random.PCG64(79))
    offset = np.arange(n * nr, dtype=np.int64) * 3
    gp = rng.integers(0, n, n * nr * 3).astype(np.int32)
    xyz = rng.uniform(0.0, 1.0, (n * nr * 3, 3))
    epray = rng.integers(0, 3, n * nr).astype(np.int32)
    r = dict(ncell=n, nrays=nr, ngrid=n, npoint=len(gp), epray=epray, offset=offset, xyz=xyz, gridpoint=gp)
    rho = 10.0 ** rng.uniform(2.0, 3.0, n)
    rays, keep = G.device_rays(r, cuda)
    got = [g.cpu().numpy() for g in G.uvfield(rays, torch.as_tensor(rho, device=cuda), 0, (10.0, 0.0, 0.0), np.zeros((nr, 3)))]
    col = np.zeros((n, nr))
    for c in range(n):
        for j in range(nr):
            p = int(offset[c * nr + j])
            for i in range(1, int(epray[c * nr + j]) + 1):
                d = xyz[p + i - 1] - xyz[p + i]
                step = np.sqrt((d[0] * d[0] + d[1] * d[1]) + d[2] * d[2])
                col[c, j] += ((rho[gp[p + i - 1]] + rho[gp[p + i]]) * 0.5 * step) * 3.08568025e+18
    assert np.array_equal(got[0], col)
    av = col * float(np.float32(6.289e-22))
    uv = np.zeros(n)
    for j in range(nr):
        uv += (10.0 / nr) * np.exp(-av[:, j] * float(np.float32(3.02)))
        uv[uv < 1e-50] = 0.0
    assert np.allclose(got[3], uv, rtol=1e-13, atol=0)
