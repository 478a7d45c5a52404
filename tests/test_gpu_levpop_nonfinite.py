"""Mixed CO level populations of cells whose rate matrix FP32 cannot hold (NaN,
infinite, or beyond 3.4e38): the FP32 factors must not settle them.  Such a cell
is re-solved in FP64 (status 2, or 1 where that finds it singular) and has the FP64 form's populations, whatever
those are; its neighbours are as they are without it."""
import numpy as np
import pytest

import pdrgpu as G
from test_gpu_levpop import case, dev

pytestmark = pytest.mark.gpu


def solve(cuda, lp, dens, spop, tau, precision):
    pop, cool, _, st = G.level_populations(G.Coolant("CO"), dev(lp["n_H"], cuda), dev(lp["T"], cuda), dev(lp["Td"], cuda),
                                           dev(lp["partner5"], cuda), dev(dens, cuda), dev(spop, cuda), dev(tau, cuda),
                                           precision=precision)
    return pop.cpu().numpy(), cool.cpu().numpy(), st.cpu().numpy()


def test_cells_beyond_fp32(cuda):
    _, lp, tau, dens, spop = case("CO", 64, seed=43)
    clean = solve(cuda, lp, dens, spop, tau, "mixed")
    assert np.isin(clean[2], (0, 2)).all()
    cells = {3: "T", 8: "tau", 13: "one tau", 18: "partner", 23: "infinite partner", 28: "populations", 33: "huge partners",
             38: "one huge tau rate", 43: "Td", 48: "just beyond"}
    lp["T"][3] = np.nan
    tau[8] = np.nan
    tau[13, 0, 0] = np.nan
    lp["partner5"][18, 4] = np.nan
    lp["partner5"][23, 4] = np.inf
    spop[28] = np.nan
    lp["partner5"][33] *= 1.0e60
    spop[38, 5] = np.inf
    lp["Td"][43] = np.nan
    lp["partner5"][48] *= 1.0e44
    mixed, fp64 = solve(cuda, lp, dens, spop, tau, "mixed"), solve(cuda, lp, dens, spop, tau, "fp64")
    bad = np.array(sorted(cells))
    rest = np.setdiff1d(np.arange(64), bad)
    for a, b in zip(mixed, clean):
        assert np.array_equal(a[rest], b[rest])
    for c in bad:
        finite = np.isfinite(fp64[0][c]).all()
        same = np.array_equal(mixed[0][c], fp64[0][c], equal_nan=True)
        redone = 1 if fp64[2][c] == 1 else 2   # 1: singular in FP64 too
        assert mixed[2][c] == redone or (finite and mixed[2][c] == 0), cells[c]
        if mixed[2][c] == redone:
            assert same, cells[c]
        else:
            m = fp64[0][c] > 1e-6 * dens[c]
            assert (np.abs(mixed[0][c] - fp64[0][c])[m] / fp64[0][c][m]).max() < 1e-6, cells[c]
    assert mixed[2][3] == mixed[2][18] == mixed[2][33] == 2
