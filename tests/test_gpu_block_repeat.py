"""The block integrator gives the same bits on a second run: a block's shared
arrays must not overlap (the 57-species network's two warps drift apart enough
to show it)."""
import numpy as np
import pytest

from test_gpu_block import gpu_run, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("network,ncell,precision", [("mynetwork", 700, "mixed"), ("mynetwork", 300, "fp64"),
                                                     ("full", 64, "mixed")])
def test_repeated_solve_bitwise(cuda, network, ncell, precision):
    w, _, rates, ab0 = inputs(network, ncell, seed=17)
    a1, st1, s1 = gpu_run(network, cuda, ab0, rates, w.n_H, precision)
    a2, st2, s2 = gpu_run(network, cuda, ab0, rates, w.n_H, precision)
    assert (st1 == 0).all() and (st2 == 0).all()
    assert (s1 == s2).all()
    assert (a1.view(np.int64) == a2.view(np.int64)).all()
