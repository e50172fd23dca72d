"""The CUDA adjoint over the lattice sizes at which its threads take one, two or
four cells along z, with remainders, against the FP64 oracle; tolerances of
tests/test_adjoint.py."""
import numpy as np
import pytest

from oracle.oracle import frozen_bed_drag
from tests.test_adjoint import OMEGA, _bed, _channel, _gpu_problem

pytestmark = pytest.mark.gpu


# (Nx, Ny, Nz): 8 x 23 blocks (one cell), 8 x 61 (two), 2 x 8195 (four)
@pytest.mark.parametrize("shape,n,steps", [((40, 32, 23), 5, 20), ((40, 32, 61), 6, 20), ((12, 12, 8195), 40, 8)])
def test_cells_along_z(shape, n, steps):
    pos, rad = _bed(8, shape, n, 5.0, 6.0)
    F = np.array([2e-6, 1e-6, 0.0])
    Lo, gFo, gPo = frozen_bed_drag(shape, OMEGA, _channel(*shape), rad, pos, F, steps, grad=True)
    prob = _gpu_problem(*shape, pos, rad, F, steps, every=6)
    L = prob.forward()
    gF, gP = prob.backward()
    assert abs(L - Lo) <= 2e-5 * abs(Lo)
    assert np.abs(gF - gFo)[:2].max() <= 1e-4 * np.abs(gFo).max()
    assert np.abs(gP - gPo).max() <= 1e-4 * np.abs(gPo).max()
