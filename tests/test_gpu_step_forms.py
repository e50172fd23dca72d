"""The form of the gathered step that the size rule picks for 16-bit storage
(two cells per thread where rows fill a block, gathers elsewhere) against the
gathers, at the edges of the rule: width 228 (a partial eighth block), 226 (not
a multiple of 4), 224 (seven blocks), 256, and 8192 rows or one fewer.

Both forms do the same arithmetic on the same inputs, so populations, lagged
state and moments agree exactly; forces are grouped differently in FP32 (two
cells before the warp's sum) and are held to 1e-5 of the largest, the bound of
tests/test_gpu_rows.py.
"""
import numpy as np
import pytest

from tests.test_gpu_rows import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,storage,walls,nsp", [
    ((228, 64, 128), "f16", None, 12),
    ((228, 64, 128), "bf16", "obstacle", 12),
    ((256, 64, 128), "f16", "moving", 12),
    ((256, 127, 64), "f16", None, 12),
    ((226, 64, 128), "f16", None, 12),
    ((224, 64, 128), "bf16", None, 12),
    ((45, 33, 31), "f16", None, 3),
])
def test_chosen_form_equals_gathers(shape, storage, walls, nsp):
    f0, rho0, vel0, aux0, F0 = _run("simt", shape, storage, "reference", walls, nsp, 3)
    f1, rho1, vel1, aux1, F1 = _run("auto", shape, storage, "reference", walls, nsp, 3)
    assert np.array_equal(f0, f1)
    assert np.array_equal(rho0, rho1)
    assert np.array_equal(vel0, vel1)
    assert np.array_equal(aux0, aux1)
    assert np.abs(F0 - F1).max() <= 1e-5 * np.abs(F0).max()
