"""The one-launch DEM form's workspace: held where that form can run, not
elsewhere, with the same results."""
import numpy as np
import pytest

from tests.gpu_util import HertzContactConfig, make_dem

pytestmark = pytest.mark.gpu


def _spheres(side, box, periodic, radius=1.0):
    pos = 2.0 + 4.0 * np.stack(np.meshgrid(*[np.arange(s) for s in side], indexing="ij"), -1).reshape(-1, 3)
    n = len(pos)
    return make_dem((0, box[0], 0, box[1], 0, box[2]), 0.05, (0, 0, -1e-3), HertzContactConfig(0.3, 0.3, 0.9, 0.9),
                    np.full(n, radius), np.full(n, 8.0), pos, np.zeros((n, 3)), periodic=periodic)


@pytest.mark.parametrize("side,box,periodic,held", [
    ((4, 4, 4), (16, 16, 16), (True, True, False), True),
    ((4, 4, 1), (16, 16, 9), (False, False, True), False),      # periodic axis below 2.5 broad-phase cells
    ((60, 50, 20), (240, 200, 80), (True, True, False), False),   # 60,000: more than one resident wave
])
def test_workspace_only_where_the_form_can_run(side, box, periodic, held):
    dem = _spheres(side, box, periodic)
    assert (dem.flow is not None) == held
    z = dem.gf.position.to_numpy()[:, 2]
    dem.run_substeps(5)
    dem.check_status()
    # free fall: velocity Verlet of a constant acceleration whose first half step has none
    v = dem.gf.velocity.to_numpy()[:, 2]
    np.testing.assert_allclose(v, -1e-3 * 0.05 * 4.5, rtol=1e-12)
    assert (dem.gf.position.to_numpy()[:, 2] < z).all()
