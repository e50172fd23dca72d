"""FP64 divisions and roots of the DEM, rounded as IEEE division and square
root round them, and their special values -- through what the solver shows of
them, against NumPy."""
import numpy as np
import pytest

from tests.gpu_util import HertzContactConfig, LinearContactConfig, make_dem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", ["hertz", "linear"])
@pytest.mark.parametrize("mode", ["flow", "split"])
@pytest.mark.parametrize("first", [True, False])
def test_frozen_sphere_of_infinite_mass(model, mode, first, monkeypatch):
    """An immovable sphere given an infinite mass: the effective mass of a
    contact with it, 1 / (1/m_i + 1/m_j), is the other sphere's mass."""
    monkeypatch.setenv("LBDEM_DEM_KERNELS", mode)
    contact = (HertzContactConfig(0.3, 0.3, 0.9, 0.9) if model == "hertz" else
               LinearContactConfig(stiffness_normal=50.0, stiffness_tangential=30.0, damping_normal=0.2,
                                   damping_tangential=0.1, pp_friction=0.3, pw_friction=0.3))
    out = []
    for heavy in (np.inf, 1e250):
        mass = np.array([heavy, 8.0] if first else [8.0, heavy])
        pos = np.array([[5.0, 5.0, 5.0], [6.99, 5.0, 5.0]])
        vel = np.array([[0.0, 0.0, 0.0], [-0.01, 0.02, 0.0]]) * (1 if first else -1)
        if not first:
            vel = vel[::-1].copy()
        dem = make_dem((0, 20, 0, 20, 0, 20), 0.05, (0, 0, 0), contact, np.ones(2), mass, pos, vel, E=1e3, wall_E=1e3,
                       model=model, freeze=np.array([1, 0] if first else [0, 1]))
        dem.run_substeps(9)
        dem.check_status()
        free = 1 if first else 0
        out.append(np.concatenate([getattr(dem.gf, k).to_numpy()[free] for k in ("position", "velocity", "force", "omega")]))
    assert np.isfinite(out[0]).all() and np.abs(out[0][6:9]).max() > 0
    np.testing.assert_allclose(out[0], out[1], rtol=1e-14, atol=0)
