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


@pytest.mark.parametrize("mode,nsub", [("flow", 3), ("split", 1)])
def test_quotients_round_as_division(mode, nsub, monkeypatch):
    """acceleration = force / mass bit for bit; quaternion = q / |q| to 3.5 units
    of 2^-53: three roundings in the sum of squares, halved by the root, one of
    the reciprocal root and one of the product (a root and a division of a sum
    added term by term: 4)."""
    monkeypatch.setenv("LBDEM_DEM_KERNELS", mode)
    rng = np.random.default_rng(11)
    side = 12
    pos = 3.0 + 6.0 * np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    n, L = len(pos), 6.0 * side
    mass = 10.0 ** rng.uniform(-6, 6, n)
    dem = make_dem((0, L, 0, L, 0, L), 1e-6, (0, 0, 0), HertzContactConfig(0.3, 0.3, 0.9, 0.9), np.ones(n), mass, pos,
                   np.zeros((n, 3)))
    force = rng.normal(0, 1, (n, 3)) * 1e-4 * mass[:, None]
    dem.gf.force_fluid.from_numpy(force)
    q = rng.normal(0, 1, (n, 4)) * 10.0 ** rng.uniform(-3, 3, (n, 1))
    dem.gf.quaternion.from_numpy(q)
    dem.run_substeps(nsub)
    dem.check_status()
    np.testing.assert_array_equal(dem.gf.acceleration.to_numpy(), force / mass[:, None])
    got = dem.gf.quaternion.to_numpy()
    e = q.astype(np.longdouble)
    e /= np.sqrt((e * e).sum(1, keepdims=True))
    assert np.abs((got.astype(np.longdouble) - e) / e).max() <= 3.5 * nsub * 2.0 ** -53


@pytest.mark.parametrize("mode", ["flow", "split"])
def test_contact_geometry_rounds_as_division(mode, monkeypatch):
    """Contact point p_i + n (r_i - overlap) with n = d / |d|, bit for bit, on
    pairs in random directions (the last sub-step's, so one)."""
    monkeypatch.setenv("LBDEM_DEM_KERNELS", mode)
    rng = np.random.default_rng(12)
    side = 10
    p = 4.0 + 8.0 * np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    d = rng.normal(0, 1, p.shape)
    d *= (1.0 / np.linalg.norm(d, axis=1) * rng.uniform(1.8, 1.99, len(p)))[:, None]
    pos, n, L = np.concatenate([p, p + d]), len(p), 8.0 * side
    dem = make_dem((0, L, 0, L, 0, L), 1e-6, (0, 0, 0), HertzContactConfig(0.3, 0.3, 0.9, 0.9), np.ones(2 * n),
                   np.full(2 * n, 8.0), pos, np.zeros((2 * n, 3)), E=1e3)
    dem.run_substeps(1)
    dem.check_status()
    dv = (p + d) - p
    dist = np.sqrt((dv[:, 0] * dv[:, 0] + dv[:, 1] * dv[:, 1]) + dv[:, 2] * dv[:, 2])
    overlap = -(dist - 1.0 - 1.0)
    cp = p + dv / dist[:, None] * (1.0 - overlap)[:, None]
    con = dem.active_contacts()
    assert len(con) == n
    np.testing.assert_array_equal(np.array([con[(i, i + n)][0] for i in range(n)]), cp)
