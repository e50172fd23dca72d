"""What the partner search of the one-launch DEM form assumes, at its edges,
against two launches per sub-step (which look every pair up afresh): a chunk
whose particles break an assumption is left to the two-phase form, in the same
launch, with the same contact sets and states.

States are held to the bounds of tests/test_gpu_dem_flow.py: the forms differ
in the order of FP64 force sums only.
"""
import numpy as np
import pytest

from tests.gpu_util import HertzContactConfig, make_dem

pytestmark = pytest.mark.gpu

STATE = ("position", "velocity", "force", "omega", "moment")


def _solver(L, pos, rad, vel, compat="reference", freeze=None, g=(0, 0, 0)):
    rad = np.asarray(rad, float)
    return make_dem((0, L, 0, L, 0, L), 0.05, g, HertzContactConfig(0.3, 0.3, 0.9, 0.9), rad,
                    2.0 * 4.0 / 3.0 * np.pi * rad ** 3, pos, vel, periodic=(True,) * 3, E=1e3, wall_E=1e3, max_coord=24,
                    compat=compat, freeze=freeze)


def _columns(p, q, side=4, step=4.0):
    """Copies of the pair (p, q) in the y-z plane: more than one block of particles."""
    k = step * np.stack(np.meshgrid(np.arange(side), np.arange(side), indexing="ij"), -1).reshape(-1, 2)
    off = np.concatenate([np.zeros((len(k), 1)), k], 1)
    return np.concatenate([p + off, q + off])


def _run(monkeypatch, mode, dem, nsub):
    if mode is None:
        monkeypatch.delenv("LBDEM_DEM_KERNELS", raising=False)
    else:
        monkeypatch.setenv("LBDEM_DEM_KERNELS", mode)
    dem.run_substeps(nsub)
    monkeypatch.delenv("LBDEM_DEM_KERNELS", raising=False)
    dem.check_status()


def _same(a, b):
    ca, cb = a.active_contacts(), b.active_contacts()
    assert set(ca) == set(cb)
    np.testing.assert_array_equal(a.cfn.cpu().numpy(), b.cfn.cpu().numpy())
    for q in range(3):
        x, y = np.array([ca[p][q] for p in sorted(ca)]), np.array([cb[p][q] for p in sorted(cb)])
        if len(ca):
            assert np.abs(x - y).max() <= 1e-8 * max(np.abs(y).max(), 1e-12)
    for k in STATE:
        x, y = getattr(a.gf, k).to_numpy(), getattr(b.gf, k).to_numpy()
        assert np.abs(x - y).max() <= (1e-11 if k == "position" else 1e-8 * max(np.abs(y).max(), 1e-12)), k


@pytest.mark.parametrize("compat", ["reference", "wrapped"])
@pytest.mark.parametrize("frozen", [False, True])
@pytest.mark.parametrize("pairs", [1, 16])
def test_centres_outside_a_periodic_face(compat, frozen, pairs, monkeypatch):
    """A centre outside a periodic face (an unwrapped packing, or a frozen
    particle, which is never wrapped) touches one at the opposite face."""
    pos = _columns([-0.5, 2.0, 2.0], [17.505, 2.0, 2.0], 1 if pairs == 1 else 4)
    n = len(pos)
    rng = np.random.default_rng(7)
    vel = rng.normal(0, 0.02, (n, 3))
    freeze = np.zeros(n, np.int32)
    if frozen:
        freeze[:n // 2] = 1
        vel[:n // 2] = 0.0
    a, b = (_solver(20.0, pos, np.ones(n), vel, compat, freeze) for _ in range(2))
    for nsub in (4, 17):
        _run(monkeypatch, "flow", a, nsub)
        _run(monkeypatch, "split", b, nsub)
        _same(a, b)
    if compat == "wrapped":                # (no gravity: only contacts change a velocity)
        assert np.abs(b.gf.velocity.to_numpy() - vel).max() > 0


@pytest.mark.parametrize("pairs", [1, 16])
@pytest.mark.parametrize("x", [9.6, 10.2])
def test_radius_above_the_broad_phase(x, pairs, monkeypatch):
    """A radius written above the largest one that the broad-phase cells were
    made for: the small sphere's search box (centre 9.6, cells of 4) ends short
    of the large one's cell."""
    pos = _columns([x, 2.0, 2.0], [x + 3.0, 2.0, 2.0], 1 if pairs == 1 else 4, 5.0)
    n = len(pos)
    vel = np.zeros((n, 3))
    vel[n // 2:, 0] = -0.04                # (closes the gap of 0.01 in half of the second call)
    a, b = (_solver(20.0, pos, np.ones(n), vel) for _ in range(2))
    for dem in (a, b):
        rad = np.ones(n)
        rad[n // 2:] = 1.99
        dem.gf.radius.from_numpy(rad)
    for nsub in (4, 17):
        _run(monkeypatch, "flow", a, nsub)
        _run(monkeypatch, "split", b, nsub)
        _same(a, b)


@pytest.mark.parametrize("compat", ["reference", "wrapped"])
@pytest.mark.parametrize("pairs", [1, 16])
def test_contacts_opened_by_a_write(pairs, compat, monkeypatch):
    """A touching pair is moved apart by a write, farther than the search lists
    but within the probed cells, and back: the contact ends in between, so the
    second one starts from no shear."""
    near = _columns([9.0, 2.0, 2.0], [10.995, 2.0, 2.0], 1 if pairs == 1 else 4)
    far = _columns([9.0, 2.0, 2.0], [11.2, 2.0, 2.0], 1 if pairs == 1 else 4)
    n = len(near)
    vel = np.zeros((n, 3))
    vel[n // 2:, 1] = 2e-3                 # tangential: builds up shear
    a, b = (_solver(20.0, near, np.ones(n), vel, compat) for _ in range(2))
    for where, touching in ((None, True), (far, False), (near, True)):
        for mode, dem in (("flow", a), ("split", b)):
            if where is not None:
                dem.gf.position.from_numpy(where)
                dem.gf.velocity.from_numpy(vel)
                dem.gf.omega.from_numpy(np.zeros((n, 3)))
            _run(monkeypatch, mode, dem, 5)
        assert (len(b.active_contacts()) > 0) == touching
        _same(a, b)
    # moved out of every probed cell the slot stays, as the reference's does
    away = near.copy()
    away[n // 2:, 0] = 19.5 - 3.0 if pairs == 1 else 3.0
    for mode, dem in (("flow", a), ("split", b)):
        dem.gf.position.from_numpy(away)
        _run(monkeypatch, mode, dem, 5)
    _same(a, b)


@pytest.mark.parametrize("side", [2, 6])
def test_chunks_that_keep_failing(side, monkeypatch):
    """A particle whose velocity no search covers (frozen, apart from the rest):
    chunk after chunk fails and the next ones are left to the two-phase form
    without a search, within a call and across calls; when the cause is gone
    the searches come back."""
    pos = 2.0 + 1.995 * np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos[0] = 20.0
    n = len(pos)
    rng = np.random.default_rng(4)
    vel = rng.normal(0, 0.005, (n, 3))
    vel[0] = (50.0, 0.0, 0.0)
    freeze = np.zeros(n, np.int32)
    freeze[0] = 1
    a, b = (_solver(24.0, pos, np.ones(n), vel, freeze=freeze) for _ in range(2))
    hold = lambda: a.flow[24:32].cpu().numpy().view(np.uint32)   # chunks left, their number
    seen = []
    for nsub in (5, 3, 3, 3, 3, 100, 7):
        _run(monkeypatch, "flow", a, nsub)
        _run(monkeypatch, "split", b, nsub)
        _same(a, b)
        seen.append(tuple(hold()))
    # chunks of at most 16: fail | held | fail | held | held | held, fail, 5 of 7 held | held
    assert seen == [(1, 1), (0, 1), (3, 3), (2, 3), (1, 3), (2, 7), (1, 7)]
    for dem in (a, b):
        v = dem.gf.velocity.to_numpy()
        v[0] = 0.0
        dem.gf.velocity.from_numpy(v)
    for nsub in (4, 4, 4):
        _run(monkeypatch, "flow", a, nsub)
        _run(monkeypatch, "split", b, nsub)
        _same(a, b)
    assert tuple(hold()) == (0, 0)
    assert not a.flow[:8].any() and not a.sync.any()
