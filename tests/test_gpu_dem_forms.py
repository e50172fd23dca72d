"""The one-launch DEM form at the particle counts where it changes its lanes per
particle and blocks per SM (8 lanes up to 4736 particles, 4 to 9472 and, at
three blocks, to 14,208, 2 to 28,416) against two launches per sub-step, with
contacts among particles, with walls and across periodic faces.  Bounds as in
tests/test_gpu_dem_flow.py.
"""
import numpy as np
import pytest

from tests.gpu_util import HertzContactConfig, make_dem
from tests.test_gpu_dem_search import _run, _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("images", [False, True])
@pytest.mark.parametrize("side", [(17, 17, 17), (19, 18, 18), (23, 23, 23), (26, 25, 25)])
def test_bed(side, images, monkeypatch):
    from lbdem_taichi_b200 import _native as N
    spacing = 1.997                                     # every sphere overlaps six others
    side_len = spacing * np.array(side, float)
    rng = np.random.default_rng(6)
    pos = spacing * (0.5 + np.stack(np.meshgrid(*[np.arange(s) for s in side], indexing="ij"), -1).reshape(-1, 3))
    pos = np.clip(pos + rng.uniform(-1e-3, 1e-3, pos.shape), 1e-9, side_len - 1e-9)
    n = len(pos)
    vel = rng.normal(0, 0.01, (n, 3))
    a, b = (make_dem((0, side_len[0], 0, side_len[1], 0, side_len[2]), 0.02, (0, 0, -1e-3),
                     HertzContactConfig(0.3, 0.3, 0.9, 0.9), np.ones(n), np.full(n, 8.0), pos, vel,
                     periodic=(images, images, False), E=1e3, wall_E=1e3, max_coord=12,
                     compat="wrapped" if images else "reference") for _ in range(2))
    for nsub in (10, 3):
        _run(monkeypatch, None, a, nsub)
        assert N.load().lbdem_dem_launches_last() == 1
        _run(monkeypatch, "split", b, nsub)
        assert N.load().lbdem_dem_launches_last() == 2 * nsub
        _same(a, b)
    assert len(b.active_contacts()) > n
    np.testing.assert_array_equal(a.wcf_active.cpu().numpy(), b.wcf_active.cpu().numpy())
    assert b.wcf_active.any()
    assert not a.flow[24:32].any()                      # no chunk failed


@pytest.mark.parametrize("images", [False, True])
@pytest.mark.parametrize("n", [1, 2, 3, 8, 9, 16, 17])
@pytest.mark.parametrize("nsub", [1, 2, 3, 4])
def test_short_calls_of_few_particles(n, nsub, images, monkeypatch):
    """The default form of short calls, on either side of where one block's
    two-phase form gives way: 2 sub-steps of one or two particles or with
    periodic images, 3 up to 8 particles, 4 above; more than one block, 3."""
    rng = np.random.default_rng(n)
    pos = 2.0 + 1.995 * np.stack(np.meshgrid(*[np.arange(3)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    vel = rng.normal(0, 0.01, (n, 3))
    a, b = (make_dem((0, 24, 0, 24, 0, 24), 0.02, (0, 0, -1e-3), HertzContactConfig(0.3, 0.3, 0.9, 0.9), np.ones(n),
                     np.full(n, 8.0), pos, vel, periodic=(True, True, False), E=1e3, wall_E=1e3,
                     compat="wrapped" if images else "reference") for _ in range(2))
    for _ in range(3):
        _run(monkeypatch, None, a, nsub)
        _run(monkeypatch, "split", b, nsub)
    _same(a, b)
    flow = nsub >= (3 if n > 16 else 2 if images or n <= 2 else 3 if n <= 8 else 4)
    assert (a.flow[16:24].cpu().numpy().view(np.uint64)[0] > 0) == flow   # the one-launch form counts its chunks
