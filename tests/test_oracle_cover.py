"""The restated preconditioner of the FP32 and mixed solves (oracle/cover.py): symmetric,
its transfers each other's transpose, and sensitive to a mistake in them."""
import numpy as np
import pytest

import cover
from cover import CoverHierarchy


@pytest.mark.parametrize("shape", [(34, 21), (11, 14, 9)])
def test_cycle_is_symmetric_and_transfers_are_transposes(shape):
    rng = np.random.default_rng(0)
    solid = (rng.random(tuple(n + 2 for n in shape[::-1])) < 0.2).astype(np.uint8)
    H = CoverHierarchy(solid, 1.0, 1.2, 0.8)
    noise = lambda l: np.where(H.levels[l].fluid, rng.standard_normal(H.levels[l].fluid.shape), 0.0)
    for star in (True, False):
        for l in range(len(H.levels) - 1):
            r, xc = noise(l), noise(l + 1)
            assert np.isclose(2 * (H.restrict(l, r, star) * xc).sum(), (r * H.prolong(l, xc, star)).sum(),
                              rtol=1e-12, atol=1e-9)
        a, b = noise(0), noise(0)
        assert np.isclose((a * H.vcycle(b, star)).sum(), (b * H.vcycle(a, star)).sum(), rtol=1e-10)


def test_a_mistake_in_the_transfers_shows(monkeypatch):
    """What the cell-by-cell tolerance of 3e-5 has to see: another weight, one coupling gone."""
    rng = np.random.default_rng(1)
    solid = (rng.random((35, 68)) < 0.2).astype(np.uint8)
    rhs = rng.standard_normal(solid.shape)
    H = CoverHierarchy(solid, 1.0, 1.0)
    want = H.first_iterate(rhs)
    monkeypatch.setattr(cover, "W", 0.21)
    assert np.abs(H.first_iterate(rhs) - want).max() > 1e-3 * np.abs(want).max()
    monkeypatch.undo()
    c = H.levels[1].c[1]
    at = np.argwhere(c > 0)[7]
    keep, H.levels[1].c[1] = c.copy(), c.copy()
    H.levels[1].c[1][tuple(at)] = 0.0  # transfers (and the level's own operator) lose it
    assert np.abs(H.first_iterate(rhs) - want).max() > 1e-3 * np.abs(want).max()
    H.levels[1].c[1] = keep
