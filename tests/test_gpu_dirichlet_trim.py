"""Dirichlet walls and trimmed coarse boxes together: every precision runs (and reports)
the reference's hierarchy there, trimmed, with the same results as untrimmed."""
import numpy as np
import pytest

from test_gpu_trim import _case
from uaamg_b200.solver import Handle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "fp32", "mixed"])
def test_dirichlet_hierarchy_is_trimmed(prec, monkeypatch):
    solid, r, h = _case()
    out = []
    for trim in (True, False):
        if not trim:
            monkeypatch.setenv("UAAMG_NO_TRIM", "1")
        hd = Handle(0)
        try:
            hd.set_dirichlet_walls(True)
            hd.set_problem(solid, h, h, h)
            z = hd.precond_apply(r, prec)
            p = np.zeros_like(r)
            st = hd.solve(r, p, hd.options(prec, 1e-6, 300, "rel"), strict=True)
            out.append((hd.level_trim(1, prec), z, p, st.iterations))
        finally:
            hd.close()
    (boxes, trimmed), (_, none) = out[0][0], out[1][0]
    # no box whose tile and ring touch a wall or a sphere: at most the inner 4^3 of 6^3
    assert boxes == 6 ** 3 and 0 < trimmed <= 4 ** 3 and none == 0
    assert np.array_equal(out[0][1], out[1][1])
    assert np.array_equal(out[0][2], out[1][2])
    assert out[0][3] == out[1][3]
