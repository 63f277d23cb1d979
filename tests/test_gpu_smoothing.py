"""V(nu, nu) cycles are symmetric: what uaamg_set_smoothing promises, on the reference's
hierarchy (precond_apply; FP64 to rounding)."""
import numpy as np
import pytest

from test_gpu_parity import connected, fluid_interior

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-12), ("mixed", 1e-4)])
@pytest.mark.parametrize("nu", [(1, 1), (1, 2), (2, 1), (3, 2)])
@pytest.mark.parametrize("shape", [(120, 70), (70, 66, 67), (40, 33, 20)])
def test_cycle_is_symmetric(handle, shape, nu, prec, tol):
    rng = np.random.default_rng(7)
    padded = tuple(n + 2 for n in shape[::-1])
    solid = connected((rng.random(padded) < 0.1).astype(np.uint8))
    fl = fluid_interior(solid)
    a, b = (np.where(fl, rng.standard_normal(padded), 0.0) for _ in range(2))
    handle.set_problem(solid, 1.0, 1.2, 0.9)
    handle.set_smoothing(*nu)
    try:
        za, zb = handle.precond_apply(a, prec), handle.precond_apply(b, prec)
    finally:
        handle.set_smoothing(1, 1)
    scale = np.sqrt((za * a).sum() * (zb * b).sum())
    assert abs((za * b).sum() - (zb * a).sum()) <= tol * scale
