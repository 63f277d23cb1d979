"""The V-cycle that the FP32 and mixed solves run, cell by cell against its FP64 restatement
(oracle/cover.py): a solve of one iteration from p = 0 returns alpha (M b - mean), so the
whole cycle shows -- the finest level by quads, boxes or (2D) one tile, the coarse marches,
the dense tail, odd sizes, and in every kernel mode the transfers it uses.

Tolerance: an FP32 cell update rounds about ten times (3e-7 of the values it adds up), and
a cycle is at most eight levels of four such passes: 1e-5 of the largest value, 3e-5 with
the mean, alpha and the reciprocals.  A weight 1/5 taken as 0.21, or one face's coupling
bit missing, is 1e-3 and more (test_oracle_cover.py)."""
import numpy as np
import pytest

from cover import CoverHierarchy
from test_gpu_parity import connected, fluid_interior

pytestmark = pytest.mark.gpu

# 70 x 66 x 67: the finest level marches (more than 64^3 cells), the next are boxes;
# 130 x 129 x 131: level 1 marches too; the smaller 3D ones are boxes from the finest on;
# tiles are 32 x 16 and 8^3, the tail takes over at 1024 cells
SHAPES = [(5, 3), (33, 17), (100, 37), (129, 31), (777, 333), (9, 7, 5), (33, 17, 9), (40, 64, 24),
          (70, 66, 67), (130, 129, 131)]


def _case(shape, seed):
    rng = np.random.default_rng(seed)
    padded = tuple(n + 2 for n in shape[::-1])
    solid = (rng.random(padded) < (0.1, 0.25)[seed % 2]).astype(np.uint8)
    if shape[0] > 16:  # a plate one cell thick, open at one end
        solid[..., 1 + shape[1] // 4:, 1 + shape[0] // 3] = 1
    solid = connected(solid)
    fl = fluid_interior(solid)
    x = sum(np.cos(2.0 * ix / n) for ix, n in zip(np.indices(padded), padded))
    rhs = np.where(fl, rng.standard_normal(padded) + 0.3 * x, 0.0)
    rhs[fl] -= rhs[fl].mean()
    return solid, rhs, tuple(rng.uniform(0.7, 1.4, 3))


def _check(handle, H, rhs, precision, **kw):
    p = np.zeros_like(rhs)
    st = handle.solve(rhs, p, handle.options(precision, 0.0, 1, "rel"))
    assert st.iterations == 1
    want = H.first_iterate(rhs, **kw)
    assert np.abs(p - want).max() <= 3e-5 * np.abs(want).max()


@pytest.mark.parametrize("precision", ["mixed", "fp32"])
@pytest.mark.parametrize("shape", SHAPES)
def test_solve_cycle_is_the_restated_one(handle, shape, precision):
    solid, rhs, sp = _case(shape, SHAPES.index(shape))
    handle.set_problem(solid, *sp)
    _check(handle, CoverHierarchy(solid, *sp), rhs, precision)


@pytest.mark.parametrize("mode", [1, 2, 3, 4])
@pytest.mark.parametrize("shape", [(129, 31), (33, 17, 9), (70, 66, 67)])
def test_kernel_modes(handle, shape, mode):
    """Mode 2 has the star transfers on every level, 3 in the tail only, 1 and 4 nowhere."""
    solid, rhs, sp = _case(shape, 3)
    H = CoverHierarchy(solid, *sp)
    star = [mode == 2 or (mode == 3 and l >= H.tail_level()) for l in range(len(H.levels))]
    handle.set_problem(solid, *sp)
    handle.set_vcycle_kernels(mode)
    try:
        _check(handle, H, rhs, "mixed", star=star)
    finally:
        handle.set_vcycle_kernels(0)


@pytest.mark.parametrize("nu", [(1, 2), (2, 1), (2, 2)])
@pytest.mark.parametrize("shape", [(129, 31), (70, 66, 67)])
def test_smoothing_schedules(handle, shape, nu):
    """A level with more than one sweep has constant transfers to the next; the tail keeps
    one sweep and star transfers."""
    solid, rhs, sp = _case(shape, 2)
    H = CoverHierarchy(solid, *sp)
    tail = H.tail_level()
    star = [l >= tail or (nu[0] if l == 0 else nu[1]) == 1 for l in range(len(H.levels))]
    handle.set_problem(solid, *sp)
    handle.set_smoothing(*nu)
    try:
        _check(handle, H, rhs, "mixed", star=star, nu=nu, tail=tail)
    finally:
        handle.set_smoothing(1, 1)
