"""Covering aggregates of the FP32 and mixed solves: odd sizes (the last aggregate has
one child along an axis, the last z chunk ends on the ghost plane), solids that leave
coarse cells with few fluid children, thin plates, and every V-cycle implementation
against the FP64 solution.  V-cycles applied by themselves keep the reference's
hierarchy (tests/test_gpu_parity.py)."""
import numpy as np
import pytest

import oracle as O
from test_gpu_parity import connected, fluid_interior, rel_l2_meanfree

pytestmark = pytest.mark.gpu

# tile edges are 32 x 16 (marches), 8^3 (boxes) and chunks of 2 or more planes
SHAPES = [(2, 2), (5, 3), (33, 17), (63, 49), (129, 31), (3, 2, 2), (9, 7, 5), (33, 17, 9),
          (17, 33, 31), (65, 67, 69), (131, 65, 67)]


def _case(shape, seed):
    rng = np.random.default_rng(seed)
    padded = tuple(n + 2 for n in shape[::-1])
    solid = (rng.random(padded) < (0.0, 0.1, 0.2)[seed % 3]).astype(np.uint8)
    if seed % 2 and shape[0] > 16:  # a plate one cell thick, open at one end
        solid[..., 1 + shape[1] // 4:, 1 + shape[0] // 3] = 1
    solid = connected(solid)
    fl = fluid_interior(solid)
    b = np.zeros(padded)
    b[fl] = rng.standard_normal(int(fl.sum()))
    if fl.any():
        b[fl] -= b[fl].mean()
    return solid, b, tuple(rng.uniform(0.7, 1.4, 3))


@pytest.mark.parametrize("mode", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("shape", SHAPES)
def test_covering_solves_match_fp64(handle, shape, mode):
    seed = SHAPES.index(shape)
    solid, b, sp = _case(shape, seed)
    handle.set_problem(solid, *sp)
    handle.set_vcycle_kernels(mode)
    try:
        p64 = np.zeros_like(b)
        handle.solve(b, p64, handle.options("fp64", 1e-11, 800, "rel"))
        p = np.zeros_like(b)
        st = handle.solve(b, p, handle.options("mixed", 1e-6, 200, "rel"))
        assert st.status == 0, st.iterations
        res, bn = O.true_residual(solid, b, p, *sp)
        assert res <= 1e-6 * bn
        # noise right-hand side: the error is within a few times the residual's 1e-6
        # times the grid's condition (at most about 1e4 here)
        assert rel_l2_meanfree(p, p64, solid) <= 1e-5 if np.any(p64) else np.all(p == 0)
        p32 = np.zeros_like(b)
        s32 = handle.solve(b, p32, handle.options("fp32", 1e-5, 200, "rel"))
        assert s32.status == 0
    finally:
        handle.set_vcycle_kernels(0)


def test_few_iterations_next_to_solids_and_on_odd_sizes(handle):
    """The point of the covering aggregates: as many iterations as a box without solids
    needs (about 10; the reference's aggregates need 50 to 200 here)."""
    from uaamg_b200 import workloads
    solid, rhs = workloads.spheres_3d(65, 65, 65, nspheres=5, rmin=3, rmax=9, seed=3)
    handle.set_problem(solid, *(1 / 65,) * 3)
    p = np.zeros_like(rhs)
    st = handle.solve(rhs, p, handle.options("mixed", 1e-6, 200, "rel"), strict=True)
    assert st.iterations <= 20
    st64 = handle.solve(rhs, np.zeros_like(rhs), handle.options("fp64", 1e-6, 200, "rel"), strict=True)
    assert st64.iterations > st.iterations


def test_inconsistent_chambers_fall_back(handle):
    """Two chambers with a net source each: no solution exists, the covering aggregates
    join the chambers on coarse levels, CG's residual grows and the solve is repeated on
    the reference's hierarchy.  It ends unconverged and finite, alone and in a batch the
    same, and a consistent right-hand side on the same mask converges before and after."""
    n, m = 90, 70
    solid = np.zeros((m + 2, n + 2), np.uint8)
    solid[:, 45] = 1
    rng = np.random.default_rng(3)
    b = np.zeros(solid.shape)
    fl = fluid_interior(solid)
    b[fl] = rng.standard_normal(int(fl.sum()))
    b[fl] -= b[fl].mean()
    c = b.copy()
    for sl in (slice(1, 45), slice(46, n + 1)):
        c[1:-1, sl] -= c[1:-1, sl].mean()
    opts = handle.options("mixed", 1e-6, 100, "rel")
    handle.set_problem(solid, 1.0, 1.0)
    pc = [np.zeros_like(b) for _ in range(2)]
    assert handle.solve(c, pc[0], opts).status == 0
    p, q = np.zeros_like(b), np.zeros_like(b)
    st = handle.solve(b, p, opts)
    assert st.status == 1 and st.iterations == 100 and np.isfinite(p).all()
    sb = handle.solve_batch([(solid, b, q, 1.0, 1.0, 1.0)], opts)[0]
    assert sb.status == 1 and sb.iterations == 100 and np.array_equal(p, q)
    assert handle.solve(c, pc[1], opts).status == 0 and np.array_equal(*pc)


@pytest.mark.parametrize("members", [2, 5])
def test_inconsistent_member_of_a_group_falls_back(handle, members):
    """In a grouped batch (one graph a step) the inconsistent member, repeated by itself
    after the group, ends as the same problem solved alone; the others converge."""
    n, m = 90, 70
    solid = np.zeros((m + 2, n + 2), np.uint8)
    solid[:, 45] = 1
    fl = fluid_interior(solid)
    rng = np.random.default_rng(4)
    b = np.zeros(solid.shape)
    b[fl] = rng.standard_normal(int(fl.sum()))
    c = b.copy()
    b[fl] -= b[fl].mean()
    for sl in (slice(1, 45), slice(46, n + 1)):
        c[1:-1, sl] -= c[1:-1, sl].mean()
    opts = handle.options("mixed", 1e-6, 60, "rel")
    handle.set_problem(solid, 1.0, 1.0)
    alone = np.zeros_like(b)
    ref = handle.solve(b, alone, opts)
    ps = [np.zeros_like(b) for _ in range(members)]
    handle.set_batch_group(1 << 20)
    try:
        st = handle.solve_batch([(solid, b if k == 1 else c, ps[k], 1.0, 1.0, 1.0) for k in range(members)], opts)
    finally:
        handle.set_batch_group(0)
    assert st[1].status == ref.status == 1 and st[1].iterations == ref.iterations
    assert np.array_equal(ps[1], alone)
    assert all(st[k].status == 0 for k in range(members) if k != 1)
