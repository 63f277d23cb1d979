"""The FP64 form's coarsest-level division (a corrected product with the reciprocal, and the
division itself outside its range) and its tile-wise z sums: V-cycles bit-exact against the
oracle at scales where either branch runs, and solves on march levels as with the
step-by-step V-cycle."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-300, 1e-249, 1e-12, 1.0, 3e200, 1e248])
@pytest.mark.parametrize("shape", [(11, 13), (35, 19), (10, 12, 9), (18, 19, 21)])
def test_tail_division_is_exact(handle, shape, scale):
    rng = np.random.default_rng(len(shape) * 7 + shape[0])
    solid = (rng.random(shape) < 0.15).astype(np.uint8)
    r = rng.standard_normal(shape) * scale
    sp = (0.7, 1.3, 0.9)
    handle.set_problem(solid, *sp)
    z = handle.precond_apply(r, "fp64")
    zr = O.Hierarchy(solid, *sp).vcycle(r)
    sl = tuple(slice(1, -1) for _ in shape)
    assert np.array_equal(z[sl], zr[sl])


@pytest.mark.parametrize("dims", [(66, 65, 67), (33, 130, 66)])
def test_tile_sums_match_the_separate_pass(handle, dims):
    from uaamg_b200 import workloads
    solid, rhs = workloads.spheres_3d(*dims, nspheres=4, rmin=4, rmax=9, seed=5)
    h = 1.0 / max(dims)
    handle.set_problem(solid, h, h, h)
    out = []
    for mode in (0, 1):  # marches with the tile sums; sweeps with the flat ones
        handle.set_vcycle_kernels(mode)
        p = np.zeros_like(rhs)
        st = handle.solve(rhs, p, handle.options("fp64", 1e-11, 400, "rel"), strict=True)
        out.append((p, st.iterations))
    handle.set_vcycle_kernels(0)
    assert abs(out[0][1] - out[1][1]) <= 1
    # both to 1e-11 of ||b||: the solutions agree to that times the grid's condition
    assert np.abs(out[0][0] - out[1][0]).max() <= 1e-7 * np.abs(out[1][0]).max()
