"""FP64 solves keep their bits: the dot products' partition (blocks of a march) does not
follow the chunk lengths of the V-cycle's marches, in any kernel mode and with Dirichlet
walls.  Digests of the pressure from the build before those lengths became a rule."""
import hashlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (shape, Dirichlet walls, kernel mode): iterations and SHA-256 of the pressure
DIGESTS = {
    ((70, 66, 67), 0, 0): "87:3d8b51e149976ebc",
    ((70, 66, 67), 0, 3): "87:a3a3ff46ed9948c6",
    ((70, 66, 67), 0, 4): "87:a3a3ff46ed9948c6",
    ((70, 66, 67), 1, 0): "35:970503b426b3a0d3",
    ((70, 66, 67), 1, 3): "35:970503b426b3a0d3",
    ((96, 96, 96), 0, 0): "34:d6940c1f019bc7fa",
    ((96, 96, 96), 0, 3): "34:7eaa03159cbe8553",
    ((96, 96, 96), 0, 4): "34:7eaa03159cbe8553",
    ((96, 96, 96), 1, 0): "35:1846d1520b7b0737",
    ((96, 96, 96), 1, 3): "35:1846d1520b7b0737",
    ((129, 64, 65), 0, 0): "98:9df47d37f01256d5",
    ((129, 64, 65), 0, 3): "98:c691f3cc2bc2ce8f",
    ((129, 64, 65), 0, 4): "98:c691f3cc2bc2ce8f",
    ((129, 64, 65), 1, 0): "37:b4a3631f8896af40",
    ((129, 64, 65), 1, 3): "37:b4a3631f8896af40",
}

# (shape, variable operator), 60 iterations
DIGESTS_2D = {
    ((512, 512), False): "60:7462cc25f0",
    ((512, 512), True): "60:1e0e846812",
    ((1024, 640), False): "60:e5b18fd8f0",
    ((1024, 640), True): "60:7dc67cd2fb",
    ((777, 1555), False): "60:61bb727bc4",
    ((777, 1555), True): "60:a419a1da47",
}


def _case(shape):
    k, j, i = np.indices(tuple(n + 2 for n in shape[::-1]))
    solid = np.zeros(i.shape, np.uint8)
    solid[20:25, 10:30, 12:28] = 1
    inner = np.zeros(i.shape, bool)
    inner[1:-1, 1:-1, 1:-1] = solid[1:-1, 1:-1, 1:-1] == 0
    b = np.where(inner, ((i * 7919 + j * 104729 + k * 1299709) % 1009 - 504).astype(float), 0.0)
    return solid, b


@pytest.mark.parametrize("walls,mode", [(0, 0), (0, 3), (0, 4), (1, 0), (1, 3)])
@pytest.mark.parametrize("shape", [(70, 66, 67), (96, 96, 96), (129, 64, 65)])
def test_fp64_bits(handle, shape, walls, mode):
    solid, b = _case(shape)
    handle.set_dirichlet_walls(bool(walls))
    handle.set_problem(solid, 1.0, 1.0, 1.0)
    handle.set_vcycle_kernels(mode)
    try:
        p = np.zeros_like(b)
        st = handle.solve(b, p, handle.options("fp64", 1e-9, 200, "rel"), strict=True)
    finally:
        handle.set_vcycle_kernels(0)
        handle.set_dirichlet_walls(False)
    got = f"{st.iterations}:{hashlib.sha256(p.tobytes()).hexdigest()[:16]}"
    assert got == DIGESTS[shape, walls, mode]


@pytest.mark.parametrize("layered", [False, True])
@pytest.mark.parametrize("shape", [(512, 512), (1024, 640), (777, 1555)])
def test_fp64_bits_2d(handle, shape, layered):
    """Grids whose search direction fills every SM: its partition is not left to how many
    blocks the compiler's register count lets reside."""
    j, i = np.indices((shape[1] + 2, shape[0] + 2))
    solid = np.zeros(i.shape, np.uint8)
    solid[50:90, 100:170] = 1
    inner = np.zeros(i.shape, bool)
    inner[1:-1, 1:-1] = solid[1:-1, 1:-1] == 0
    b = np.where(inner, ((i * 7919 + j * 104729) % 1009 - 504).astype(float), 0.0)
    handle.set_problem(solid, 1.0, 1.0)
    if layered:
        w = np.ones(i.shape)
        handle.set_variable_laplacian(4.2 * w, -1.0 * w, -1.1 * w)
    p = np.zeros_like(b)
    st = handle.solve(b, p, handle.options("fp64", 1e-9, 60, "rel"))
    handle.set_variable_laplacian()
    assert f"{st.iterations}:{hashlib.sha256(p.tobytes()).hexdigest()[:10]}" == DIGESTS_2D[shape, layered]
