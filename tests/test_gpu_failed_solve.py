"""A solve that fails on the host leaves no residual history behind."""
import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def memory_taken(piece):
    """The device's memory, taken until no allocation of `piece` bytes is left (blocks that
    the driver keeps for this process included)."""
    from cuda.bindings import runtime as rt
    ok, held, size = rt.cudaError_t.cudaSuccess, [], 1 << 36
    try:
        while size >= piece:
            err, p = rt.cudaMalloc(size)
            if err == ok:
                held.append(p)
            else:
                rt.cudaGetLastError()
                size = size // 2 if size // 2 >= piece or size == piece else piece
        yield
    finally:
        for p in held:
            rt.cudaFree(p)


def test_no_history_after_a_failed_solve(handle):
    """The FP32 copies of a variable operator find no device memory: the solve fails, and the
    history is refused instead of the previous solve's entries."""
    n, m = 2000, 1500
    solid = np.zeros((m + 2, n + 2), np.uint8)
    rng = np.random.default_rng(0)
    b = np.zeros(solid.shape)
    b[1:-1, 1:-1] = rng.standard_normal((m, n))
    opts = handle.options("mixed", 1e-3, 30, "rel")
    handle.set_problem(solid, 1.0, 1.0)
    st = handle.solve(b, np.zeros_like(b), opts, strict=True)
    assert handle.residual_history(31)[st.iterations] > 0
    lap = np.ones_like(b)
    handle.set_variable_laplacian(4 * lap, lap, lap)
    try:
        with memory_taken(4 << 20):
            with pytest.raises(Exception, match="allocation"):
                handle.solve(b, np.zeros_like(b), opts)
            with pytest.raises(Exception, match="no solve yet"):
                handle.residual_history(31)
    finally:
        handle.set_variable_laplacian()
    st = handle.solve(b, np.zeros_like(b), opts, strict=True)
    assert handle.residual_history(31)[st.iterations] > 0
