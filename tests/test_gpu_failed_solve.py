"""A solve that fails on the host leaves no residual history behind."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_no_history_after_a_failed_solve(handle):
    """The FP32 copies of a variable operator find no device memory: the solve fails, and the
    history is refused instead of the previous solve's entries."""
    import torch
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
    torch.cuda.init()
    free, _ = torch.cuda.mem_get_info(0)
    hog = torch.empty(free - (6 << 20), dtype=torch.uint8, device="cuda:0")
    try:
        with pytest.raises(Exception, match="allocation"):
            handle.solve(b, np.zeros_like(b), opts)
        with pytest.raises(Exception, match="no solve yet"):
            handle.residual_history(31)
    finally:
        del hog
        torch.cuda.empty_cache()
        handle.set_variable_laplacian()
    st = handle.solve(b, np.zeros_like(b), opts, strict=True)
    assert handle.residual_history(31)[st.iterations] > 0
