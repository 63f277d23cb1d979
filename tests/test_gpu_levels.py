"""The level count of a solve's statistics is the inspected hierarchy's in every precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 2), (4, 9), (5, 5), (9, 9), (65, 33), (100, 37), (5, 5, 5), (9, 17, 33),
                                   (65, 65, 65), (64, 64, 64), (129, 9, 20)])
def test_stats_levels_agree_with_num_levels(handle, shape):
    b = np.zeros(tuple(n + 2 for n in shape[::-1]))
    b[(1,) * b.ndim], b[(2,) * b.ndim] = 1.0, -1.0
    handle.set_problem(np.zeros(b.shape, np.uint8), 1.0, 1.0, 1.0)
    n = handle.num_levels()
    assert handle.level_dims(0)[:2] == shape[:2]
    for prec in ("fp64", "fp32", "mixed"):
        st = handle.solve(b, np.zeros_like(b), handle.options(prec, 1e-3, 5, "rel"))
        assert st.levels == n, prec
    for st in handle.solve_batch([(np.zeros(b.shape, np.uint8), b, np.zeros_like(b), 1.0, 1.0, 1.0)],
                                 handle.options("mixed", 1e-3, 5, "rel")):
        assert st.levels == n
