"""When a solve on the covering aggregates is repeated on the reference's hierarchy: the
solves that must not be (plain CG, consistent right-hand sides cut off by max_iter), those
that must (every way a run-away solve can end), and what the repeat's own engine has to
follow (stream, kernel mode, memory)."""
import numpy as np
import pytest

from test_gpu_parity import connected, fluid_interior

pytestmark = pytest.mark.gpu


def _smooth(shape, seed, solids=0.2):
    """A connected mask with scattered solids and a smooth consistent right-hand side: the
    2-norm of the first CG residuals lies above the one of the right-hand side."""
    rng = np.random.default_rng(seed)
    padded = tuple(n + 2 for n in shape[::-1])
    solid = connected((rng.random(padded) < solids).astype(np.uint8))
    fl = fluid_interior(solid)
    x = np.arange(padded[-1]) / shape[0]
    b = np.where(fl, np.sin(3.0 * x) + 0.5 * np.arange(padded[0]).reshape((-1,) + (1,) * (len(shape) - 1)) / padded[0], 0.0)
    b[fl] -= b[fl].mean()
    return solid, b


@pytest.mark.parametrize("precision", ["mixed", "fp32"])
def test_plain_cg_is_never_repeated(handle, precision):
    """Without a preconditioner the hierarchy plays no part: a residual above the first one
    at max_iter is the end of the solve, in one engine."""
    solid, b = _smooth((200, 60), 1)
    handle.set_problem(solid, 1.0, 1.0)
    grew = False
    # the engine and a history of ten entries
    handle.solve(b, np.zeros_like(b), handle.options(precision, 0.9, 9, "rel"), strict=True)
    held = handle.device_bytes()
    for max_iter in (1, 2, 3, 4, 6, 9):
        st = handle.solve(b, np.zeros_like(b),
                          handle.options(precision, 0.0, max_iter, "rel", preconditioner=False))
        hist = handle.residual_history(max_iter + 1)
        grew |= hist[max_iter] > hist[0]
        assert st.status == 1 and st.iterations == max_iter
        assert handle.device_bytes() == held
    assert grew  # the case is one where it happens
