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


@pytest.mark.parametrize("precision", ["mixed", "fp32"])
@pytest.mark.parametrize("shape", [(200, 60), (40, 30, 30)])
def test_consistent_solves_cut_off_early_are_not_repeated(handle, shape, precision):
    """A consistent right-hand side and a max_iter of one to four iterations: the residual may
    lie above the first one, and the solve ends there."""
    solid, b = _smooth(shape, 1)
    handle.set_problem(solid, 1.0, 1.0, 1.0)
    handle.solve(b, np.zeros_like(b), handle.options(precision, 0.9, 9, "rel"), strict=True)
    held, grew = handle.device_bytes(), False
    for max_iter in (1, 2, 3, 4):
        st = handle.solve(b, np.zeros_like(b), handle.options(precision, 1e-12, max_iter, "rel"))
        hist = handle.residual_history(max_iter + 1)
        grew |= hist[max_iter] > hist[0]
        assert st.status == 1 and st.iterations == max_iter
        assert handle.device_bytes() == held
    assert grew


@pytest.mark.parametrize("shape", [(20000, 6), (8, 30000), (5, 5, 20000)])
def test_consistent_channels_are_not_repeated(handle, shape):
    """Long channels with a smooth right-hand side: the residual rises several thousand times
    before it falls, and the solve goes on where it is."""
    padded = tuple(n + 2 for n in shape[::-1])
    solid = np.zeros(padded, np.uint8)
    ax = int(np.argmax(padded))
    v = np.linspace(0, 1, padded[ax]).reshape([-1 if a == ax else 1 for a in range(len(padded))])
    fl = fluid_interior(solid)
    b = np.where(fl, np.cos(np.pi * v), 0.0)
    b[fl] -= b[fl].mean()
    handle.set_problem(solid, 1.0, 1.0, 1.0)
    rough = np.where(fl, np.random.default_rng(2).standard_normal(padded), 0.0)
    handle.solve(rough, np.zeros_like(b), handle.options("mixed", 0.9, 60, "rel"), strict=True)
    held = handle.device_bytes()
    handle.solve(b, np.zeros_like(b), handle.options("mixed", 1e-4, 60, "rel"))
    hist = handle.residual_history(61)
    assert hist.max() > 1e3 * hist[0]
    assert handle.device_bytes() == held
