"""When a solve on the covering aggregates is repeated on the reference's hierarchy: the
solves that must not be (plain CG, consistent right-hand sides cut off by max_iter), those
that must (every way a run-away solve can end), and what the repeat's own engine has to
follow (stream, kernel mode, memory)."""
import numpy as np
import pytest

from test_gpu_failed_solve import memory_taken
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


def _rooms(dim):
    """A closed room inside the domain, and its label (1: outside, 2: inside)."""
    if dim == 2:
        solid = np.zeros((258, 386), np.uint8)
        solid[100:160, 100:160] = 1
        solid[103:157, 103:157] = 0
        inside = np.zeros(solid.shape, bool)
        inside[103:157, 103:157] = True
    else:
        solid = np.zeros((72, 74, 78), np.uint8)
        solid[20:40, 20:40, 20:40] = 1
        solid[22:38, 22:38, 22:38] = 0
        inside = np.zeros(solid.shape, bool)
        inside[22:38, 22:38, 22:38] = True
    fl = fluid_interior(solid)
    return solid, np.where(fl, np.where(inside, 2, 1), 0)


def _inconsistent(solid, lab, share, seed=5):
    """Noise that sums to zero in every room, plus a net source of the given share."""
    rng = np.random.default_rng(seed)
    b = np.where(lab > 0, rng.standard_normal(lab.shape), 0.0)
    for q in range(1, lab.max() + 1):
        b[lab == q] -= b[lab == q].mean()
    src = (lab == 2).astype(float)
    src[lab > 0] -= src[lab > 0].mean()
    return b + share * src * np.linalg.norm(b) / np.linalg.norm(src)


@pytest.mark.parametrize("precision", ["mixed", "fp32"])
@pytest.mark.parametrize("dim,share,max_iter", [(2, 1.0, 3), (3, 1.0, 3), (2, 1e-4, 12), (2, 1e-6, 25), (2, 1e-6, 40), (3, 1e-2, 12),
                                                (3, 1e-4, 6), (3, 1e-4, 12), (3, 1e-6, 25)])
def test_inconsistent_share_ends_as_on_the_reference_hierarchy(handle, dim, share, max_iter, precision):
    """A net source of a share of b, cut off by max_iter: the residual rises from the start,
    or falls to a small share and then rises.  The solve ends about where the FP64 form (on the reference's hierarchy) does: the two
    differ by the oscillation of CG on such a system, a factor of up to four."""
    solid, lab = _rooms(dim)
    b = _inconsistent(solid, lab, share)
    handle.set_problem(solid, 1.0, 1.0, 1.0)
    ref = handle.solve(b, np.zeros_like(b), handle.options("fp64", 1e-7, max_iter, "rel"))
    st = handle.solve(b, np.zeros_like(b), handle.options(precision, 1e-7, max_iter, "rel"))
    assert st.rel_residual <= max(6.0 * ref.rel_residual, 1e-5)
    assert st.status == 0 or st.iterations == max_iter


@pytest.mark.parametrize("dim", [2, 3])
def test_a_run_away_that_overflows_is_repeated(handle, dim):
    """A large right-hand side: the run-away iterates overflow FP32 before the residual has
    grown enough, and the solve used to end with NaN.  On the reference's hierarchy it ends
    at max_iter, finite."""
    solid, lab = _rooms(dim)
    b = _inconsistent(solid, lab, 1e-2) * 1e32
    handle.set_problem(solid, 1.0, 1.0, 1.0)
    p = np.zeros_like(b)
    st = handle.solve(b, p, handle.options("fp32", 1e-8, 40, "rel"))
    assert st.status == 1 and st.iterations == 40


@pytest.mark.parametrize("precision", ["mixed", "fp32"])
def test_not_finite_and_tiny_right_hand_sides_are_not_repeated(handle, precision):
    """NaN in the right-hand side ends as NaN, and one whose p.Ap lies below the absolute
    threshold as a breakdown, in one engine."""
    solid, b = _smooth((70, 50), 3)
    handle.set_problem(solid, 1.0, 1.0)
    handle.solve(b, np.zeros_like(b), handle.options(precision, 1e-3, 30, "rel"), strict=True)
    held = handle.device_bytes()
    st = handle.solve(1e-12 * b, np.zeros_like(b), handle.options(precision, 1e-20, 30, "abs"))
    assert st.status == 2
    bad = b.copy()
    bad[20, 20] = np.nan
    with pytest.raises(Exception, match="nan"):
        handle.solve(bad, np.zeros_like(b), handle.options(precision, 1e-6, 30, "rel"))
    bad[20, 20] = np.inf
    with pytest.raises(Exception, match="nan"):
        handle.solve(bad, np.zeros_like(b), handle.options(precision, 1e-6, 30, "rel"))
    assert handle.device_bytes() == held


def _two_chambers():
    """Two chambers with a net source each (no solution exists)."""
    solid = np.zeros((72, 92), np.uint8)
    solid[:, 45] = 1
    fl = fluid_interior(solid)
    b = np.where(fl, np.random.default_rng(3).standard_normal(solid.shape), 0.0)
    b[:, :45][fl[:, :45]] += 1.0
    b[fl] -= b[fl].mean()
    return solid, b


@pytest.mark.parametrize("modes", [(0, 1), (0, 4), (3, 0), (2, 1)])
def test_repeat_follows_the_kernel_mode(handle, modes):
    """The repeat's engine, kept while the mask stays, runs the V-cycle kernels that are set
    now: as many launches as in a handle where it was made with them."""
    from uaamg_b200.solver import Handle
    solid, b = _two_chambers()
    opts = handle.options("mixed", 1e-6, 40, "rel")
    other = Handle(0)
    try:
        got = []
        for h, ms in ((handle, modes), (other, modes[1:])):
            h.set_problem(solid, 1.0, 1.0)
            for m in ms:
                h.set_vcycle_kernels(m)
                p = np.zeros_like(b)
                st = h.solve(b, p, opts)
            assert st.status == 1 and st.iterations == 40
            got.append((st.kernel_launches, p))
        assert got[0][0] == got[1][0]
        assert np.array_equal(got[0][1], got[1][1])
    finally:
        handle.set_vcycle_kernels(0)
        other.close()


def test_repeat_follows_the_stream(handle):
    """The stream a solve was repeated on is gone before the next mask and the next repeat."""
    from cuda.bindings import runtime as rt
    solid, b = _two_chambers()
    opts = handle.options("mixed", 1e-6, 40, "rel")
    handle.set_problem(solid, 1.0, 1.0)
    p, q = np.zeros_like(b), np.zeros_like(b)
    handle.solve(b, p, opts)
    err, stream = rt.cudaStreamCreate()
    assert err == rt.cudaError_t.cudaSuccess
    try:
        handle.set_stream(int(stream))
        st = handle.solve(b, q, opts)
        assert st.status == 1 and np.array_equal(p, q)
    finally:
        handle.set_stream(0)
        rt.cudaStreamDestroy(stream)
    handle.set_problem(solid, 1.0, 1.0)  # releases the repeat's engine
    q[:] = 0
    st = handle.solve(b, q, opts)
    assert st.status == 1 and np.array_equal(p, q)


def test_repeat_without_room_for_a_second_engine(handle):
    """With the device's memory taken, a run-away solve is repeated in its own engine: the
    same result as with a second one, and the next mask is on covering aggregates again."""
    solid = np.zeros((1502, 2002), np.uint8)
    solid[:, 1000] = 1
    fl = fluid_interior(solid)
    rng = np.random.default_rng(8)
    b = np.where(fl, rng.standard_normal(solid.shape), 0.0)
    c = b.copy()
    b[:, :1000][fl[:, :1000]] += 1.0
    b[fl] -= b[fl].mean()
    for sl in (slice(1, 1000), slice(1001, 2001)):
        c[1:-1, sl] -= c[1:-1, sl].mean()
    opts = handle.options("mixed", 1e-6, 40, "rel")
    handle.set_problem(solid, 1.0, 1.0)
    want, good = np.zeros_like(b), np.zeros_like(b)
    ref = handle.solve(b, want, opts)
    st = handle.solve(c, good, opts, strict=True)
    two = handle.device_bytes()
    handle.set_problem(solid, 1.0, 1.0)  # the second engine is gone
    q = np.zeros_like(b)
    handle.solve(c, q, opts, strict=True)
    one = handle.device_bytes()
    assert two > one and np.array_equal(q, good)
    p = np.zeros_like(b)
    with memory_taken((two - one) // 2):
        got = handle.solve(b, p, opts)
    assert handle.device_bytes() <= one
    assert got.status == ref.status == 1 and got.iterations == ref.iterations
    assert np.array_equal(p, want)
    handle.set_problem(solid, 1.0, 1.0)
    q[:] = 0
    again = handle.solve(c, q, opts, strict=True)
    assert again.iterations == st.iterations and np.array_equal(q, good)


def _serve(srv, sim_id, solid, b):
    t = srv.submit(sim_id, solid, b, 1.0, 1.0)
    srv.drain()
    return srv.poll(t)


def test_server_counts_the_engine_of_a_repeat(handle):
    """The resident bytes grow by the repeat's engine, and idle ids make room for it."""
    from uaamg_b200.solver import Server
    solid, b = _two_chambers()
    c = np.zeros_like(b)
    for sl in (slice(1, 45), slice(46, 91)):
        c[1:-1, sl] = np.random.default_rng(4).standard_normal(c[1:-1, sl].shape)
        c[1:-1, sl] -= c[1:-1, sl].mean()
    srv = Server(0, "mixed", 1e-6, 40)
    try:
        assert _serve(srv, 1, solid, c)["status"] == 0
        one = srv.info()["device_bytes"]
        assert _serve(srv, 1, solid, b)["status"] == 1
        two = srv.info()["device_bytes"]
        assert two > 1.2 * one
    finally:
        srv.stop()
    # room for two ids, not for a third engine
    srv = Server(0, "mixed", 1e-6, 40, hbm_budget_bytes=2 * one + (two - one) // 2)
    try:
        assert _serve(srv, 1, solid, c)["status"] == 0
        assert _serve(srv, 2, solid, c)["status"] == 0
        assert srv.info()["device_bytes"] <= 2 * one
        assert _serve(srv, 2, solid, b)["status"] == 1
        info = srv.info()
        assert info["resident"] == 1 and info["device_bytes"] == two
    finally:
        srv.stop()


@pytest.mark.parametrize("shape", [(48, 48), (64, 64), (70, 33)])
def test_server_budget_holds_for_small_ids(shape):
    """Small grids hold the dense tail's matrix, many times the grid: a budget for one and a
    half of them admits one at a time."""
    from uaamg_b200.solver import Server
    solid, b = _smooth(shape, 2)
    srv = Server(0, "mixed", 1e-6, 100)
    try:
        assert _serve(srv, 1, solid, b)["status"] == 0
        one = srv.info()["device_bytes"]
    finally:
        srv.stop()
    srv = Server(0, "mixed", 1e-6, 100, hbm_budget_bytes=one + one // 2)
    try:
        for sim in (1, 2, 3):
            assert _serve(srv, sim, solid, b)["status"] == 0
            assert srv.info()["device_bytes"] <= one + one // 2
    finally:
        srv.stop()


@pytest.mark.parametrize("shape,max_iter,reached", [((65, 33), 60, 1e-6), ((130, 70), 20, 1e-10), ((130, 70), 60, 1e-6),
                                                    ((70, 66, 67), 60, 1e-10), ((70, 66, 67), 100, 1e-6)])
def test_converged_chambers_with_a_tolerance_out_of_reach(handle, shape, max_iter, reached):
    """Two chambers, each with a consistent right-hand side, and a tolerance of 0: the solve
    gets far below 1e-6 and keeps it, whatever its rounding does until max_iter."""
    padded = tuple(n + 2 for n in shape[::-1])
    solid = np.zeros(padded, np.uint8)
    solid[..., shape[0] // 2] = 1
    fl = fluid_interior(solid)
    b = np.where(fl, np.random.default_rng(4).standard_normal(padded), 0.0)
    for part in (np.s_[..., :shape[0] // 2], np.s_[..., shape[0] // 2 + 1:]):
        v, f = b[part], fl[part]
        v[f] -= v[f].mean()
    handle.set_problem(solid, 1.0, 1.0, 1.0)
    st = handle.solve(b, np.zeros_like(b), handle.options("mixed", 0.0, max_iter, "rel"))
    assert st.iterations == max_iter and st.rel_residual <= reached


@pytest.mark.parametrize("warm", [False, True])
@pytest.mark.parametrize("precision", ["mixed", "fp32"])
@pytest.mark.parametrize("wall,share,max_iter", [(10, 1e-4, 12), (10, 1e-6, 25), (80, 1e-4, 25), (80, 1e-6, 12)])
def test_chambers_of_different_size(handle, wall, share, max_iter, precision, warm):
    """A small chamber beside a large one, an absolute tolerance, from zero and from a warm
    start: as test_inconsistent_share_ends_as_on_the_reference_hierarchy."""
    solid = np.zeros((72, 92), np.uint8)
    solid[:, wall] = 1
    fl = fluid_interior(solid)
    lab = np.where(fl, 1 + (np.arange(92) > wall)[None, :], 0)
    b = _inconsistent(solid, lab, share)
    p0 = np.where(fl, np.random.default_rng(6).standard_normal(solid.shape), 0.0) * warm
    handle.set_problem(solid, 1.0, 1.0)
    opts = lambda prec: handle.options(prec, 1e-6, max_iter, "abs", warm_start=warm)
    ref = handle.solve(b, p0.copy(), opts("fp64"))
    st = handle.solve(b, p0.copy(), opts(precision))
    assert st.status == 1 and st.iterations == max_iter
    assert st.rel_residual <= 6.0 * ref.rel_residual
