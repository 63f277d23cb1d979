"""One host thread per handle (uaamg.h): handles on the default stream in several threads,
each with changing masks and grids -- set-up, graph captures and releases side by side --
give the results they give alone."""
import threading

import numpy as np
import pytest

from test_gpu_parity import fluid_interior

pytestmark = pytest.mark.gpu

SHAPES = [(64, 48), (130, 70), (40, 33, 20), (33, 17, 9)]


def _case(n):
    shape = SHAPES[n % 4]
    rng = np.random.default_rng(n)
    solid = np.zeros(tuple(v + 2 for v in shape[::-1]), np.uint8)
    at = 2 + n // 4
    solid[tuple(slice(at, at + v // 5 + 1) for v in solid.shape)] = 1
    fl = fluid_interior(solid)
    b = np.where(fl, rng.standard_normal(solid.shape), 0.0)
    b[fl] -= b[fl].mean()
    return solid, b


def _run(h, cases, order, prec, out):
    for n in order:
        solid, b = cases[n]
        p = np.zeros_like(b)
        if n % 3 == 2:
            h.solve_batch([(solid, b, p, 1.0, 1.0, 1.0)], h.options(prec, 1e-6, 60, "rel"), strict=True)
        else:
            h.set_problem(solid, 1.0, 1.0, 1.0)
            h.solve(b, p, h.options(prec, 1e-6, 60, "rel"), strict=True)
        out.append((n, p))


@pytest.mark.parametrize("prec", ["mixed", "fp32"])
def test_handles_in_threads(handle, prec):
    from uaamg_b200.solver import Handle
    cases = [_case(n) for n in range(12)]
    alone = []
    _run(handle, cases, range(12), prec, alone)
    want = dict(alone)
    outs, errors = [[] for _ in range(4)], []

    def work(k):
        h = Handle(0)
        try:
            order = np.random.default_rng(k).integers(0, 12, 60)
            _run(h, cases, [int(n) for n in order], prec, outs[k])
        except Exception as e:  # reported by the main thread
            errors.append(e)
        finally:
            h.close()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for out in outs:
        assert len(out) == 60
        for n, p in out:
            assert np.array_equal(p, want[n])
