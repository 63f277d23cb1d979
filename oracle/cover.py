"""The preconditioner of the FP32 and mixed solves, restated in numpy and FP64: one V-cycle
over aggregates that cover every fluid cell, and a solve's first iteration with it.

A level holds arrays over its interior cells (the last axis is x).  Sizes halve rounding
up; a coarse cell is fluid when any of its children is; coarse couplings are the sums of
the fine ones across the shared face.  Smoothing is red-black (forward: colour 1 then 0,
backward: 0 then 1), the coarsest level ten forward and backward sweeps.  The prolongation
adds 2 (x_c + w sum_a (x_n - x_c)), x_n the coarse neighbour on the cell's own side along
axis a where the coarse level couples the two; the restriction is half its transpose.
w is 1/5 on star transfers and 0 on constant ones (per level, `star`)."""
from __future__ import annotations

import numpy as np

W = 0.2


def _shift(a, axis, by, fill=0):
    """a[i + by] along axis, fill outside."""
    out = np.full_like(a, fill)
    n = a.shape[axis]
    src, dst = [slice(None)] * a.ndim, [slice(None)] * a.ndim
    src[axis] = slice(max(by, 0), n + min(by, 0))
    dst[axis] = slice(max(-by, 0), n + min(-by, 0))
    out[tuple(dst)] = a[tuple(src)]
    return out


class Level:
    """fluid: bool per cell; c[axis]: coupling to the next cell along the axis."""

    def __init__(self, fluid, c):
        self.fluid, self.c = fluid, c
        self.d = sum(c[a] + _shift(c[a], a, -1) for a in range(fluid.ndim))
        self.relax = fluid & (self.d >= 1e-30)
        self.colour = (np.indices(fluid.shape).sum(0) + fluid.ndim) & 1  # of 1-based indices

    def neighbours(self, x):
        return sum(self.c[a] * _shift(x, a, 1) + _shift(self.c[a], a, -1) * _shift(x, a, -1)
                   for a in range(x.ndim))

    def sweep(self, x, b, colour):
        m = self.relax & (self.colour == colour)
        x[m] = ((b + self.neighbours(x)) / np.where(self.relax, self.d, 1.0))[m]

    def residual(self, x, b):
        return np.where(self.fluid, b - self.d * x + self.neighbours(x), 0.0)


def _children(a, coarse):
    """The array extended to even sizes, axes split as (coarse, child)."""
    e = np.zeros(tuple(2 * n for n in coarse), a.dtype)
    e[tuple(slice(0, n) for n in a.shape)] = a
    return e.reshape([v for n in coarse for v in (n, 2)])


class CoverHierarchy:
    def __init__(self, solid, *spacing):
        """solid: padded mask (ghost ring); spacing dx, dy[, dz]."""
        nd = solid.ndim
        sp = spacing[:nd][::-1]  # per array axis
        fluid = (np.asarray(solid) == 0)[(slice(1, -1),) * nd]
        c = []
        for a in range(nd):
            both = fluid & _shift(fluid, a, 1, False)
            c.append(np.where(both, 1.0 / (sp[a] * sp[a]), 0.0))
        self.levels = [Level(fluid, c)]
        while min(self.levels[-1].fluid.shape) > 4:
            f = self.levels[-1]
            n = tuple((v + 1) // 2 for v in f.fluid.shape)
            kids = tuple(range(1, 2 * nd, 2))
            cc = []
            for a in range(nd):
                last = np.take(_children(f.c[a], n), 1, axis=2 * a + 1)  # children at the + face
                cc.append(last.sum(axis=tuple(k - (k > 2 * a + 1) for k in kids if k != 2 * a + 1)))
            self.levels.append(Level(_children(f.fluid, n).any(axis=kids), cc))

    def prolong(self, l, xc, star):
        """P x_c on the cells of level l."""
        f, c = self.levels[l], self.levels[l + 1]
        nd = xc.ndim
        out = np.zeros(tuple(2 * n for n in xc.shape))
        child = np.indices(out.shape) & 1
        up = lambda a: np.kron(a, np.ones((2,) * nd, a.dtype))
        v = xc.copy()
        out += up(v)
        if star:
            for a in range(nd):
                hi = np.where(c.c[a] > 0, _shift(xc, a, 1) - xc, 0.0)
                lo = np.where(_shift(c.c[a], a, -1) > 0, _shift(xc, a, -1) - xc, 0.0)
                out += W * np.where(child[a] == 1, up(hi), up(lo))
        out = 2.0 * out[tuple(slice(0, n) for n in f.fluid.shape)]
        return np.where(f.fluid, out, 0.0)

    def restrict(self, l, r, star):
        """Half the transpose of prolong."""
        c = self.levels[l + 1]
        nd = r.ndim
        k = _children(r, c.fluid.shape)
        kids = tuple(range(1, 2 * nd, 2))
        s = k.sum(axis=kids)
        if star:
            t = np.zeros_like(s)
            for a in range(nd):
                rest = tuple(q - (q > 2 * a + 1) for q in kids if q != 2 * a + 1)
                lo = np.take(k, 0, axis=2 * a + 1).sum(axis=rest)  # children at the - side
                hi = np.take(k, 1, axis=2 * a + 1).sum(axis=rest)
                t += np.where(c.c[a] > 0, _shift(lo, a, 1) - hi, 0.0)
                t += np.where(_shift(c.c[a], a, -1) > 0, _shift(hi, a, -1) - lo, 0.0)
            s = s + W * t
        return np.where(c.fluid, s, 0.0)

    def vcycle(self, b, star=True, nu=(1, 1), l=0, tail=None):
        """M b.  star: a flag, or one per level; nu: smoothing sweeps of the finest and of
        the coarser levels (level `tail` and below: one sweep)."""
        L = self.levels[l]
        x = np.zeros_like(b)
        if l == len(self.levels) - 1:
            for _ in range(10):
                for colour in (1, 0, 0, 1):
                    L.sweep(x, b, colour)
            return x
        st = star if isinstance(star, bool) else star[l]
        n = 1 if tail is not None and l >= tail else nu[0] if l == 0 else nu[1]
        for _ in range(n):
            L.sweep(x, b, 1)
            L.sweep(x, b, 0)
        xc = self.vcycle(self.restrict(l, L.residual(x, b), st), star, nu, l + 1, tail)
        x += self.prolong(l, xc, st)
        for _ in range(n):
            L.sweep(x, b, 0)
            L.sweep(x, b, 1)
        return x

    def first_iterate(self, rhs, **kw):
        """x after one CG iteration on lap(x) = rhs (padded in, padded out)."""
        L = self.levels[0]
        inner = (slice(1, -1),) * rhs.ndim
        f = L.fluid
        b = np.where(f, -rhs[inner], 0.0)
        b[f] -= b[f].mean()
        z = self.vcycle(b, **kw)
        z = np.where(f, z - z[f].mean(), 0.0)
        az = np.where(f, L.d * z - L.neighbours(z), 0.0)
        out = np.zeros_like(rhs)
        out[inner] = z * ((b * z).sum() / (z * az).sum())
        return out

    def tail_level(self):
        """First level (>= 1) of at most 1024 cells: from there on the cycle is one product."""
        for l, L in enumerate(self.levels[1:], 1):
            if L.fluid.size <= 1024:
                return l
        return len(self.levels) - 1
