"""NumPy restatement of the library's multigrid V-cycle (csrc/vfs_mg.cu) in FP64, from the 19
operator coefficients per cell.

TEST INFRASTRUCTURE ONLY.  The levels, couplings, Thomas factors and zebra sweeps are those of
poisson_mg.MGSolver; what differs is restated here: coarse levels are smoothed, not solved, a
level whose odd cell count along a periodic i or k cannot be two-coloured takes damped line Jacobi
sweeps, and inactive cells (no coupling to any neighbour) take part in neither transfer.
"""
import numpy as np

from .poisson_mg import MGSolver, _Level

CP, EP, WP, NP, SP, TP, BP = range(7)
OMEGA = 0.8


class VCycle(MGSolver):
    def __init__(self, coef, periodic, pre=3, post=3, coarse=4, levels=0):
        """coef: (19, mz, my, mx) in the slot order of PoissonLHSNew (poisson.c:951-969)."""
        self.ip, self.jp, self.kp = periodic
        self.pre, self.post, self.coarse, self.max_levels = pre, post, coarse, levels
        self.levels = []
        self._build(coef[:, 1:-1, 1:-1, 1:-1])

    def _fine_couplings(self, c):
        out = []
        fluid = c[CP] != 0
        for axis, per, up, down in ((2, self.ip, EP, WP), (1, self.jp, NP, SP), (0, self.kp, TP, BP)):
            g = np.maximum(0.0, 0.5 * (c[up] + np.roll(c[down], -1, axis=axis)))
            g[~(fluid & np.roll(fluid, -1, axis=axis))] = 0.0
            if not per:
                last = [slice(None)] * 3
                last[axis] = -1
                g[tuple(last)] = 0.0
            out.append(g)
        return out

    def _build(self, c):
        ce, cn, ct = self._fine_couplings(c)
        while True:
            L = _Level()
            L.ce, L.cn, L.ct = ce, cn, ct
            L.shape = nz, ny, nx = ce.shape
            self._finish_level(L)
            L.act = L.dg != 0
            L.zebra = not ((self.ip and nx % 2) or (self.kp and nz % 2))
            self.levels.append(L)
            if len(self.levels) == self.max_levels or not all(d % 2 == 0 and d >= 4 for d in L.shape):
                return
            ce = 0.5 * L.ce[:, :, 1::2].reshape(nz // 2, 2, ny // 2, 2, nx // 2).sum(axis=(1, 3))
            cn = 0.5 * L.cn[:, 1::2, :].reshape(nz // 2, 2, ny // 2, nx // 2, 2).sum(axis=(1, 4))
            ct = 0.5 * L.ct[1::2, :, :].reshape(nz // 2, ny // 2, 2, nx // 2, 2).sum(axis=(2, 4))

    def _sweeps(self, L, x, b, n):
        for _ in range(n):
            if L.zebra:
                x = self._smooth(L, x, b)
                continue
            # every column from the previous iterate: a zebra sweep per colour on a copy of it
            old, new = x, np.empty_like(x)
            for colour in (0, 1):
                keep, L.colour = L.colour, np.where(L.colour == colour, 0, 2)
                y = self._smooth(L, old.copy(), b)
                L.colour = keep
                sel = np.broadcast_to((L.colour == colour)[:, None, :], L.shape)
                new[sel] = y[sel]
            x = old + OMEGA * (new - old)
        return x

    def _restrict_active(self, L, r):
        return self._restrict(L, np.where(L.act, r, 0.0))

    def _prolong_active(self, L, C, e):
        """Trilinear from the cell's eight nearest coarse cells; one that does not exist or is
        inactive gives its weight to the parent."""
        out = np.zeros(L.shape)

        def neighbour(a, axis, shift, per, fill):
            b = np.roll(a, -shift, axis=axis)
            if not per:
                edge = [slice(None)] * 3
                edge[axis] = -1 if shift > 0 else 0
                b[tuple(edge)] = fill
            return b

        for ak in (0, 1):
            for aj in (0, 1):
                for ai in (0, 1):
                    s, own = np.zeros(C.shape), np.full(C.shape, 27.0 / 64.0)
                    for n in range(1, 8):
                        w = np.prod([1.0 if n >> q & 1 else 3.0 for q in range(3)]) / 64.0
                        v, ok = e, C.act
                        for q, (axis, per, up) in enumerate(((2, self.ip, ai), (1, self.jp, aj), (0, self.kp, ak))):
                            if n >> q & 1:
                                shift = 1 if up else -1
                                v, ok = neighbour(v, axis, shift, per, 0.0), neighbour(ok, axis, shift, per, False)
                        s += np.where(ok, w * v, 0.0)
                        own += np.where(ok, 0.0, w)
                    out[ak::2, aj::2, ai::2] = s + own * e
        return np.where(L.act, out, 0.0)

    def vcycle(self, b, l=0):
        L = self.levels[l]
        x = np.zeros(L.shape)
        if l == len(self.levels) - 1:
            return self._sweeps(L, x, b, self.coarse)
        x = self._sweeps(L, x, b, self.pre)
        e = self.vcycle(self._restrict_active(L, b - self._apply(L, x)), l + 1)
        x = x + self._prolong_active(L, self.levels[l + 1], e)
        return self._sweeps(L, x, b, self.post)

    def line_condition(self):
        """Bound of the condition numbers of the columns' line systems over the levels: the largest
        diagonal over the smallest coupling of a row out of its column."""
        worst = 1.0
        for L in self.levels:
            out = (L.ce + L.cw + L.ct + L.cb)[L.act]
            worst = max(worst, 2.0 * np.abs(L.dg).max() / out.min()) if out.size and out.min() > 0 else np.inf
        return worst
