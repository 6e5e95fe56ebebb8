"""One V-cycle of the reference (apply_preconditioner, src/apic.rs:1788-1821, with
smooth_level :471-535, restrict :537-594, prolongate :596-616 and
solve_coarse_exact :618-704, its sums serial) in numpy, on levels given as
arrays: what the mask leaves out takes no part, whatever the coefficients hold
there."""
import numpy as np

F = np.float32


def fma(a, b, c):
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(F)


class Level:
    """Padded arrays (index = cell + w, cells + 2 w entries)."""

    def __init__(self, w, h, bits, diag, inv, px, py):
        self.w, self.h, self.cells = w, h, w * h
        on = np.unpackbits(np.asarray(bits).view(np.uint8), bitorder="little")[:self.cells].astype(bool)
        self.on = np.concatenate([np.zeros(w, bool), on, np.zeros(w, bool)])
        self.diag, self.inv, self.px, self.py = (np.asarray(a, F) for a in (diag, inv, px, py))
        self.res, self.err = np.zeros(self.cells + 2 * w, F), np.zeros(self.cells + 2 * w, F)
        self.fluid = np.nonzero(self.on)[0]
        raw = self.fluid - w
        self.red = (raw % w + raw // w) % 2 == 0

    def neighbours(self, c):
        """(index, coupling) of the right, upper, left and lower cell, in the reference's order."""
        w = self.w
        return ((c + 1, self.px[c]), (c + w, self.py[c]), (c - 1, self.px[c - 1]), (c - w, self.py[c - w]))

    def smooth(self, red):
        c = self.fluid[self.red == red]
        s = self.res[c]
        for n, k in self.neighbours(c):
            s = np.where(self.on[n], fma(-k, self.err[n], s), s)
        old = self.err[c]
        new = old + F(1.2) * (s * self.inv[c] - old)
        self.err[c] = np.where(self.inv[c] == 0, old, new)

    def restrict(self, coarse):
        c = self.fluid
        ax = self.diag[c] * self.err[c]
        for n, k in self.neighbours(c):
            ax = np.where(self.on[n], ax + k * self.err[n], ax)
        left = np.zeros_like(self.res)
        left[c] = self.res[c] - ax
        raw = coarse.fluid - coarse.w
        x, y, s = raw % coarse.w, raw // coarse.w, np.zeros(raw.size, F)
        for dy in (0, 1):
            for dx in (0, 1):
                p = (2 * y + dy) * self.w + 2 * x + dx + self.w
                s = np.where(self.on[p], s + left[p], s)
        coarse.res[coarse.fluid] = s

    def prolong(self, coarse, extra=0):
        raw = self.fluid - self.w
        ec = coarse.err[(raw // self.w >> 1) * coarse.w + (raw % self.w >> 1) + coarse.w]
        self.err[self.fluid] += ec
        for _ in range(extra):
            self.err[self.fluid[-1]] += ec[-1]

    def solve(self, total=lambda q: np.cumsum(q, dtype=F)[-1]):
        """CG; total: the sum of an FP32 array, rounded to FP32."""
        c = self.fluid
        r, x = self.res[c].copy(), np.zeros(c.size, F)
        s = np.zeros_like(self.res)
        s[c] = r
        gamma = total(r * r)
        if gamma < F(1e-12):
            return
        order = (0, 2, 1, 3)  # the matrix product takes right, left, upper, lower
        for _ in range(min(c.size, 100)):
            ap = self.diag[c] * s[c]
            nb = self.neighbours(c)
            for i in order:
                n, k = nb[i]
                ap = np.where(self.on[n], fma(k, s[n], ap), ap)
            delta = total(s[c] * ap)
            if abs(delta) < F(1e-5):
                break
            alpha = F(gamma / delta)
            x = x + alpha * s[c]
            r = r - alpha * ap
            if not (np.abs(r) >= F(1e-6)).any():
                break
            new = total(r * r)
            beta, gamma = F(new / gamma), new
            s[c] = r + beta * s[c]
        self.err[c] = x


def vcycle(levels, residual, total=None):
    """The base level's error (padded) for its padded residual; levels finest first."""
    levels[0].res = np.asarray(residual, F).copy()
    for f, c in zip(levels, levels[1:]):
        f.smooth(True)
        f.smooth(False)
        f.restrict(c)
    levels[-1].solve(total) if total else levels[-1].solve()
    for k in range(len(levels) - 2, -1, -1):
        extra = (8 - levels[0].fluid.size % 8) % 8 if k == 0 else 0
        levels[k].prolong(levels[k + 1], extra)
        levels[k].smooth(False)
        levels[k].smooth(True)
    return levels[0].err
