"""The Cartesian operator and predictor in numpy's extended precision (quad on aarch64, 64
significant bits on x86), with the magnitudes that bound the rounding of the same sums in
FP64.  Fields are (3, nk, nj, ni), materials (nk, nj, ni), stretching three 1-D arrays."""
import numpy as np

L = np.longdouble


def _at(a, m, ax):
    return np.roll(a, -m, axis=-1 - ax)


def _line(s, ax):
    return np.asarray(s, dtype=L).reshape([-1 if d == 2 - ax else 1 for d in range(3)])


def _interior(a):
    out = np.zeros_like(a)
    out[..., 2:-2, 2:-2, 2:-2] = a[..., 2:-2, 2:-2, 2:-2]
    return out


def operator(u, mu, la, st, h, differences=False):
    """(L(u), terms): terms sums, per component, the magnitudes that one rounding of each
    product and sum is relative to: of a second difference every part of its weight times
    both values (times their difference, if differences), of a mixed term its coefficient
    times the inner differences."""
    u, mu, la = [np.asarray(a, dtype=L) for a in (u, mu, la)]
    s = [_line(a, ax) for ax, a in enumerate(st)]
    out, terms = [], []
    for c in range(3):
        r, t = L(0), L(0)
        for ax in range(3):
            f = u[c]
            a = {m: _at((2 * mu + la if ax == c else mu) * s[ax], m, ax) for m in range(-2, 3)}
            w = {-2: (a[-1], -0.75 * (a[0] + a[-2])), -1: (a[-2] + a[1], 3 * (a[0] + a[-1])),
                 1: (a[-1] + a[2], 3 * (a[1] + a[0])), 2: (a[1], -0.75 * (a[0] + a[2]))}
            for m, (p, q) in w.items():
                r = r + s[ax] * (p + q) * (_at(f, m, ax) - f) / 6
                size = abs(_at(f, m, ax) - f) if differences else abs(_at(f, m, ax)) + abs(f)
                t = t + abs(s[ax]) * (abs(p) + abs(q)) * size / 6
        for ax in range(3):
            if ax == c:
                continue
            for coef, v, outer, inner in ((la, u[ax], c, ax), (mu, u[ax], ax, c)):
                d = _at(v, 1, inner) - _at(v, -1, inner)
                e = _at(v, -2, inner) - _at(v, 2, inner)
                g, m = coef * (8 * d + e), abs(coef) * (8 * abs(d) + abs(e))
                x = s[c] * s[ax] / 144
                r = r + x * (8 * (_at(g, 1, outer) - _at(g, -1, outer)) + _at(g, -2, outer) - _at(g, 2, outer))
                t = t + abs(x) * (8 * (_at(m, 1, outer) + _at(m, -1, outer)) + _at(m, -2, outer) + _at(m, 2, outer))
        out.append(r)
        terms.append(t)
    h2 = L(h) ** 2
    return _interior(np.stack(out)) / h2, _interior(np.stack(terms)) / h2
