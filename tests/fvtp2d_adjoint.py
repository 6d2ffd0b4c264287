"""The transposed fvtp2d in numpy, in passes: each PPM sweep's transpose over the whole field, the
fluxes and quotients between them as fields of their own (the order of operations of the FP64
kernels in csrc/k_fvtp2d.cu), every operation rounded to the arrays' type."""
from __future__ import annotations

import numpy as np

H = 3  # halo of every array
_M = 9  # margin of a sweep's window


def fma32(a, b, c):
    """a b + c in float32, rounded once: the product is exact in float64; the sum there is rounded to
    odd, so that rounding it to float32 is the one rounding of the exact sum."""
    p = np.float64(a) * np.float64(b)
    c = np.float64(c)
    s = p + c
    bb = s - p
    err = (p - (s - bb)) + (c - bb)
    s = np.array(s)
    odd = np.isfinite(err) & (err != 0) & ((s.view(np.int64) & 1) == 0)
    s.view(np.int64)[odd] += np.where((err > 0) == (s > 0), 1, -1)[odd]
    return s.astype(np.float32)


def _sweep(state, courant, flux, lo, hi, p1, p2):
    """The transposed sweep along the last axis: `state` is defined on [lo, hi), `flux` is the flux
    adjoint (zero off the flux points), `courant` the Courant number of each point's low face."""
    n = state.shape[-1]
    pad = lambda a, v: np.pad(a, [(0, 0), (0, 0), (_M, _M)], constant_values=a.dtype.type(v))  # noqa: E731
    gs = np.pad(state[..., lo + H:hi + H], [(0, 0), (0, 0), (_M + lo + H, _M + n - hi - H)], mode="edge")
    c, f = pad(courant, 1), pad(flux, 0)
    at = lambda a, d: np.roll(a, -d, axis=-1)  # noqa: E731  (wraps into the margin only)
    one, zero = f.dtype.type(1), f.dtype.type(0)
    als = p1 * (at(gs, -1) + gs) + p2 * (at(gs, -2) + at(gs, 1))
    m, r = als - gs, at(als, 1) - gs
    smt = ((m < 0) & (r > 0)) | ((m > 0) & (r < 0))
    up = c > 0
    t = np.where((f != 0) & (at(smt, -1) | smt), f * (one + -np.abs(c)), zero)
    t1, c1 = at(t, 1), at(c, 1)
    below, above = (t1 != 0) & at(up, 1), (t != 0) & ~up
    b0 = np.where(below, -c1 * t1, zero)
    b0 = np.where(above, b0 + c * t, b0)
    alm, br = np.where(above, t, zero) + b0, np.where(below, t1, zero) + b0
    al = alm + at(br, -1)
    g = fma32(p1, at(al, 1) + al, fma32(p2, at(al, 2) + at(al, -1), -alm)) - br
    f1 = at(f, 1)
    g = np.where((f1 != 0) & at(up, 1), g + f1, g)
    g = np.where((f != 0) & ~up, g + f, g)
    return g[..., _M:-_M]


def adjoint(x, q_i, q_j, fx1b, fy1b, nx, ny, p1, p2):
    """qb over q's whole box [-3, n + 3)^2 on every level, of float32 arrays with halo 3: the state x,
    its q_i and q_j, the seeds."""
    p1, p2, half = np.float32(p1), np.float32(p2), np.float32(0.5)
    T = lambda a: np.ascontiguousarray(a.swapaxes(1, 2))  # noqa: E731
    shape = q_i.shape
    jj, ii = np.meshgrid(np.arange(shape[1]) - H, np.arange(shape[2]) - H, indexing="ij")

    def box(ilo, ihi, jlo, jhi):
        return (ii >= ilo) & (ii < ihi) & (jj >= jlo) & (jj < jhi)

    def on(where, a):
        return np.where(where, a, np.float32(0))

    inner, bi, bj = box(0, nx, 0, ny), box(-3, nx + 2, 0, ny), box(0, nx, -3, ny + 2)
    gx, gy = on(inner, (half * x["xfx"]) * fx1b), on(inner, (half * x["yfx"]) * fy1b)
    qib = on(bi, _sweep(q_i, x["crx"], gx, -3, nx + 2, p1, p2))
    qjb = on(bj, T(_sweep(T(q_j), T(x["cry"]), T(gy), -3, ny + 2, p1, p2)))
    ry, rx = on(bi, qib / x["ra_y"]), on(bj, qjb / x["ra_x"])
    fy2b = on(box(-3, nx + 2, 0, ny + 1), gy + x["yfx"] * (ry - np.roll(ry, 1, axis=1)))
    fx2b = on(box(0, nx + 1, -3, ny + 2), gx + x["xfx"] * (rx - np.roll(rx, 1, axis=2)))
    qb = _sweep(x["q"], x["crx"], fx2b, -3, nx + 3, p1, p2)
    qb = np.where(bi, qb + (x["area"] / x["ra_y"]) * qib, qb)
    qb = np.where(bj, qb + (x["area"] / x["ra_x"]) * qjb, qb)
    return qb + T(_sweep(T(x["q"]), T(x["cry"]), T(fy2b), -3, ny + 3, p1, p2))
