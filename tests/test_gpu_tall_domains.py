"""Domains of more levels, or of more rows of tiles, than the 65535 a launch's grid takes along z and y:
what the stencils give there is what they give on a window of the same fields."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NZ, ROWS16, ROWS8 = 65600, 16 * 65535 + 40, 8 * 65535 + 40
# (form, stencil, dtype, axis, extent, halo, levels a CTA or 0).  With levels a CTA: the kernels whose
# default is one level, which took such domains only so.
CASES = ([("call", n, "f32", "k", NZ, 3, 0) for n in ("laplace", "hdiffsa", "nh_p_grad", "fvtp2d")] +
         [("call", n, "f32", "k", NZ, 3, 2) for n in ("hdiffsmag", "hadvuv", "hadvuv5th", "fastwavesuv", "p_grad_c")] +
         [("adjoint", "hdiffsmag", "f32", "k", NZ, 3, 2)] +
         [(f, "hdiffsa", "f64", "j", ROWS16, 2, 0) for f in ("call", "tl", "adjoint")] +
         [(f, "hdiffsmag", "f64", "j", ROWS16, 1, 0) for f in ("call", "tl")] +
         [("adjoint", "fastwavesuv", p, "j", ROWS8, 1, 0) for p in ("f64", "f32")])


def _run(pkg, form, name, arrays, out, h, nx, domain):
    st = {k: pkg.Storage(v, h, nx=nx if v.ndim == 3 else None) for k, v in {**arrays, **out}.items()}
    spec = pkg.KERNELS[name]
    sc = {s.name: 0.0625 for s in spec.scalars}
    group = lambda p: {n[1]: s for n, s in st.items() if n[0] == p}  # noqa: E731
    if form == "call":
        pkg.call(name, {**group("in"), **group("out")}, sc, domain=domain)
    else:
        getattr(pkg, "tangent_linear" if form == "tl" else "adjoint")(name, group("in"), group("seed"), group("out"), sc,
                                                                     domain=domain)


@pytest.mark.parametrize("case", CASES, ids=["-".join(map(str, c)) for c in CASES])
def test_a_window_of_a_tall_domain(pkg, cuda, case):
    import torch
    form, name, prec, axis, extent, h, kb = case
    nx, ny, nz = (3, 2, extent) if axis == "k" else (1, extent, 1)
    spec = pkg.KERNELS[name]
    dt = torch.float32 if prec == "f32" else torch.float64
    gen = torch.Generator(device=cuda).manual_seed(71)
    make = lambda *s: torch.rand(s, generator=gen, device=cuda, dtype=dt) + 0.5  # noqa: E731
    shape = (nz + 2 * h, ny + 2 * h, nx + 2 * h)
    arrays = {("in", a.name): make(ny + 2 * h) if a.role == "in1" else make(*shape)
              for a in spec.args if a.role in ("in1", "in3")}
    if form != "call":
        arrays.update({("seed", n): make(*shape) for n in (pkg.ACTIVE[name] if form == "tl" else spec.semantic_outputs)})
    out = {("out", n): torch.zeros(shape, device=cuda, dtype=dt)
           for n in (pkg.ACTIVE[name] if form == "adjoint" else [a.name for a in spec.by_role("out3")])}
    lib = pkg.load_library()
    try:
        assert lib.oeb_set_kblock(ctypes.c_int(kb)) == 0
        _run(pkg, form, name, arrays, out, h, nx, (nx, ny, nz))
    finally:
        lib.oeb_set_kblock(ctypes.c_int(0))
    torch.cuda.synchronize()
    n, edge = 24, 8  # rows or levels of a window, and of it those that its own edges reach
    for first in (0, extent // 2, extent - n):
        part = slice(first, first + n + 2 * h)
        cut = lambda v: (v[part] if v.ndim == 1 or axis == "k" else v[:, part]).contiguous()  # noqa: E731
        small = {q: v if axis == "k" and v.ndim == 1 else cut(v) for q, v in arrays.items()}
        got = {q: torch.zeros_like(cut(v)) for q, v in out.items()}
        _run(pkg, form, name, small, got, h, nx, (nx, ny, n) if axis == "k" else (nx, n, nz))
        torch.cuda.synchronize()
        a, b = h + edge, h + n - edge
        for q, v in got.items():
            whole = cut(out[q])
            same = torch.equal(v[a:b], whole[a:b]) if axis == "k" else torch.equal(v[h:-h, a:b], whole[h:-h, a:b])
            assert same, "%s at %d" % (q[1], first)
            assert v.abs().max() > 0
