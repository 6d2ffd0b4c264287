"""The FP64 point loops' tiles of 32 rows, which large grids take, against the 8 rows of small ones: a
domain of many levels, and windows of its levels, give the same bits, forward, tangent-linear and
adjoint, with a tile at the far edge of one column, of a few, of 23, of 24 and of 31 (TileCells)."""
from __future__ import annotations

import pytest

from test_gpu_tall_domains import _run

pytestmark = pytest.mark.gpu

H = 3
SIZES = [(33, 33), (37, 5), (55, 31), (56, 40), (63, 64)]
NAMES = ("laplace", "hdiffsmag", "hadvuv", "hadvuv5th", "fastwavesuv", "uvbke", "nh_p_grad", "p_grad_c")
MANY = 18 * 152  # tiles from which every form has 32-row ones (forward from 8 * 152)


@pytest.mark.parametrize("size", SIZES, ids=["x".join(map(str, s)) for s in SIZES])
@pytest.mark.parametrize("form", ("call", "tl", "adjoint"))
@pytest.mark.parametrize("name", NAMES)
def test_windows_of_many_levels(pkg, cuda, name, form, size):
    import torch
    nx, ny = size
    nz = MANY // (-(-nx // 32) * -(-ny // 32)) + 40
    spec = pkg.KERNELS[name]
    gen = torch.Generator(device=cuda).manual_seed(109)
    make = lambda *s: torch.rand(s, generator=gen, device=cuda, dtype=torch.float64) + 0.5  # noqa: E731
    shape = (nz + 2 * H, ny + 2 * H, nx + 2 * H)
    arrays = {("in", a.name): make(ny + 2 * H) if a.role == "in1" else make(*shape)
              for a in spec.args if a.role in ("in1", "in3")}
    if form != "call":
        arrays.update({("seed", n): make(*shape) for n in (pkg.ACTIVE[name] if form == "tl" else spec.semantic_outputs)})
    names = pkg.ACTIVE[name] if form == "adjoint" else [a.name for a in spec.by_role("out3")]
    out = {("out", n): torch.full(shape, 7.0, device=cuda, dtype=torch.float64) for n in names}
    _run(pkg, form, name, arrays, out, H, nx, (nx, ny, nz))
    n, edge = 12, 4  # levels of a window, and of it those that its own ends reach
    for first in (0, nz // 2, nz - n):
        part = slice(first, first + n + 2 * H)
        small = {q: v if v.ndim == 1 else v[part].contiguous() for q, v in arrays.items()}
        got = {q: torch.full_like(v[part], 7.0) for q, v in out.items()}
        _run(pkg, form, name, small, got, H, nx, (nx, ny, n))
        torch.cuda.synchronize()
        for q, v in got.items():
            a, b = H + edge, H + n - edge
            assert torch.equal(v[a:b], out[q][part][a:b]), "%s at %d" % (q[1], first)
