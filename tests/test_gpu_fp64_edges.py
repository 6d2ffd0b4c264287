"""Two things the FP64 kernels do apart from the plain loop: operands that are exactly zero take the
integer-pipe products and quotients' fast path with a stand-in (mul_zero, div_zero), and the tiles at
the far edge of a box deal their few columns to whole warps (TileCells)."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_adjoint import H, Case, _dot_test

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(33, 31, 2), (64, 40, 1), (5, 3, 2)], ids=["33x31x2", "64x40x1", "5x3x2"])
def test_zero_operands_are_the_oracle(pkg, fields, orc, cuda, size):
    """FP64 hdiffsmag where the clamped coefficient is zero, next to finite and not finite sums: the
    oracle's bits (a zero times an infinite or undefined sum is undefined)."""
    import torch
    nx, ny, nz = size
    spec = pkg.KERNELS["hdiffsmag"]
    inputs = fields.make_inputs("hdiffsmag", nx, ny, nz, seed=41, workload="fronts", halo=H)
    sc = fields.make_scalars("hdiffsmag", seed=41)
    rng = np.random.default_rng(43)
    mask = inputs["mask"]
    mask[rng.random(mask.shape) < 0.4] = 1e6   # the weight outweighs the deformation: clamped to zero
    mask[rng.random(mask.shape) < 0.3] = -1e6  # clamped from above
    odd = rng.random(inputs["uin"].shape)
    inputs["uin"][odd < 0.01] = np.inf
    inputs["vin"][odd > 0.99] = np.nan
    inputs["vin"][(odd > 0.5) & (odd < 0.6)] = 0.0
    outs = fields.make_outputs("hdiffsmag", nx, ny, nz, halo=H)
    want = {k: v.copy() for k, v in {**inputs, **outs}.items()}
    dev = {k: pkg.Storage(torch.from_numpy(v.copy()).to(cuda), H, nx=nx if v.ndim == 3 else None)
           for k, v in want.items()}
    with np.errstate(all="ignore"):
        orc.run_oracle(spec, want, sc, nx, ny, nz, H)
    pkg.call("hdiffsmag", dev, sc, domain=(nx, ny, nz))
    torch.cuda.synchronize()
    for a in spec.by_role("out3"):
        got, w = dev[a.name].numpy(), want[a.name]
        assert np.isnan(w).any() or nx < 10
        np.testing.assert_array_equal(np.isnan(got), np.isnan(w), err_msg=a.name)
        ok = ~np.isnan(w)
        np.testing.assert_array_equal(got[ok].view(np.uint64), w[ok].view(np.uint64), err_msg=a.name)


# widths and heights that leave a box of each adjoint (the interior widened by 1 to 6) one column or
# row into a tile, one short of it, and in the middle
EDGES = [(1, 1, 1), (26, 27, 2), (27, 58, 2), (29, 31, 3), (31, 26, 1), (32, 32, 2), (33, 65, 2), (60, 30, 4),
         (95, 33, 2), (50, 3, 70)]


@pytest.mark.parametrize("size", EDGES, ids=["x".join(map(str, s)) for s in EDGES])
@pytest.mark.parametrize("name", ("laplace", "hdiffsa", "hadvuv", "hadvuv5th", "hdiffsmag", "fastwavesuv", "uvbke",
                                  "nh_p_grad", "p_grad_c", "fvtp2d"))
def test_fp64_edge_tiles(pkg, fields, cuda, name, size):
    """<J dx, y> = <dx, J^T y> with y = J dx.  A cell missed, visited twice or at another's place would
    be an error of the order of one over the number of cells, at least 1e-5; the sums' roundings are
    about 60 a cell at 1.1e-16, cancelling terms a thousand times the result at most: 1e-11."""
    _dot_test(Case(pkg, fields, cuda, name, *size, seed=47), 1e-11)


@pytest.mark.parametrize("name", ("fvtp2d", "hdiffsmag"))
def test_zero_seeds(pkg, fields, cuda, name):
    """Seeds that are zero in half of the columns: the adjoint is linear in them, so the two halves add
    up to the whole (60 roundings of 1.1e-16 on terms a thousand times the largest gradient at most),
    and where no seed reaches, the gradient is exactly zero."""
    case = Case(pkg, fields, cuda, name, 70, 35, 2, seed=53, workload="fronts")
    rng = np.random.default_rng(59)
    y = {n: rng.normal(size=case.shape3()) for n in case.spec.semantic_outputs}
    half = np.arange(case.shape3()[2]) < 38
    lo = {n: np.where(half, v, 0.0) for n, v in y.items()}
    hi = {n: np.where(half, 0.0, v) for n, v in y.items()}
    g, gl, gh = case.adj(y), case.adj(lo), case.adj(hi)
    for n in case.active:
        w, a, b = (case.sem_box(n, v[n]) for v in (g, gl, gh))
        assert np.abs(w - (a + b)).max() <= 1e-11 * np.abs(w).max()
        assert (a[..., 52:] == 0.0).all() and (b[..., :25] == 0.0).all()


# both tile heights of hdiffsa and hdiffsmag: 8 rows where the grid is small, 16 where it fills the GPU
TILES = [(32, 7, 2), (33, 8, 2), (31, 9, 1), (1, 16, 3), (64, 17, 2), (40, 15, 500), (33, 16, 500), (20, 17, 520),
         (65, 33, 140)]


@pytest.mark.parametrize("size", TILES, ids=["x".join(map(str, s)) for s in TILES])
@pytest.mark.parametrize("name", ("hdiffsa", "hdiffsmag"))
def test_tile_heights_are_the_oracle(pkg, fields, orc, cuda, name, size):
    import torch
    nx, ny, nz = size
    spec = pkg.KERNELS[name]
    want = {**fields.make_inputs(name, nx, ny, nz, seed=61, workload="fronts", halo=H),
            **fields.make_outputs(name, nx, ny, nz, halo=H)}
    sc = fields.make_scalars(name, seed=61)
    dev = {k: pkg.Storage(torch.from_numpy(v.copy()).to(cuda), H, nx=nx if v.ndim == 3 else None)
           for k, v in want.items()}
    orc.run_oracle(spec, want, sc, nx, ny, nz, H)
    pkg.call(name, dev, sc, domain=(nx, ny, nz))
    torch.cuda.synchronize()
    for a in spec.by_role("out3"):
        np.testing.assert_array_equal(dev[a.name].numpy().view(np.uint64), want[a.name].view(np.uint64), err_msg=a.name)


@pytest.mark.parametrize("size", [(31, 26, 2), (27, 29, 3), (33, 12, 400), (60, 61, 330)],
                         ids=["31x26x2", "27x29x3", "33x12x400", "60x61x330"])
def test_hdiffsa_f32_adjoint_tiles(pkg, fields, cuda, size):
    """The FP32 hdiffsa adjoint in tiles of 16 rows (small grids) and of 32: <J dx, y> = <dx, J^T y> with
    y = J dx, to 1e-5, which a cell missed or visited twice would exceed at the small sizes and the
    existing FP32 bound holds for roundings."""
    _dot_test(Case(pkg, fields, cuda, "hdiffsa", *size, seed=67, dtype=np.float32), 1e-5)
