"""The marching FP32 kernels (csrc/march.cuh) at the sizes where a strip or a chunk can go wrong:
one column or row, a strip's width and one beside it, a chunk's rows and one beside them, padded
and larger halos.  Every output cell is the oracle's, compiled for float, bit for bit (the same
operations in the same order; the limiter and monotonicity signs are decided on exact products, which
agree with the float products wherever those do not underflow), and nothing outside the written
boxes changes.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (nx, ny, nz, halo, columns of row padding)
SIZES = [(1, 1, 1, 3, 0), (5, 3, 2, 3, 0), (26, 4, 3, 3, 0), (27, 5, 2, 4, 1), (30, 33, 2, 3, 0), (31, 9, 2, 3, 2),
         (32, 8, 1, 4, 0), (33, 31, 2, 3, 3), (52, 65, 2, 3, 0), (53, 12, 5, 4, 0), (61, 129, 1, 3, 0),
         (127, 70, 3, 3, 0), (209, 17, 2, 3, 1)]
NAMES = ("fvtp2d", "hadvuv", "hadvuv5th", "hdiffsa", "hdiffsmag", "fastwavesuv")


@pytest.mark.parametrize("size", SIZES, ids=["x".join(map(str, s)) for s in SIZES])
@pytest.mark.parametrize("name", NAMES)
def test_marching_kernel_is_the_float_oracle(pkg, fields, orc, cuda, name, size):
    import torch
    nx, ny, nz, h, pad = size
    spec = pkg.KERNELS[name]
    inputs = fields.make_inputs(name, nx, ny, nz, seed=23, workload="fronts", halo=h)
    sc = fields.make_scalars(name, seed=23)
    sc32 = {s.name: (sc[s.name] if s.always_double else float(np.float32(sc[s.name]))) for s in spec.scalars}
    outs = fields.make_outputs(name, nx, ny, nz, halo=h)
    want = {k: v.astype(np.float32) for k, v in {**inputs, **outs}.items()}
    dev = {}
    for k, v in want.items():
        a = np.full(v.shape[:-1] + (v.shape[-1] + pad,), np.float32(fields.SENTINEL)) if v.ndim == 3 else v.copy()
        if v.ndim == 3:
            a[..., :v.shape[-1]] = v
        dev[k] = pkg.Storage(torch.from_numpy(a).to(cuda), h, nx=nx if v.ndim == 3 else None)
    orc.run_oracle(spec, want, sc32, nx, ny, nz, h)
    pkg.call(name, dev, sc32, domain=(nx, ny, nz))
    torch.cuda.synchronize()
    for a in spec.by_role("out3"):
        got = dev[a.name].numpy()
        np.testing.assert_array_equal(got[..., :nx + 2 * h].copy().view(np.uint32), want[a.name].view(np.uint32),
                                      err_msg="%s.%s %s vs the float oracle" % (name, a.name, size))
        assert (got[..., nx + 2 * h:] == np.float32(fields.SENTINEL)).all(), "%s.%s wrote its row padding" % (name, a.name)


@pytest.mark.parametrize("size", SIZES, ids=["x".join(map(str, s)) for s in SIZES])
@pytest.mark.parametrize("name", ("laplace", "p_grad_c", "nh_p_grad"))
def test_row_kernels_match_the_plain_kernels(pkg, fields, cuda, name, size):
    """The FP32 stencils whose arithmetic is not the reference's float sequence: the plain kernels,
    which run where the fields lie in host memory, give the same bits."""
    import torch
    nx, ny, nz, h, pad = size
    spec = pkg.KERNELS[name]
    inputs = fields.make_inputs(name, nx, ny, nz, seed=29, workload="fronts", halo=h)
    sc = {k: float(np.float32(v)) for k, v in fields.make_scalars(name, seed=29).items()}
    arrays = {k: np.pad(v.astype(np.float32), ((0, 0), (0, 0), (0, pad)), constant_values=fields.SENTINEL)
              for k, v in {**inputs, **fields.make_outputs(name, nx, ny, nz, halo=h)}.items()}
    assert pkg.load_library().oeb_set_host_direct(1) == 0
    host = {k: pkg.Storage(torch.from_numpy(v.copy()).pin_memory(), h, nx=nx) for k, v in arrays.items()}
    dev = {k: pkg.Storage(torch.from_numpy(v.copy()).to(cuda), h, nx=nx) for k, v in arrays.items()}
    pkg.call(name, host, sc, domain=(nx, ny, nz))
    pkg.call(name, dev, sc, domain=(nx, ny, nz))
    torch.cuda.synchronize()
    for a in spec.by_role("out3"):
        np.testing.assert_array_equal(dev[a.name].numpy().view(np.uint32), host[a.name].numpy().view(np.uint32),
                                      err_msg="%s.%s %s vs the plain kernel" % (name, a.name, size))


def _state(pkg, fields, cuda, name, nx, ny, nz, h, dtype):
    import torch
    inputs = fields.make_inputs(name, nx, ny, nz, seed=31, workload="physical", halo=h)
    dev = lambda v: pkg.Storage(torch.from_numpy(v.astype(np.float32).astype(dtype)).to(cuda), h,  # noqa: E731
                                nx=nx if v.ndim == 3 else None)
    rng = np.random.default_rng(37)
    shape = (nz + 2 * h, ny + 2 * h, nx + 2 * h)
    ybar = {n: dev(rng.normal(size=shape)) for n in pkg.KERNELS[name].semantic_outputs}
    xbar = {n: dev(np.full(shape, fields.SENTINEL)) for n in pkg.ACTIVE[name]}
    sc = {k: float(np.float32(v)) for k, v in fields.make_scalars(name, seed=31).items()}
    pkg.adjoint(name, {k: dev(v) for k, v in inputs.items()}, ybar, xbar, sc, domain=(nx, ny, nz))
    torch.cuda.synchronize()
    return {n: s.numpy().astype(np.float64) for n, s in xbar.items()}


@pytest.mark.parametrize("size", SIZES, ids=["x".join(map(str, s)) for s in SIZES])
@pytest.mark.parametrize("name", ("fvtp2d", "fastwavesuv", "hdiffsmag"))
def test_marching_adjoint_matches_fp64(pkg, fields, cuda, name, size):
    """The FP32 adjoint against the FP64 one on the same (FP32) inputs and seeds.  About forty roundings
    of 6e-8 enter a gradient cell, on terms no larger than a few times the largest gradient: 1e-5
    of it bounds their sum.  A monotonicity flag decided within a rounding of zero may differ: with
    |m|, |r| of order 0.05 and values of order 1 that is about 1e-5 of the flags, six cells each."""
    nx, ny, nz, h, _ = size
    got = _state(pkg, fields, cuda, name, nx, ny, nz, h, np.float32)
    want = _state(pkg, fields, cuda, name, nx, ny, nz, h, np.float64)
    reach = {a.name: a.reach for a in pkg.KERNELS[name].args}
    for n in want:
        ilo, ihi, jlo, jhi, klo, khi = reach[n]
        box = (slice(h - klo, h + nz + khi), slice(h - jlo, h + ny + jhi), slice(h - ilo, h + nx + ihi))
        off = np.ones(want[n].shape, dtype=bool)
        off[box] = False
        assert (got[n][off] == fields.SENTINEL).all(), "%s: %sb written outside its box" % (name, n)
        err = np.abs(got[n][box] - want[n][box])
        assert np.isfinite(got[n][box]).all()
        bad = np.count_nonzero(err > 1e-5 * np.abs(want[n][box]).max())
        assert bad <= 8 + 1e-3 * err.size, "%s: %d of %d cells of %sb differ" % (name, bad, err.size, n)
