"""Infinite and undefined parameters in the FP32 adjoints: a product with a term that is exactly zero,
or that the transpose has no place for, is not formed, so such a parameter reaches only the cells
that its own terms reach."""
from __future__ import annotations

import numpy as np
import pytest

H = 3
pytestmark = pytest.mark.gpu


def _adjoint(pkg, cuda, name, inputs, ybar, sc, nx, ny, nz, fill):
    import torch
    dev = lambda v: pkg.Storage(torch.from_numpy(v.astype(np.float32)).to(cuda), H,  # noqa: E731
                                nx=nx if v.ndim == 3 else None)
    shape = (nz + 2 * H, ny + 2 * H, nx + 2 * H)
    xbar = {n: dev(np.full(shape, fill)) for n in pkg.ACTIVE[name]}
    pkg.adjoint(name, {k: dev(v) for k, v in inputs.items()}, {k: dev(v) for k, v in ybar.items()}, xbar, sc,
                domain=(nx, ny, nz))
    torch.cuda.synchronize()
    return {n: s.numpy() for n, s in xbar.items()}


@pytest.mark.parametrize("value", (np.inf, -np.inf, np.nan), ids=("inf", "-inf", "nan"))
@pytest.mark.parametrize("field", ("crx", "cry"))
def test_fvtp2d_courant_numbers_where_no_seed_enters(pkg, fields, cuda, field, value):
    """Seeds in the western half only; the Courant numbers that are not finite lie beyond the reach of
    the terms these give (5 cells a sweep, two sweeps and one face): every gradient is the one with
    finite numbers there."""
    nx, ny, nz = 61, 40, 2
    inputs = fields.make_inputs("fvtp2d", nx, ny, nz, seed=53, workload="fronts", halo=H)
    sc = fields.make_scalars("fvtp2d", seed=53)
    rng = np.random.default_rng(59)
    shape = (nz + 2 * H, ny + 2 * H, nx + 2 * H)
    ybar = {n: rng.normal(size=shape) for n in pkg.KERNELS["fvtp2d"].semantic_outputs}
    for v in ybar.values():
        v[..., H + nx // 2:] = 0.0
    want = _adjoint(pkg, cuda, "fvtp2d", inputs, ybar, sc, nx, ny, nz, fields.SENTINEL)
    bad = rng.random(shape) < 0.05
    bad[..., :H + nx // 2 + 12] = False
    inputs[field][bad] = value
    got = _adjoint(pkg, cuda, "fvtp2d", inputs, ybar, sc, nx, ny, nz, fields.SENTINEL)
    assert np.isfinite(want["q"]).all()
    np.testing.assert_array_equal(got["q"], want["q"])


@pytest.mark.parametrize("value", (np.inf, np.nan), ids=("inf", "nan"))
@pytest.mark.parametrize("field", ("crlato", "crlatu", "crlavo", "crlavu", "acrlat0"))
@pytest.mark.parametrize("size", [(37, 29, 3), (28, 70, 2), (5, 3, 2)], ids=["37x29x3", "28x70x2", "5x3x2"])
def test_hdiffsmag_metric_terms(pkg, fields, cuda, size, field, value):
    """A latitude whose metric term is not finite (the first, the last, one between): the one-launch
    adjoint gives what the passes with their terms in scratch give, which skip the points off the
    interior."""
    import ctypes
    nx, ny, nz = size
    inputs = fields.make_inputs("hdiffsmag", nx, ny, nz, seed=61, workload="fronts", halo=H)
    sc = {k: float(np.float32(v)) for k, v in fields.make_scalars("hdiffsmag", seed=61).items()}
    rng = np.random.default_rng(67)
    ybar = {n: rng.normal(size=(nz + 2 * H, ny + 2 * H, nx + 2 * H)) for n in ("uout", "vout")}
    lib = pkg.load_library()
    for row in sorted({0, ny // 2, ny - 1}):
        odd = {**inputs, field: inputs[field].copy()}
        odd[field][H + row] = value
        got = {}
        try:
            for one in (1, 0):
                assert lib.oeb_set_adjoint_tiles(ctypes.c_int(one)) == 0
                got[one] = _adjoint(pkg, cuda, "hdiffsmag", odd, ybar, sc, nx, ny, nz, fields.SENTINEL)
        finally:
            lib.oeb_set_adjoint_tiles(ctypes.c_int(1))
        for n in ("uin", "vin"):
            np.testing.assert_array_equal(got[1][n], got[0][n], err_msg="%sb, row %d" % (n, row))
