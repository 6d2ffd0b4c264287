"""The marching FP32 kernels (csrc/march.cuh) with the rows a warp takes and the strips a CTA holds
forced: short and long chunks, one row, chunks of 32 rows and one beside it (where the metric terms
held one a lane are read anew), remainders.  Domains small enough to compare would choose four rows
by themselves; large ones choose up to 64.  Every form is held to the bits of another one: the
forward kernels to the float oracle or the plain kernels, the adjoints to the passes with their
terms in scratch, fvtp2d's to the same passes in numpy."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

import fvtp2d_adjoint

pytestmark = pytest.mark.gpu

H = 3
NX, NY, NZ = 59, 150, 2  # strips of 22 to 32 columns and chunks of rows that leave a remainder
SHAPES = [(1, 0), (5, 1), (31, 2), (32, 3), (33, 0), (37, 1), (64, 2), (64, 3), (32, 0)]
IDS = ["%drows-%dstrips" % (r, 1 << w) for r, w in SHAPES]


@pytest.fixture
def march_shape(pkg):
    lib = pkg.load_library()

    def force(rows, wx_log):
        assert lib.oeb_selftest_march_shape(ctypes.c_int(rows), ctypes.c_int(wx_log)) == 0

    yield force
    force(0, 0)


def _scalars32(fields, name, seed):
    return {k: float(np.float32(v)) for k, v in fields.make_scalars(name, seed=seed).items()}


@pytest.mark.parametrize("shape", SHAPES, ids=IDS)
@pytest.mark.parametrize("name", ("fvtp2d", "hadvuv", "hadvuv5th", "hdiffsa", "hdiffsmag", "fastwavesuv"))
def test_forward_is_the_float_oracle(pkg, fields, orc, cuda, march_shape, name, shape):
    import torch
    spec = pkg.KERNELS[name]
    inputs = fields.make_inputs(name, NX, NY, NZ, seed=73, workload="fronts", halo=H)
    sc = _scalars32(fields, name, 73)
    want = {k: v.astype(np.float32) for k, v in {**inputs, **fields.make_outputs(name, NX, NY, NZ, halo=H)}.items()}
    dev = {k: pkg.Storage(torch.from_numpy(v.copy()).to(cuda), H, nx=NX if v.ndim == 3 else None)
           for k, v in want.items()}
    orc.run_oracle(spec, want, sc, NX, NY, NZ, H)
    march_shape(*shape)
    pkg.call(name, dev, sc, domain=(NX, NY, NZ))
    torch.cuda.synchronize()
    for a in spec.by_role("out3"):
        np.testing.assert_array_equal(dev[a.name].numpy().view(np.uint32), want[a.name].view(np.uint32), err_msg=a.name)


@pytest.mark.parametrize("shape", SHAPES, ids=IDS)
@pytest.mark.parametrize("name", ("p_grad_c", "nh_p_grad"))
def test_forward_is_the_plain_kernel(pkg, fields, cuda, march_shape, name, shape):
    """Where the fields lie in host memory the plain kernels run."""
    import torch
    inputs = fields.make_inputs(name, NX, NY, NZ, seed=79, workload="fronts", halo=H)
    sc = _scalars32(fields, name, 79)
    arrays = {k: v.astype(np.float32)
              for k, v in {**inputs, **fields.make_outputs(name, NX, NY, NZ, halo=H)}.items()}
    host = {k: pkg.Storage(torch.from_numpy(v.copy()).pin_memory(), H, nx=NX) for k, v in arrays.items()}
    dev = {k: pkg.Storage(torch.from_numpy(v.copy()).to(cuda), H, nx=NX) for k, v in arrays.items()}
    pkg.call(name, host, sc, domain=(NX, NY, NZ))
    march_shape(*shape)
    pkg.call(name, dev, sc, domain=(NX, NY, NZ))
    torch.cuda.synchronize()
    for a in pkg.KERNELS[name].by_role("out3"):
        np.testing.assert_array_equal(dev[a.name].numpy().view(np.uint32), host[a.name].numpy().view(np.uint32),
                                      err_msg=a.name)


def _adjoint(pkg, fields, cuda, name, nx, ny, nz, seed):
    """xbar of an FP32 adjoint, and its inputs."""
    import torch
    x = {k: v.astype(np.float32)
         for k, v in fields.make_inputs(name, nx, ny, nz, seed=seed, workload="fronts", halo=H).items()}
    sc = _scalars32(fields, name, seed)
    rng = np.random.default_rng(seed + 1)
    shape = (nz + 2 * H, ny + 2 * H, nx + 2 * H)
    ybar = {n: rng.normal(size=shape).astype(np.float32) for n in pkg.KERNELS[name].semantic_outputs}
    dev = lambda v: pkg.Storage(torch.from_numpy(v.copy()).to(cuda), H, nx=nx if v.ndim == 3 else None)  # noqa: E731
    xbar = {n: dev(np.full(shape, np.float32(fields.SENTINEL))) for n in pkg.ACTIVE[name]}
    pkg.adjoint(name, {k: dev(v) for k, v in x.items()}, {k: dev(v) for k, v in ybar.items()}, xbar, sc,
                domain=(nx, ny, nz))
    torch.cuda.synchronize()
    return {n: s.numpy() for n, s in xbar.items()}, x, ybar, sc


@pytest.mark.parametrize("shape", SHAPES, ids=IDS)
def test_hdiffsmag_adjoint_is_the_passes(pkg, fields, cuda, march_shape, shape):
    lib = pkg.load_library()
    march_shape(*shape)
    got = _adjoint(pkg, fields, cuda, "hdiffsmag", NX, NY, NZ, 83)[0]
    try:
        assert lib.oeb_set_adjoint_tiles(ctypes.c_int(0)) == 0
        want = _adjoint(pkg, fields, cuda, "hdiffsmag", NX, NY, NZ, 83)[0]
    finally:
        lib.oeb_set_adjoint_tiles(ctypes.c_int(1))
    for n in want:
        np.testing.assert_array_equal(got[n].view(np.uint32), want[n].view(np.uint32), err_msg=n)


@pytest.mark.parametrize("kb", (1, 2, 7, 25, 40, 64))
def test_fastwavesuv_adjoint_is_the_passes(pkg, fields, cuda, kb):
    """The march over levels: every split of 40 of them (and the two beyond) is the same bits."""
    lib = pkg.load_library()
    got = {}
    try:
        assert lib.oeb_set_kblock(ctypes.c_int(kb)) == 0
        for one in (1, 0):
            assert lib.oeb_set_adjoint_tiles(ctypes.c_int(one)) == 0
            got[one] = _adjoint(pkg, fields, cuda, "fastwavesuv", 61, 19, 40, 89)[0]
    finally:
        lib.oeb_set_adjoint_tiles(ctypes.c_int(1))
        lib.oeb_set_kblock(ctypes.c_int(0))
    for n in got[1]:
        np.testing.assert_array_equal(got[1][n].view(np.uint32), got[0][n].view(np.uint32), err_msg=n)


def _fvtp2d_adjoint_is_the_passes(pkg, fields, orc, cuda, nx, ny, nz, seed):
    got, x, ybar, sc = _adjoint(pkg, fields, cuda, "fvtp2d", nx, ny, nz, seed)
    fwd = {**{k: v.copy() for k, v in x.items()},
           **{k: v.astype(np.float32) for k, v in fields.make_outputs("fvtp2d", nx, ny, nz, halo=H).items()}}
    orc.run_oracle(pkg.KERNELS["fvtp2d"], fwd, sc, nx, ny, nz, H)
    with np.errstate(all="ignore"):
        want = fvtp2d_adjoint.adjoint(x, fwd["q_i"], fwd["q_j"], ybar["fx1"], ybar["fy1"], nx, ny, sc["p1"], sc["p2"])
    want[:H] = want[H + nz:] = fields.SENTINEL
    np.testing.assert_array_equal(got["q"], want)


@pytest.mark.parametrize("shape", SHAPES, ids=IDS)
def test_fvtp2d_adjoint_is_the_passes(pkg, fields, orc, cuda, march_shape, shape):
    march_shape(*shape)
    _fvtp2d_adjoint_is_the_passes(pkg, fields, orc, cuda, NX, NY, NZ, 97)


# the smallest boxes, a strip's width (22 and 26 columns) and beside it, and the split large domains choose
SIZES = [(1, 1, 1), (5, 3, 2), (16, 4, 3), (17, 5, 2), (22, 7, 1), (23, 33, 2), (26, 9, 2), (27, 31, 2), (38, 65, 1),
         (127, 70, 3), (209, 17, 2), (256, 256, 80)]


@pytest.mark.parametrize("size", SIZES, ids=["x".join(map(str, s)) for s in SIZES])
def test_fvtp2d_adjoint_sizes(pkg, fields, orc, cuda, size):
    _fvtp2d_adjoint_is_the_passes(pkg, fields, orc, cuda, *size, 101)


@pytest.mark.parametrize("size", [(1, 1, 1), (5, 3, 2), (26, 4, 3), (31, 9, 2), (256, 256, 80), (320, 304, 20)],
                         ids=["1x1x1", "5x3x2", "26x4x3", "31x9x2", "256x256x80", "320x304x20"])
@pytest.mark.parametrize("name", ("hdiffsmag", "fastwavesuv"))
def test_adjoint_sizes(pkg, fields, cuda, name, size):
    lib = pkg.load_library()
    got = _adjoint(pkg, fields, cuda, name, *size, 103)[0]
    try:
        assert lib.oeb_set_adjoint_tiles(ctypes.c_int(0)) == 0
        want = _adjoint(pkg, fields, cuda, name, *size, 103)[0]
    finally:
        lib.oeb_set_adjoint_tiles(ctypes.c_int(1))
    for n in want:
        np.testing.assert_array_equal(got[n].view(np.uint32), want[n].view(np.uint32), err_msg=n)


def test_shape_limits(pkg, march_shape):
    lib = pkg.load_library()
    for rows, wx in ((-1, 0), (65, 0), (8, -1), (8, 4)):
        assert lib.oeb_selftest_march_shape(ctypes.c_int(rows), ctypes.c_int(wx)) != 0
