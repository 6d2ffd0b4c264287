"""Fields in host memory that the device reads in place: the kernels and splits taken there, on both
sides of the sizes where they change (fewer 32 x 32 tiles than SMs; a wave of 16-row tiles), give the
device call's bits."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1, 3), (5, 3, 2, 3), (33, 20, 10, 4), (48, 40, 20, 3), (64, 64, 60, 3), (70, 97, 9, 3), (130, 67, 31, 4)]


@pytest.mark.parametrize("size", SIZES, ids=["x".join(map(str, s)) for s in SIZES])
@pytest.mark.parametrize("dtype", (np.float32, np.float64), ids=("f32", "f64"))
@pytest.mark.parametrize("name", ("laplace", "hdiffsa", "hdiffsmag", "hadvuv", "hadvuv5th", "fastwavesuv", "uvbke",
                                  "nh_p_grad", "p_grad_c", "fvtp2d"))
def test_in_place_is_the_device_call(pkg, fields, cuda, name, dtype, size):
    import torch
    nx, ny, nz, h = size
    sc = {k: float(np.float32(v)) for k, v in fields.make_scalars(name, seed=107).items()}
    arrays = {k: v.astype(dtype) for k, v in
              {**fields.make_inputs(name, nx, ny, nz, seed=107, workload="fronts", halo=h),
               **fields.make_outputs(name, nx, ny, nz, halo=h)}.items()}
    assert pkg.load_library().oeb_set_host_direct(1) == 0
    host = {k: pkg.Storage(torch.from_numpy(v.copy()).pin_memory(), h, nx=nx if v.ndim == 3 else None)
            for k, v in arrays.items()}
    dev = {k: pkg.Storage(torch.from_numpy(v.copy()).to(cuda), h, nx=nx if v.ndim == 3 else None)
           for k, v in arrays.items()}
    pkg.call(name, host, sc, domain=(nx, ny, nz))
    pkg.call(name, dev, sc, domain=(nx, ny, nz))
    torch.cuda.synchronize()
    word = np.uint32 if dtype == np.float32 else np.uint64
    for a in pkg.KERNELS[name].by_role("out3"):
        np.testing.assert_array_equal(host[a.name].numpy().view(word), dev[a.name].numpy().view(word), err_msg=a.name)
