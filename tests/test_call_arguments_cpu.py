"""What a call hands to the library, with the library replaced by a recorder: scalars in every form
that ``dict.update`` takes, the tables of defaults and active inputs as they are at the call, and the
descriptors of a Storage subclass."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

H = 3


@pytest.fixture
def calls(pkg, monkeypatch):
    import importlib
    kernels = importlib.import_module("oeb_gb300.kernels")
    seen = []
    monkeypatch.setattr(kernels, "entry", lambda name: lambda *args: seen.append((name, args)) or 0)
    monkeypatch.setattr(kernels, "_device_fields", lambda kernel, flat: "f64")
    monkeypatch.setattr(kernels, "_current_stream", lambda: 0)
    return seen


def _fields(pkg, kernel, names, cls=None):
    one = {a.name for a in pkg.KERNELS[kernel].args if a.role == "in1"}
    cls = cls or pkg.Storage
    return {n: cls(np.zeros((11,) if n in one else (11, 11, 11)), H) for n in names}


def _scalars(args):
    return [a.value for a in args if isinstance(a, (ctypes.c_double, ctypes.c_float))]


@pytest.mark.parametrize("form", ["dict", "pairs", "mapping", "none"])
def test_scalars_in_every_form(pkg, calls, form):
    from types import MappingProxyType
    mine = {"p1": 0.25}
    scalars = {"dict": mine, "pairs": list(mine.items()), "mapping": MappingProxyType(mine), "none": None}[form]
    names = [a.name for a in pkg.KERNELS["fvtp2d"].abi_args]
    pkg.call("fvtp2d", _fields(pkg, "fvtp2d", names), scalars, domain=(5, 5, 5))
    defaults = pkg.DRIVER_SCALARS["fvtp2d"]
    assert _scalars(calls[0][1]) == [defaults["p1"] if form == "none" else 0.25, defaults["p2"]]


def test_defaults_are_read_at_the_call(pkg, calls, monkeypatch):
    names = [a.name for a in pkg.KERNELS["fvtp2d"].abi_args]
    f = _fields(pkg, "fvtp2d", names)
    pkg.call("fvtp2d", f, domain=(5, 5, 5))
    monkeypatch.setitem(pkg.DRIVER_SCALARS, "fvtp2d", {"p1": 0.5, "p2": 0.125})
    pkg.call("fvtp2d", f, domain=(5, 5, 5))
    assert _scalars(calls[1][1]) == [0.5, 0.125]


def test_active_inputs_are_read_at_the_call(pkg, calls, monkeypatch):
    names = [a.name for a in pkg.KERNELS["laplace"].args]
    f = _fields(pkg, "laplace", names)
    pkg.adjoint("laplace", f, f, f, domain=(5, 5, 5))
    monkeypatch.setitem(pkg.ACTIVE, "laplace", ("out",))
    with pytest.raises(KeyError):
        pkg.adjoint("laplace", f, f, {"in": f["in"]}, domain=(5, 5, 5))


def test_a_subclass_describes_itself(pkg, calls):
    class Shifted(pkg.Storage):
        def memref(self):
            m = super().memref()
            m.offset += 1
            return m

    class Late(pkg.Storage):  # a constructor of its own, and an address of its own
        def __init__(self, data, halo):
            self.data, self.halo, self.rank = data, halo, data.ndim
            self.dtype, self.szi, self.pitch = data.dtype, data.shape[-1], data.shape[-1]

        def data_ptr(self):
            return super().data_ptr() + 8

    names = [a.name for a in pkg.KERNELS["laplace"].abi_args]
    plain = _fields(pkg, "laplace", names)
    for cls in (Shifted, Late):
        f = {n: cls(s.data, H) for n, s in plain.items()}
        for _ in range(2):
            pkg.call("laplace", f, domain=(5, 5, 5))
            for n, arg in zip(names, calls[-1][1]):
                m, p = arg._obj, plain[n].memref()
                assert m.offset == p.offset + (cls is Shifted)
                assert m.aligned == p.aligned + 8 * (cls is Late)
