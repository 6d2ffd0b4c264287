"""Storage.packed(): the kept descriptor is the one memref() builds, and is built again when the
buffer, its shape, the halo or the row length is another."""
from __future__ import annotations

import numpy as np
import pytest


def _same(a, b):
    names = [n for n, _ in a._fields_]
    return all((list(getattr(a, n)) if n in ("sizes", "strides") else getattr(a, n)) ==
               (list(getattr(b, n)) if n in ("sizes", "strides") else getattr(b, n)) for n in names)


@pytest.mark.parametrize("kind", ["numpy", "torch"])
@pytest.mark.parametrize("shape", [(7, 9, 12), (11,)])
def test_packed_follows_the_buffer(pkg, kind, shape):
    torch = pytest.importorskip("torch")
    new = (lambda s: np.zeros(s, np.float32)) if kind == "numpy" else (lambda s: torch.zeros(s))
    st = pkg.Storage(new(shape), 2, nx=6 if len(shape) == 3 else None)
    m, _ = st.packed()
    assert _same(m, st.memref()) and st.packed()[0] is m
    keep = st.data
    st.data = new(shape)
    assert st.packed()[0] is not m and _same(st.packed()[0], st.memref())
    st.data = new(tuple(n + 3 for n in shape))
    assert _same(st.packed()[0], st.memref())
    st.data, st.halo = keep, 1
    assert _same(st.packed()[0], st.memref())
    if len(shape) == 3:
        st.szi = shape[2]
        assert _same(st.packed()[0], st.memref()) and list(st.packed()[0].sizes)[2] == shape[2]
