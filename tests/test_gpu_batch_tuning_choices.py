"""What the batch autotuner chooses among: a launch that no k-blocking changes is timed once, and the
fastwavesuv adjoint's own levels a chunk, more than any k-blocking's, are among the candidates."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_batch import _member

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def chain(pkg):
    import importlib
    return importlib.import_module("oeb_gb300.chain")


def test_launches_without_a_k_blocking(pkg, fields, chain, cuda):
    """The FP32 forward step marches one level a CTA but for the update: the first candidate stands."""
    members = [_member(pkg, fields, chain, cuda, nx, 48, 20, np.float32, 113 + nx) for nx in (48, 64, 80)]
    plan = chain.BatchPlan(members, chain.FORWARD)
    for _ in range(3):
        plan.autotune()
        kbs = [kb for kb, _, _ in plan.tuning()]
        assert sum(kb == 1 for kb in kbs) >= len(kbs) - 1, kbs
    plan.close()


@pytest.mark.parametrize("dtype", (np.float32, np.float64), ids=("f32", "f64"))
def test_long_chunks_give_the_same_bits(pkg, fields, chain, cuda, dtype):
    """A domain whose fastwavesuv adjoint takes 11 or 14 levels a chunk by itself: recorded with
    k-blocking 8, which stands for those, with 1 and by default."""
    import torch
    m = _member(pkg, fields, chain, cuda, 128, 128, 40, dtype, 127)
    plan = chain.BatchPlan([m], chain.FORWARD | chain.ADJOINT)
    plan.run()
    torch.cuda.synchronize()
    want = {n: s.numpy().copy() for n, s in m["grads"].items()}
    n = len(plan.tuning())
    for kb in (8, 1, 8):
        plan.apply_tuning([(kb, 0, 0)] * n)
        for s in m["grads"].values():
            s.data.fill_(0)
        plan.run()
        torch.cuda.synchronize()
        for g, s in m["grads"].items():
            np.testing.assert_array_equal(s.numpy()[8:-8, 8:-8, 8:-8], want[g][8:-8, 8:-8, 8:-8], err_msg=g)
    plan.close()
