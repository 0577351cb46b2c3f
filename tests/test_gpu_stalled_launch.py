"""Failure detection in every launch of a pair of sweeps (gpu): a cluster tail
whose first level is never solved, and a dataflow launch whose first claim unit
is not, each end in APXB_ERR_TIMEOUT after the wait's budget, before or behind
the other launches of the pair; the next pair has the bits of the first."""
import numpy as np
import pytest

from apxchol_b200 import native
from tests.test_gpu_tail import SHAPES, layered

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    import torch
    torch.cuda.init()
    e = native.Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("precision,k", [("FP64", 1), ("FP32", 1), ("FP32", 8), ("FP32", 16), ("FP16", 1)])
@pytest.mark.parametrize("shape,tail", [("levels_at_the_limit", 1), ("levels_at_the_limit", 0), ("rows_over_a_batch", 1),
                                        ("wide_then_narrow", 0), ("a_chain", 1)])
def test_a_stalled_launch_ends_in_a_timeout(eng, shape, tail, precision, k):
    import torch
    _, F = layered(*SHAPES[shape], seed=5)
    D = native.DeviceFactor(eng, F, drop_rel=0.0, precision=getattr(native, "PREC_" + precision))
    x = torch.from_numpy(np.random.default_rng(1).standard_normal((F.m, k))).cuda()

    def pair():
        z = torch.empty_like(x)
        torch.cuda.synchronize()
        if k == 1:
            D.sweep_pair(x, z)
        else:
            D.sweep_pair_multi(k, x, z)
        eng.sync()
        return z

    want = pair()
    assert torch.isfinite(want).all()
    for direction in (0, 1):
        with pytest.raises(native.ApxbError) as ei:
            native.check(eng.lib.apxb_test_stalled_launch(eng.h, D.h, direction, k, tail, 20_000_000))   # 20 ms
        assert ei.value.code == native.ERR_TIMEOUT
        assert torch.equal(pair(), want), direction


def test_a_launch_that_is_not_there_is_refused(eng):
    _, F = layered(*SHAPES["all_in_the_tail"], seed=5)
    D = native.DeviceFactor(eng, F)
    assert eng.lib.apxb_test_stalled_launch(eng.h, D.h, 0, 1, 0, 1_000_000) == native.ERR_INVALID   # no dataflow launch
    _, F = layered(*SHAPES["too_few_levels"], seed=5)
    D = native.DeviceFactor(eng, F)
    assert eng.lib.apxb_test_stalled_launch(eng.h, D.h, 1, 1, 1, 1_000_000) == native.ERR_INVALID   # no tail
