"""The time budget of a sweep's waits (gpu): it limits the time without
progress. A warp whose operands keep arriving, each well inside the budget,
does not run out however long it waits for all of them."""
import time

import numpy as np
import pytest

from apxchol_b200 import native
from apxchol_b200.refsetup import Factor

pytestmark = pytest.mark.gpu

ROWS = 2000   # fewer than the resident warps: nearly every row is waited for from the start


@pytest.fixture(scope="module")
def eng():
    import torch
    torch.cuda.init()
    e = native.Engine(0)
    yield e
    e.close()


def staircase(direction):
    """One row a level. Row i (in the direction's order) needs the row before it and rows i/8, 2i/8, ... 7i/8, so
    that a waiting row sees an operand arrive every eighth of the time up to its turn."""
    n = ROWS
    cols = [[] for _ in range(n)]
    for i in range(1, n):
        for d in sorted({i - 1} | {i * q // 8 for q in range(1, 8)}):
            if direction == 0:
                cols[d].append(i)
            else:
                cols[n - 1 - i].append(n - 1 - d)
    ptr, idx, val = [0], [], []
    for j in range(n):
        idx += [j] + sorted(cols[j])
        val += [1.0 + len(cols[j])] + [-0.5] * len(cols[j])
        ptr.append(len(idx))
    return Factor(n=n, colptr=np.array(ptr, np.uint32), rowidx=np.array(idx, np.uint32), vals=np.array(val, np.float32),
                  perm=np.arange(n, dtype=np.uint32), sddm=True, rounds=np.ones(n, np.uint64))


@pytest.mark.parametrize("limit", ["0", None])                     # dataflow kernels alone; cluster tail
@pytest.mark.parametrize("direction", [0, 1])
@pytest.mark.parametrize("precision", [native.PREC_FP64, native.PREC_FP32])
def test_a_wait_that_progresses_does_not_run_out(eng, precision, direction, limit, monkeypatch):
    import torch
    if limit is not None:
        monkeypatch.setenv("APXB_SEG_LEVEL_ROWS", limit)
    D = native.DeviceFactor(eng, staircase(direction), drop_rel=0.0, precision=precision)
    x = torch.randn(ROWS, dtype=torch.float64, device="cuda")
    z = torch.empty_like(x)
    torch.cuda.synchronize()

    def sweep():
        t = time.perf_counter()
        D.sweep(direction, x, z)
        eng.sync()
        return time.perf_counter() - t

    took = min(sweep() for _ in range(4))
    want = z.clone()
    # operands come an eighth of the sweep apart (a quarter where the early rows are slowed by all the others'
    # polls); the last row waits for nearly all of it
    eng.set_spin_budget(int(0.45 * took * 1e9))
    try:
        for _ in range(3):
            sweep()
            assert torch.equal(z, want)
    finally:
        eng.set_spin_budget(2_000_000_000)
