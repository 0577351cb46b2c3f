"""The cluster tail of the sweeps (gpu): the narrow last levels of a factor are
solved by one thread-block cluster from shared memory, the others by the
dataflow kernels. Where the two meet, and at rows shorter and longer than a
batch of operands, the fp64 pair stays the reference's bytes and the fp32
sweeps stay within the rounding of their sums."""
import numpy as np
import pytest

from apxchol_b200 import native
from apxchol_b200.gen import Matrix
from apxchol_b200.refsetup import Factor

import oracle

pytestmark = pytest.mark.gpu



def fp32_rtol(shape):
    """fp32 sums of up to `reach` products in any order beside three more roundings (right-hand side, subtraction,
    division), two sweeps: 2 * (reach + 3) * 2^-24 of the absolute sums bounds the relative error of a row; the rows
    are diagonally dominant (off-diagonals sum to at most half the diagonal), so the sweeps do not amplify it by more
    than 2 each."""
    return 4 * 2 * (SHAPES[shape][1] + 3) * 2.0 ** -24



@pytest.fixture(scope="module")
def eng():
    import torch
    torch.cuda.init()
    e = native.Engine(0)
    yield e
    e.close()


def layered(widths, reach, seed, sddm=True):
    """A factor whose levels have the given widths: every row depends on a row of the level before it and on up
    to reach - 1 more of any earlier level."""
    rng = np.random.default_rng(seed)
    bounds = np.concatenate([[0], np.cumsum(widths)])
    m = int(bounds[-1])
    n = m if sddm else m + 1
    cols = [[] for _ in range(m)]
    for lv in range(1, len(widths)):
        for r in range(bounds[lv], bounds[lv + 1]):
            deps = {int(rng.integers(bounds[lv - 1], bounds[lv]))}
            deps.update(int(q) for q in rng.integers(0, bounds[lv], size=min(reach - 1, 4 * int(bounds[lv]))))
            for j in deps:
                cols[j].append(r)
    ptr, idx, val = [0], [], []
    for j in range(m):
        rows = sorted(cols[j]) + ([] if sddm else [m])
        w = rng.uniform(0.1, 1.0, size=len(rows))
        idx += [j] + rows
        val += [2.0 * max(w.sum(), 1.0)] + list(-w)
        ptr.append(len(idx))
    if not sddm:
        idx.append(m); val.append(1.0); ptr.append(len(idx))
    fac = Factor(n=n, colptr=np.array(ptr, np.uint32), rowidx=np.array(idx, np.uint32), vals=np.array(val, np.float32),
                 perm=rng.permutation(n).astype(np.uint32), sddm=sddm, rounds=np.array(widths, np.uint64))
    eye = Matrix(n=n, colptr=np.arange(n + 1, dtype=np.int32), rowidx=np.arange(n, dtype=np.int32), vals=np.ones(n))
    return eye, fac


SHAPES = {
    "all_in_the_tail": ([5, 3, 2, 1, 1], 4),
    "too_few_levels": ([901, 300, 2, 1], 6),
    "levels_at_the_limit": ([701, 513, 512, 512, 33, 17, 16, 9, 8, 5, 4, 3, 2, 1], 9),
    "wide_then_narrow": ([6000, 2000, 400, 31, 1, 1, 1, 30, 12, 1, 2, 3], 40),
    "rows_over_a_batch": ([800, 300, 20, 3, 1, 1, 2, 1, 1], 700),
    "a_chain": ([1] * 300, 1),
}


@pytest.mark.parametrize("limit", [None, "0", "4096"])
@pytest.mark.parametrize("shape", list(SHAPES))
def test_sweeps_through_the_tail(eng, shape, limit, monkeypatch):
    import torch
    if limit is not None:
        monkeypatch.setenv("APXB_SEG_LEVEL_ROWS", limit)
    A, F = layered(*SHAPES[shape], seed=len(shape), sddm=len(shape) % 2 == 0)
    x = np.random.default_rng(9).standard_normal(F.m)
    want = oracle.Oracle(A, F).pair(x)
    D = native.DeviceFactor(eng, F)
    assert np.array_equal(D.sweep_pair_host(x), want)
    assert np.array_equal(D.sweep_pair_host(x), want)        # the buffers are armed again
    D32 = native.DeviceFactor(eng, F, precision=native.PREC_FP32)
    one = D32.sweep_pair_host(x)
    assert np.linalg.norm(one - want) <= fp32_rtol(shape) * np.linalg.norm(want)
    for k in (2, 4, 8, 16):                                   # a column does not depend on the others
        X = np.random.default_rng(k).standard_normal((F.m, k))
        X[:, k - 1] = x
        dX = torch.from_numpy(X).cuda()
        dZ = torch.empty_like(dX)
        torch.cuda.synchronize()
        D32.sweep_pair_multi(k, dX, dZ)
        eng.sync()
        assert np.array_equal(dZ.cpu().numpy()[:, k - 1], one), k


@pytest.mark.parametrize("limit", [None, "0"])
@pytest.mark.parametrize("shape", ["levels_at_the_limit", "wide_then_narrow", "rows_over_a_batch"])
def test_the_sweep_grid_sizes_the_clusters_and_not_the_bits(eng, shape, limit, monkeypatch):
    """From one block a column slice (1, 2 and 4 of them at k = 1, 2 and 4) to clusters of 16; without tails, from
    one block to the resident grid."""
    import torch
    if limit is not None:
        monkeypatch.setenv("APXB_SEG_LEVEL_ROWS", limit)
    _, F = layered(*SHAPES[shape], seed=7)
    D = native.DeviceFactor(eng, F)
    D32 = native.DeviceFactor(eng, F, precision=native.PREC_FP32)
    D16 = native.DeviceFactor(eng, F, precision=native.PREC_FP16)
    x = {k: torch.from_numpy(np.random.default_rng(k).standard_normal((F.m, k))).cuda() for k in (1, 2, 4, 16)}

    def pairs():
        out = []
        for k in x:
            z = torch.empty_like(x[k])
            torch.cuda.synchronize()
            D32.sweep_pair_multi(k, x[k], z)
            eng.sync()
            out.append(z)
        for one in (D, D16):
            z = torch.empty_like(x[1])
            torch.cuda.synchronize()
            one.sweep_pair(x[1], z)
            eng.sync()
            out.append(z)
        return out

    want = pairs()
    try:
        for grid in (1, 3, 7, 8, 31, 64):
            eng.set_sweep_grid(grid)
            for got, ref in zip(pairs(), want):
                assert torch.equal(got, ref), (grid, got.shape)
    finally:
        eng.set_sweep_grid(0)


@pytest.mark.parametrize("limit", [None, "0"])
@pytest.mark.parametrize("shape", list(SHAPES))
def test_fp16_sweeps_through_the_tail(eng, shape, limit, monkeypatch):
    """Each sweep over the stored binary16 values against the same sweep in fp64, and the columns of a block."""
    import torch
    if limit is not None:
        monkeypatch.setenv("APXB_SEG_LEVEL_ROWS", limit)
    _, F = layered(*SHAPES[shape], seed=len(shape), sddm=len(shape) % 2 == 0)
    h = native.prepare_host_fp16(F, 0.0)
    D = native.DeviceFactor(eng, F, drop_rel=0.0, precision=native.PREC_FP16)
    x = np.random.default_rng(12).standard_normal(F.m).astype(np.float32)

    def run(fn, v):
        dv = torch.from_numpy(np.ascontiguousarray(v, np.float64)).cuda()
        dz = torch.empty_like(dv)
        torch.cuda.synchronize()
        fn(dv, dz)
        eng.sync()
        return dz.cpu().numpy()

    y = run(lambda a, b: D.sweep(0, a, b), x)
    want = oracle.sweep16(0, h, x)
    assert np.linalg.norm(y - want) <= fp32_rtol(shape) / 2 * np.linalg.norm(want)
    z = run(lambda a, b: D.sweep(1, a, b), y)
    want = oracle.sweep16(1, h, y.astype(np.float32), h["inv_scale"].astype(np.float64) ** 2)
    assert np.linalg.norm(z - want) <= fp32_rtol(shape) / 2 * np.linalg.norm(want)
    one = run(D.sweep_pair, x)
    for k in (2, 4, 8, 16):
        X = np.random.default_rng(k).standard_normal((F.m, k))
        X[:, 0] = x
        assert np.array_equal(run(lambda a, b: D.sweep_pair_multi(k, a, b), X)[:, 0], one), k


@pytest.mark.parametrize("limit", [None, "0"])
def test_infinities_and_nan_reach_the_rows_that_depend_on_them(eng, limit, monkeypatch):
    """In the first, a middle and the last rows of the elimination: the fp64 pair is the reference's (NaN by place),
    the fp32 and fp16 sweeps are finite, infinite and NaN in the same places."""
    if limit is not None:
        monkeypatch.setenv("APXB_SEG_LEVEL_ROWS", limit)
    A, F = layered(*SHAPES["wide_then_narrow"], seed=2)
    O = oracle.Oracle(A, F)
    Ds = {p: native.DeviceFactor(eng, F, precision=p) for p in (native.PREC_FP64, native.PREC_FP32, native.PREC_FP16)}
    for at in (0, F.m // 2, F.m - 90, F.m - 1):
        for bad in (np.inf, -np.inf, np.nan):
            x = np.random.default_rng(at).standard_normal(F.m)
            x[at] = bad
            with np.errstate(all="ignore"):
                want = O.pair(x)
            for p, D in Ds.items():
                got = D.sweep_pair_host(x)
                assert np.array_equal(np.isnan(got), np.isnan(want)), (at, bad, p)
                assert np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isneginf(got), np.isneginf(want))
                if p == native.PREC_FP64:
                    assert np.array_equal(got, want, equal_nan=True)
            x[at] = 1.0                                       # nothing of it stays behind
            assert np.array_equal(Ds[native.PREC_FP64].sweep_pair_host(x), O.pair(x))


@pytest.mark.parametrize("precision", ["FP32", "FP16"])
@pytest.mark.parametrize("shapes", [("levels_at_the_limit", "too_few_levels", "all_in_the_tail"),
                                    ("wide_then_narrow", "a_chain", "rows_over_a_batch")])
@pytest.mark.parametrize("k", [1, 2, 4, 8, 16, 32])
def test_batches_of_instances_with_and_without_tails(eng, k, shapes, precision):
    """Instances with a tail, without one and wholly inside theirs share a batch: each gives the bytes it gives alone.
    (Even sizes: with one column the vector passes sum elements in pairs from an even offset, so an instance that
    starts at an odd row has other partial sums than alone, whatever its sweeps.)"""
    made = [layered(*SHAPES[s], seed=3 + i) for i, s in enumerate(shapes)]
    Ds = [native.DeviceFactor(eng, F, precision=getattr(native, "PREC_" + precision)) for _, F in made]
    Ops = [native.DeviceOperator(eng, A, F.perm) for A, F in made]
    rhs = [np.random.default_rng(20 + i).standard_normal((k, F.n)) for i, (_, F) in enumerate(made)]
    bt = native.Batch(eng, Ds, Ops, k)
    xs, _ = bt.solve(rhs, tol=1e-10, max_iter=3)
    for i in range(len(made)):
        alone = native.Batch(eng, [Ds[i]], [Ops[i]], k)
        xa, _ = alone.solve([rhs[i]], tol=1e-10, max_iter=3)
        assert np.array_equal(xs[i], xa[0]), i
        assert np.isfinite(xs[i]).all()
