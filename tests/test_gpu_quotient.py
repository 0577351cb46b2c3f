"""The sweeps' quotients (gpu): a row's last step is a division that the
kernels replace by products with a reciprocal formed ahead of the operands.
Factors of diagonal entries alone make a sweep that division and nothing else:
every result has the bits that IEEE division gives, over both ends of the
exponent ranges in which the short way is taken, and for zeros, subnormals,
infinities and NaN."""
import numpy as np
import pytest

from apxchol_b200 import native
from apxchol_b200.refsetup import Factor

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    import torch
    torch.cuda.init()
    e = native.Engine(0)
    yield e
    e.close()


def diagonal(d, widths):
    n = len(d)
    return Factor(n=n, colptr=np.arange(n + 1, dtype=np.uint32), rowidx=np.arange(n, dtype=np.uint32),
                  vals=d.astype(np.float32), perm=np.arange(n, dtype=np.uint32), sddm=True,
                  rounds=np.array(widths, np.uint64))


def widths_of(n, route):
    """Rounds of n rows: one wide level (dataflow kernels), or levels that the cluster tail takes, some of
    more and some of at most eight rows (one and several lanes a row)."""
    if route == "dataflow":
        return [n]
    w, cycle, left = [], (500, 9, 8, 33, 4, 1, 3, 2), n
    while left:
        w.append(min(left, cycle[len(w) % len(cycle)]))
        left -= w[-1]
    return w


# Biased exponents on both sides of the short way's limits (192 and 1873 for the fp64 dividend, 903 and 1143 for
# its fp32 divisor; 67 and 187, 87 and 167 in fp32), where a * l or a remainder would leave the normal range,
# where the result does, and the ordinary ones.
EXP64 = (0, 1, 52, 108, 122, 123, 124, 136, 148, 171, 191, 192, 193, 1022, 1023, 1872, 1873, 1874, 2046)
EXP32_OF_64 = (0, 1, 6, 7, 8, 126, 127, 245, 246, 247, 254)
EXP32 = (0, 1, 66, 67, 68, 127, 186, 187, 188, 254)
EXP32_DIV = (0, 1, 86, 87, 88, 127, 166, 167, 168, 254)


def mantissas(rng, bits, count):
    m = rng.integers(0, 1 << bits, size=count, dtype=np.uint64)
    m[:4] = (0, 1, (1 << bits) - 1, 1 << (bits - 1))
    return m


def pairs(ea, ed, bits, per, dtype, seed):
    rng = np.random.default_rng(seed)
    a, d = [], []
    word = np.uint64 if bits == 52 else np.uint32
    for x in ea:
        for y in ed:
            ma, md = mantissas(rng, bits, per), rng.permutation(mantissas(rng, 23, per))
            sign = rng.integers(0, 2, size=per).astype(np.uint64) << np.uint64(63 if bits == 52 else 31)
            a.append((sign | np.uint64(x << bits) | ma).astype(word).view(dtype))
            d.append((np.uint64(y << 23) | md).astype(np.uint32).view(np.float32))
    a, d = np.concatenate(a), np.concatenate(d)
    a[:6] = (0.0, -0.0, np.inf, -np.inf, np.nan, 1.0)
    d[d == 0] = 1.0
    return a, d


def same_bits(got, want):
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    bad = np.flatnonzero(got[~nan].view(np.int64) != want[~nan].view(np.int64))
    assert bad.size == 0, (bad.size, got[~nan][bad[:4]], want[~nan][bad[:4]])


def sweeps(eng, D, x):
    import torch
    dx = torch.from_numpy(x).cuda()
    dy = torch.empty_like(dx)
    torch.cuda.synchronize()
    for direction in (0, 1):
        D.sweep(direction, dx, dy)
        eng.sync()
        yield dy.cpu().numpy()


@pytest.mark.parametrize("route", ["dataflow", "tail"])
def test_fp64_quotients_are_the_divisions(eng, route):
    a, d = pairs(EXP64, EXP32_OF_64, 52, 96, np.float64, 1)
    # quotients just above the subnormal range, whose correction term would be subnormal
    a[6:8] = float.fromhex("0x1.c4db8e4f939e6p-900"), float.fromhex("0x1.ae5c58b12db15p-900")
    d[6:8] = float.fromhex("0x1.e02d0cp+119"), float.fromhex("0x1.f6fafap+119")
    D = native.DeviceFactor(eng, diagonal(d, widths_of(len(d), route)))
    with np.errstate(all="ignore"):
        want = a / d.astype(np.float64)
    for got in sweeps(eng, D, a):
        same_bits(got, want)


@pytest.mark.parametrize("route", ["dataflow", "tail"])
def test_fp32_quotients_are_the_divisions(eng, route):
    a, d = pairs(EXP32, EXP32_DIV, 23, 120, np.float32, 2)
    D = native.DeviceFactor(eng, diagonal(d, widths_of(len(d), route)), precision=native.PREC_FP32)
    with np.errstate(all="ignore"):
        want = (a / d).astype(np.float64)
    for got in sweeps(eng, D, a.astype(np.float64)):
        same_bits(got, want)
