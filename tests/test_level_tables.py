"""The level tables of the sweep plans: a sweep leaves the items behind one of
their bounds to its cluster tail, so a bound off by one would leave rows
unsolved. The host preparation checks its own tables (no GPU); on the GPU the
device preparation's are compared with them."""
import numpy as np
import pytest

from apxchol_b200 import native
from tests.test_gpu_tail import SHAPES, layered

# what the caller's rounds may look like: as they are, with empty ones in between and behind, without the last two
# (every row left over is a level of its own), with more rows than the factor has, none (topological levels)
ROUNDS = {
    "as_they_are": lambda r: r,
    "empty_between": lambda r: np.insert(r, [0, len(r) // 2, len(r) // 2, len(r) - 1], 0),
    "empty_behind": lambda r: np.append(r, [0, 0, 0, 0, 0]),
    "cut_short": lambda r: r[:-2],
    "too_long": lambda r: np.append(r, [7, 0, 9]),
    "none": lambda r: r[:0],
}


def factor_args(shape, rounds):
    _, F = layered(*SHAPES[shape], seed=11, sddm=len(rounds) % 2 == 0)
    keep = [np.ascontiguousarray(F.colptr, np.uint32), np.ascontiguousarray(F.rowidx, np.uint32),
            np.ascontiguousarray(F.vals, np.float32), np.ascontiguousarray(F.perm, np.uint32),
            np.ascontiguousarray(ROUNDS[rounds](F.rounds), np.uint64)]
    return F, keep


@pytest.mark.parametrize("rounds", list(ROUNDS))
@pytest.mark.parametrize("shape", ["levels_at_the_limit", "wide_then_narrow", "a_chain"])
def test_host_tables_hold(shape, rounds):
    lib = native.load()
    F, keep = factor_args(shape, rounds)
    items, chunks = np.zeros(2, np.uint32), np.zeros(2, np.uint32)
    for k in (1, 4, 8, 64):
        native.check(lib.apxb_batch_plan_host(F.n, *[native.ptr(a) for a in keep[:4]], int(F.sddm), native.ptr(keep[4]),
                                              keep[4].size, 0.0, k, native.ptr(items), native.ptr(chunks)))
        assert (items >= chunks).all() and chunks.all()


@pytest.mark.gpu
@pytest.mark.parametrize("rounds", [r for r in ROUNDS if r != "none"])
@pytest.mark.parametrize("shape", ["levels_at_the_limit", "wide_then_narrow", "a_chain"])
def test_device_tables_are_the_host_ones(shape, rounds):
    eng = native.Engine(0)
    F, keep = factor_args(shape, rounds)
    for k in (0, 1, 4, 16):
        native.check(eng.lib.apxb_test_prep_compare(eng.h, F.n, *[native.ptr(a) for a in keep[:4]], int(F.sddm),
                                                    native.ptr(keep[4]), keep[4].size, 0.0, k, None, None, None))
    eng.close()
