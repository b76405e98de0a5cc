"""A batch's EM-ICP teams (csrc/cesa_emicp.cu, plan_teams), checked on the host by
cesa_self_test_teams: every registration runs once, its blocks depend on its size and not
on where it stands, and no batch leaves the chip half idle. Needs no GPU."""
import ctypes

import numpy as np
import pytest

GRID = 304


def plan(cesa, sizes, grid=GRID):
    n = len(sizes)
    arr = [np.ascontiguousarray([s[k] for s in sizes], dtype=np.int32) for k in range(3)]
    blocks, ms = np.zeros(n, np.int32), ctypes.c_double(0)
    rc = cesa.lib().cesa_self_test_teams(n, *(a.ctypes.data_as(ctypes.c_void_p) for a in arr), grid,
                                         blocks.ctypes.data_as(ctypes.c_void_p), ctypes.byref(ms))
    assert rc == cesa.CESA_OK
    return blocks, ms.value


def evenly_ms(sizes, grid=GRID):
    """All affinities of the batch at 0.095 ns a block, evenly divided."""
    return sum(n * m * s for n, m, s in sizes) * 0.095e-6 / grid


def mixed(n, seed, lo=500, hi=4000):
    rng = np.random.default_rng(seed)
    return [(int(a), int(b), int(s)) for (a, b), s in zip(np.exp(rng.uniform(np.log(lo), np.log(hi), (n, 2))),
                                                          rng.choice([20, 66, 66, 66], n))]


@pytest.mark.parametrize("n", [1, 2, 3, 151, 152, 153, 160, 303, 304, 305, 310, 600, 1024])
@pytest.mark.parametrize("size", [1, 8, 300, 2000, 20000])
def test_equal_pairs(cesa, n, size):
    blocks, _ = plan(cesa, [(size, size, 66)] * n)
    assert len(set(blocks)) == 1


@pytest.mark.parametrize("grid", [2, 3, 16, 296, 304])
@pytest.mark.parametrize("n", [1, 5, 40, 300, 1000])
def test_uneven_pairs_wherever_they_stand(cesa, n, grid):
    sizes = mixed(n, n)
    blocks, ms = plan(cesa, sizes, grid)
    order = np.random.default_rng(1).permutation(n)
    again, ms2 = plan(cesa, [sizes[i] for i in order], grid)
    assert np.array_equal(again, blocks[order]) and ms == ms2


@pytest.mark.parametrize("sizes", [[(2000, 2000, 66)] * 153, [(2000, 2000, 66)] * 160, [(5000, 5000, 66)] * 160,
                                   [(2000, 2000, 66)] * 305, [(5000, 5000, 66)] * 310,
                                   [(6000, 6000, 66)] * 4 + [(2000, 2000, 66)] * 150])
def test_pairs_a_few_more_than_the_blocks(cesa, sizes):
    """(a team each took 2.3 times the evenly divided affinities' time and more)"""
    _, ms = plan(cesa, sizes)
    assert ms < 1.8 * evenly_ms(sizes)
