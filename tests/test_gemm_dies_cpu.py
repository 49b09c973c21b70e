"""How the two-SM GEMM's host side numbers the pairs of SMs from their latencies to words of memory."""
import ctypes

import numpy as np
import pytest

from flextrain_b200.ops.cuda import load


def _numbers(cycles):
    cycles = np.ascontiguousarray(cycles, dtype=np.float32)
    out = (ctypes.c_ubyte * cycles.shape[0])()
    first = load("gemm_tcgen05").ftb_gemm_dies_from_latencies(cycles.ctypes.data_as(ctypes.c_void_p), cycles.shape[0], out)
    return first, list(out)


@pytest.mark.parametrize("pairs,share", [(74, 0.5), (74, 0.45), (66, 0.3), (2, 0.5)])
def test_pairs_are_numbered_die_by_die(pairs, share):
    rng = np.random.default_rng(pairs)
    die = np.zeros(pairs, dtype=int)
    die[rng.permutation(np.arange(1, pairs))[: pairs - max(1, round(share * pairs))]] = 1
    home = rng.integers(0, 2, 32)
    home[:2] = 0, 1
    cycles = np.where(die[:, None] == home[None], 16 * 270.0, 16 * 650.0) + rng.normal(0, 300, (pairs, 32))
    first, number = _numbers(cycles)
    assert first == int((die == 0).sum())
    assert sorted(number) == list(range(pairs))
    assert all((n < first) == (d == 0) for n, d in zip(number, die))
    for d in (0, 1):                               # in order within a die
        mine = [n for n, dd in zip(number, die) if dd == d]
        assert mine == sorted(mine)


def test_patterns_that_are_not_two_dies_give_no_order():
    rng = np.random.default_rng(0)
    assert _numbers(np.full((74, 32), 300.0))[0] == 0                       # all alike, nothing to tell by
    assert _numbers(300 + rng.normal(0, 10, (74, 32)))[0] == 0              # noise
    one = np.tile(rng.normal(400, 100, 32), (74, 1))
    assert _numbers(one)[0] == 0                                            # one die
    one[5] = 800 - one[5]
    assert _numbers(one)[0] == 0                                            # one pair against the rest
    one[:, 3] = np.nan
    assert _numbers(one)[0] == 0
