"""The temporaries that the kernels' bindings allocate by themselves stay inside what a plan sets aside for them."""
import random

import pytest

from flextrain_b200 import ops
from flextrain_b200.core.working_set import WORKSPACE_ALLOWANCE
from flextrain_b200.ops import cuda as k


def _shapes(seed, top):
    rng = random.Random(seed)
    return [tuple(8 * rng.randint(8, top // 8) for _ in range(2)) for _ in range(200)]


@pytest.mark.parametrize("seed", range(3))
def test_slabs_of_cut_gemms(seed):
    """Two GEMMs with a cut reduction do not run at once, and one takes at most half of the allowance."""
    rng = random.Random(seed)
    cut = 0
    for m, n in _shapes(seed, 16384):
        splits = k._k_splits(m, n, 8 * rng.randint(1, 32768))
        cut += splits > 1
        assert splits == 1 or splits * m * n * 4 <= k.GEMM_SLAB_BYTES <= WORKSPACE_ALLOWANCE // 2
    assert cut


@pytest.mark.parametrize("seed", range(3))
def test_batches_of_the_muon_iteration(seed):
    """Two buffers of the iterate and two of its product with itself, in bf16; a single matrix that is larger takes 8 bytes an
    element (its rows padded)."""
    for m, n in _shapes(seed, 16384) + [(65, 64), (72, 64), (128, 64), (64, 72)]:
        nb, rows, side = ops._muon_batch_size(m, n), (m + 63) // 64 * 64 if m > n else m, min(m, n)
        nbytes = 2 * nb * (2 * rows * n + 2 * side * side)
        assert nbytes <= (WORKSPACE_ALLOWANCE if nb > 1 else max(WORKSPACE_ALLOWANCE, 8 * rows * n))
        assert nb >= 1
