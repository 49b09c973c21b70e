"""The temporaries that the kernels' bindings allocate by themselves stay inside what a plan sets aside for them."""
import ctypes
import math
import random
import types

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


@pytest.mark.parametrize("seed", range(3))
def test_parts_of_adapter_gradients(seed):
    """Not at once with a GEMM whose reduction is cut: at most half of the allowance, too."""
    lib = k.load("lora")
    lib.ftb_lora_wgrad_bytes.restype = ctypes.c_long
    rng = random.Random(seed)
    log = lambda lo, hi: int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))
    shapes = [(rng.randint(1, 3), log(1, 131072), 32 * log(1, 1024), rng.choice((8, 16, 32))) for _ in range(3000)]
    for n, T, K, R in shapes + [(3, 59205, 23360, 32), (3, 131072, 32768, 32)]:
        N = (ctypes.c_int * n)(*(32 * log(1, 2048) for _ in range(n)))
        assert 0 < lib.ftb_lora_wgrad_bytes(n, T, K, N, R) <= WORKSPACE_ALLOWANCE // 2


@pytest.mark.parametrize("seed", range(3))
def test_chunks_of_gated_deltanet(seed):
    """A plan counts them, for as many sequences as the chunked kernels take."""
    from flextrain_b200.core.working_set import _workspace_bytes
    from flextrain_b200.ops import linattn_cuda as la
    lib = k.load("gdn_chunk")
    lib.ftb_gdn_chunk_bytes.restype = ctypes.c_long
    rng = random.Random(seed)
    for _ in range(1000):
        T, HV = rng.randint(1, 65536), rng.choice((1, 4, 16, 32, 64))
        S = rng.randint(0, T // 40)
        took = lib.ftb_gdn_chunk_bytes(ctypes.c_long(T), S, HV) + S * HV * 4
        assert took <= la.chunk_work_most(T, HV, 128, 128)
    assert la.chunk_work_most(4096, 8, 64, 128) == 0                              # other heads go token by token
    with_, without = (_plan_workspace(_workspace_bytes, dim) for dim in (128, 64))
    assert with_ - without >= lib.ftb_gdn_chunk_bytes(ctypes.c_long(8192), 8192 // 40, 32)


def _plan_workspace(workspace_bytes, head_dim):
    layer = types.SimpleNamespace(cfg=types.SimpleNamespace(
        d_model=2048, attn=None, moe=None, ffn=types.SimpleNamespace(ffn_dim=6144),
        gdn=types.SimpleNamespace(n_v_heads=32, head_k_dim=head_dim, head_v_dim=head_dim)))
    return workspace_bytes([layer], types.SimpleNamespace(head_chunk_size=1024, vocab_size=32000), 8192)
