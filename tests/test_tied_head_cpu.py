"""A tied head: its gradient added to the embedding's where that lies, against the two summed afterwards."""
import pytest
import torch

import flextrain_b200 as ft
from conftest import build_tiny

DIMS = dict(vocab_size=512, n_layers=1, d_model=64, n_heads=2, n_kv_heads=1, head_dim=32, expert_dim=128, ffn_dim=128,
            num_routed_experts=0, num_shared_experts=0, top_k=0, is_causal=True)


def _train(in_place, steps=3, calls=2, optimizer=None):
    torch.manual_seed(0)
    am = build_tiny(arch="gemma3", dims=DIMS, hyper={"sliding_window": 16, "layer_pattern": "SF"}, max_seq_len=48, batch_tokens=96,
                    optimizer=optimizer and optimizer())
    assert am.head.tied and am._tied_in_place()
    if not in_place:
        am._tied_in_place = lambda: False
        am._head_update_spec = lambda: am.head.param_spec
    g = torch.Generator().manual_seed(1)
    for _ in range(steps):
        for n in (48, 20)[:calls]:
            am.fwd_bwd([ft.Sequence(torch.randint(0, 512, (n,), generator=g))])
        assert not am.buffers.head_grads()["g_head_proj"].any()
        grad = am.buffers.embed_grads()["g_tok_embeddings"].clone()
        am.step()
        assert torch.equal(am.buffers.head_params()["w_head_proj"], am.buffers.embed_params()["w_tok_embeddings"])
    weights = {(s, l, n): t.clone() for s, l, n, t in am.named_master_params()}
    return grad, weights, {k: v.clone() for k, v in am.buffers.head_opt().items()}


@pytest.mark.parametrize("optimizer", [None, lambda: ft.AdamW(lr=1e-3, weight_decay=0.1, check_error=True)])
def test_tied_gradient_in_place(optimizer):
    g, w, o = _train(True, optimizer=optimizer)
    g1, w1, o1 = _train(False, optimizer=optimizer)
    # fp32 on both sides: the same two shares of a gradient, added in another order, through three updates
    assert (g - g1).norm() <= 1e-5 * g1.norm()
    for k in w1:
        torch.testing.assert_close(w[k], w1[k], rtol=1e-4, atol=1e-5)
    assert o.keys() == o1.keys()
    for k in o:                                    # the head's own state: zero for the projection, updated for the norm
        torch.testing.assert_close(o[k], o1[k], rtol=1e-3, atol=1e-6)


def _table_gradient(calls, seqs, chunk, *, grad_dtype=torch.bfloat16, in_place=True):
    from flextrain_b200.engine.host_memory import UnpinnedHostBackend
    torch.manual_seed(0)
    am = ft.from_dims(DIMS, arch="gemma3", optimizer=ft.AdamW(lr=1e-3), max_seq_len=48, max_global_batch_tokens=96,
                      max_gpu_mem_bytes=8 << 30, max_host_mem_bytes=8 << 30, hyperparams={"sliding_window": 16, "layer_pattern": "SF"},
                      device="cpu", compute_dtype=torch.bfloat16, master_dtype=torch.bfloat16, grad_dtype=grad_dtype,
                      working_set=ft.WorkingSetConfig.simple(max_seq_len=48, max_global_batch_tokens=96, chunk=chunk),
                      host_backend=UnpinnedHostBackend())
    if not in_place:
        am._tied_in_place = lambda: False
    g = torch.Generator().manual_seed(1)
    chunks = 0
    for _ in range(calls):
        ids = [torch.randint(0, 32, (n,), generator=g) for n in seqs]             # few token ids: rows that many tokens add to
        chunks += am.fwd_bwd([ft.Sequence(i, targets=torch.roll(i, -1)) for i in ids], loss_scale_factor=1.0).n_chunks
    return am.buffers.embed_grads()["g_tok_embeddings"].double(), chunks


@pytest.mark.parametrize("calls,seqs,chunk", [(1, (48,), 48), (1, (40, 40), 48), (8, (48,), 48), (8, (40, 40), 48)])
def test_bf16_table_gradient_over_several_calls(calls, seqs, chunk):
    """bf16 gradients against the same sums in fp32: adding the head's share where the embedding's lies costs no precision over
    adding up each by itself, however many calls and chunks a step has."""
    want, n = _table_gradient(calls, seqs, chunk, grad_dtype=torch.float32)
    assert n == calls * len(seqs)
    err = [float((_table_gradient(calls, seqs, chunk, in_place=p)[0] - want).norm() / want.norm()) for p in (True, False)]
    # each sum of a call is rounded once and each call's total once: 2^-9 of an element's size at the most, added up over the calls
    assert err[1] <= 2.0 ** -9 * (1 + calls * len(seqs))
    assert err[0] <= 1.02 * err[1]
