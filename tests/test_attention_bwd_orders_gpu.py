"""Attention backward at the sizes where its order of work and its pipeline change: one tile pair, few pairs (the software
pipeline's start and end), many short sequences (the warp-wide tile search crosses 32), and both fixed orders of dQ."""

import pytest
import torch

from flextrain_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"

CASES = {                                       # lens_q, lens_k, H, KV, window, softcap
    "one_pair": ([128], [128], 1, 1, 0, 0.0),
    "one_token": ([1, 2], [1, 2], 2, 1, 0, 0.0),
    "two_pairs": ([129], [129], 1, 1, 0, 0.0),
    "rep_three": ([257, 5], [257, 5], 3, 1, 0, 0.0),
    "more_than_32_sequences": ([3 + 5 * i for i in range(70)], [3 + 5 * i for i in range(70)], 4, 2, 0, 0.0),
    "prior": ([130, 64], [700, 300], 4, 2, 0, 0.0),
    "more_queries_than_keys": ([300], [100], 2, 1, 0, 0.0),
    # (past 4096 keys, or 1024 at head dim 64, the fixed order is the other one)
    "in_step": ([4200], [4200], 2, 1, 0, 0.0),
    "in_step_prior": ([500, 77], [4333, 99], 4, 1, 0, 0.0),
    "in_step_window": ([4200, 300], [4200, 300], 2, 1, 200, 0.0),
    "in_step_softcap": ([4200], [4200], 2, 1, 0, 20.0),
    "in_step_window_prior": ([600], [4500], 4, 2, 129, 0.0),
    "in_step_waves": ([4224], [4224], 8, 8, 0, 0.0),                    # 264 CTAs, more than run at once
}


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("name", list(CASES))
def test_attention_bwd(hd, name):
    """dQ, dK, dV against the fp32 reference: P and dS are rounded to bf16 (2^-9 relative each) before products whose
    terms add up at random, and the results once more, so the relative error of a whole tensor stays below 2^-6.  The fixed
    order repeats bit for bit and agrees with the free one to fp32 rounding before the result is rounded to bf16: each element
    to a neighbouring bf16 value (2^-7 relative), or where the tiles' shares cancel to 36 additions' roundings of them (2^-14 of
    the tensor's root mean square has room for shares of 28 times it)."""
    from flextrain_b200.ops import attention_cuda as fa
    from flextrain_b200.ops import cuda as kk
    lens_q, lens_k, H, KV, window, softcap = CASES[name]
    torch.manual_seed(1)
    cu = lambda n: torch.tensor([0] + list(torch.tensor(n).cumsum(0)), dtype=torch.int32, device=DEV)
    cu_q, cu_k = cu(lens_q), cu(lens_k)
    mk = lambda n, h: torch.randn(n, h, hd, device=DEV).to(torch.bfloat16)
    q, do, k, v = mk(sum(lens_q), H), mk(sum(lens_q), H), mk(sum(lens_k), KV), mk(sum(lens_k), KV)
    kw = dict(scale=hd ** -0.5, window=window, softcap=softcap)
    o, lse = fa.fwd(q, k, v, cu_q, cu_k, max(lens_q), max(lens_k), **kw)
    blind = max(lens_q[0] - lens_k[0], 0)       # queries that see no key: the reference is given the others alone
    cu_w = (cu_q - blind).clamp_min(0)
    ow, lw = ref.attention_fwd(q[blind:], k, v, cu_w, cu_k, **kw)
    want = list(ref.attention_bwd(do[blind:], q[blind:], k, v, ow, lw, cu_w, cu_k, **kw))
    want[0] = torch.cat([want[0].new_zeros(blind, H, hd), want[0]])
    got = [fa.bwd(do, q, k, v, o, lse, cu_q, cu_k, max(lens_q), max(lens_k), deterministic=d, **kw)
           for d in (True, True, False)]
    assert kk.device_error_words().get("attention", 0) == 0
    for first, again, free, w in zip(*got, want):
        assert torch.equal(first, again)
        a, b = first.float(), free.float()
        assert torch.all((a - b).abs() <= 2.0 ** -7 * torch.maximum(a.abs(), b.abs()) + 2.0 ** -14 * w.float().square().mean().sqrt())
        for g in (first, free):
            assert torch.isfinite(g).all()
            assert float((g.float() - w.float()).norm()) <= 2.0 ** -6 * float(w.float().norm()) + 1e-6


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("shift", [2, 4])
@pytest.mark.parametrize("which", ["dout", "q", "k", "v", "out"])
def test_operands_off_the_16_byte_grid(which, shift, hd):
    """A contiguous operand that starts ``shift`` elements past a 16-byte boundary gives the aligned one's bits."""
    from flextrain_b200 import ops
    torch.manual_seed(0)
    cu = torch.tensor([0, 150, 200], dtype=torch.int32, device=DEV)
    t = {n: torch.randn(200, h, hd, device=DEV).to(torch.bfloat16) for n, h in (("q", 4), ("k", 2), ("v", 2), ("dout", 4))}
    kw = dict(scale=hd ** -0.5)
    t["out"], lse = ops.attention_fwd(t["q"], t["k"], t["v"], cu, cu, 150, 150, **kw)
    run = lambda: ops.attention_bwd(t["dout"], t["q"], t["k"], t["v"], t["out"], lse, cu, cu, 150, 150, **kw)
    want = run()
    off = torch.empty(t[which].numel() + shift, dtype=torch.bfloat16, device=DEV)[shift:].view(t[which].shape)
    t[which] = off.copy_(t[which])
    assert off.is_contiguous() and off.data_ptr() % 16 == 2 * shift
    for g, w in zip(run(), want):
        assert torch.equal(g, w)
    assert torch.equal(ops.attention_fwd(t["q"], t["k"], t["v"], cu, cu, 150, 150, **kw)[0], t["out"])


@pytest.mark.parametrize("deterministic", [False, True])
def test_more_key_tiles_than_the_second_grid_dimension_holds(deterministic):
    """66000 sequences of one token: every query sees its own key alone, so out = v, dv = dout, and dq and dk are what is left
    of dP - delta: two fp32 sums of the same 64 products of at most 25 in size, one of them as three bf16 terms, which differ by
    2^-20 of the sum of the sizes at most; times a key or query (at most 5) and the scale."""
    from flextrain_b200.ops import attention_cuda as fa
    from flextrain_b200.ops import cuda as kk
    torch.manual_seed(0)
    n, hd = 66000, 64
    q, k, v, do = (torch.randn(n, 1, hd, device=DEV).to(torch.bfloat16) for _ in range(4))
    cu = torch.arange(n + 1, dtype=torch.int32, device=DEV)
    out, lse = fa.fwd(q, k, v, cu, cu, 1, 1, scale=hd ** -0.5)
    dq, dk, dv = fa.bwd(do, q, k, v, out, lse, cu, cu, 1, 1, scale=hd ** -0.5, deterministic=deterministic)
    assert kk.device_error_words().get("attention", 0) == 0
    assert torch.equal(out, v) and torch.equal(dv, do)
    room = 2.0 ** -20 * 64 * 25 * 5 * hd ** -0.5
    assert float(dq.float().abs().max()) <= room and float(dk.float().abs().max()) <= room


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("scale", [0.0, 1e-30, -0.1])
def test_unusual_scales(scale, hd):
    """Uniform attention (a scale of 0) and scores that fall as the product grows, against the fp32 reference and its lse, with
    the bound of the other cases."""
    from flextrain_b200.ops import attention_cuda as fa
    torch.manual_seed(2)
    cu = torch.tensor([0, 150, 450], dtype=torch.int32, device=DEV)
    q, do, k, v = (torch.randn(450, h, hd, device=DEV).to(torch.bfloat16) for h in (4, 4, 2, 2))
    o, lse = ref.attention_fwd(q, k, v, cu, cu, scale=scale)
    want = ref.attention_bwd(do, q, k, v, o, lse, cu, cu, scale=scale)
    for g, w in zip(fa.bwd(do, q, k, v, o.to(torch.bfloat16), lse.contiguous(), cu, cu, 300, 300, scale=scale), want):
        assert torch.isfinite(g).all()
        assert float((g.float() - w.float()).norm()) <= 2.0 ** -6 * float(w.float().norm()) + 1e-6
