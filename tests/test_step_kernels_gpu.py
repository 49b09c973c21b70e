"""Kernels of the optimizer step against the plain PyTorch reference, at the sizes where the vector paths end."""

import itertools

import pytest
import torch

from flextrain_b200 import ops
from flextrain_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF16, F32 = torch.bfloat16, torch.float32


@pytest.mark.parametrize("pdt,gdt,sdt", list(itertools.product((BF16, F32), repeat=3)))
@pytest.mark.parametrize("shift", [0, 1, 8])
def test_adamw_types_tails_and_alignment(pdt, gdt, sdt, shift):
    """Every type combination, lengths around a group of 8 and around a block of 2048, and tensors that start off the
    16-byte grid (``shift`` elements into their buffer): update and state as in the fp32 reference.  The momentum has
    the gradient's sign, so nothing cancels but the weight against its update: the fp32 values before the last rounding
    differ by some ten roundings of 2^-24, of the weight and of the update, and by 1 - 0.95 in fp32 (2^-22 off); a bf16
    result may then round to the neighbouring value.
    """
    torch.manual_seed(0)
    sizes = (1, 7, 8, 9, 2040, 2047, 2048, 2049, 5003)
    mk = lambda n, dt, f: f(torch.randn(n + shift, device=DEV)).to(dt)[shift:]
    same = lambda t: t
    P, G = [mk(n, pdt, same) for n in sizes], [mk(n, gdt, same) for n in sizes]
    M = [(mk(n, F32, torch.abs) * g.float().sign()).to(sdt) for n, g in zip(sizes, G)]
    M = [torch.cat([m.new_zeros(shift), m])[shift:] for m in M]
    V = [mk(n, sdt, torch.square) for n in sizes]
    before = [p.clone() for p in P]
    want = [[t.clone() for t in ts] for ts in (P, M, V)]
    kw = dict(beta1=0.9, beta2=0.95, eps=1e-8, step=3, grad_scale=0.5)
    ops.adamw_multi(P, G, M, V, lrs=[1e-2] * len(sizes), wds=[0.1] * len(sizes), **kw)
    for p, g, m, v in zip(want[0], G, want[1], want[2]):
        ref.adamw_step(p, g, m, v, lr=1e-2, weight_decay=0.1, **kw)
    for got, new, old, dt in ((P, want[0], before, pdt), (M, want[1], want[1], sdt), (V, want[2], want[2], sdt)):
        for a, b, o in zip(got, new, old):
            room = 2.0 ** -20 * (b.float().abs() + o.float().abs()) + (2.0 ** -7 * b.float().abs() if dt == BF16 else 0)
            assert torch.all((a.float() - b.float()).abs() <= room)


@pytest.mark.parametrize("shift", [0, 1])
def test_sum_of_squares_sizes_types_and_alignment(shift):
    """More tensors than one launch takes, lengths around a group of 8 and a block of 16384, both types, off the 16-byte
    grid, next to tensors the kernel does not take (host, strided).  Blocks add in fp32 (64 terms a thread and a tree of
    8 levels: 2^-24 * 72 relative at most, all terms being positive) and the blocks in double."""
    torch.manual_seed(0)
    sizes = (1, 7, 8, 9, 16383, 16384, 16385, 40003)
    ts = [torch.randn(n + shift, device=DEV).to(dt)[shift:] for n in sizes * 5 for dt in (BF16, F32)]
    ts += [torch.randn(33), torch.randn(64, 32, device=DEV)[:, :7], torch.empty(0, device=DEV)]
    want = sum(float(t.double().square().sum()) for t in ts)
    got = float(ops.sum_of_squares(ts, torch.device(DEV, 0)))
    assert abs(got - want) <= 2.0 ** -24 * 80 * want
    assert float(ops.sum_of_squares([], torch.device(DEV, 0))) == 0.0
    ts[3][0] = float("inf")
    assert float(ops.sum_of_squares(ts, torch.device(DEV, 0))) == float("inf")
    ts[3][0] = float("nan")
    assert ops.sum_of_squares(ts, torch.device(DEV, 0)).isnan()


@pytest.mark.parametrize("nesterov", [True, False])
@pytest.mark.parametrize("gdt,mdt", [(BF16, BF16), (F32, F32)])
def test_muon_batches_match_the_reference(nesterov, gdt, mdt):
    """Matrices of several sizes (wide, tall with a row count that needs padding, square), 2-D and stacked, more of one size
    than one launch takes, one off the 16-byte grid and one transposed, in one call: momentum as the fp32 reference's to the
    rounding of its type, and the step within the 2 % that bf16 iterates of five Newton-Schulz steps keep (the reference
    iterates in fp32; the polynomial's slope at small singular values is 3.4 per step)."""
    torch.manual_seed(0)
    shapes = [(256, 512), (328, 64), (200, 200)] + [(64, 72)] * 70 + [(3, 128, 256)]
    mk = lambda s, dt, k: (torch.randn(*s, device=DEV) * k).to(dt)
    P, G, M = ([mk(s, dt, k) for s in shapes] for dt, k in ((BF16, 0.05), (gdt, 0.01), (mdt, 0.01)))
    P[0] = (torch.randn(256 * 512 + 1, device=DEV) * 0.05).to(BF16)[1:].view(256, 512)
    P[2] = mk((200, 200), BF16, 0.05).t()
    start = [p.float().clone() for p in P]
    want = [(p.float().contiguous(), m.float().clone()) for p, m in zip(P, M)]
    kw = dict(lr=0.02, beta=0.95, weight_decay=0.01, nesterov=nesterov, grad_scale=0.5)
    ops.muon_multi(P, G, M, **kw)
    for p, g, m, p0, (pw, mw) in zip(P, G, M, start, want):
        ref.muon_step(pw, g.float(), mw, **kw)
        assert torch.all((m.float() - mw).abs() <= (2.0 ** -8 if mdt == BF16 else 2.0 ** -21) * (mw.abs() + g.float().abs()))
        step, step_want = p.float() - p0, pw - p0
        cos = torch.nn.functional.cosine_similarity(step.flatten(), step_want.flatten(), dim=0)
        assert float(cos) > 0.98, (tuple(p.shape), float(cos))


@pytest.mark.parametrize("shape", [(64, 4096), (4104, 64), (2, 64, 65536), (30, 64, 8192), (128, 20000), (20000, 512)])
def test_muon_long_matrices(shape):
    """Few matrices with a long side, whose products with themselves are cut along it, and as many as are not: the step within
    the 2 % of the batches above."""
    torch.manual_seed(0)
    p, g, m = ((torch.randn(*shape, device=DEV) * k).to(BF16) for k in (0.05, 0.01, 0.01))
    start, pw, mw = p.float(), p.float(), m.float()
    kw = dict(lr=0.02, beta=0.95, weight_decay=0.01)
    ops.muon_step(p, g, m, **kw)
    ref.muon_step(pw, g.float(), mw, **kw)
    for a, b in zip((p.float() - start).view(-1, *shape[-2:]), (pw - start).view(-1, *shape[-2:])):
        assert float(torch.nn.functional.cosine_similarity(a.flatten(), b.flatten(), dim=0)) > 0.98


@pytest.mark.parametrize("V", [8, 1000, 16384, 16392, 32771, 50257])
@pytest.mark.parametrize("softcap", [0.0, 30.0])
def test_cross_entropy_batches_and_loss_only(V, softcap):
    """Vocabularies around what a block reads at once (4 x 512 x 8 = 16384), not a multiple of 8, with ignored and masked
    rows: loss and gradient as the fp32 reference's, and the loss-only form equal to it bit for bit, logits untouched."""
    torch.manual_seed(0)
    T, ld = 37, (V + 15) // 8 * 8
    z = (torch.randn(T, ld, device=DEV) * 3).to(BF16)[:, :V]
    tgt = torch.randint(0, V, (T,), device=DEV)
    tgt[3] = -100
    mask = torch.ones(T, device=DEV)
    mask[5] = 0
    kw = dict(softcap=softcap, loss_mask=mask)
    before = z.clone()
    alone = ops.softmax_ce_loss(z, tgt, **kw)
    assert torch.equal(z, before)
    lw, dw = ref.softmax_ce_fwd_bwd(z, tgt, grad_scale=0.25, ignore_index=-100, **kw)
    loss = ops.softmax_ce_(z, tgt, grad_scale=0.25, **kw)
    assert torch.equal(loss, alone) and torch.allclose(loss, lw, rtol=1e-5, atol=1e-4)      # lse of |z| < 20 in fp32
    assert torch.all((z.float() - dw.float()).abs() <= 2.0 ** -7 * dw.float().abs() + 1e-6)
