"""The output gate of gated attention and norms of heads that lie apart ([query | gate] of one projection) against fp64."""
import pytest
import torch

from flextrain_b200 import ops

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _close(got, want, ulps=1.0):
    """bf16 results of fp32 arithmetic: one rounding (2^-9 of the value; 2^-8 allows for a double one at a tie), fp32 below it."""
    assert ((got.double() - want).abs() <= ulps * 2.0 ** -8 * want.abs() + 1e-6).all()


@pytest.mark.parametrize("T,H,hd,tail", [(1, 1, 8, 0), (3, 2, 64, 8), (257, 3, 128, 16), (1000, 16, 256, 512), (65, 4, 72, 4)])
def test_gate(T, H, hd, tail):
    torch.manual_seed(T)
    mk = lambda *s: torch.randn(*s, device="cuda").mul(3).to(BF)
    wide = mk(T, 2 * H * hd + tail)
    heads = wide[:, :2 * H * hd].unflatten(1, (H, 2 * hd))
    gate = torch.empty(T, H * hd, dtype=BF, device="cuda")
    ops.copy_heads(heads[:, :, hd:], gate)
    assert torch.equal(gate.view(T, H, hd), heads[:, :, hd:])
    x, d = mk(T, H * hd), mk(T, H * hd)
    gate[0, 0], gate[-1, -1] = 200.0, -200.0                       # the sigmoid's ends: 1 and 0 exactly, no NaN from inf
    s = torch.sigmoid(gate.double())
    _close(ops.attn_gate_fwd(x, gate), x.double() * s)
    dwide = torch.full_like(wide, 7.0)
    dst = dwide[:, :2 * H * hd].unflatten(1, (H, 2 * hd))[:, :, hd:]
    want = d.double() * s, x.double() * s, (d.double() * x.double() * s * (1 - s)).view(T, H, hd)
    dx, y = ops.attn_gate_bwd(d.clone(), x, gate, dst)
    _close(dx, want[0])
    _close(y, want[1])
    # 1 - s is taken in fp32: off by 2^-24 of 1, which is |d x s| * 2^-23 with the product's own roundings
    assert ((dst.double() - want[2]).abs() <= 2.0 ** -8 * want[2].abs() + 2.0 ** -20 * (d.double() * x.double()).abs().view(T, H, hd) + 1e-6).all()
    assert (dwide[:, :2 * H * hd].unflatten(1, (H, 2 * hd))[:, :, :hd] == 7).all() and (dwide[:, 2 * H * hd:] == 7).all()


@pytest.mark.parametrize("T,H,hd", [(1, 1, 64), (33, 3, 128), (300, 16, 256)])
def test_norm_of_heads_apart(T, H, hd):
    """The same bits as heads side by side, forward and in dx; the gain's gradient up to the order of its sums."""
    torch.manual_seed(T)
    wide, dwide = torch.randn(T, H, 2 * hd, device="cuda").to(BF), torch.zeros(T, H, 2 * hd, device="cuda", dtype=BF)
    x, dy, w = wide[:, :, :hd], torch.randn(T, H, hd, device="cuda").to(BF), torch.randn(hd, device="cuda")
    y, r = ops.rmsnorm_fwd(x, w, 1e-6)
    y1, r1 = ops.rmsnorm_fwd(x.contiguous(), w, 1e-6)
    assert torch.equal(y, y1) and torch.equal(r, r1)
    dw, dw1, dx1 = torch.zeros(hd, device="cuda"), torch.zeros(hd, device="cuda"), torch.empty(T, H, hd, device="cuda", dtype=BF)
    ops.rmsnorm_bwd(dy, x, w, r, dw_out=dw, dx_out=dwide[:, :, :hd])
    ops.rmsnorm_bwd(dy, x.contiguous(), w, r, dw_out=dw1, dx_out=dx1)
    assert torch.equal(dwide[:, :, :hd], dx1) and (dwide[:, :, hd:] == 0).all()
    xh = x.double() * r.double()[:, :, None]
    n = T * H                                                      # n fp32 additions of |dy xh|, in any order
    assert ((dw.double() - (dy.double() * xh).sum((0, 1))).abs() <= n * 2.0 ** -23 * (dy.double() * xh).abs().sum((0, 1)) + 1e-6).all()
    assert ((dw - dw1).abs() <= n * 2.0 ** -22 * (dy.double() * xh).abs().sum((0, 1)) + 1e-6).all()


@pytest.mark.parametrize("span", [1, 10, 40, 80])
def test_gate_is_rounded_as_the_fp32_chain_is(span):
    """Results that are not the correctly rounded ones: fp32 is off by some 2^-24, a bf16 boundary lies every 2^-8, so there are
    some 1e-5 of them; not more than 1.5 times as many as in the tensor library's chain of fp32 operations (and 40, by chance)."""
    torch.manual_seed(span)
    T, H, hd = 2048, 16, 128
    x, d = (torch.randn(T, H * hd, device="cuda").to(BF) for _ in range(2))
    gate = ((torch.rand(T, H * hd, device="cuda") * 2 - 1) * span).to(BF)
    s, s32 = torch.sigmoid(gate.double()), torch.sigmoid(gate.float())
    dst = torch.empty(T, H, hd, device="cuda", dtype=BF)
    fwd = ops.attn_gate_fwd(x, gate)
    dx, y = ops.attn_gate_bwd(d.clone(), x, gate, dst)
    for got, t in ((fwd, x), (y, x), (dx, d)):
        want = (t.double() * s).float().to(BF)
        off, chain = (int((r != want).sum()) for r in (got, (t.float() * s32).to(BF)))
        assert off <= 1.5 * chain + 40
    want = (d.double() * x.double() * s * (1 - s32.double())).float().to(BF).view_as(dst)      # (1 - s in fp32 on both sides)
    off, chain = (int((r != want).sum()) for r in (dst, (d.float() * x.float() * s32 * (1 - s32)).to(BF).view_as(dst)))
    assert off <= 1.5 * chain + 0.02 * dst.numel()     # (a fp32 sigmoid next to 1 that is one unit off changes 1 - s by far more)


def test_gate_that_is_not_finite():
    gate = torch.tensor([float("nan"), float("inf"), float("-inf"), 3e38, -3e38, 89.0, -89.0, 0.0], device="cuda").to(BF)[None]
    x = torch.full_like(gate, 2.0)
    want = (x.float() * torch.sigmoid(gate.float())).to(BF)
    for got in (ops.attn_gate_fwd(x, gate), ops.attn_gate_bwd(x.clone(), x, gate, torch.empty(1, 1, 8, device="cuda", dtype=BF))[0]):
        assert got[0, 0].isnan() and torch.allclose(got[0, 1:], want[0, 1:], rtol=0, atol=1e-37)
