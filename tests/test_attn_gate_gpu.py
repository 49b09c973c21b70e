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
