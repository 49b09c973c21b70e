"""Kernels that take rows in 16-byte pieces: against float64, and against the general kernels that rows off the grid still take."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16


def _randn(*s, scale=1.0):
    return (torch.randn(*s, device=DEV) * scale).to(BF)


@pytest.mark.parametrize("D", [8, 248, 256, 264, 520, 768, 776, 1024, 1032, 1536, 1544, 2040, 2048, 2056, 3072, 3080])
@pytest.mark.parametrize("T", [1, 7, 8, 9, 5000])
def test_rmsnorm_rows_by_warps(D, T):
    """Around 256 elements a piece of a lane, the last widths of one, two and four warps a row, and rows around the eight of a block.  A bf16
    result is off by 2^-9 of itself; a sum of n fp32 terms by n 2^-24 of its terms' magnitudes."""
    from flextrain_b200 import ops
    torch.manual_seed(D + T)
    x, dy, add = (_randn(T, D) for _ in range(3))
    w = torch.rand(D, device=DEV) + 0.5
    dw0 = torch.randn(D, device=DEV)
    dw = dw0.clone()
    y, rstd = ops.rmsnorm_fwd(x, w, 1e-6)
    dx, y2 = ops.rmsnorm_bwd(dy, x, w, rstd, dx_add=add, emit_y=True, dw_out=dw)
    X, W = x.double(), w.double()
    R = torch.rsqrt(X.pow(2).mean(-1, keepdim=True) + 1e-6)
    want_y = X * R * W
    G = dy.double() * W
    want_dx = R * (G - X * R * (G * X * R).mean(-1, keepdim=True)) + add.double()
    terms = dy.double() * X * R
    near = lambda a, b, room: bool(((a.double() - b).abs() <= room).all())
    assert near(rstd.view(-1, 1), R, R * (2.0 ** -20 + D * 2.0 ** -24))
    assert near(y, want_y, want_y.abs() * 2.0 ** -8) and near(y2, want_y, want_y.abs() * 2.0 ** -8)
    size = R * (G.abs() + (X * R).abs() * (G * X * R).abs().mean(-1, keepdim=True)) + add.double().abs()
    assert near(dx, want_dx, want_dx.abs() * 2.0 ** -8 + size * (D + 32) * 2.0 ** -23)
    assert near(dw, dw0.double() + terms.sum(0), (terms.abs().sum(0) + dw0.double().abs()) * (T + 32) * 2.0 ** -23)
    dx, none = ops.rmsnorm_bwd(dy, x, None, rstd)
    assert none is None
    G = dy.double()
    want = R * (G - X * R * (G * X * R).mean(-1, keepdim=True))
    size = R * (G.abs() + (X * R).abs() * (G * X * R).abs().mean(-1, keepdim=True))
    assert near(dx, want, want.abs() * 2.0 ** -8 + size * (D + 32) * 2.0 ** -23)
