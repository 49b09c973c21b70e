"""Norms that read and write views of a fused projection in place, against the plain PyTorch fp32 reference."""

import pytest
import torch

from flextrain_b200 import ops
from flextrain_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _check(x, dy, w, dst, keep):
    """One bf16 rounding of each result (2^-8 covers it and the fp32 sums before it), the gain's gradient to fp32 sums."""
    before = keep.clone()
    y, r = ops.rmsnorm_fwd(x, w, 1e-6)
    yw, rw = ref.rmsnorm_fwd(x, w, 1e-6)
    near = lambda a, b: torch.all((a.float() - b.float()).abs() <= 2.0 ** -8 * b.float().abs() + 2.0 ** -10 * b.float().abs().max())
    assert y.is_contiguous() and y.shape == x.shape and r.shape == rw.shape and near(y, yw)
    assert torch.allclose(r, rw, rtol=1e-5)
    dw = torch.randn(w.shape, device=DEV) if w is not None else None
    dw0 = dw.clone() if dw is not None else None
    dx, _ = ops.rmsnorm_bwd(dy, x, w, r, dw_out=dw, dx_out=dst)
    dxw, dww = ref.rmsnorm_bwd(dy, x, w, r)
    assert dx.data_ptr() == dst.data_ptr() and near(dst, dxw)
    if dw is not None:
        mag = (dy.float() * x.float() * r.unsqueeze(-1)).abs().reshape(-1, x.shape[-1]).sum(0)
        assert torch.all((dw - dw0 - dww).abs() <= 2.0 ** -16 * mag + 1e-5)
    dst.fill_(0)                                        # nothing around the view was written
    mask = keep != before
    assert not mask.any() or torch.all(keep[mask] == 0)


@pytest.mark.parametrize("hd", [64, 96, 128, 256])
@pytest.mark.parametrize("T,H", [(1, 1), (3, 5), (33, 8), (257, 3)])
@pytest.mark.parametrize("gain", [True, False])
@pytest.mark.parametrize("shift", [0, 4])
def test_norm_of_heads_in_a_wider_row(hd, T, H, gain, shift):
    """Heads inside rows of a wider tensor, on and off the 16-byte grid, at row counts that leave a block partly empty; a head
    dim without a kernel of its own takes the copying path."""
    torch.manual_seed(0)
    mk = lambda: torch.randn(T, H * hd + 64, device=DEV).bfloat16()
    cut = lambda t: t[:, 8 + shift:8 + shift + H * hd].unflatten(1, (H, hd))
    x, g, out = mk(), mk(), torch.full((T, H * hd + 64), 7.0, device=DEV).bfloat16()
    w = torch.randn(hd, device=DEV) if gain else None
    _check(cut(x), cut(g).contiguous(), w, cut(out), out)


@pytest.mark.parametrize("D", [512, 520, 2048, 4104])
@pytest.mark.parametrize("T", [1, 5, 700])
@pytest.mark.parametrize("shift", [0, 4])
def test_norm_of_rows_in_a_wider_row(D, T, shift):
    torch.manual_seed(0)
    x, out = torch.randn(T, D + 64, device=DEV).bfloat16(), torch.full((T, D + 64), 7.0, device=DEV).bfloat16()
    cut = lambda t: t[:, 8 + shift:8 + shift + D]
    _check(cut(x), torch.randn(T, D, device=DEV).bfloat16(), torch.randn(D, device=DEV), cut(out), out)
