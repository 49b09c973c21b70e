"""RMSNorm of rows in which one element outweighs all others: their squares are not lost one by one beside it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [256, 264, 768, 1024, 1536, 2048, 2056, 3072, 4096, 8192])
def test_an_element_that_outweighs_its_row(D):
    """4096^2 = 2^24, whose units are 2: a square of 0.98 added to it alone is lost.  That may happen to the seven of its own piece of
    eight, and half a unit, 1, to each of the sums that follow: of a lane's pieces (7 at most), over a warp (5) and over a block
    (8), so 27 of 2^24, half of it in the root; the reciprocal root has 2^-22."""
    from flextrain_b200 import ops
    x = torch.full((D, D), 0.98828125, device="cuda", dtype=torch.bfloat16).fill_diagonal_(4096.0)   # every place in turn
    y, rstd = ops.rmsnorm_fwd(x, None, 1e-6)
    want = (x.double().pow(2).mean(-1) + 1e-6).rsqrt()
    assert ((rstd.view(-1).double() - want).abs() <= want * (27 * 2.0 ** -25 + 2.0 ** -22)).all()
    assert ((y.double() - x.double() * want[:, None]).abs() <= 2.0 ** -8 * (x.double() * want[:, None]).abs()).all()
