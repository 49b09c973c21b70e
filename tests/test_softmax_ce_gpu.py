"""Cross entropy around the row length and the number of rows from which a row takes 256 threads, not 512, and around what a block
reads at once (16384 and 32768)."""
import pytest
import torch

from flextrain_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("softcap", [0.0, 30.0])
@pytest.mark.parametrize("V,T", [(7, 300), (16384, 296), (16385, 296), (32768, 295), (32776, 300), (57344, 300), (57345, 300), (57352, 9),
                                 (7, 9), (16384, 9), (32768, 9), (98309, 9), (131072, 9)])
def test_loss_and_gradient(V, T, softcap):
    torch.manual_seed(V)
    ld = (V + 7) // 8 * 8
    buf = torch.full((T, ld), 5.0, device="cuda", dtype=torch.bfloat16)
    z = buf[:, :V]
    z.copy_(torch.randn(T, V, device="cuda") * 3)
    tgt = torch.tensor([0, V - 1, V // 8 * 8 - 1 if V >= 8 else 0, min(V - 1, 255), -100, V // 2, V, min(V - 1, 57344), 1], device="cuda")
    tgt = torch.cat([tgt, torch.randint(0, V, (T - 9,), device="cuda")])
    d = z.double()
    zc = softcap * torch.tanh(d / softcap) if softcap else d
    lse, on = zc.logsumexp(1), (tgt >= 0) & (tgt < V)
    at = tgt.clamp(0, V - 1)
    want = (lse - zc.gather(1, at[:, None])[:, 0]) * on
    p = (zc - lse[:, None]).exp()
    p.scatter_add_(1, at[:, None], -torch.ones(T, 1, device="cuda", dtype=torch.double))
    g = 0.25 * p * (1 - (zc / softcap) ** 2 if softcap else 1.0) * on[:, None]
    loss = ops.softmax_ce_loss(z, tgt, softcap=softcap)
    got = ops.softmax_ce_(z, tgt, grad_scale=0.25, softcap=softcap)
    assert torch.equal(loss, got)
    # |z| < 20: sums of V / 256 terms a thread in fp32, exponentials to some 2^-21
    assert ((got.double() - want).abs() <= 1e-4).all()
    # one rounding to bf16, and the tanh of the fast kind (2^-10.9 of 1 - t^2 where t is near 1) under a soft-cap
    assert ((z.double() - g).abs() <= 2.0 ** -8 * g.abs() * (4 if softcap else 1.02) + 1e-7).all()
    assert (buf[:, V:] == 5).all()
