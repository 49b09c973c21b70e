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


@pytest.mark.parametrize("hd,HQ,HK", [(64, 3, 1), (128, 6, 2), (256, 2, 2)])
@pytest.mark.parametrize("T", [1, 5, 301])
@pytest.mark.parametrize("inverse", [False, True])
def test_rope_qkv_equals_its_parts(hd, HQ, HK, T, inverse):
    """One launch for Q, K and V against the rotation of each and a copy: the same bits; fp32 queries against rounded ones within
    the rounding of the input."""
    from flextrain_b200 import ops
    torch.manual_seed(0)
    qkv = _randn(T, (HQ + 2 * HK) * hd)
    q, k, v = (t.unflatten(1, (-1, hd)) for t in qkv.split([HQ * hd, HK * hd, HK * hd], 1))
    pos = torch.randint(0, 5000, (T,), device=DEV)
    inv = 1.0 / 10000 ** (torch.arange(hd // 2, device=DEV) / (hd // 2))
    want = [ops.rope(t.contiguous(), pos, inv, inverse=inverse) for t in (q.clone(), k.clone())] + [v]
    out = torch.full((T, (HQ + 2 * HK) * hd + 8), 3.0, device=DEV, dtype=BF)
    dst = [t.unflatten(1, (-1, hd)) for t in out[:, :-8].split([HQ * hd, HK * hd, HK * hd], 1)]
    before = ops.launch_count()
    ops.rope_qkv(q, k, v, pos, inv, q_out=dst[0], k_out=dst[1], v_out=dst[2], inverse=inverse)
    assert ops.launch_count() == before + 1
    assert all(torch.equal(a, b) for a, b in zip(dst, want)) and bool((out[:, -8:] == 3.0).all())
    some = torch.empty(T, HK, hd, device=DEV, dtype=BF)
    ops.rope_qkv(None, k, None, pos, inv, q_out=None, k_out=some, v_out=None, inverse=inverse)
    assert torch.equal(some, want[1])
    got = torch.empty(T, HQ, hd, device=DEV, dtype=BF)
    ops.rope_qkv(q.float().contiguous(), k, v, pos, inv, q_out=got, k_out=some, v_out=torch.empty_like(some), inverse=inverse)
    assert torch.equal(got, want[0])
    odd = torch.empty(T * HK * hd + 1, device=DEV, dtype=BF)[1:].view(T, HK, hd).copy_(k)      # off the grid: by parts
    ops.rope_qkv(q, odd, v, pos, inv, q_out=got, k_out=some, v_out=dst[2], inverse=inverse)
    near = lambda a, b: torch.allclose(a.float(), b.float(), rtol=2.0 ** -7, atol=1e-3)         # (other roundings in fp32)
    assert near(some, want[1]) and near(got, want[0])


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("T,H", [(1, 1), (5, 3), (700, 4)])
def test_l2_and_gated_norm_rows(D, T, H):
    """The 16-byte kernels against the general ones (rows one element off the grid), and the heads that share a key head.  Two
    roundings to bf16 of values that differ in the last bits of fp32: one unit in 2^-7 of each at most."""
    from flextrain_b200.ops import linattn_cuda as la
    torch.manual_seed(0)
    x, z = _randn(T, H * D + 8), _randn(T, H * D + 16)
    off = lambda t: torch.empty(t.shape[0], t.shape[1] + 1, device=DEV, dtype=t.dtype)[:, 1:].copy_(t)
    (y, rn), (y1, rn1) = (la.l2norm_heads_fwd(t, H, D) for t in (x, off(x)))
    assert torch.allclose(rn, rn1, rtol=1e-6) and torch.allclose(y.float(), y1.float(), rtol=2.0 ** -7, atol=1e-6)
    dy = torch.randn(T, 2 * H, D, device=DEV)
    dx, dx1 = torch.empty_like(x), torch.empty_like(x)
    la.l2norm_heads_bwd(dy, x, rn, dx[:, :H * D], H, D)
    la.l2norm_heads_bwd(dy.view(T, H, 2, D).sum(2), off(x), rn, dx1[:, :H * D], H, D)
    assert torch.allclose(dx[:, :H * D].float(), dx1[:, :H * D].float(), rtol=2.0 ** -7, atol=1e-5)
    la.l2norm_heads_bwd(dy, off(x), rn, dx1[:, :H * D], H, D)                      # general rows, two heads a key head
    assert torch.allclose(dx[:, :H * D].float(), dx1[:, :H * D].float(), rtol=2.0 ** -7, atol=1e-5)
    o, w, g = _randn(T, H, D), torch.rand(D, device=DEV) + 0.5, _randn(T, H, D)
    a, b = (la.gated_rmsnorm_fwd(o, t[:, :H * D], w, 1e-6) for t in (z, off(z)))
    assert torch.allclose(a.float(), b.float(), rtol=2.0 ** -7, atol=1e-6)
    got = []
    for zz in (z, off(z)):
        dz, dw = torch.empty(T, H * D, device=DEV, dtype=BF), torch.ones(D, device=DEV)
        got.append((la.gated_rmsnorm_bwd(g, o, zz[:, :H * D], w, dz, dw, H, D, 1e-6), dz, dw))
    for u, v in zip(got[0][:2], got[1][:2]):
        assert torch.allclose(u.float(), v.float(), rtol=2.0 ** -7, atol=1e-5)
    assert torch.allclose(got[0][2], got[1][2], rtol=1e-4, atol=T * H * 2.0 ** -20)
