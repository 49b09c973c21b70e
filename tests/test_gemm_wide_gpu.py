"""Tiles of 512 x 256 of the two-SM GEMM, several to a pair of SMs: every layout of the operands, both output types, C, bias, rows
and sums that end inside a tile, and slices of a sum; and the order of tiles by dies in the gated-FFN epilogues.  Against fp64, all
elements."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _operands(M, N, K, ta, tb):
    torch.manual_seed(M + N + K + 2 * ta + tb)
    a = torch.randn(*((K, M) if ta else (M, K)), device="cuda").to(BF)
    b = torch.randn(*((N, K) if tb else (K, N)), device="cuda").to(BF)
    return a, b, (a.t() if ta else a).double() @ (b.t() if tb else b).double()


def _sms():
    return torch.cuda.get_device_properties(0).multi_processor_count & ~1


def _close(got, want, K):
    """fp32 sums of K products of normal numbers: an error of 2^-24 of the running sum (some sqrt K) at each of K / 16 steps, all of
    one sign at worst, so K sqrt(K) 2^-28, and as much for the truncated products within a step; then one rounding of the result."""
    ulp = 2.0 ** -8 if got.dtype == BF else 2.0 ** -23
    assert ((got.double() - want).abs() <= ulp * want.abs() + K ** 1.5 * 2.0 ** -27).all()


@pytest.mark.parametrize("dtype", [BF, torch.float32])
@pytest.mark.parametrize("ta,tb", [(False, True), (False, False), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K", [(4056, 9464, 8200), (4096, 9472, 8192), (1000, 37880, 8264)])
def test_wide_tiles(M, N, K, ta, tb, dtype):
    from flextrain_b200.ops import cuda as k
    lib, pairs = k.load("gemm_tcgen05"), _sms() // 2
    assert lib.ftb_gemm_wide_tiles(M, N, K, 1, _sms())
    assert -(-M // 512) * -(-N // 256) > 2 * pairs                 # three tiles and more to a pair
    a, b, want = _operands(M, N, K, ta, tb)
    assert k._k_splits(M, N, K) == 1
    bias = torch.randn(N, device="cuda")
    wide = torch.randn(M, N + 24, device="cuda").to(dtype)
    keep = wide.clone()
    k.gemm(a, b, trans_a=ta, trans_b=tb, alpha=0.5, beta=1.0, bias=bias, out=wide[:, 8:8 + N])
    _close(wide[:, 8:8 + N], 0.5 * want + bias.double() + keep[:, 8:8 + N].double(), K)
    assert torch.equal(wide[:, :8], keep[:, :8]) and torch.equal(wide[:, 8 + N:], keep[:, 8 + N:])
    _close(k.gemm(a, b, trans_a=ta, trans_b=tb, out_dtype=dtype), want, K)
    assert k.device_error_words().get("gemm_tcgen05", 0) == 0


@pytest.mark.parametrize("dtype", [BF, torch.float32])
@pytest.mark.parametrize("ta,tb", [(False, True), (False, False), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K,splits", [(3000, 2040, 32832, 4), (2040, 4600, 16456, 2)])
def test_slices_of_wide_tiles(M, N, K, splits, ta, tb, dtype, monkeypatch):
    """Two and three tiles to a pair, the last slice shorter."""
    from flextrain_b200.ops import cuda as k
    lib = k.load("gemm_tcgen05")
    k_slice = -(-K // splits)
    a, b, want = _operands(M, N, K, ta, tb)
    monkeypatch.setattr(k, "_k_splits", lambda *s: splits)
    assert lib.ftb_gemm_wide_tiles(M, N, k_slice, splits, _sms())
    c = torch.randn(M, N, device="cuda").to(dtype)
    got = k.gemm(a, b, trans_a=ta, trans_b=tb, beta=1.0, c=c, out_dtype=dtype)
    _close(got, want + c.double(), K)
    assert k.device_error_words().get("gemm_tcgen05", 0) == 0


@pytest.mark.parametrize("M,F,K", [(2560, 2560, 4096), (2500, 2432, 4104)])
def test_gated_ffn_by_dies(M, F, K, monkeypatch):
    """More than two tiles a pair.  The same bits as tiles in the order of blocks (on fewer pairs), and against fp64."""
    from flextrain_b200.ops import cuda as k
    assert -(-M // 256) * (F // 128) > _sms()                      # forward; the backward has half as many
    torch.manual_seed(M)
    x, w = torch.randn(M, K, device="cuda").to(BF), (torch.randn(2 * F, K, device="cuda") / K ** 0.5).to(BF)
    dy, w2 = torch.randn(M, K, device="cuda").to(BF), (torch.randn(K, F, device="cuda") / K ** 0.5).to(BF)
    runs = []
    for ctas in (0, _sms() - 2):
        monkeypatch.setattr(k, "GEMM_MAX_CTAS", ctas)
        x13, act = k.gemm_glu_fwd(x, w)
        runs.append((x13, act, *k.gemm_glu_bwd(dy, w2, x13)))
    assert all(torch.equal(p, q) for p, q in zip(*runs))
    x13, act, dx13, act2 = runs[0]
    _close(x13, x.double() @ w.double().t(), K)
    g, u = x13[:, :F].double(), x13[:, F:].double()                # (the rounded values are what the backward reads)
    s = torch.sigmoid(g)
    assert torch.equal(act, act2) or ((act.double() - act2.double()).abs() <= 2.0 ** -7 * act.double().abs()).all()
    # the forward's activation is taken from the sums before they are rounded: 2^-9 each of g and u, and its own rounding
    assert ((act2.double() - g * s * u).abs() <= 2.0 ** -8 * (g * s * u).abs() + 1e-6).all()
    assert ((act.double() - g * s * u).abs() <= 2.0 ** -7 * ((g * s * u).abs() + (u * (s + g * s * (1 - s)) * g).abs()) + 1e-6).all()
    dact = dy.double() @ w2.double()
    want = torch.cat([dact * u * (s + g * s * (1 - s)), dact * g * s], 1)
    size = K ** 1.5 * 2.0 ** -27 / K ** 0.5 * torch.cat([u.abs() * 1.1, g.abs()], 1)
    assert ((dx13.double() - want).abs() <= 2.0 ** -8 * want.abs() + size + 1e-5).all()
    assert k.device_error_words().get("gemm_tcgen05", 0) == 0
