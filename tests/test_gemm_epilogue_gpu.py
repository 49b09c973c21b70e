"""The two-SM GEMM's epilogue (rows turned over in shared memory, 128 bytes at a time) and its grouped forms, at the sizes
where pieces, row tiles and groups end.  Operands are bf16, sums fp32: against float64 a bf16 result is off by half a unit in
the last place (2^-9 relative) and an fp32 one by the order of the additions (K * 2^-24 of the sum of magnitudes)."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _close(got, want, mag, K):
    room = (2.0 ** -8 * want.abs() if got.dtype == torch.bfloat16 else 0) + K * 2.0 ** -23 * mag + 1e-6
    assert torch.all((got.double() - want).abs() <= room)


@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N,K", [(512, 512, 64), (513, 520, 72), (767, 584, 136), (640, 1000, 64), (1025, 776, 200)])
@pytest.mark.parametrize("ta,tb", [(False, True), (False, False), (True, False)])
def test_two_sm_epilogue(out_dtype, M, N, K, ta, tb):
    """Plain, with bias, with C in place, with C of another row stride, into a strided D whose neighbours stay as they are."""
    from flextrain_b200.ops import cuda as k
    torch.manual_seed(0)
    Mp = (M + 7) // 8 * 8
    a = torch.randn(K, Mp, device=DEV).bfloat16()[:, :M] if ta else torch.randn(M, K, device=DEV).bfloat16()
    b = (torch.randn(N, K, device=DEV) if tb else torch.randn(K, N, device=DEV)).bfloat16()
    A, B = (a.t() if ta else a).double(), (b.t() if tb else b).double()
    prod, mag = A @ B, A.abs() @ B.abs()
    _close(k.gemm(a, b, trans_a=ta, trans_b=tb, out_dtype=out_dtype, bn=512), prod, mag, K)
    bias = torch.randn(N, device=DEV)
    got = k.gemm(a, b, trans_a=ta, trans_b=tb, out_dtype=out_dtype, alpha=0.5, bias=bias, bn=512)
    _close(got, 0.5 * prod + bias.double(), mag, K)
    wide = torch.randn(M, N + 24, device=DEV).to(out_dtype)
    keep = wide.clone()
    k.gemm(a, b, trans_a=ta, trans_b=tb, beta=1.0, out=wide[:, 8:8 + N], bn=512)
    _close(wide[:, 8:8 + N], prod + keep[:, 8:8 + N].double(), mag, K)
    assert torch.equal(wide[:, :8], keep[:, :8]) and torch.equal(wide[:, 8 + N:], keep[:, 8 + N:])
    c = torch.randn(M, N + 16, device=DEV).to(out_dtype)[:, 16:]
    got = k.gemm(a, b, trans_a=ta, trans_b=tb, beta=-2.0, c=c, out_dtype=out_dtype, bn=512)
    _close(got, prod - 2.0 * c.double(), mag, K)
    assert k.device_error_words().get("gemm_tcgen05", 0) == 0


COUNTS = {"even": [512] * 6, "odd_tiles": [128, 384, 640, 0, 1152, 256], "one_holds_all": [0, 0, 3072, 0, 0, 0]}


@pytest.mark.parametrize("counts", list(COUNTS))
@pytest.mark.parametrize("N,K", [(256, 64), (520, 136), (776, 1024)])
def test_grouped_two_sm(counts, N, K):
    """Row groups of multiples of 128 rows, some empty, in a buffer with room behind them that is not written."""
    from flextrain_b200.ops import cuda as k
    torch.manual_seed(0)
    cnt = COUNTS[counts]
    E, used = len(cnt), sum(cnt)
    R = used + 256
    off = torch.tensor([0] + list(torch.tensor(cnt).cumsum(0)), dtype=torch.int32, device=DEV)
    x = torch.randn(R, K, device=DEV).bfloat16()
    x[used:] = float("nan")
    for trans_w in (True, False):
        w = torch.randn(*((E, N, K) if trans_w else (E, K, N)), device=DEV).bfloat16()
        for beta in (0.0, 1.0):
            out = torch.randn(R, N, device=DEV).bfloat16()
            before = out.clone()
            k.grouped_gemm(x, w, off, trans_w=trans_w, out=out, beta=beta)
            for e in range(E):
                s = slice(int(off[e]), int(off[e + 1]))
                W = (w[e].t() if trans_w else w[e]).double()
                _close(out[s], x[s].double() @ W + beta * before[s].double(), x[s].double().abs() @ W.abs(), K)
            assert torch.equal(out[used:], before[used:])
    dy = torch.randn(R, N, device=DEV).bfloat16()
    x[used:] = 0
    Kd = max(K, 256)
    xx = torch.randn(R, Kd, device=DEV).bfloat16()
    for dt in (torch.bfloat16, torch.float32):
        for acc in (False, True):
            g = torch.randn(E, N, Kd, device=DEV).to(dt)
            before = g.clone()
            k.grouped_wgrad(dy, xx, off, g, accumulate=acc)
            for e in range(E):
                s = slice(int(off[e]), int(off[e + 1]))
                if cnt[e] == 0:
                    assert torch.equal(g[e], before[e])
                    continue
                want = dy[s].double().t() @ xx[s].double() + (before[e].double() if acc else 0)
                _close(g[e], want, dy[s].double().abs().t() @ xx[s].double().abs(), cnt[e])
    assert k.device_error_words().get("gemm_tcgen05", 0) == 0


@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N,K", [(512, 512, 4096), (768, 520, 8200), (1000, 776, 16384)])
@pytest.mark.parametrize("ta,tb", [(True, False), (False, False), (False, True)])
def test_two_sm_split_k(out_dtype, M, N, K, ta, tb):
    """Few tiles and a long reduction: slices of K on two-SM tiles, the last one shorter, with C, bias and a strided D."""
    from flextrain_b200.ops import cuda as k
    assert k._two_sm_splits(M, N, K) > 1
    torch.manual_seed(0)
    a = (torch.randn(K, M, device=DEV) if ta else torch.randn(M, K, device=DEV)).bfloat16()
    b = (torch.randn(N, K, device=DEV) if tb else torch.randn(K, N, device=DEV)).bfloat16()
    A, B = (a.t() if ta else a).double(), (b.t() if tb else b).double()
    prod, mag = A @ B, A.abs() @ B.abs()
    bias = torch.randn(N, device=DEV)
    wide = torch.randn(M, N + 24, device=DEV).to(out_dtype)
    keep = wide.clone()
    k.gemm(a, b, trans_a=ta, trans_b=tb, alpha=0.5, beta=1.0, bias=bias, out=wide[:, 8:8 + N])
    _close(wide[:, 8:8 + N], 0.5 * prod + bias.double() + keep[:, 8:8 + N].double(), mag, K)
    assert torch.equal(wide[:, :8], keep[:, :8]) and torch.equal(wide[:, 8 + N:], keep[:, 8 + N:])
    assert k.device_error_words().get("gemm_tcgen05", 0) == 0
