"""Gradients of adapters that share an input (csrc/lora.cu) against fp64 and against the four GEMMs that they stand in for."""
import pytest
import torch

from flextrain_b200 import ops
from flextrain_b200.ops import cuda

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _inputs(T, K, N, R, gt, pad=0):
    torch.manual_seed(T + K + R)
    x = torch.randn(T, K + pad, device="cuda").to(BF)[:, :K]
    dy = torch.randn(T, sum(N) + pad, device="cuda").to(BF)
    adapters, c = [], 0
    for n in N:
        a, b = (torch.randn(R, K, device="cuda") / K ** 0.5).to(BF), (torch.randn(n, R, device="cuda") / n ** 0.5).to(BF)
        adapters.append((dy[:, c:c + n], a, b, torch.randn(R, K, device="cuda").to(gt), torch.randn(n, R, device="cuda").to(gt)))
        c += n
    return x, adapters


def _check(x, adapters, run, scale=0.7):
    want, size = [], []
    for dy, a, b, ga, gb in adapters:
        d, X, dyb, xa = dy.double(), x.double(), dy.double() @ b.double(), x.double() @ a.double().t()
        want.append((ga.double() + scale * dyb.t() @ X, gb.double() + scale * d.t() @ xa))
        # what can be off: the rank-r intermediates are rounded to bf16 (2^-9 each, an error that adds up over the tokens like the
        # root of the sum of squares; 6 of those for the largest of all elements), sums in fp32, the gradient rounded once
        size.append((scale * 6 * 2.0 ** -9 * ((dyb ** 2).t() @ X ** 2).sqrt(), scale * 6 * 2.0 ** -9 * ((d ** 2).t() @ xa ** 2).sqrt()))
    run(x, adapters, scale)
    for ad, w, e in zip(adapters, want, size):
        for g, v, err in zip(ad[3:], w, e):
            ulp = 2.0 ** -8 if g.dtype == BF else 2.0 ** -16
            assert ((g.double() - v).abs() <= err + ulp * v.abs() + 1e-6).all()


@pytest.mark.parametrize("gt", [BF, torch.float32])
@pytest.mark.parametrize("R", [8, 16, 32])
@pytest.mark.parametrize("T,K,N", [(1, 32, (32,)), (31, 64, (160, 32)), (65, 96, (32, 96, 128)), (257, 128, (416, 64, 64)),
                                   (700, 2080, (96,)), (8191, 96, (32, 64)), (8193, 96, (128, 32, 32)), (8320, 544, (1056,))])
def test_adapter_gradients(T, K, N, R, gt):
    x, ad = _inputs(T, K, N, R, gt, pad=8)
    assert cuda.lora_wgrad_supported(x, ad)
    again = [t[:3] + (t[3].clone(), t[4].clone()) for t in ad]
    _check(x, ad, ops.lora_wgrad)
    ops.lora_wgrad(x, again, 0.7)
    assert all(torch.equal(p, q) for s, t in zip(ad, again) for p, q in zip(s[3:], t[3:]))


@pytest.mark.parametrize("case", ["rank 4", "40 columns", "four", "odd stride", "gradient types", "rows apart", "turned rows"])
def test_other_forms_keep_the_gemms(case):
    """What the kernels do not take runs as four GEMMs per adapter, with the same result."""
    T, K, N, R = 96, 64, (64, 32), 16
    if case == "rank 4":
        R = 4
    elif case == "40 columns":
        K = 40
    elif case == "four":
        N = (32, 32, 32, 32)
    x, ad = _inputs(T, K, N, R, BF, pad=1 if case == "odd stride" else 8)
    if case == "gradient types":
        ad[0] = ad[0][:4] + (ad[0][4].float(),)
    elif case == "rows apart":
        ad[1] = (ad[1][0].contiguous(),) + ad[1][1:]
    elif case == "turned rows":
        ad = [(d.t().contiguous().t(),) + tuple(r) for d, *r in ad]
        assert ad[0][0].stride(-1) != 1
        _check(x, ad, ops.lora_wgrad)
        return
    assert not cuda.lora_wgrad_supported(x, ad)
    _check(x, ad, ops.lora_wgrad)


@pytest.mark.parametrize("rows", [(64, 32, 32), (1000,), (2048, 256)])
def test_merged_weight_from_the_base_in_place(rows):
    """The same bits as the product added to a copy of the weight, the base untouched; a member without an adapter is copied."""
    from flextrain_b200.nn.blocks.linear import LinearGroup, LoRAConfig
    torch.manual_seed(0)
    names = [f"w_{i}" for i in range(len(rows))]
    lora = LoRAConfig(targets=tuple(names[:2]), rank=16, alpha=8.0)
    p = {n: torch.randn(r, 256, device="cuda").to(BF) for n, r in zip(names, rows)}
    for n, r in zip(names[:2], rows):
        p[n + "_lora_a"], p[n + "_lora_b"] = torch.randn(16, 256, device="cuda").to(BF), torch.randn(r, 16, device="cuda").to(BF)
    base = {n: p[n].clone() for n in names}
    want = torch.cat([base[n] for n in names])
    for n, o in zip(names[:2], (0, rows[0])):
        ops.gemm(p[n + "_lora_b"], p[n + "_lora_a"], alpha=lora.scale, beta=1.0, out=want[o:o + p[n].shape[0]])
    assert torch.equal(LinearGroup(names, lora).weight(p), want)
    assert all(torch.equal(p[n], base[n]) for n in names)


def test_two_threads():
    """One adapter in one thread and three in another, whose launches take different amounts of shared memory."""
    import threading
    errors = []

    def work(N):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                x, ad = _inputs(64, 64, N, 32, torch.float32)
                want = [t.clone() for a in ad for t in a[3:]]
                ops.lora_wgrad(x, ad, 1.0)
                step = [t - w for t, w in zip((t for a in ad for t in a[3:]), want)]
                for _ in range(1500):
                    ops.lora_wgrad(x, ad, 1.0)
                for t, w, s in zip((t for a in ad for t in a[3:]), want, step):       # 1501 additions, each rounded in fp32
                    assert (t - w - 1501 * s).abs().max() <= 1501 * 2.0 ** -22 * (w.abs() + 1501 * s.abs()).max()
        except Exception as e:                     # noqa: BLE001 (reported in the main thread)
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(n,)) for n in ((32,), (32, 32, 32), (32,))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
