"""Which pair of SMs works out which tile does not change a bit: products on all pairs, numbered die by die, against the same on
fewer pairs, which take the tiles in order; around one and two waves of the 74 pairs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles_m,tiles_n", [(2, 2), (73, 1), (37, 2), (5, 15), (49, 3), (74, 2), (149, 1), (9, 33)])
@pytest.mark.parametrize("K", [72, 8192])
def test_order_of_tiles(tiles_m, tiles_n, K, monkeypatch):
    from flextrain_b200.ops import cuda as kernels
    torch.manual_seed(0)
    M, N = tiles_m * 256 - 40, tiles_n * 256 - 8
    if M < 512 or N < 512:
        M, N = max(M, 512), max(N, 512)
    a, b, c = (torch.randn(*s, device="cuda").to(torch.bfloat16) for s in ((M, K), (N, K), (M, N)))
    monkeypatch.setattr(kernels, "_k_splits", lambda *s: 1)
    got = []
    for ctas in (0, 146):
        monkeypatch.setattr(kernels, "GEMM_MAX_CTAS", ctas)
        d = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
        got.append(kernels.gemm(a, b, trans_b=True, beta=1.0, c=c, out=d))
    assert torch.equal(*got)
    rows = torch.tensor([0, M // 2, M - 1], device="cuda")
    want = a[rows].double() @ b.double().t() + c[rows].double()
    assert (got[0][rows].double() - want).abs().max() <= 2.0 ** -8 * want.abs().max() + K * 2.0 ** -22


def test_pairs_have_one_number_each():
    import ctypes
    from flextrain_b200.ops.cuda import _stream, load
    out, n = (ctypes.c_ubyte * 80)(), ctypes.c_int(0)
    first = load("gemm_tcgen05").ftb_gemm_dies(out, ctypes.byref(n), _stream())
    assert n.value == torch.cuda.get_device_properties(0).multi_processor_count // 2
    assert first == 0 or (0 < first < n.value and sorted(out[:n.value]) == list(range(n.value)))
