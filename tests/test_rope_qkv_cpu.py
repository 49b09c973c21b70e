"""``rope_qkv``: which tensors it takes.  The kernel reads and writes all of them for the tokens and heads of one, so what does not
fit together is refused before it."""
import pytest
import torch

from flextrain_b200 import ops
from flextrain_b200.ops import cuda

HD = 64


class OnGpu:
    """The properties of a tensor on a GPU that the predicate looks at."""
    is_cuda = True

    def __init__(self, *shape, dtype=torch.bfloat16):
        self._t = torch.empty(shape, dtype=dtype)
        self.shape, self.dtype, self.stride = self._t.shape, dtype, self._t.stride

    def data_ptr(self):
        return 1024


def _call(T=4, q=None, k=None, v=None, q_out=None, k_out=None, v_out=None, new=torch.zeros):
    one = lambda given, heads: new(*(given or (T, heads, HD)))
    return dict(q=one(q, 4), k=one(k, 2), v=one(v, 2), q_out=one(q_out, 4), k_out=one(k_out, 2), v_out=one(v_out, 2))


WRONG = [dict(k=(3, 2, HD)), dict(k=(5, 2, HD)), dict(k=(1, 2, HD)), dict(v=(5, 2, HD)), dict(v=(1, 2, HD)), dict(q=(1, 4, HD)),
         dict(q_out=(3, 4, HD)), dict(k_out=(4, 1, HD)), dict(v=(4, 1, HD)), dict(q=(4, 1, HD))]


@pytest.mark.parametrize("wrong", WRONG)
def test_shapes_that_do_not_fit(wrong):
    inv = torch.ones(HD // 2)
    with pytest.raises(ValueError):
        ops.rope_qkv(positions=torch.arange(4), inv_freq=inv, **_call(**wrong))
    t = _call(**wrong, new=OnGpu)
    assert not cuda.rope_qkv_supported(t["q"], t["k"], t["v"], t["q_out"], t["k_out"], t["v_out"], torch.arange(4), inv, None)


@pytest.mark.parametrize("positions", [1, 3, 5])
def test_positions_that_do_not_fit(positions):
    inv = torch.ones(HD // 2)
    with pytest.raises(ValueError):
        ops.rope_qkv(positions=torch.arange(positions), inv_freq=inv, **_call())
    t = _call(new=OnGpu)
    assert not cuda.rope_qkv_supported(t["q"], t["k"], t["v"], t["q_out"], t["k_out"], t["v_out"], torch.arange(positions), inv, None)


def test_shapes_that_fit():
    inv = torch.ones(HD // 2)
    t = _call()
    for x in (t["q"], t["k"], t["v"]):
        x.normal_()
    ops.rope_qkv(positions=torch.arange(4), inv_freq=inv, **t)
    assert torch.equal(t["v_out"], t["v"]) and not torch.equal(t["k_out"], t["k"])
    torch.testing.assert_close(t["q_out"].norm(), t["q"].norm())
    ops.rope_qkv(None, t["k"], None, torch.stack([torch.arange(4)] * 3, 1), inv, q_out=None, k_out=t["k_out"], v_out=None,
                 mrope_sections=(16, 8, 8))
    t = _call(new=OnGpu)
    assert cuda.rope_qkv_supported(t["q"], t["k"], t["v"], t["q_out"], t["k_out"], t["v_out"], torch.arange(4), inv, None)
    assert cuda.rope_qkv_supported(None, t["k"], None, None, t["k_out"], None, torch.arange(4), inv, None)
