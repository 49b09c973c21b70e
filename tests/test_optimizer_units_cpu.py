"""The update of all resident layers at once does what ``optimizer.step`` on each layer does: finite-gradient checks of the
optimizer and of the ones it delegates to, replaced ``step`` methods and optimizers without a batched form are honoured."""
import pytest
import torch

import flextrain_b200 as ft
from conftest import build_tiny

F32 = torch.float32


def hybrid(**kw):
    kw = {"muon": ft.Muon(lr=1e-2), "adamw": ft.AdamW(lr=1e-3, state_dtype=F32), **kw}
    return ft.HybridMuonAdamW(**kw)


def model(optimizer):
    """Two layers with the gradients of one step."""
    am = build_tiny(optimizer=optimizer)
    am.fwd_bwd(ft.SyntheticTokenSource(1024, 128, seed=0).get_sequences(256))
    return am


def weights(am, l):
    return {k: v.clone() for k, v in am.buffers.params(l).items()}


CHECKED = {
    "hybrid": lambda: hybrid(check_error=True),
    "hybrid_muon": lambda: hybrid(muon=ft.Muon(lr=1e-2, check_error=True)),
    "hybrid_adamw": lambda: hybrid(adamw=ft.AdamW(lr=1e-3, state_dtype=F32, check_error=True)),
    "hybrid_both": lambda: hybrid(muon=ft.Muon(lr=1e-2, check_error=True),
                                  adamw=ft.AdamW(lr=1e-3, state_dtype=F32, check_error=True)),
    "adamw": lambda: ft.AdamW(lr=1e-3, state_dtype=F32, check_error=True),
}


@pytest.mark.parametrize("name", list(CHECKED))
def test_nan_gradient_is_reported_and_reaches_no_weight(name):
    """A NaN in the second layer's gradient of a tensor that the checking optimizer updates: the first layer is updated, the
    step reports an error, and of the second layer the weights that this optimizer updates stay as they are (all of them, when
    the outer optimizer checks)."""
    am = model(CHECKED[name]())
    g, owned = ("g_attn_norm", ("w_attn_norm", "w_ffn_norm")) if name == "hybrid_adamw" else ("g_q", ("w_q", "w_k", "w_1"))
    am.buffers.grads(1)[g].view(-1)[3] = float("nan")
    first, second = weights(am, 0), weights(am, 1)
    assert am.step() != 0
    assert any(not torch.equal(first[k], v) for k, v in am.buffers.params(0).items())
    for k, v in am.buffers.params(1).items():
        assert torch.isfinite(v).all()
        if k in owned or name in ("hybrid", "adamw"):
            assert torch.equal(second[k], v)


class CountedMuon(ft.Muon):
    def step(self, *args, **kw):
        self.calls = getattr(self, "calls", 0) + 1
        return super().step(*args, **kw)


class StepOnly:
    """An inner optimizer with ``step`` and no batched form."""

    def __init__(self):
        self.real, self.calls, self.lr = ft.Muon(lr=1e-2), 0, 1e-2

    def state_specs(self, param_spec):
        return self.real.state_specs(param_spec)

    def step(self, *args, **kw):
        self.calls += 1
        return self.real.step(*args, **kw)


@pytest.mark.parametrize("inner", [CountedMuon, StepOnly])
def test_a_replaced_inner_step_is_called_for_every_unit(inner):
    muon = inner() if inner is StepOnly else inner(lr=1e-2)
    am, plain = model(hybrid(muon=muon)), model(hybrid())
    assert am.step() == 0 and plain.step() == 0
    assert muon.calls == 2 + 2                      # embedding, head and two layers
    for l in range(2):
        for k, v in am.buffers.params(l).items():
            assert torch.equal(v, plain.buffers.params(l)[k])


def test_a_step_replaced_on_the_inner_object_is_called():
    opt = hybrid()
    seen, step = [], opt.adamw.step
    opt.adamw.step = lambda *a, **kw: (seen.append(1), step(*a, **kw))[1]
    am = model(opt)
    assert am.step() == 0 and len(seen) == 4


def test_a_subclass_may_split_the_tensors_its_own_way():
    class Rows(ft.HybridMuonAdamW):
        def _split(self, param_spec):
            names = [t.name for t in param_spec.trainable()]
            return [n for n in names if n in ("w_q", "w_k")], [n for n in names if n not in ("w_q", "w_k")]

    am = model(Rows(muon=ft.Muon(lr=1e-2), adamw=ft.AdamW(lr=1e-3, state_dtype=F32)))
    assert set(k for k in am.buffers.opt_state(0) if "muon" in k) == {"o_muon_q", "o_muon_k"}
    before = weights(am, 1)
    assert am.step() == 0
    assert all(not torch.equal(before[k], v) for k, v in am.buffers.params(1).items())


@pytest.mark.parametrize("shape", [(64, 96), (96, 64), (64, 64)])
def test_one_matrix_is_orthogonalised(shape):
    """The op on one matrix, bf16 iterates here through the plain GEMM, against the fp32 iteration (2 % from five steps)."""
    from flextrain_b200 import ops
    from flextrain_b200.ops import reference as ref
    torch.manual_seed(0)
    u = torch.randn(*shape)
    got, want = ops.newton_schulz_bf16(u), ref.newton_schulz(u)
    assert got.dtype == torch.bfloat16 and got.shape == u.shape
    assert float(torch.nn.functional.cosine_similarity(got.float().flatten(), want.flatten(), dim=0)) > 0.98
