"""Infinities and NaN in the chunked Gated DeltaNet: they reach the same elements as in the recurrence token by token (which takes
tensors that do not start on 16 bytes), tokens before them and other sequences and heads keep their values."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16
LENS, HK, HV = [100, 70, 133], 2, 4
BAD = 100 + 35                                     # a token of the second sequence, amid a block of 16, and a value head
HEAD = 1


def _inputs():
    g = torch.Generator(device=DEV).manual_seed(0)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)
    T, S = sum(LENS), len(LENS)
    q, k = (F.normalize(r(T, HK, 128) + 0.2, dim=-1).to(BF) for _ in range(2))
    return dict(q=q, k=k, v=r(T, HV, 128).to(BF), g=-torch.rand(T, HV, device=DEV, generator=g) * 0.3,
                beta=torch.rand(T, HV, device=DEV, generator=g), d_o=r(T, HV, 128).to(BF), state=r(S, HV, 128, 128) * 0.2,
                dstate=r(S, HV, 128, 128) * 0.1)


def _odd(x):
    return torch.empty(x.numel() + 1, dtype=x.dtype, device=DEV)[1:].view_as(x).copy_(x)


def _same(a, b, tol):
    """The same elements are finite, NaN, or an infinity of one sign; the finite ones are as close as the two forms are."""
    assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf())
    assert torch.equal(a[a.isinf()], b[b.isinf()])
    a, b = (torch.where(x.isfinite(), x, 0).double() for x in (a, b))
    assert (a - b).norm() <= tol * b.norm()


@pytest.mark.parametrize("where", ["v", "q", "k", "g", "beta", "d_o", "state", "dstate", "none"])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf")])
def test_non_finite_values(where, value):
    from flextrain_b200.ops import linattn_cuda as la
    t = _inputs()
    if where in ("state", "dstate"):
        t[where][1, HEAD, 5, 77] = value
    elif where in ("g", "beta"):
        t[where][BAD, HEAD] = value
    elif where != "none":
        t[where][BAD, 0 if where in "qk" else HEAD, 77] = value
    cu = torch.tensor([0] + list(torch.tensor(LENS).cumsum(0)), dtype=torch.int32, device=DEV)
    first = [t[n] for n in ("q", "k", "v", "g", "beta")]
    odd = first[:2] + [_odd(t["v"])] + first[3:]
    T, S = sum(LENS), len(LENS)
    assert la._chunked(S, *(first[i] for i in (0, 2, 1))) and not la._chunked(S, *(odd[i] for i in (0, 2, 1)))
    got, want = (la.gdn_fwd(*x, cu, t["state"], want_r=True) for x in (first, odd))
    for a, b, tol in zip(got, want, (2.0 ** -8, 2e-5, 2e-5)):
        _same(a, b, tol)
    o = got[0]
    if where != "state":
        assert o[:BAD].isfinite().all()
    assert o[:100].isfinite().all() and o[170:].isfinite().all() and o[:, 2:].isfinite().all()
    _, fin, r = want
    wide = torch.full((T, 3 * HV * 128), 7.0, dtype=BF, device=DEV)               # v and dv as columns of wider tensors
    columns = [wide[:, i * HV * 128:(i + 1) * HV * 128].unflatten(1, (HV, 128)) for i in range(3)]
    first[2] = columns[1].copy_(t["v"])
    again = la.gdn_fwd(*first, cu, t["state"], want_r=True)
    assert all(torch.equal(a.nan_to_num(), b.nan_to_num()) for a, b in zip(again, got))
    back = lambda x: la.gdn_bwd(*x, cu, t["state"], fin, r, t["d_o"], dstate_final=t["dstate"],
                                dv_out=columns[2] if x is first else None)
    for a, b, tol in zip(back(first), back(odd), (2e-5, 2e-5, 2.0 ** -8, 1e-4, 2e-5, 2e-5)):
        _same(a, b, tol)
    assert bool((columns[0] == 7.0).all()) and torch.equal(columns[1].nan_to_num(), t["v"].nan_to_num())


def test_a_product_that_overflows():
    """Values near the largest of fp32's range: a state that becomes infinite does so at its own token."""
    from flextrain_b200.ops import linattn_cuda as la
    t = _inputs()
    t["v"][BAD, HEAD, 3], t["g"][BAD + 1:, HEAD] = 3e38, 2.0
    cu = torch.tensor([0] + list(torch.tensor(LENS).cumsum(0)), dtype=torch.int32, device=DEV)
    first = [t[n] for n in ("q", "k", "v", "g", "beta")]
    got = la.gdn_fwd(*first, cu, t["state"], want_r=True)
    want = la.gdn_fwd(*first[:2], _odd(t["v"]), *first[3:], cu, t["state"], want_r=True)
    assert not want[1].isfinite().all() and got[0][:BAD].isfinite().all()
    for a, b, tol in zip(got, want, (2.0 ** -8, 2e-5, 2e-5)):
        _same(a, b, tol)
