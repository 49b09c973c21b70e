"""Gated DeltaNet in chunks (heads of 128 x 128) against the token recurrence in float64, at sequence lengths around the chunk
of 64 tokens and its 16-token blocks."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV, BF, F64 = "cuda", torch.bfloat16, torch.float64


def _cu(lens):
    return torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)


def _inputs(lens, HK, HV, decay, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)
    T = sum(lens)
    q, k = (F.normalize(r(T, HK, 128) + 0.2, dim=-1).to(BF) for _ in range(2))
    beta = torch.rand(T, HV, device=DEV, generator=g)
    return q, k, r(T, HV, 128).to(BF), -torch.rand(T, HV, device=DEV, generator=g) * decay, beta, r(T, HV, 128).to(BF)


def _recurrence(q, k, v, g, beta, s0, lens, scale):
    rep = v.shape[1] // q.shape[1]
    q, k = q.repeat_interleave(rep, 1) * scale, k.repeat_interleave(rep, 1)
    out, fin, a = [], [], 0
    for i, n in enumerate(lens):
        S = s0[i]
        for t in range(a, a + n):
            S = S * g[t].exp()[:, None, None]
            e = beta[t][:, None] * (v[t] - torch.einsum("hk,hkv->hv", k[t], S))
            S = S + k[t][:, :, None] * e[:, None]
            out.append(torch.einsum("hk,hkv->hv", q[t], S))
        fin.append(S)
        a += n
    return torch.stack(out), torch.stack(fin)


def _rel(a, b):
    a, b = a.detach().double(), b.detach().double()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


@pytest.mark.parametrize("lens,HK,HV,decay,with_state", [
    ([1], 1, 1, 0.2, True),                        # token by token
    ([63, 64, 65, 1, 17], 2, 4, 0.2, True),
    ([40], 1, 1, 0.2, True),                       # the shortest that goes in a chunk
    ([128, 0, 129], 1, 3, 0.2, True),              # an empty sequence, an odd number of value heads
    ([200], 2, 2, 0.0, False),                     # no decay at all
    ([150, 90], 1, 2, 5.0, True),                  # strong decay: most of a chunk forgotten inside it
])
def test_chunks_against_the_recurrence(lens, HK, HV, decay, with_state):
    from flextrain_b200.ops import linattn_cuda as la
    q, k, v, g, beta, do = _inputs(lens, HK, HV, decay)
    beta[0] = 0                                    # a token that writes nothing still has a gradient of its gate
    if sum(lens) > 70:
        g[70] = -1e4                               # a token that forgets everything before it
    S, scale = len(lens), 128 ** -0.5
    s0 = torch.randn(S, HV, 128, 128, device=DEV) * 0.2 if with_state else None
    df = torch.randn(S, HV, 128, 128, device=DEV) * 0.1 if with_state else None
    wide = torch.empty(sum(lens), 3 * HV * 128, dtype=BF, device=DEV)              # v and dv as columns of wider tensors
    vv = wide[:, HV * 128:2 * HV * 128].unflatten(1, (HV, 128))
    vv.copy_(v)
    dwide = torch.full_like(wide, 7.0)
    cu = _cu(lens)
    o, fin, r = la.gdn_fwd(q, k, vv, g, beta, cu, s0, want_r=True)
    dq, dk, dv, dg, db, ds = la.gdn_bwd(q, k, vv, g, beta, cu, s0, fin, r, do, dstate_final=df,
                                        dv_out=dwide[:, :HV * 128].unflatten(1, (HV, 128)))
    assert bool((dwide[:, HV * 128:] == 7.0).all()) and dv.data_ptr() == dwide.data_ptr()
    zero = torch.zeros(S, HV, 128, 128, device=DEV, dtype=F64)
    leaves = [t.double().requires_grad_(True) for t in (q, k, v, g, beta)]
    leaves.append((zero if s0 is None else s0.double()).requires_grad_(True))
    ow, fw = _recurrence(*leaves, lens, scale)
    wq, wk, wv, wg, wb, ws = torch.autograd.grad([ow, fw], leaves, [do.double(), zero if df is None else df.double()])
    # bf16 results: half a unit in the last of 8 bits, 2^-9 of each element at most.  fp32 results: sums of up to a few hundred
    # products through a solve whose factors stay below 1; 2e-5 leaves two orders over 2^-24.  dg sums over all later tokens
    # differences of terms that nearly cancel.
    assert _rel(o, ow) < 2.0 ** -9 and _rel(dv, wv) < 2.0 ** -9
    for got, want in ((fin, fw), (dq, wq), (dk, wk), (db, wb), (ds, ws)):
        assert _rel(got, want) < 2e-5
    assert _rel(dg, wg) < 1e-4


def test_chunks_run_twice_give_the_same_bits():
    from flextrain_b200.ops import linattn_cuda as la
    lens = [300, 40, 1000]
    q, k, v, g, beta, do = _inputs(lens, 2, 4, 1.0)
    cu, runs = _cu(lens), []
    for _ in range(2):
        o, fin, r = la.gdn_fwd(q, k, v, g, beta, cu, want_r=True)
        runs.append((o, fin, r) + la.gdn_bwd(q, k, v, g, beta, cu, None, fin, r, do))
    assert all(torch.equal(a, b) for a, b in zip(*runs))


def test_sequences_do_not_meet_and_heads_add_up():
    """A sequence alone gives what it gives among others, and the value heads' dq / dk add up to their key head's."""
    from flextrain_b200.ops import linattn_cuda as la
    lens = [100, 64, 333]
    q, k, v, g, beta, do = _inputs(lens, 2, 4, 0.5)
    cu = _cu(lens)
    o, fin, r = la.gdn_fwd(q, k, v, g, beta, cu, want_r=True)
    all_ = la.gdn_bwd(q, k, v, g, beta, cu, None, fin, r, do)
    per_head = la.gdn_bwd(q, k, v, g, beta, cu, None, fin, r, do, sum_heads=False)
    for i in (0, 1):
        assert torch.equal(all_[i], per_head[i].view(sum(lens), 2, 2, 128).sum(2))
    w = slice(100, 164)
    part = [t[w].contiguous() for t in (q, k, v, g, beta, do)]
    o1, fin1, r1 = la.gdn_fwd(*part[:5], _cu([64]), want_r=True)
    one = la.gdn_bwd(*part[:5], _cu([64]), None, fin1, r1, part[5])
    assert torch.equal(o[w], o1) and torch.equal(fin[1], fin1[0])
    for a, b in zip(all_[:5], one[:5]):
        assert torch.equal(a[w], b)


@pytest.mark.parametrize("ends", [[3, 64, 200], [0, 64, 150], [70, 130, 190]])
def test_tokens_of_no_sequence(ends):
    """Sequences that leave tokens out: their gradients are 0, the others' as without them, and the error word says so."""
    from flextrain_b200.ops import linattn_cuda as la
    from flextrain_b200.ops.cuda import device_error_words
    T = 200
    q, k, v, g, beta, do = _inputs([T], 2, 4, 0.5)
    cu = torch.tensor(ends, dtype=torch.int32, device=DEV)
    device_error_words()
    o, fin, r = la.gdn_fwd(q, k, v, g, beta, cu, want_r=True)
    dq, dk, dv, dg, db, _ = la.gdn_bwd(q, k, v, g, beta, cu, None, fin, r, do)
    assert device_error_words()["gdn"] == 3300
    w = slice(ends[0], ends[-1])
    part = [t[w].contiguous() for t in (q, k, v, g, beta, do)]
    o1, fin1, r1 = la.gdn_fwd(*part[:5], cu - ends[0], want_r=True)
    one = la.gdn_bwd(*part[:5], cu - ends[0], None, fin1, r1, part[5])
    assert torch.equal(o[w], o1)
    for got, want in zip((dq, dk, dv, dg, db), one):
        assert torch.equal(got[w], want)
    for t in (dq, dk, dg, db):
        assert float(t[:ends[0]].abs().sum() + t[ends[-1]:].abs().sum()) == 0.0


def test_rows_off_the_16_byte_grid_take_the_recurrent_kernels():
    from flextrain_b200.ops import linattn_cuda as la
    lens = [90]
    q, k, v, g, beta, do = _inputs(lens, 1, 2, 0.5)
    buf = torch.empty(v.numel() + 1, dtype=BF, device=DEV)
    odd = buf[1:].view_as(v).copy_(v)
    a, b = la.gdn_fwd(q, k, v, g, beta, _cu(lens))[:2], la.gdn_fwd(q, k, odd, g, beta, _cu(lens))[:2]
    assert _rel(a[0], b[0]) < 2.0 ** -8 and _rel(a[1], b[1]) < 2e-5


@pytest.mark.parametrize("gates", ["strong", "model", "slow", "none"])
def test_precision_is_that_of_fp32(gates):
    """Errors in units of 2^-24, the rounding of fp32, over sequences of several chunks.  A result goes through some ten roundings
    (16 allowed; measured 1 to 5); a product that kept two bf16 terms of an fp32 operand, 2^-16 of it cut off, would be off by a
    hundred.  dg adds up, over all later tokens, differences that cancel to a tenth and less (256 allowed; measured 7 to 60)."""
    from flextrain_b200.ops import linattn_cuda as la
    lens, HK, HV = [256, 200, 300], 2, 4
    T = sum(lens)
    q, k, v, _, beta, do = _inputs(lens, HK, HV, 1.0)
    gen = torch.Generator(device=DEV).manual_seed(1)
    n = torch.randn(T, HV, device=DEV, generator=gen)
    g = {"strong": -F.softplus(n + 1), "model": -F.softplus(n - 4) * torch.tensor([1.0, 4, 9, 16], device=DEV),
         "slow": -0.01 * n.abs(), "none": torch.zeros_like(n)}[gates]
    cu = _cu(lens)
    o, fin, r = la.gdn_fwd(q, k, v, g, beta, cu, want_r=True)
    got = la.gdn_bwd(q, k, v, g, beta, cu, None, fin, r, do)
    leaves = [t.double().requires_grad_(True) for t in (q, k, v, g, beta)]
    zero = torch.zeros(len(lens), HV, 128, 128, device=DEV, dtype=F64)
    ow, fw = _recurrence(*leaves, zero, lens, 128 ** -0.5)
    wq, wk, _, wg, wb = torch.autograd.grad(ow, leaves, do.double())
    for a, w, units in ((fin, fw, 16), (got[0], wq, 16), (got[1], wk, 16), (got[4], wb, 16), (got[3], wg, 256)):
        assert _rel(a, w) <= units * 2.0 ** -24
