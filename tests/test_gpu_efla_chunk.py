"""Chunked EFLA kernels at the edges of a chunk (32 tokens) and of the one-launch form (112 tokens of few states), against the fp32 token loop.

Bounds: outputs and k / v gradients are rounded to bf16 once (2^-9 of the value; 2^-8 of the largest allows for the fp32 noise of both
sides), states and their gradients stay in fp32 on both sides, where each of the T updates rounds at 2^-24: 1e-5 of the largest covers
T <= 130 updates of each side.
"""
import pytest
import torch

from elfa_b200 import native
from elfa_b200.ops import efla as eops

pytestmark = pytest.mark.gpu


def _inputs(dev, B, T, H, d, with_state, seed=0):
    g = torch.Generator(device=dev).manual_seed(seed)
    k = (torch.randn(B, T, H, d, generator=g, device=dev) * 0.4).bfloat16()
    v = torch.randn(B, T, H, d, generator=g, device=dev).bfloat16()
    s0 = 0.3 * torch.randn(B, H, d, d, generator=g, device=dev) if with_state else None
    return k, v, torch.tensor([0.3], device=dev), s0


def _close(a, b, rel):
    assert (a.float() - b.float()).abs().max() <= rel * b.float().abs().max()


@pytest.mark.parametrize("T", [1, 16, 17, 31, 32, 33, 65, 130])
@pytest.mark.parametrize("d", [32, 64, 96, 128])
def test_forward_at_chunk_edges(cuda_device, T, d):
    k, v, beta, s0 = _inputs(cuda_device, 2, T, 3, d, T % 2 == 1, seed=T + d)
    o, s = eops.efla_scan(k, v, beta, s0)
    o_ref, s_ref = eops.efla_scan_ref(k, v, beta, s0)
    assert native.status() == 0
    _close(o, o_ref, 2 ** -8)
    _close(s, s_ref, 1e-5)


def test_forward_takes_any_layout_and_offset(cuda_device):
    k, v, beta, _ = _inputs(cuda_device, 2, 40, 2, 64, False)
    want = eops.efla_scan(k, v, beta)
    odd = torch.empty(k.numel() + 1, dtype=k.dtype, device=cuda_device)[1:].view(k.shape)     # 2-byte aligned only
    odd.copy_(k)
    wide = torch.empty(2, 40, 2, 128, dtype=v.dtype, device=cuda_device)[..., :64]
    wide.copy_(v)
    got = eops.efla_scan(odd, wide, beta)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_a_bad_token_leaves_the_earlier_ones_alone(cuda_device, bad):
    k, v, beta, _ = _inputs(cuda_device, 1, 64, 1, 64, False)
    o0, _ = eops.efla_scan(k, v, beta)
    for which in (0, 1):
        kv = [k.clone(), v.clone()]
        kv[which][0, 40, 0, 5] = bad
        o, _ = eops.efla_scan(*kv, beta)
        assert torch.equal(o[0, :40], o0[0, :40])
        assert not torch.isfinite(o[0, 40, 0]).all()
        if which == 1:                      # a value touches its own column only
            keep = [j for j in range(64) if j != 5]
            assert torch.equal(o[0, :, 0, keep], o0[0, :, 0, keep])


@pytest.mark.parametrize("T", [1, 31, 32, 33, 65, 130])
@pytest.mark.parametrize("d", [32, 64, 96, 128])
def test_backward_at_chunk_edges(cuda_device, T, d):
    with_state = T % 2 == 1
    k, v, beta, s0 = _inputs(cuda_device, 2, T, 3, d, with_state, seed=T + d)
    go, gs = torch.randn_like(v), 0.1 * torch.randn(2, 3, d, d, device=cuda_device)
    grads = []
    for fn, cast in ((eops.efla_scan, lambda t: t), (eops.efla_scan_ref, lambda t: t.float())):
        ins = [t.detach().clone().requires_grad_(True) for t in (cast(k), cast(v), beta, s0) if t is not None]
        o, s = fn(*ins)
        grads.append(torch.autograd.grad([o, s], ins, [go.to(o.dtype), gs]))
    assert native.status() == 0
    got, ref = grads
    _close(got[0], ref[0], 2 ** -8)
    _close(got[1], ref[1], 2 ** -8)
    # beta: a sum over all tokens whose terms cancel; each term is off by at most 2^-20 of its size (about d products)
    assert abs(got[2] - ref[2]).item() <= 2e-5 * max(1.0, ref[2].abs().item()) + 1e-6 * T * d
    if with_state:
        _close(got[3], ref[3], 1e-5)


def test_backward_of_one_output_only(cuda_device):
    k, v, beta, _ = _inputs(cuda_device, 1, 50, 2, 64, False)
    k.requires_grad_(True)
    kr = k.detach().float().requires_grad_(True)
    eops.efla_scan(k, v, beta)[1].square().sum().backward()
    eops.efla_scan_ref(kr, v, beta)[1].square().sum().backward()
    _close(k.grad, kr.grad, 2 ** -8)


@pytest.mark.parametrize("d", [32, 64, 96, 128])
def test_an_infinite_value_gives_an_infinite_output(cuda_device, d):
    """o = p + c lam (v - p) is infinite for its token, the state gets the sign of the key, later outputs of the column are NaN; a column
    of a finite chunk keeps its bits. Token 40 is the last one, or one in the middle of its chunk."""
    for T in (41, 64):
        k, v, beta, s0 = _inputs(cuda_device, 1, T, 2, d, True)
        run = lambda: [x.detach() for x in eops.efla_scan(k.detach().requires_grad_(True), v, beta, s0)]      # a gradient: the chunked form
        o0, f0 = run()
        v[0, 40, 0, 5] = float("inf")
        o, s = run()
        assert o[0, 40, 0, 5] == float("inf") and o[0, 41:, 0, 5].isnan().all()
        o[0, 40:, 0, 5] = o0[0, 40:, 0, 5]
        assert torch.equal(o, o0)
        if T == 41:
            assert torch.equal(s[0, 0, :, 5], torch.copysign(torch.full((d,), float("inf"), device=cuda_device), k[0, 40, 0].float()))
        s[0, 0, :, 5] = f0[0, 0, :, 5]
        assert torch.equal(s, f0)


@pytest.mark.parametrize("d", [32, 64, 96, 128])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_backward_keeps_a_bad_token_to_its_side(cuda_device, d, bad):
    """A bad value touches the key gradients of its own and later tokens only and no value gradient; a bad output gradient touches its own
    and earlier tokens only, and its own column of the value gradients. The finite ones are those of the clean call, up to the bf16 rounding
    of sums taken in another order."""
    T = 100
    k, v, beta, s0 = _inputs(cuda_device, 1, T, 2, d, True)
    torch.manual_seed(d)
    go, gs = torch.randn_like(v), 0.1 * torch.randn(1, 2, d, d, device=cuda_device)

    def grads(v, go):
        ins = [t.detach().clone().requires_grad_(True) for t in (k, v, s0)]
        o, s = eops.efla_scan(ins[0], ins[1], beta, ins[2])
        return torch.autograd.grad([o, s], ins, [go, gs])

    dk0, dv0, ds0 = grads(v, go)
    v1 = v.clone()
    v1[0, 41, 0, 5] = bad
    dk, dv, ds = grads(v1, go)
    assert torch.equal(dv, dv0) and torch.equal(ds, ds0) and torch.equal(dk[:, :, 1], dk0[:, :, 1])
    _close(dk[:, :41, 0], dk0[:, :41, 0], 2 ** -8)
    assert not dk[0, 41:, 0].isfinite().any()
    g1 = go.clone()
    g1[0, 41, 0, 5] = bad
    dk, dv, ds = grads(v, g1)
    assert torch.equal(dk[:, :, 1], dk0[:, :, 1])
    _close(dk[:, 42:, 0], dk0[:, 42:, 0], 2 ** -8)
    _close(dv[:, 42:, 0], dv0[:, 42:, 0], 2 ** -8)
    assert not dk[0, :42, 0].isfinite().any() and not dv[0, :42, 0, 5].isfinite().any()
    keep = [j for j in range(d) if j != 5]
    _close(dv[:, :, 0, keep], dv0[:, :, 0, keep], 2 ** -8)
    _close(ds[:, :, :, keep], ds0[:, :, :, keep], 1e-5)


@pytest.mark.parametrize("T", [1, 16, 17, 31, 32, 33, 65, 112, 113])
@pytest.mark.parametrize("d", [32, 64, 96, 128])
def test_both_forms_at_the_line(cuda_device, monkeypatch, T, d):
    """Blocks without a gradient go token by token while whole calls are faster that way (few states: up to 112 tokens), with a gradient never."""
    k, v, beta, s0 = _inputs(cuda_device, 1, T, 2, d, T % 2 == 1, seed=T + d)
    names, call = [], eops.lib.call
    monkeypatch.setattr(eops.lib, "call", lambda name, *a: names.append(name) or call(name, *a))
    o, s = eops.efla_scan(k, v, beta, s0)
    o2, s2 = (x.detach() for x in eops.efla_scan(k.detach().requires_grad_(True), v, beta, s0))
    assert names == ["elfa_efla_scan_fwd" if T <= 112 else "elfa_efla_chunk_fwd", "elfa_efla_chunk_fwd"]
    o_ref, s_ref = eops.efla_scan_ref(k, v, beta, s0)
    for a, b in ((o, s), (o2, s2)):
        _close(a, o_ref, 2 ** -8)
        _close(b, s_ref, 1e-5)
    assert [eops._efla_step_tokens(1 << n) for n in range(12, 27, 2)] == [112, 112, 112, 112, 96, 32, 16, 16]


@pytest.mark.parametrize("T", [8, 17, 113])
@pytest.mark.parametrize("std", [0.0, 1e-5, 2e-4, 3e-3, 0.05])
def test_short_keys_have_the_same_coefficient_in_both_forms(cuda_device, T, std):
    """c = (1 - exp(-beta lam)) / lam cancels for short keys. 64-bit loop; the state is a sum of T terms that fp32 rounds a handful of times each."""
    g = torch.Generator(device=cuda_device).manual_seed(T)
    k = (torch.randn(1, T, 2, 64, generator=g, device=cuda_device) * std).bfloat16()
    v = torch.randn(1, T, 2, 64, generator=g, device=cuda_device).bfloat16()
    S = torch.zeros(1, 2, 64, 64, dtype=torch.float64, device=cuda_device)
    for t in range(T):
        kt, vt = k[:, t].double(), v[:, t].double()
        lam = (kt * kt).sum(-1)
        c = torch.where(lam == 0, torch.full_like(lam, 0.3), -torch.expm1(-0.3 * lam) / lam.clamp_min(1e-300))
        S = S + c[..., None, None] * kt[..., :, None] * (vt - torch.einsum("bhi,bhij->bhj", kt, S))[..., None, :]
    beta = torch.tensor([0.3], device=cuda_device)
    for want in (False, True):
        s = eops.efla_scan(k.detach().requires_grad_(want), v, beta)[1].detach()
        assert (s.double() - S).abs().max() <= 2e-6 * S.abs().max()


@pytest.mark.parametrize("d", [32, 64, 96, 128])
def test_a_key_whose_square_overflows_changes_nothing(cuda_device, d):
    """|k|^2 past the largest float makes c zero: the state passes by, and later tokens are those of a call in which that key is zero. (5e37: the
    products of that key with the state stay finite, their sums over the value columns do not.)"""
    T = 130
    for seed in range(6):
        k, v, beta, s0 = _inputs(cuda_device, 1, T, 2, d, True, seed=seed)
        torch.manual_seed(seed)
        go, gs = 50 * torch.randn_like(v), 0.1 * torch.randn(1, 2, d, d, device=cuda_device)
        got = []
        for low in (True, False):
            kk = k.clone()
            kk[0, 41, 0] = 0.0
            if low:
                kk[0, 41, 0, 3] = -5e37
            ins = [t.detach().requires_grad_(True) for t in (kk, v)]
            o, s = eops.efla_scan(*ins, beta, s0)
            got.append([o.detach(), s.detach(), *torch.autograd.grad([o, s], ins, [go, gs])])
        (o, s, dk, dv), (o0, s0_, dk0, dv0) = got
        _close(o[:, 42:], o0[:, 42:], 2 ** -8)
        _close(s, s0_, 1e-5)
        _close(dk[:, 42:], dk0[:, 42:], 2 ** -8)
        _close(dv[:, 42:], dv0[:, 42:], 2 ** -8)
