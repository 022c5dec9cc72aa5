"""The EFLA walk in segments: joined at every kind of boundary, against the token-by-token recurrence.

Bounds: states are fp32 sums; a segment adds the roundings of its start (2^-24 a term) to the errors of its own walk, and the maps contract, so
1e-5 of the largest value that the state (or its gradient) had on its way covers both forms. That is what it starts from for the gradient, which
only shrinks where the outputs' gradient is smaller. Outputs and k / v gradients are rounded to bf16 once (2^-8 of the largest).
"""
import pytest
import torch

from elfa_b200 import native
from elfa_b200.native import lib, stream_ptr
from elfa_b200.ops import efla as eops

pytestmark = pytest.mark.gpu


def _inputs(dev, B, T, H, d):
    g = torch.Generator(device=dev).manual_seed(T + d)
    r = lambda *s, std=1.0: torch.randn(*s, generator=g, device=dev) * std
    return (r(B, T, H, d, std=0.4).bfloat16(), r(B, T, H, d).bfloat16(), torch.tensor([0.3], device=dev), r(B, H, d, d, std=0.3),
            r(B, T, H, d).bfloat16(), r(B, H, d, d, std=0.1))


def _run(P, k, v, beta, s0, do, ds):
    """Forward and backward through the native entry points with the walk in P segments; backward in both of its forms, with beta's terms per token and, as
    training calls it, with their sum (bounded as below)."""
    B, T, H, d = k.shape
    n = (T + 31) // 32
    new = lambda *s, dt=torch.float32: torch.empty(*s, dtype=dt, device=k.device)
    ckpt, dckpt, coef, nmat = new(B * H * n * d * d), new(B * H * n * d * d), new(B, H, n, 4, 32), new(B, H, n, 3, 32, 32, dt=torch.bfloat16)
    work = new(3 * P * B * H * d * d) if P > 1 else None
    o, s, dk, dv, ds0, db = torch.empty_like(k), torch.empty_like(s0), torch.empty_like(k), torch.empty_like(k), torch.empty_like(s0), new(B * T * H)
    lib.call("elfa_efla_chunk_fwd_cut", k, v, beta, s0, o, s, ckpt, nmat, coef, work, P, B, T, H, d, stream_ptr(k))
    lib.call("elfa_efla_chunk_bwd_cut", k, v, nmat, coef, ckpt, do, ds, dk, dv, db, ds0, dckpt, work, P, B, T, H, d, stream_ptr(k))
    dk2, dv2, ds2, terms, total = torch.empty_like(dk), torch.empty_like(dv), torch.empty_like(ds0), new(B * H * n), new(1)
    lib.call("elfa_efla_chunk_bwd_sum", k, v, nmat, coef, ckpt, do, ds, dk2, dv2, terms, total, ds2, dckpt, work, P, B, T, H, d, stream_ptr(k))
    assert native.status() == 0
    for a, b in ((dk, dk2), (dv, dv2), (ds0, ds2)):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))
    db = db.double()
    if torch.isfinite(db).all():
        assert abs(total.item() - db.sum().item()) <= 2 ** -24 * (db.abs().sum() + db.sum().abs()).item()
    return o, s, dk, dv, ds0


@pytest.mark.parametrize("d", [32, 64, 96, 128])
@pytest.mark.parametrize("T,P", [(64, 2), (96, 3), (97, 3), (160, 4), (200, 5), (512, 16), (530, 16), (33, 16)])
def test_segments(cuda_device, d, T, P):
    ins = _inputs(cuda_device, 2, T, 3, d)
    got = _run(P, *ins)
    want = [t.detach().double().requires_grad_(True) for t in ins[:4]]
    o, s = eops.efla_scan_ref(*want)                                    # fp32 inside
    ref = [o, s, *torch.autograd.grad([o, s], [want[0], want[1], want[3]], [ins[4].to(o.dtype), ins[5].to(s.dtype)])]
    for a, b, rel, top in zip(got, ref, (2 ** -8, 1e-5, 2 ** -8, 2 ** -8, 1e-5), (0, 0, 0, 0, ins[5].abs().max())):
        assert (a.double() - b).abs().max() <= rel * max(b.abs().max(), top)


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("at", [0, 70, 128, 255, 256, 511])
def test_a_bad_value_stays_behind_its_token_and_in_its_column(cuda_device, bad, at):
    k, v, beta, s0, do, ds = _inputs(cuda_device, 1, 512, 2, 64)
    clean = _run(4, k, v, beta, s0, do, ds)
    v[0, at, 0, 5] = bad
    o, s, _, dv, _ = _run(4, k, v, beta, s0, do, ds)
    assert not torch.isfinite(o[0, at:, 0, 5]).any() and not torch.isfinite(s[0, 0, :, 5]).any()
    o[0, at:, 0, 5] = clean[0][0, at:, 0, 5]
    s[0, 0, :, 5] = clean[1][0, 0, :, 5]
    assert torch.equal(o, clean[0]) and torch.equal(s, clean[1]) and torch.equal(dv, clean[3])
    v[0, at, 0, 5] = 1.0
    clean = _run(4, k, v, beta, s0, do, ds)
    do[0, at, 0, 5] = bad                                               # backward: its own and earlier tokens
    _, _, _, dv, ds0 = _run(4, k, v, beta, s0, do, ds)
    assert not torch.isfinite(dv[0, :at + 1, 0, 5]).any() and not torch.isfinite(ds0[0, 0, :, 5]).any()
    dv[0, :at + 1, 0, 5] = clean[3][0, :at + 1, 0, 5]
    ds0[0, 0, :, 5] = clean[4][0, 0, :, 5]
    # the chunk with the bad value is walked token by token in all columns: other fp32 roundings
    for a, b, rel in ((dv, clean[3], 2 ** -8), (ds0, clean[4], 1e-5)):
        assert (a.float() - b.float()).abs().max() <= rel * b.float().abs().max()


@pytest.mark.parametrize("d", [32, 128])
@pytest.mark.parametrize("beta,first", [(-3.0, 500), (-0.02, 0), (-1e-6, 0)])
def test_negative_beta_is_walked_in_one_piece(cuda_device, d, beta, first):
    """Its maps grow: those of a whole segment leave fp32 where the zero states before the first value would not."""
    k, v, b, s0, do, ds = _inputs(cuda_device, 2, 530, 3, d)
    v[:, :first] = 0
    if first:
        s0.zero_()
        do[:, first:], ds = 0, torch.zeros_like(ds)
        k[:, first:] *= 0.1
    ins = (k, v, torch.full_like(b, beta), s0, do, ds)
    want = _run(1, *ins)
    assert torch.isfinite(want[0]).all() and torch.isfinite(want[1]).all()
    for P in (2, 3, 16):
        for x, y in zip(_run(P, *ins), want):
            torch.testing.assert_close(x, y, rtol=0, atol=0, equal_nan=True)


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), 1e30])
@pytest.mark.parametrize("at", [0, 70, 128, 255, 256, 511])
def test_a_bad_key_reaches_what_it_reaches_in_one_walk(cuda_device, bad, at):
    """1e30: its square overflows, which leaves the token without an effect. The segments are joined by maps made from such keys."""
    k, v, beta, s0, do, ds = _inputs(cuda_device, 1, 512, 2, 64)
    k[0, at, 0, 5] = bad
    for got, want, rel in zip(_run(4, k, v, beta, s0, do, ds), _run(1, k, v, beta, s0, do, ds), (2 ** -8, 1e-5, 2 ** -8, 2 ** -8, 1e-5)):
        ok = torch.isfinite(want)
        assert torch.equal(torch.isfinite(got), ok)
        got, want = got[ok].float(), want[ok].float()
        # of the second head's and the other tokens' largest: the overflowing key itself gives outputs and gradients of its own size
        assert ((got - want).abs() <= rel * want.abs().clamp(min=want.abs().quantile(0.999).item())).all()


def test_the_rule_gives_segments_that_fit(cuda_device):
    for B, T, H, d in ((1, 8192, 16, 64), (2, 1531, 8, 128), (8, 2048, 16, 64), (1, 113, 4, 32), (1, 1, 1, 64), (64, 4096, 16, 64)):
        n = lib.raw("elfa_efla_segments")(B, T, H, d)
        assert 1 <= n <= 16 and (n == 1 or (T + 31) // 32 >= 4 * n)
    assert lib.raw("elfa_efla_segments")(1, 8192, 16, 64) > 1 and lib.raw("elfa_efla_segments")(64, 4096, 16, 64) == 1


@pytest.mark.parametrize("B,T,H,d", [(1, 1, 1, 32), (3, 33, 5, 64), (2, 300, 4, 96), (1, 97, 2, 128), (8, 1100, 16, 32)])
def test_beta_gradient_is_the_sum_of_its_terms(cuda_device, B, T, H, d):
    """Added up per chunk and then over the chunks (1, few and more than 4096 of them), in 64 bits: a rounding of each chunk's sum and one of the result,
    2^-24 of what they are."""
    k, v, beta, _, do, _ = _inputs(cuda_device, B, T, H, d)
    n = (T + 31) // 32
    new = lambda *s, dt=torch.float32: torch.empty(*s, dtype=dt, device=k.device)
    ckpt, dckpt, coef, nmat, s = new(B * H * n * d * d), new(B * H * n * d * d), new(B, H, n, 4, 32), new(B, H, n, 3, 32, 32, dt=torch.bfloat16), new(B, H, d, d)
    o, dk, dv, terms, tok, db = torch.empty_like(k), torch.empty_like(k), torch.empty_like(k), new(B * H * n), new(B * T * H), new(1)
    lib.call("elfa_efla_chunk_fwd", k, v, beta, None, o, s, ckpt, nmat, coef, B, T, H, d, stream_ptr(k))
    lib.call("elfa_efla_chunk_bwd", k, v, nmat, coef, ckpt, do, None, dk, dv, tok, None, dckpt, B, T, H, d, stream_ptr(k))
    lib.call("elfa_efla_chunk_bwd_sum", k, v, nmat, coef, ckpt, do, None, dk, dv, terms, db, None, dckpt, None, 1, B, T, H, d, stream_ptr(k))
    tok = tok.double()
    assert abs(db.item() - tok.sum().item()) <= 2 ** -24 * (tok.abs().sum() + tok.sum().abs()).item()

