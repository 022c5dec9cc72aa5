"""PRISM gate from its weights (one GEMM, one kernel per direction) against the plain PyTorch form.

The oracle is fp32 throughout except for the logits, which both sides round to bf16. The kernels round results to bf16, and the input
gradient twice more on its way (its two addends): at most three roundings of 2^-9, 2^-7 of the largest.
"""
import pytest
import torch

from elfa_b200 import native
from elfa_b200.native import lib, stream_ptr
from elfa_b200.ops import efla as eops, linear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,G,d,L", [(1, 1, 8, 1), (33, 3, 32, 2), (64, 16, 64, 3), (7, 5, 64, 4), (20, 2, 128, 8), (19, 4, 24, 5)])
def test_gated_refine(cuda_device, T, G, d, L):
    torch.manual_seed(T)
    D = G * d
    u = torch.randn(2, T, D, device=cuda_device).bfloat16().requires_grad_(True)
    v = torch.randn(2, T, D, device=cuda_device).bfloat16().requires_grad_(True)
    ws = [(torch.randn(D, d, device=cuda_device) * D ** -0.5).bfloat16().requires_grad_(True) for _ in range(L)]
    assert eops.prism_gated_native(u, v, ws, d)
    dy = torch.randn(2, T, D, device=cuda_device).bfloat16()
    y = eops.prism_gated_refine(u, v, ws, d)
    got = torch.autograd.grad(y, [u, v, *ws], dy)
    uf, vf, *wf = (t.detach().float().requires_grad_(True) for t in (u, v, *ws))
    zs = [uf @ w for w in wf]
    zs = [z + (linear(u, w).detach().float() - z).detach() for z, w in zip(zs, ws)]       # the value of the bf16 logits
    ref_y = eops.prism_refine_ref(uf, vf, [torch.sigmoid(z) for z in zs], d)
    ref = torch.autograd.grad(ref_y, [uf, vf, *wf], dy.float())
    assert native.status() == 0
    for a, b in zip([y, *got], [ref_y, *ref]):
        assert a.shape == b.shape and a.dtype == torch.bfloat16
        assert (a.float() - b).abs().max() <= 2 ** -7 * b.abs().max()


def test_other_calls_keep_the_general_path(cuda_device):
    u = torch.randn(1, 4, 12, device=cuda_device).bfloat16()                       # groups of 12 channels
    w = torch.randn(12, 12, device=cuda_device).bfloat16()
    assert not eops.prism_gated_native(u, u, [w], 12)
    cpu = torch.randn(1, 4, 16)
    wc = torch.randn(16, 8)
    assert not eops.prism_gated_native(cpu, cpu, [wc], 8)
    want = eops.prism_refine_ref(cpu, cpu + 1, [torch.sigmoid(cpu @ wc)], 8)
    assert torch.allclose(eops.prism_gated_refine(cpu, cpu + 1, [wc], 8), want, atol=1e-6)


def _weight_call(cuda_device, T, G, d, L):
    torch.manual_seed(T)
    D = G * d
    u, v, dy = (torch.randn(2, T, D, device=cuda_device).bfloat16() for _ in range(3))
    ws = [(torch.randn(D, d, device=cuda_device) * D ** -0.5).bfloat16().requires_grad_(True) for _ in range(L)]
    return u, v, dy, ws


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("T,G,d,L", [(1, 1, 8, 1), (700, 3, 24, 3), (4100, 16, 64, 2), (2048, 5, 128, 8)])
def test_weight_gradients_have_one_order(cuda_device, T, G, d, L, deterministic):
    """Every call gives the same bits, with the deterministic mode and without; a main_grad is overwritten when fresh and added to when not,
    with the fp32 sum whose rounding is the gradient returned otherwise; inputs that want no gradient change nothing for the others."""
    u, v, dy, ws = _weight_call(cuda_device, T, G, d, L)
    native.set_deterministic(deterministic)
    try:
        def run(*wrt):
            return torch.autograd.grad(eops.prism_gated_refine(u, v, ws, d), wrt, dy, allow_unused=True)

        first = run(*ws)
        for _ in range(3):
            assert all(torch.equal(a, b) for a, b in zip(run(*ws), first))
        ws[0].requires_grad_(False)
        assert all(torch.equal(a, b) for a, b in zip(run(*ws[1:]), first[1:])) if L > 1 else True
        ws[0].requires_grad_(True)
        for w in ws:
            w.main_grad = torch.full(w.shape, 7.0, device=cuda_device)
            w._grad_fresh = True
        assert all(g is None for g in run(*ws))
        once = [w.main_grad.clone() for w in ws]
        assert all(torch.equal(a.bfloat16(), b) for a, b in zip(once, first)) and not any(w._grad_fresh for w in ws)
        run(*ws)
        assert all(torch.equal(w.main_grad, a + a) for w, a in zip(ws, once))
        assert native.status() == 0
    finally:
        native.set_deterministic(False)


def test_one_weight_for_two_iterations(cuda_device):
    u, v, dy, (w, _) = _weight_call(cuda_device, 50, 2, 32, 2)
    copy = w.detach().clone().requires_grad_(True)
    a, b = torch.autograd.grad(eops.prism_gated_refine(u, v, [w, copy], 32), [w, copy], dy)
    w.main_grad, w._grad_fresh = torch.zeros(w.shape, device=cuda_device), True
    torch.autograd.grad(eops.prism_gated_refine(u, v, [w, w], 32), [w], dy, allow_unused=True)
    want = a.float() + b.float()
    assert (w.main_grad - want).abs().max() <= 2 ** -8 * want.abs().max()            # the two addends are rounded to bf16


@pytest.mark.parametrize("M,N,K,pieces", [(8, 8, 1, 1), (128, 64, 512, 1), (136, 24, 700, 1), (1024, 128, 8200, 9), (640, 1024, 1500, 3), (4736, 1024, 256, 1)])
def test_split_product_adds_up(cuda_device, M, N, K, pieces):
    """Every tile width of the split product (64, 128, 256 columns), ragged rows, columns and contraction: the pieces add up to the product. fp32
    sums of exact bf16 products: 2^-20 of the largest for 8200 terms in blocks of 16 and a few pieces."""
    torch.manual_seed(M)
    a, b = torch.randn(K, M, device=cuda_device).bfloat16(), torch.randn(K, N, device=cuda_device).bfloat16()
    n = native.lib.raw("elfa_gemm_bf16_parts_count")(M, N, K)
    assert n == pieces                               # on 148 SMs
    parts = torch.full((n, (M + 127) // 128 * 128, N), float("nan"), device=cuda_device)
    native.lib.call("elfa_gemm_bf16_parts", a, b, parts, M, N, K, M, N, native.stream_ptr(a))
    want = a.double().t() @ b.double()
    assert native.status() == 0
    assert (parts.double().sum(0)[:M] - want).abs().max() <= 2 ** -20 * want.abs().max() * max(1, K / 256) ** 0.5


@pytest.mark.parametrize("tokens,G,d,L", [(1, 16, 64, 2), (37, 5, 32, 1), (129, 3, 64, 8), (40, 1, 128, 3), (700, 16, 64, 2), (1200, 7, 8, 4)])
def test_few_tokens_spread_their_groups(cuda_device, tokens, G, d, L):
    """A call of few tokens spreads the groups over threads: the bits of the same rows inside a call that does not."""
    g = torch.Generator(device=cuda_device).manual_seed(tokens)
    rows = 148 * 2 * 256 // (d // 8) + tokens + 8                     # two blocks per SM without spreading
    u, v, z = (torch.randn(rows, n, generator=g, device=cuda_device).bfloat16() for n in (G * d, G * d, L * d))
    whole, few = torch.empty_like(u), torch.full_like(u[:tokens + 1], 7.0)
    for y, n in ((whole, rows), (few, tokens)):
        lib.call("elfa_prism_gated_fwd", u, v, z, z.stride(0), y, n, G, d, L, stream_ptr(u))
    assert native.status() == 0 and torch.equal(few[:tokens], whole[:tokens]) and (few[tokens:] == 7).all()


@pytest.mark.parametrize("d,L", [(32, 1), (64, 2), (96, 3), (128, 8)])          # the last one: tiles of twelve tokens
@pytest.mark.parametrize("T", [1, 5, 64, 65, 131])
def test_the_state_does_not_depend_on_the_tiles(cuda_device, d, L, T):
    """Tiles of up to 64 tokens; one call and calls of a few tokens each leave the same state."""
    B, G = 2, 3
    g = torch.Generator(device=cuda_device).manual_seed(T + d)
    u, v, z = (torch.randn(B, T, n, generator=g, device=cuda_device).bfloat16() for n in (G * d, G * d, 3 * L * d))
    s0 = torch.randn(B, G, d, d, generator=g, device=cuda_device)

    def state(lo, hi, s):
        a, b, c = (x[:, lo:hi].contiguous() for x in (u, v, z))
        out = torch.empty_like(s)
        lib.call("elfa_prism_state", a, b, c, 3 * L * d, L * d, 2 * L * d, s, out, B, hi - lo, G, d, L, 0.9, stream_ptr(a))
        return out
    cut = s0
    for lo in range(0, T, 7):
        cut = state(lo, min(T, lo + 7), cut)
    assert native.status() == 0 and torch.equal(state(0, T, s0), cut) and torch.isfinite(cut).all()
