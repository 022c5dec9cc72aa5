"""PRISM state carry in one kernel against the token-by-token update. fp32 on both sides: 1e-5 of the largest covers 40 tokens."""
import pytest
import torch

from elfa_b200 import native, ops
from elfa_b200.ops import efla as eops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,G,d,L", [(1, 2, 32, 1), (8, 3, 64, 2), (9, 2, 96, 3), (40, 2, 128, 8)])
def test_state_carry(cuda_device, T, G, d, L):
    torch.manual_seed(T + d)
    B, D = 2, G * d
    u, v = (torch.randn(B, T, D, device=cuda_device).bfloat16() for _ in range(2))
    wp, wb, wk = ([(torch.randn(D, d, device=cuda_device) * D ** -0.5).bfloat16() for _ in range(L)] for _ in range(3))
    s0 = torch.randn(B, G, d, d, device=cuda_device)
    assert eops.prism_stream_native(u, v, wp, wb, wk, s0, d)
    y, s = eops.prism_stream(u, v, wp, wb, wk, s0, 0.97, d)
    r = (v.float() - u.float()).view(B, T, G, d)
    deltas, betas, ks = [], [], []
    for l in range(L):
        delta = ops.gelu_tanh_ref(torch.sigmoid(ops.linear(u, wp[l]).float()).unsqueeze(2) * r)
        r = r - delta
        deltas.append(delta)
        betas.append(torch.sigmoid(ops.linear(u, wb[l]).float().mean(-1)))
        ks.append(torch.nn.functional.normalize(ops.linear(u, wk[l]).float(), dim=-1))
    want = eops.prism_state_update(s0, deltas, betas, ks, 0.97)
    assert native.status() == 0
    assert (s - want).abs().max() <= 1e-5 * want.abs().max()
    ref = u.float() + sum(deltas).view(B, T, D)
    assert (y.float() - ref).abs().max() <= 2 ** -8 * ref.abs().max()


@pytest.mark.parametrize("order", [(1, 0, 2, 3), (0, 2, 1, 3), (0, 1, 3, 2)])
def test_state_of_any_stride(cuda_device, order):
    torch.manual_seed(0)
    B, T, G, d, L = 2, 5, 32, 32, 2
    u, v = (torch.randn(B, T, G * d, device=cuda_device).bfloat16() for _ in range(2))
    wp, wb, wk = ([(torch.randn(G * d, d, device=cuda_device) * (G * d) ** -0.5).bfloat16() for _ in range(L)] for _ in range(3))
    s0 = torch.randn(B, G, d, d, device=cuda_device)
    view = s0.permute(order).contiguous().permute(order)          # the same values, dense in another order (each order is its own inverse)
    assert not view.is_contiguous() and torch.equal(view, s0)
    want = eops.prism_stream(u, v, wp, wb, wk, s0, 0.97, d)
    got = eops.prism_stream(u, v, wp, wb, wk, view, 0.97, d)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
