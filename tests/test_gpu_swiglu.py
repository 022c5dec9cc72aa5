"""Gated activation against fp32 PyTorch; at most two bf16 roundings per result (the general path rounds silu too): 2^-7 of the largest."""
import pytest
import torch

from elfa_b200 import native, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 16), (3, 5, 48), (257, 4096), (2, 3, 20)])      # the last one keeps the general path (F = 10)
@pytest.mark.parametrize("offset", [0, 1])
def test_swiglu(cuda_device, shape, offset):
    n = torch.Size(shape).numel()
    h = torch.empty(n + offset, dtype=torch.bfloat16, device=cuda_device)[offset:].view(shape)
    h.copy_(torch.randn(shape, device=cuda_device) * 3)
    h.requires_grad_(True)
    hr = h.detach().float().requires_grad_(True)
    a = ops.swiglu(h)
    g, u = hr.chunk(2, -1)
    ar = torch.nn.functional.silu(g) * u
    da = torch.randn_like(ar).bfloat16()
    (dh,) = torch.autograd.grad(a, h, da)
    (dr,) = torch.autograd.grad(ar, hr, da.float())
    assert native.status() == 0
    for x, r in ((a, ar), (dh, dr)):
        assert x.shape == r.shape and (x.float() - r).abs().max() <= 2 ** -7 * r.abs().max()
