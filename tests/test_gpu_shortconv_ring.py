"""ShortConv at the edges of the register ring (windows 4, 8, 16; spans of 16 to 64 steps) and at windows that keep the general kernels.

fp32 sums on both sides, outputs and gradients rounded to bf16 once: 2^-8 of the largest.
"""
import pytest
import torch

from elfa_b200 import native
from elfa_b200.ops import efla as eops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W", [4, 5, 8, 16, 64])
@pytest.mark.parametrize("B,T,C", [(1, 1, 2), (2, 15, 66), (3, 17, 64), (1, 65, 130), (4, 200, 1024)])
@pytest.mark.parametrize("bias", [False, True])
def test_shortconv_edges(cuda_device, B, T, C, W, bias):
    torch.manual_seed(T + W)
    x = torch.randn(B, T, C, device=cuda_device).bfloat16().requires_grad_(True)
    w = (torch.randn(C, W, device=cuda_device) * W ** -0.5).bfloat16().requires_grad_(True)
    b = torch.randn(C, device=cuda_device).bfloat16().requires_grad_(True) if bias else None
    dy = torch.randn(B, T, C, device=cuda_device).bfloat16()
    ins = [t for t in (x, w, b) if t is not None]
    y = eops.shortconv(x, w, b)
    got = torch.autograd.grad(y, ins, dy)
    fins = [t.detach().float().requires_grad_(True) for t in ins]
    yr = eops.shortconv_ref(*fins)
    ref = torch.autograd.grad(yr, fins, dy.float())
    assert native.status() == 0
    for a, r in zip([y, *got], [yr, *ref]):
        assert (a.float() - r).abs().max() <= 2 ** -8 * r.abs().max()
