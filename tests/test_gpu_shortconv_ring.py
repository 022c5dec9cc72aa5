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


@pytest.mark.parametrize("W", [4, 5, 8, 16])
@pytest.mark.parametrize("T", [1, 3, 16, 17, 40, 65, 130])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_nothing_beyond_the_sequence_is_multiplied(cuda_device, T, W, bad):
    """Terms that reach outside the sequence do not exist; formed with zeros they would make NaN of a value that is not finite."""
    torch.manual_seed(T + W)
    C, c = 66, 9
    other = [i for i in range(C) if i != c]
    x0, dy0 = (torch.randn(2, T, C, device=cuda_device).bfloat16() for _ in range(2))
    w0 = torch.randn(C, W, device=cuda_device).bfloat16()

    def run(x, w, dy):
        ins = [t.clone().requires_grad_(True) for t in (x, w)]
        y = eops.shortconv(*ins)
        return [y.detach(), *torch.autograd.grad(y, ins, dy)]

    clean = run(x0, w0, dy0)
    taps, times = torch.arange(W, device=cuda_device), torch.arange(T, device=cuda_device)
    for what in range(3):
        x, w, dy = x0.clone(), w0.clone(), dy0.clone()
        if what == 0:
            x[0, T - 1, c] = bad             # the last input meets the last output gradient through tap 0 only
        elif what == 1:
            dy[0, 0, c] = bad                # the first output gradient meets the first input through tap 0 only
        else:
            w[c, W - 1] = bad                # the last tap: outputs from W - 1 on, input gradients up to T - W
        y, dx, dw = run(x, w, dy)
        ok_y = (times < T - 1 if what == 0 else torch.full_like(times, what == 1) > 0) if what < 2 else times < W - 1
        ok_dx = (torch.full_like(times, 1) > 0 if what == 0 else times > 0) if what < 2 else times > T - W
        assert torch.equal(y[0, :, c].isfinite(), ok_y) and torch.equal(dx[0, :, c].isfinite(), ok_dx)
        assert torch.equal(dw[c].isfinite(), taps > 0 if what < 2 else taps >= 0)
        for got, ref in zip((y, dx), clean):
            assert torch.equal(got[:, :, other], ref[:, :, other])
        assert torch.equal(dw[other], clean[2][other])
