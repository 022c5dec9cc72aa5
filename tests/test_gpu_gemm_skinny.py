"""Products of one to eight rows (plain loads, no tensor-core tile) against fp64 and against the tensor-core form.

Bound: bf16 operands, fp32 sums of K terms in any order (K 2^-24 of the sum of magnitudes at worst; 2^-12 of the largest output covers K <= 11008 of
random signs) and one rounding of the output to bf16 (2^-9 of itself): 2^-8 of the largest.
"""
import os
import subprocess
import sys

import pytest
import torch

from elfa_b200 import native, ops
from elfa_b200.ops.gemm import gelu_tanh_ref, gemm

pytestmark = pytest.mark.gpu


def _operands(dev, M, N, K, bmn):
    g = torch.Generator(device=dev).manual_seed(M * 7 + N + K)
    r = lambda *s: torch.randn(*s, generator=g, device=dev)
    return r(M, K).bfloat16(), (r(K, N) if bmn else r(N, K)).mul(K ** -0.5).bfloat16()


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9])                    # 9: the tensor-core form
@pytest.mark.parametrize("N,K", [(8, 8), (64, 256), (72, 264), (1000, 1104), (1536, 1024), (256, 11008), (32000, 128), (30000, 520), (9480, 1104),
                                 (11008, 776), (6144, 2056), (14336, 8192)])
@pytest.mark.parametrize("bmn", [True, False])
def test_matches_the_product(cuda_device, M, N, K, bmn):
    a, b = _operands(cuda_device, M, N, K, bmn)
    want = a.double() @ (b.double() if bmn else b.double().t())
    y = gemm(a, b, b_mn=bmn)
    assert native.status() == 0
    assert (y.double() - want).abs().max() <= 2 ** -8 * want.abs().max()
    assert torch.equal(y, gemm(a, b, b_mn=bmn))


@pytest.mark.parametrize("bmn", [True, False])
def test_epilogue_and_pitches(cuda_device, bmn):
    a, b = _operands(cuda_device, 5, 136, 320, bmn)
    wide = torch.randn(5, 400, device=cuda_device).bfloat16()
    wide[:, 8:328] = a
    bias = torch.randn(136, device=cuda_device).bfloat16()
    out = torch.full((5, 200), 7.0, dtype=torch.bfloat16, device=cuda_device)
    pre = torch.full((5, 144), 7.0, dtype=torch.bfloat16, device=cuda_device)
    gemm(wide[:, 8:328], b, b_mn=bmn, bias=bias, gelu=True, preact=pre[:, :136], out=out[:, 64:], alpha=0.5)
    want = 0.5 * (a.double() @ (b.double() if bmn else b.double().t())) + bias.double()
    assert (pre[:, :136].double() - want).abs().max() <= 2 ** -8 * want.abs().max()
    # the activation uses the hardware tanh: 2^-11 of its own besides the rounding
    assert (out[:, 64:].double() - gelu_tanh_ref(want)).abs().max() <= 2 ** -7 * want.abs().max()
    assert (out[:, :64] == 7).all() and (pre[:, 136:] == 7).all()


def test_not_finite_values_stay_in_their_row_and_column(cuda_device):
    for bmn in (True, False):
        a, b = _operands(cuda_device, 3, 64, 256, bmn)
        y = gemm(a, b, b_mn=bmn)
        a[1, 200] = float("nan")
        (b if bmn else b.t())[17, 40] = float("inf")
        z = gemm(a, b, b_mn=bmn)
        assert z[1].isnan().all() and not torch.isfinite(z[:, 40]).any()
        keep = [j for j in range(64) if j != 40]
        assert torch.equal(z[::2, keep], y[::2, keep])


def test_linear_backward_of_a_few_rows(cuda_device):
    x = torch.randn(4, 256, device=cuda_device).bfloat16().requires_grad_(True)
    w = (torch.randn(256, 512, device=cuda_device) / 16).bfloat16().requires_grad_(True)
    dy = torch.randn(4, 512, device=cuda_device).bfloat16()
    dx, dw = torch.autograd.grad(ops.linear(x, w), [x, w], dy)
    for got, want in ((dx, dy.double() @ w.double().t()), (dw, x.double().t() @ dy.double())):
        assert (got.double() - want).abs().max() <= 2 ** -8 * want.abs().max()


@pytest.mark.parametrize("bmn,M,N,K", [(False, 8, 9480, 8192), (False, 1, 11008, 4096), (False, 8, 18944, 1024), (True, 8, 6144, 1024), (True, 8, 9480, 1024),
                                       (True, 8, 14336, 8192), (True, 1, 12288, 4096)])
def test_no_slower_than_the_tiles(cuda_device, bmn, M, N, K):
    """The cuts of a matrix at which one round too many, or too few warps, once cost up to three times the tensor-core tiles' time."""
    ops_ = [_operands(cuda_device, M, N, K, bmn) for _ in range(max(2, min(8, 300_000_000 // (N * K * 2))))]
    out = torch.empty(M, N, dtype=torch.bfloat16, device=cuda_device)

    def us(bn):
        run = lambda: [gemm(a, b, b_mn=bmn, out=out, force_bn=bn) for a, b in ops_]
        run()
        g, best = torch.cuda.CUDAGraph(), []
        with torch.cuda.graph(g):
            run()
        for _ in range(6):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            g.replay()
            e[1].record()
            torch.cuda.synchronize()
            best.append(e[0].elapsed_time(e[1]))
        return min(best)
    assert us(0) < 1.15 * us(512 if N >= 18944 else 128)


def test_first_few_rows_of_a_process_under_capture(cuda_device):
    """The clusters that run at once are asked for on the first such call, which may be inside a graph capture (the library's status word is made by
    the product of 16 rows before it)."""
    code = ("import torch\nfrom elfa_b200.ops.gemm import gemm\n"
            "a, b = torch.randn(4, 1024, device='cuda').bfloat16(), torch.randn(1024, 4096, device='cuda').bfloat16()\n"
            "y = torch.zeros(4, 4096, dtype=torch.bfloat16, device='cuda')\ng = torch.cuda.CUDAGraph()\n"
            "gemm(torch.cat([a] * 4), b, b_mn=True)\n"
            "with torch.cuda.graph(g):\n    gemm(a, b, b_mn=True, out=y)\n"
            "g.replay()\nz = gemm(a, b, b_mn=True)\ntorch.cuda.synchronize()\nassert torch.equal(y, z) and y.abs().max() > 0\n")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0, r.stderr[-2000:]
