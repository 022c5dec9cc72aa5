"""PRISM state carry in one kernel against the token-by-token update. fp32 on both sides: 1e-5 of the largest covers 40 tokens."""
import sys
import threading

import pytest
import torch

from elfa_b200 import native, ops
from elfa_b200.native import lib, stream_ptr
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


def _state_us(dev, B, G, d, L, T):
    u, v, z = (torch.randn(B, T, n, device=dev).bfloat16() for n in (G * d, G * d, 3 * L * d))
    s0, best = torch.randn(B, G, d, d, device=dev), []
    s1 = torch.empty_like(s0)
    for _ in range(5):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        torch.cuda._sleep(4_000_000)
        e[0].record()
        for _ in range(40):
            lib.call("elfa_prism_state", u, v, z, 3 * L * d, L * d, 2 * L * d, s0, s1, B, T, G, d, L, 0.9, stream_ptr(u))
        e[1].record()
        torch.cuda.synchronize()
        best.append(25 * e[0].elapsed_time(e[1]))
    return min(best)


def test_many_states_and_one_token(cuda_device):
    """2048 states of 32, eight iterations, against 128, which are one for each SM: measured 3.0 times as long, 7.1 with tiles that leave two CTAs to an SM. One token:
    eight iterations against two, 1.0 and, with their loads one behind the other, 1.6."""
    assert _state_us(cuda_device, 128, 16, 32, 8, 64) < 4.5 * _state_us(cuda_device, 8, 16, 32, 8, 64)
    assert _state_us(cuda_device, 2, 16, 64, 8, 1) < 1.45 * _state_us(cuda_device, 2, 16, 64, 2, 1)


def test_lengths_of_several_threads(cuda_device):
    """Two threads with tiles of twelve tokens, two with tiles of four: how much shared memory one call takes is no limit for another one's launch (where
    it was, one launch in sixty failed)."""
    d, L, failed = 128, 8, [0] * 4
    f = lib.raw("elfa_prism_state")

    def run(i, T):
        u, v, z = (torch.randn(1, T, n, device=cuda_device).bfloat16() for n in (d, d, 3 * L * d))
        s0 = torch.randn(1, 1, d, d, device=cuda_device)
        s1 = torch.empty_like(s0)
        with torch.cuda.stream(torch.cuda.Stream()):
            here = torch.cuda.current_stream()
            here.wait_stream(torch.cuda.default_stream())
            for k in range(4096):
                failed[i] += f(u.data_ptr(), v.data_ptr(), z.data_ptr(), 3 * L * d, L * d, 2 * L * d, s0.data_ptr(), s1.data_ptr(), 1, T, 1, d, L, 0.9,
                               here.cuda_stream) != 0
                if k % 64 == 63:
                    here.synchronize()
    threads = [threading.Thread(target=run, args=(i, T)) for i, T in enumerate((12, 1, 12, 4))]
    switch = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)
    try:
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(switch)
    assert failed == [0] * 4 and native.status() == 0
