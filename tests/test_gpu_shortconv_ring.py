"""ShortConv at the edges of the register ring (windows 4, 8, 16; spans of 16 to 64 steps) and at windows that keep the general kernels.

fp32 sums on both sides, outputs and gradients rounded to bf16 once: 2^-8 of the largest.
"""
import pytest
import torch

from elfa_b200 import native
from elfa_b200.native import lib, stream_ptr
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


def _behind_tail(tail, n, w, b):
    """The native streaming form: new outputs, and tail and inputs side by side."""
    (B, tails, C), T, W = tail.shape, n.shape[1], w.shape[1]
    xin, u = torch.empty(B, tails + T, C, dtype=n.dtype, device=n.device), torch.empty_like(n)
    rows = lib.raw("elfa_shortconv_stream_rows")(B, tails, T, C, W)
    full = torch.empty(rows, C, dtype=n.dtype, device=n.device) if rows else None
    if rows and B == 1:
        u = full[tails:].view(n.shape)
    lib.call("elfa_shortconv_stream", tail, tail.stride(0), n, w, b, xin, u, full, B, tails, T, C, W, stream_ptr(n))
    return u, xin, rows > 0


@pytest.mark.parametrize("W,B,C,short,long", [(4, 1, 1024, 2047, 2048), (4, 3, 1024, 2048, None), (5, 1, 66, 40, 31776), (8, 2, 1024, 511, 512), (16, 1, 130, 2016, 2017),
                                              (16, 3, 512, 170, 171), (24, 2, 256, 1023, 1024), (64, 1, 64, 1023, 1024), (64, 3, 128, 170, 171)])
@pytest.mark.parametrize("pitch", ["own", "wide", "shared"])
def test_behind_a_tail_on_both_sides_of_the_line(cuda_device, W, B, C, short, long, pitch):
    torch.manual_seed(W + C)
    r = lambda *s: torch.randn(*s, device=cuda_device).bfloat16()
    w, b = (r(C, W) * W ** -0.5), r(C)
    for T in (short, long):
        if T is None:
            continue
        tail = r(B, W - 1, C) if pitch == "own" else r(B, W + 3, C)[:, 2:W + 1] if pitch == "wide" else r(1, W - 1, C).expand(B, -1, -1)
        n = r(B, T, C)
        u, xin, in_full = _behind_tail(tail, n, w, b)
        assert native.status() == 0 and in_full == (T == long)
        whole = torch.cat([tail, n], 1)
        assert torch.equal(xin, whole) and torch.equal(u, eops.shortconv(whole, w, b)[:, W - 1:])


@pytest.mark.parametrize("W,C,T", [(16, 1024, 8192), (64, 1024, 2048), (4, 512, 16384)])
def test_a_long_block_behind_a_tail_costs_about_what_the_whole_costs(cuda_device, W, C, T):
    r = lambda *s: torch.randn(*s, device=cuda_device).bfloat16()
    tail, n, w, b = r(1, W - 1, C), r(1, T, C), r(C, W), r(C)
    whole = torch.cat([tail, n], 1)

    def us(f):
        best = []
        for _ in range(5):
            torch.cuda.synchronize()
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            for _ in range(10):
                f()
            e[1].record()
            torch.cuda.synchronize()
            best.append(e[0].elapsed_time(e[1]))
        return min(best)
    with torch.no_grad():       # measured 1.2 to 1.7 with the copies; one block per position was 3.5 to 23
        assert us(lambda: _behind_tail(tail, n, w, b)) < 3 * us(lambda: eops.shortconv(whole, w, b))


@pytest.mark.parametrize("B", [1, 2])
def test_a_block_of_two_gigabytes_behind_a_tail(cuda_device, B):
    """Past the largest pitch of a copy of rows. Values that bf16 sums exactly, so that a wrong place cannot hide."""
    T, C, W = (1 << 20) + 3, 1024, 16
    ramp = torch.arange(T, device=cuda_device) % 61
    n = ramp.to(torch.bfloat16).view(1, T, 1).expand(B, T, C).contiguous()
    tail = torch.full((B, W - 1, C), 7.0, dtype=torch.bfloat16, device=cuda_device)
    w = torch.zeros(C, W, dtype=torch.bfloat16, device=cuda_device)
    w[:, W - 1] = 1
    u, xin, in_full = _behind_tail(tail, n, w, torch.zeros(C, dtype=torch.bfloat16, device=cuda_device))
    assert native.status() == 0 and in_full
    assert (xin[:, :W - 1] == 7).all() and torch.equal(xin[:, W - 1:], n)
    assert (u[:, :W - 1] == 7).all() and torch.equal(u[:, W - 1:], n[:, :T - W + 1])


@pytest.mark.parametrize("W", [1, 15, 17, 32, 33, 48, 100, 128])
@pytest.mark.parametrize("B,T,C", [(1, 1, 2), (3, 16, 66), (2, 47, 64), (300, 3, 2), (1, 700, 64)])
def test_other_windows(cuda_device, B, T, C, W):
    """Windows, lengths and channels around whole blocks of 16 taps, 16 steps and 64 channels; many sequences to a slice, many slices to a sequence."""
    test_shortconv_edges(cuda_device, B, T, C, W, True)


@pytest.mark.parametrize("W", [15, 17, 33, 64])
@pytest.mark.parametrize("T", [1, 17, 40, 130])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_nothing_beyond_the_sequence_is_multiplied_by_other_windows(cuda_device, T, W, bad):
    test_nothing_beyond_the_sequence_is_multiplied(cuda_device, T, W, bad)


def test_weight_gradient_of_long_sequences_keeps_its_error(cuda_device):
    """fp32 sums against 64 bits: chains of 256 terms and a sum of their results; random signs let 2^-24 grow with the root of a chain's length (16 times),
    and the first sum is no nearer than its own rounding."""
    B, T, C, W = 4, 4096, 64, 33
    torch.manual_seed(1)
    x, dy = (torch.randn(B, T, C, device=cuda_device).bfloat16() for _ in range(2))
    w = torch.randn(C, W, device=cuda_device).bfloat16()
    slices = lib.raw("elfa_shortconv_bwd_slices")(B, T, C, W)
    part, dw, db = (torch.empty(*s, device=cuda_device) for s in ((slices, W + 1, C), (C, W), (C,)))
    lib.call("elfa_shortconv_bwd_as", x, w, dy, torch.empty_like(x), dw, db, part, 0, B, T, C, W, stream_ptr(x))
    ref = torch.stack([(dy[:, j:].double() * x[:, :T - j].double()).sum((0, 1)) for j in range(W)], 1)
    assert ((dw.double() - ref).norm() / ref.norm()).item() < 16 * 2.0 ** -24


@pytest.mark.parametrize("W", [1, 5, 15, 64])
@pytest.mark.parametrize("B,T,C", [(2500, 8, 130), (700, 9, 64), (3, 7, 2), (5000, 2, 66)])
def test_other_windows_of_short_sequences(cuda_device, B, T, C, W):
    """Up to eight steps a warp takes whole sequences, several in turn."""
    test_shortconv_edges(cuda_device, B, T, C, W, True)


@pytest.mark.parametrize("W", [5, 33])
@pytest.mark.parametrize("T", [2, 8, 9])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_nothing_beyond_a_short_sequence_is_multiplied(cuda_device, T, W, bad):
    test_nothing_beyond_the_sequence_is_multiplied(cuda_device, T, W, bad)


@pytest.mark.parametrize("W", [5, 64])
@pytest.mark.parametrize("T", [1, 2, 4, 8])
def test_short_sequences_cost_about_what_long_ones_do(cuda_device, T, W):
    """The same values in sequences of T and of 1024 steps, output and gradients. Measured 0.6 to 1.5; in blocks of 16 taps by 16 steps 2.9 to 23."""
    def us(B, T):
        x = torch.randn(B, T, 1024, device=cuda_device).bfloat16().requires_grad_(True)
        w, b = (torch.randn(*s, device=cuda_device).bfloat16().requires_grad_(True) for s in ((1024, W), (1024,)))
        dy, best = torch.randn_like(x), []
        for _ in range(5):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            torch.cuda._sleep(10_000_000)
            e[0].record()
            for _ in range(10):
                torch.autograd.grad(eops.shortconv(x, w, b), (x, w, b), dy)
            e[1].record()
            torch.cuda.synchronize()
            best.append(e[0].elapsed_time(e[1]))
        return min(best)
    assert us(12288 // T, T) < 2 * us(12, 1024)
