"""Which calls the native paths take, asked with stand-ins for CUDA tensors: nothing here touches a device."""
from types import SimpleNamespace

import pytest
import torch

from elfa_b200 import native
from elfa_b200.ops import efla as eops


def _fake(*shape, device="cuda:0", dtype=torch.bfloat16):
    return SimpleNamespace(shape=torch.Size(shape), device=torch.device(device), dtype=dtype, is_cuda=device.startswith("cuda"),
                           numel=lambda: torch.Size(shape).numel())


@pytest.mark.parametrize("other", ["cpu", "cuda:1"])
def test_prism_kernels_want_one_device(other):
    """A kernel given a host pointer, or one of another GPU, would fault: those calls belong to the general path, which refuses them."""
    d, D = 32, 64
    u, v, s = _fake(2, 3, D), _fake(2, 3, D), _fake(2, 2, d, d, dtype=torch.float32)
    ws = [[_fake(D, d) for _ in range(2)] for _ in range(3)]
    assert eops.prism_gated_native(u, v, ws[0], d) and eops.prism_stream_native(u, v, *ws, s, d)
    assert not eops.prism_gated_native(u, _fake(2, 3, D, device=other), ws[0], d)
    assert not eops.prism_stream_native(u, v, *ws, _fake(2, 2, d, d, device=other, dtype=torch.float32), d)
    for i in range(3):
        moved = [list(w) for w in ws]
        moved[i][1] = _fake(D, d, device=other)
        assert not eops.prism_stream_native(u, v, *moved, s, d)


def test_a_host_tensor_has_no_stream(monkeypatch):
    asked = []
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda i: asked.append(i) or 7, raising=False)
    assert native.stream_ptr(SimpleNamespace(get_device=lambda: 1)) == 7 and asked == [1]
    with pytest.raises(ValueError, match="cuda device"):
        native.stream_ptr(torch.zeros(1))
    assert asked == [1]


# S, B, query heads, key heads, head dimension, causal -> the fastest of 1, 2 and 4 CTAs per key head, by at least 3 %, on a B200 with 148 SMs
@pytest.mark.parametrize("shape,shares", [((512, 1, 16, 4, 64, 1), 4), ((1024, 1, 16, 4, 64, 1), 4), ((1777, 2, 16, 4, 64, 1), 2), ((2048, 1, 16, 4, 128, 1), 4),
                                          ((1024, 4, 16, 4, 128, 1), 2), ((1024, 4, 16, 4, 128, 0), 1), ((1024, 4, 32, 8, 128, 1), 1), ((2048, 2, 32, 8, 64, 1), 1),
                                          ((1152, 4, 16, 8, 128, 1), 1), ((1152, 2, 16, 4, 128, 1), 2), ((1152, 2, 16, 4, 128, 0), 2), ((384, 12, 16, 4, 128, 1), 1),
                                          ((128, 36, 16, 4, 128, 1), 1), ((128, 18, 16, 4, 64, 1), 2), ((1280, 4, 16, 4, 128, 0), 2), ((2048, 1, 16, 1, 128, 1), 4),
                                          ((4096, 1, 32, 32, 128, 1), 1), ((300, 2, 6, 2, 64, 1), 1)])
def test_shares_of_a_key_head(shape, shares):
    assert native.lib.raw("elfa_attention_bwd_shares")(*shape) == shares


@pytest.mark.parametrize("shape,forward,train", [((1, 384, 8, 64), False, False), ((1, 500, 16, 32), False, False), ((1, 1000, 2, 64), True, False), ((1, 1400, 2, 64), True, False),
                                                 ((1, 2000, 8, 64), True, True), ((1, 8192, 16, 64), True, True), ((2, 1531, 8, 128), True, True),
                                                 ((8, 1400, 8, 64), False, False), ((8, 2048, 16, 64), False, False)])
def test_walks_that_are_cut(shape, forward, train):
    """Two launches and an allocation more: not for a walk that ends before the host has issued the rest of the call."""
    assert (native.lib.raw("elfa_efla_segments")(*shape) > 1, native.lib.raw("elfa_efla_segments_train")(*shape) > 1) == (forward, train)


# M, N, most CTAs -> columns of a tile, 148 SMs
@pytest.mark.parametrize("shape,width", [((128, 4096, 0), 64), ((128, 4096, 200), 64), ((128, 4096, 64), 64), ((128, 4096, 63), 128), ((260, 4096, 0), 128),
                                         ((520, 1024, 80), 64), ((520, 1024, 79), 128), ((128, 64, 1), 64), ((4096, 4096, 0), 512), ((4096, 4096, 100), 256),
                                         ((9, 3072, 0), 64), ((16, 3080, 0), 128), ((63, 9216, 0), 128), ((64, 9216, 0), 64)])
def test_a_wave_of_narrow_tiles_is_one_of_the_launch(shape, width):
    """64 CTAs make 64 narrow tiles in one wave; fewer would go round twice. Few rows, which all of them ask for, go to fewer tiles."""
    M, N, most = shape
    tile = native.lib.raw("elfa_gemm_bf16_tile")
    assert tile(M, N, 0, 0, most) == width
    assert [tile(M, N, 0, n, most) for n in (64, 128, 256, 512)] == [64, 128, 256, 512]
