"""Decoding steps of the EFLA family, all layers in one kernel, against the layer-by-layer route: the same pieces in the same order, so the same bits. Sizes
at the edges of what the kernel takes: one to eight rows, rows whose norm takes one and two warps, one and several rounds of tiles, a ring of two and of four
half blocks, more layers than one launch holds."""
import pytest
import torch

from elfa_b200 import native
from elfa_b200.config import Config
from elfa_b200.models import streaming
from elfa_b200.models.efla_model import EflaModel
from elfa_b200.native import lib

pytestmark = pytest.mark.gpu


def _config(layers, H, hd, F, act="gelu", norm="rmsnorm", L=2, W=4, prism=True):
    cfg = Config()
    m = cfg.model
    m.dtype, m.efla.enabled, m.prism.enabled = "bf16", True, prism
    m.num_layers, m.hidden_dim, m.num_heads, m.num_kv_heads, m.head_dim = layers, H * hd, H, H, hd
    m.intermediate_dim, m.vocab_size, m.activation, m.norm_type, m.max_seq_len, cfg.data.seq_len = F, 264, act, norm, 700, 700
    m.prism.num_iterations, m.prism.shortconv_window, cfg.bench.init_std = L, W, 0.05
    return cfg


def _steps(model, ids, cuts, launches):
    """Logits and states of every call; the steps after the prompt are ``launches`` kernels each (None: not looked at)."""
    out, states = [], None
    with torch.no_grad():
        for lo, hi in zip(cuts, cuts[1:]):
            lib.raw("elfa_launch_count")(1)
            logits, states = model.forward_with_states(ids[:, lo:hi], states)
            if lo and launches:
                assert lib.raw("elfa_launch_count")(0) == launches
            out.append(logits)
            out += [t for s in states for t in s.values() if t is not None]
    return out


def _check(model, B, cuts, dev, monkeypatch, launches):
    ids = torch.randint(0, 264, (B, cuts[-1]), generator=torch.Generator().manual_seed(B)).to(dev)
    got = _steps(model, ids, cuts, launches)
    monkeypatch.setattr(streaming, "efla_stream", lambda *a: None)
    want = _steps(model, ids, cuts, None)
    assert native.status() == 0 and len(got) == len(want)
    for a, b in zip(got, want):
        assert torch.isfinite(b).all() and torch.equal(a, b)


@pytest.mark.parametrize("H,hd,F,layers,act,norm,L,W,prism,B,cuts,launches", [
    (1, 32, 8, 2, "gelu", "layernorm", 1, 4, True, 1, (0, 3, 4, 5), 2),
    (16, 64, 4096, 2, "gelu", "rmsnorm", 2, 16, True, 2, (0, 64, 65, 69), 2),
    (16, 128, 512, 1, "silu", "rmsnorm", 4, 5, True, 8, (0, 9, 10), 2),      # eight rows, 2048 wide
    (32, 96, 264, 1, "gelu", "layernorm", 8, 16, True, 1, (0, 20, 21, 23), 2),      # 3072 wide; several rounds of gate logits
    (4, 64, 256, 9, "relu", "rmsnorm", 2, 4, True, 1, (0, 4, 12), 3),      # a layer more than one launch holds, eight tokens
    (4, 64, 256, 2, "gelu", "rmsnorm", 1, 1, False, 4, (0, 2, 4), 2),
    (4, 64, 264, 1, "gelu", "layernorm", 2, 4, True, 3, (0, 6, 7), 2),      # rows that end inside a pair of the fragments' columns
    (8, 32, 256, 1, "silu", "rmsnorm", 1, 8, True, 5, (0, 7, 8), 2),
    (2, 96, 200, 1, "relu", "rmsnorm", 2, 16, True, 7, (0, 17, 18), 2),
    (2, 128, 264, 1, "gelu", "rmsnorm", 1, 1, False, 7, (0, 2, 3), 2),
])
def test_matches_the_layers(cuda_device, monkeypatch, H, hd, F, layers, act, norm, L, W, prism, B, cuts, launches):
    torch.manual_seed(0)
    cfg = _config(layers, H, hd, F, act, norm, L, W, prism)
    _check(EflaModel(cfg, device=cuda_device).eval(), B, cuts, cuda_device, monkeypatch, launches)


@pytest.mark.parametrize("H,hd,F,L,W,prism,B,cuts", [
    (20, 128, 5120, 2, 4, False, 8, (0, 3, 4, 5)),      # two and three rounds of tiles where the chain's products take one: half as long again in one kernel
    (40, 64, 10240, 2, 4, True, 4, (0, 9, 10)),
    (24, 128, 264, 2, 4, True, 8, (0, 5, 6)),      # eight rows of 3072 do not fit beside the weights
    (2, 128, 264, 8, 16, True, 1, (0, 20, 23, 26)),      # nor three tokens of eight iterations in the states' scratch
    (4, 96, 264, 8, 16, True, 1, (0, 2, 6, 10)),      # (a tail shorter than the window)
])
def test_the_chain_where_the_kernel_does_not_fit_or_is_slower(cuda_device, monkeypatch, H, hd, F, L, W, prism, B, cuts):
    torch.manual_seed(0)
    m = EflaModel(_config(1, H, hd, F, L=L, W=W, prism=prism), device=cuda_device).eval()
    ids = torch.randint(0, 264, (B, cuts[-1]), generator=torch.Generator().manual_seed(B)).to(cuda_device)
    with torch.no_grad():
        _, states = m.forward_with_states(ids[:, :cuts[1]])
        lib.raw("elfa_launch_count")(1)
        m.forward_with_states(ids[:, cuts[1]:cuts[2]], states)
        assert lib.raw("elfa_launch_count")(0) > 8
    _check(m, B, cuts, cuda_device, monkeypatch, None)


def _us(model, ids, states):
    """A step on the device, its launches queued ahead."""
    best = []
    with torch.no_grad():
        for _ in range(6):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            torch.cuda._sleep(8_000_000)
            e[0].record()
            for _ in range(10):
                model.forward_with_states(ids, states)
            e[1].record()
            torch.cuda.synchronize()
            best.append(100 * e[0].elapsed_time(e[1]))
    return min(best)


@pytest.mark.parametrize("H,hd,prism,most", [(16, 128, True, 2.1), (8, 128, False, 1.7)])
def test_scan_and_state_are_spread(cuda_device, H, hd, prism, most):
    """Eight sequences against one. 2048 wide the product beside the states leaves eight CTAs without a tile, 128 states are too many for those; without PRISM no
    product goes beside the scan. Measured 1.6 and 1.3; with everything on those few CTAs 3.0 and 2.0."""
    torch.manual_seed(0)
    m = EflaModel(_config(2, H, hd, 4 * H * hd, prism=prism), device=cuda_device).eval()
    us = []
    for B in (1, 8):
        ids = torch.randint(0, 264, (B, 5), generator=torch.Generator().manual_seed(1)).to(cuda_device)
        with torch.no_grad():
            _, states = m.forward_with_states(ids[:, :4])
        us.append(_us(m, ids[:, 4:], states))
    assert us[1] < most * us[0]


def test_under_capture_and_on_two_streams(cuda_device):
    """A captured step replays; two streams decode side by side, each call with its own barrier."""
    m = EflaModel(_config(2, 4, 64, 256), device=cuda_device).eval()
    ids = torch.randint(0, 264, (2, 12), generator=torch.Generator().manual_seed(1)).to(cuda_device)
    with torch.no_grad():
        _, states = m.forward_with_states(ids[:, :9])
        want, _ = m.forward_with_states(ids[:, 9:10], states)
        side = [torch.cuda.Stream() for _ in range(2)]
        torch.cuda.synchronize()
        got = []
        for i in range(8):
            with torch.cuda.stream(side[i % 2]):
                got.append(m.forward_with_states(ids[:, 9:10], states)[0])
        torch.cuda.synchronize()
        assert all(torch.equal(g, want) for g in got)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out, _ = m.forward_with_states(ids[:, 9:10], states)
        for _ in range(2):
            out.zero_()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(out, want)
        del graph
    assert native.status() == 0


def test_on_a_part_of_the_gpu(cuda_device):
    """A stream of a green context has fewer SMs than the one-kernel form needs at once: the chain, and no error is left behind."""
    green = pytest.importorskip("torch.cuda.green_contexts")
    m = EflaModel(_config(2, 4, 64, 256), device=cuda_device).eval()
    ids = torch.randint(0, 264, (2, 10), generator=torch.Generator().manual_seed(1)).to(cuda_device)
    with torch.no_grad():
        _, states = m.forward_with_states(ids[:, :9])
        want, _ = m.forward_with_states(ids[:, 9:], states)
        torch.cuda.synchronize()
        try:
            part = green.GreenContext.create(num_sms=32, device_id=cuda_device.index or 0)
        except RuntimeError as e:
            pytest.skip(str(e))
        with torch.cuda.stream(part.Stream()):
            got, _ = m.forward_with_states(ids[:, 9:], states)
        torch.cuda.synchronize()
        part.set_context()
        try:
            also, _ = m.forward_with_states(ids[:, 9:], states)
            torch.cuda.synchronize()
        finally:
            part.pop_context()
    assert torch.equal(got, want) and torch.equal(also, want) and native.status() == 0
