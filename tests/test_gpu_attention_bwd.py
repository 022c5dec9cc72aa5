"""Attention backward where its tiles, rings and shares end, against the fp32 formula.

Bound: P and dS are rounded to bf16 once (2^-9 of each) before products over at most S terms whose errors do not line up, and the gradients
once more: 2 % of the largest gradient, as for the other attention tests.
"""
import pytest
import torch

from elfa_b200 import native, ops

pytestmark = pytest.mark.gpu


def _check(dev, S, B, H, Hkv, hd, doc_start=None, causal=True):
    g = torch.Generator().manual_seed(S + H)
    qkv = torch.randn((S, B, H + 2 * Hkv, hd), generator=g).to(torch.bfloat16).to(dev).requires_grad_(True)
    go = torch.randn((S, B, H * hd), generator=g).to(torch.bfloat16).to(dev)
    grads = [torch.autograd.grad(ops.attention(qkv, causal=causal, num_heads=H, doc_start=doc_start), qkv, go)[0] for _ in range(2)]
    assert native.status() == 0
    assert torch.equal(*grads)                                      # fixed order of every sum
    ref_in = qkv.detach().float().requires_grad_(True)
    ref = torch.autograd.grad(ops.attention_ref(ref_in, causal=causal, num_heads=H, doc_start=doc_start), ref_in, go.float())[0]
    scale = max(ref.abs().max().item(), 1.0)
    assert (grads[0].float() - ref).abs().max().item() < 0.02 * scale + 0.02


@pytest.mark.parametrize("S", [1, 127, 129, 256, 385, 640, 897])     # one to eight inner tiles: less than, equal to and past the rings
@pytest.mark.parametrize("hd", [64, 128, 40])
def test_ring_lengths(cuda_device, S, hd):
    _check(cuda_device, S, 1, 2, 2, hd)


@pytest.mark.parametrize("H,Hkv", [(2, 1), (4, 1), (3, 1), (6, 1), (8, 1), (8, 2)])      # 1, 2 or 4 CTAs share a key head's query heads
@pytest.mark.parametrize("S,hd", [(200, 64), (330, 128), (130, 32)])
def test_shared_key_heads(cuda_device, H, Hkv, S, hd):
    _check(cuda_device, S, 2, H, Hkv, hd)


def test_key_heads_without_sharing(cuda_device):
    _check(cuda_device, 1030, 9, 8, 4, 64)                             # 9 tiles x 4 heads x 9: more CTAs than two per SM


def test_a_document_longer_than_32_tiles(cuda_device):
    """The end of a key tile's range is looked for 32 query tiles at a time."""
    S = 128 * 37 + 5
    ds = torch.zeros(1, S, dtype=torch.int32, device=cuda_device)
    ds[:, 128 * 34 + 7:] = 128 * 34 + 7
    _check(cuda_device, S, 1, 2, 1, 64, ds)


def test_not_causal(cuda_device):
    _check(cuda_device, 300, 2, 4, 2, 64, causal=False)
