"""Cached attention kernel against the fp32 formula. The output is rounded to bf16 once: 2^-8 of the largest."""
import pytest
import torch

from elfa_b200 import native, ops
from elfa_b200.models.gpt import _attend_cached

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,s,B,H,Hkv,hd", [(1, 1, 1, 1, 1, 32), (31, 1, 2, 4, 4, 64), (32, 2, 1, 8, 2, 64), (255, 1, 3, 8, 1, 128),
                                            (600, 3, 1, 4, 2, 256), (5000, 1, 1, 16, 4, 64)])
def test_attention_decode(cuda_device, t, s, B, H, Hkv, hd):
    torch.manual_seed(t + hd)
    h = torch.randn(s, B, H + 2 * Hkv, hd, device=cuda_device).bfloat16()
    q, k, v = h[:, :, :H], h[:, :, H:H + Hkv], h[:, :, H + Hkv:]
    kc, vc = (torch.randn(t, B, Hkv, hd, device=cuda_device).bfloat16() for _ in range(2))
    assert ops.attention_decode_native(q, k, v, kc, vc)
    o, ko, vo = ops.attention_decode(q, k, v, kc, vc)
    k_all, v_all = torch.cat((kc, k)), torch.cat((vc, v))
    assert torch.equal(ko, k_all) and torch.equal(vo, v_all)
    rep = H // Hkv
    ref = _attend_cached(q.float(), k_all.repeat_interleave(rep, 2).float(), v_all.repeat_interleave(rep, 2).float())
    assert native.status() == 0
    assert (o.float() - ref).abs().max() <= 2 ** -8 * ref.abs().max()
    # a cache handed in as a strided view
    o2, _, _ = ops.attention_decode(q, k, v, kc.transpose(0, 1).contiguous().transpose(0, 1), vc)
    assert torch.equal(o2, o)


def test_gradients_and_wide_blocks_keep_the_general_path(cuda_device):
    h = torch.randn(3, 1, 12, 64, device=cuda_device).bfloat16()
    kc = torch.randn(4, 1, 2, 64, device=cuda_device).bfloat16()
    q, k, v = h[:, :, :8], h[:, :, 8:10], h[:, :, 10:]
    assert not ops.attention_decode_native(q, k, v, kc, kc)                        # 3 x 4 query rows per key head
    assert not ops.attention_decode_native(q[:1].detach().requires_grad_(True), k[:1], v[:1], kc, kc)


@pytest.mark.parametrize("t,s", [(31, 1), (32, 1), (33, 1), (64, 2), (95, 2), (600, 1)])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_a_non_finite_key_is_not_dropped(cuda_device, t, s, bad):
    """At t = 32 and 95 the newest key is the first of its slice: its NaN scores are the only ones there."""
    torch.manual_seed(t)
    h = torch.randn(s, 1, 4, 64, device=cuda_device).bfloat16()
    h[-1, 0, 2, 5], h[-1, 0, 2, 6] = bad, -bad                                     # inf - inf in the score of every query
    h[:, :, :2, 5:7] = 1.0
    q, k, v = h[:, :, :2], h[:, :, 2:3], h[:, :, 3:]
    kc, vc = (torch.randn(t, 1, 1, 64, device=cuda_device).bfloat16() for _ in range(2))
    o = ops.attention_decode(q, k, v, kc, vc)[0]
    ref = _attend_cached(q.float(), torch.cat((kc, k)).repeat_interleave(2, 2).float(), torch.cat((vc, v)).repeat_interleave(2, 2).float())
    assert ref[-1].isnan().all() and (s == 1 or ref[0].isfinite().all())           # the row before the key does not see it
    assert torch.equal(o.isnan(), ref.isnan())
