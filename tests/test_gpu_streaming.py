"""``forward_with_states`` from native code against the layer-by-layer route: the same kernels in the same order, so the same bits."""
import pytest
import torch
import torch.autograd.forward_ad as fwd

from elfa_b200 import native
from elfa_b200.config import Config
from elfa_b200.models import streaming
from elfa_b200.models.efla_model import EflaModel
from elfa_b200.models.gpt import GPTModel
from elfa_b200.native import lib

pytestmark = pytest.mark.gpu


def _config(efla, act="gelu", norm="layernorm", H=4, Hkv=4, hd=64, L=2, W=4, prism=True, tie=True, positions=True):
    cfg = Config()
    m = cfg.model
    m.dtype, m.efla.enabled, m.prism.enabled = "bf16", efla, efla and prism
    m.num_layers, m.hidden_dim, m.num_heads, m.num_kv_heads, m.head_dim = 2, H * hd, H, Hkv, hd
    m.intermediate_dim, m.vocab_size, m.activation, m.norm_type, m.tie_embeddings = 256, 264, act, norm, tie
    m.prism.num_iterations, m.prism.shortconv_window, m.max_seq_len, cfg.data.seq_len = L, W, 400, 400
    cfg.bench.init_std, cfg.bench.learned_positions = 0.05, positions
    return cfg


def _stream(model, ids, cuts):
    """Logits and states of the calls that ``cuts`` splits ``ids`` into."""
    out, states = [], None
    with torch.no_grad():
        for lo, hi in zip(cuts, cuts[1:]):
            logits, states = model.forward_with_states(ids[:, lo:hi], states)
            out.append(logits)
    layers = states["layers"] if isinstance(states, dict) else states
    return out + [t for s in layers for t in s.values() if t is not None]


def _compare(monkeypatch, model, ids, cuts, native_calls):
    general = {n: getattr(streaming, n) for n in ("gpt_stream", "efla_stream")}
    taken = []

    def counting(f):
        def g(*a):
            r = f(*a)
            taken.append(r is not None)
            return r
        return g
    for n, f in general.items():
        monkeypatch.setattr(streaming, n, counting(f))
    got = _stream(model, ids, cuts)
    assert sum(taken) == native_calls
    for n in general:
        monkeypatch.setattr(streaming, n, lambda *a: None)
    want = _stream(model, ids, cuts)
    assert native.status() == 0 and len(got) == len(want)
    for a, b in zip(got, want):
        assert a.shape == b.shape and a.stride() == b.stride() and a.dtype == b.dtype and torch.equal(a, b)


def _ids(B, T, dev):
    return torch.randint(0, 264, (B, T), generator=torch.Generator().manual_seed(T)).to(dev)


@pytest.mark.parametrize("act,norm,H,Hkv,hd,tie,positions", [("gelu", "layernorm", 4, 4, 64, True, True), ("swiglu", "rmsnorm", 8, 2, 64, False, True),
                                                              ("silu", "layernorm", 4, 1, 128, True, False), ("relu", "rmsnorm", 2, 2, 32, True, True)])
@pytest.mark.parametrize("B,cuts", [(1, (0, 1, 2, 3)), (3, (0, 33, 34, 36)), (2, (0, 300, 301))])
def test_softmax_family(cuda_device, monkeypatch, act, norm, H, Hkv, hd, tie, positions, B, cuts):
    torch.manual_seed(0)
    model = GPTModel(_config(False, act, norm, H, Hkv, hd, tie=tie, positions=positions), device=cuda_device).eval()
    _compare(monkeypatch, model, _ids(B, cuts[-1], cuda_device), cuts, len(cuts) - 1)


@pytest.mark.parametrize("act,norm,hd,L,W,prism", [("gelu", "rmsnorm", 64, 2, 4, True), ("silu", "layernorm", 32, 1, 16, True), ("gelu", "rmsnorm", 128, 3, 1, True),
                                                   ("relu", "rmsnorm", 64, 2, 4, False), ("gelu", "rmsnorm", 96, 8, 5, True)])
@pytest.mark.parametrize("B,cuts", [(1, (0, 1, 2, 3)), (2, (0, 2, 5, 50)), (2, (0, 130, 131, 390))])
def test_efla_family(cuda_device, monkeypatch, act, norm, hd, L, W, prism, B, cuts):
    torch.manual_seed(0)
    model = EflaModel(_config(True, act, norm, 2, 2, hd, L, W, prism), device=cuda_device).eval()
    _compare(monkeypatch, model, _ids(B, cuts[-1], cuda_device), cuts, len(cuts) - 1)


@pytest.mark.parametrize("B,H,hd,cuts", [(2, 2, 64, (0, 100, 1137, 2210)), (1, 2, 128, (0, 1500, 1501, 2535))])
def test_efla_calls_that_are_walked_in_segments(cuda_device, monkeypatch, B, H, hd, cuts):
    """The scratch of the segments is a piece of the one workspace of all layers; carried states, ragged last chunks, a tail in front."""
    cut = [lib.raw("elfa_efla_segments")(B, hi - lo, H, hd) for lo, hi in zip(cuts, cuts[1:])]
    assert sum(c > 1 for c in cut) >= 2, cut
    torch.manual_seed(0)
    model = EflaModel(_config(True, H=H, hd=hd, W=16), device=cuda_device).eval()
    _compare(monkeypatch, model, _ids(B, cuts[-1], cuda_device), cuts, len(cuts) - 1)


def test_what_is_left_to_the_general_route(cuda_device, monkeypatch):
    ids = _ids(2, 12, cuda_device)
    cuts = (0, 8, 9)

    def left(change, calls=0, efla=False):
        model = (EflaModel if efla else GPTModel)(_config(efla), device=cuda_device).eval()
        change(model)
        with monkeypatch.context() as m:
            _compare(m, model, ids, cuts, calls)
    for efla in (False, True):
        first = lambda m: m.blocks[1]
        left(lambda m: None, 2, efla)
        left(lambda m: first(m).ln1.register_forward_hook(lambda *a: None), 0, efla)
        left(lambda m: first(m).register_forward_pre_hook(lambda *a: None), 0, efla)

        def replaced(m):
            f = first(m).ln2.forward
            first(m).ln2.forward = lambda *a, **k: f(*a, **k)
        left(replaced, 0, efla)

        if not efla:
            m2 = GPTModel(_config(False), device=cuda_device).eval()
            logits, _ = m2.forward_with_states(ids)                     # a gradient may be wanted
            assert logits.requires_grad
    # five rows of four heads to a key head: the cached kernel takes eight
    model = GPTModel(_config(False, H=4, Hkv=1), device=cuda_device).eval()
    _compare(monkeypatch, model, ids, (0, 4, 9, 10), 2)


@pytest.mark.parametrize("offset,pitch", [(1, 192), (0, 193), (3, 195)])
def test_tails_at_odd_places(cuda_device, offset, pitch):
    """A caller's own ShortConv tail may start and step anywhere: such calls go layer by layer, to the same values."""
    model = EflaModel(_config(True, H=1, hd=64), device=cuda_device).eval()
    ids = _ids(2, 9, cuda_device)
    with torch.no_grad():
        _, states = model.forward_with_states(ids[:, :5])
        want, after = model.forward_with_states(ids[:, 5:], states)
        for s in states:
            odd = torch.empty(offset + 2 * pitch, dtype=torch.bfloat16, device=cuda_device).as_strided((2, 3, 64), (pitch, 64, 1), offset)
            s["conv_tail"] = odd.copy_(s["conv_tail"])
        got, now = model.forward_with_states(ids[:, 5:], states)
    assert native.status() == 0 and torch.equal(got, want)
    assert all(torch.equal(a[n], b[n]) for a, b in zip(after, now) for n in a)


def test_a_tangent_is_not_dropped(cuda_device):
    """Forward mode stays open under ``no_grad``: the scan has no such rule and refuses a dual state."""
    model = EflaModel(_config(True), device=cuda_device).eval()
    ids = _ids(1, 4, cuda_device)
    with torch.no_grad():
        _, states = model.forward_with_states(ids[:, :3])
        with fwd.dual_level():
            states[0]["efla"] = fwd.make_dual(states[0]["efla"], torch.ones_like(states[0]["efla"]))
            with pytest.raises(NotImplementedError):
                model.forward_with_states(ids[:, 3:], states)
