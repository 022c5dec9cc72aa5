"""Which streaming calls go to native code, decided on the CPU: the native calls are only recorded, so nothing is launched and a call that must not
get there shows without a device."""
import contextlib
import ctypes

import pytest
import torch
from torch.autograd import forward_ad

from elfa_b200 import native
from elfa_b200.config import Config
from elfa_b200.models import streaming
from elfa_b200.models.efla_model import EflaModel
from elfa_b200.models.gpt import GPTModel
from elfa_b200.parallel.mesh import ParallelContext
from elfa_b200.quant.qat import QuantSpec


@pytest.fixture
def route(monkeypatch):
    """``route(model, ids, states)``: whether the call is taken by native code."""
    calls = []
    monkeypatch.setattr(streaming, "_eager", lambda ids: True)
    monkeypatch.setattr(streaming, "stream_ptr", lambda t: 0)
    monkeypatch.setattr(streaming.lib, "call", lambda name, *a: calls.append(name))
    monkeypatch.setattr(streaming.lib, "raw", lambda name: lambda *a: 1)

    def ask(model, ids, states=None):
        if states is None:
            states = fresh(model, ids.shape[0])
        calls.clear()
        with torch.no_grad():
            r = (streaming.efla_stream if isinstance(model, EflaModel) else streaming.gpt_stream)(model, ids, states)
        assert (r is not None) == (len(calls) == 1)
        return r is not None
    return ask


def fresh(model, batch):
    return model.init_states(batch) if isinstance(model, EflaModel) else {"pos": 0, "layers": [{"k": None, "v": None} for _ in model.blocks]}


def model(efla, act="gelu", layers=2, prism=True):
    cfg = Config()
    m = cfg.model
    m.dtype, m.efla.enabled, m.prism.enabled = "bf16", efla, efla and prism
    m.num_layers, m.hidden_dim, m.num_heads, m.num_kv_heads, m.head_dim = layers, 64, 2, 2, 32
    m.intermediate_dim, m.vocab_size, m.activation, m.norm_type, m.max_seq_len, cfg.data.seq_len = 64, 72, act, "rmsnorm", 32, 32
    m.prism.num_iterations, m.prism.shortconv_window = 2, 4
    return (EflaModel if efla else GPTModel)(cfg, device=torch.device("cpu")).eval()


IDS = torch.arange(6).view(2, 3)


def test_plain_calls_are_taken(route):
    assert route(model(True), IDS) and route(model(False), IDS) and route(model(True, prism=False), IDS)


def test_shortconv_tails_that_the_kernel_cannot_read(route):
    """It reads two channels at a time: an odd offset or an odd batch stride belongs to the general route."""
    m, D = model(True), 64

    def tail(offset, pitch):
        flat = torch.zeros(offset + 2 * pitch + 3 * D, dtype=torch.bfloat16)
        return flat.as_strided((2, 3, D), (pitch, D, 1), offset)
    for offset, pitch, taken in ((0, 3 * D, True), (2, 3 * D + 2, True), (1, 3 * D, False), (0, 3 * D + 1, False), (3, 3 * D + 3, False)):
        states = fresh(m, 2)
        for s in states:
            s["conv_tail"] = tail(offset, pitch)
        assert route(m, IDS, states) == taken, (offset, pitch)


def test_an_activation_that_the_block_does_not_have(route):
    """An EFLA block has one up-projection: with SwiGLU written into it the native call would read twice its columns."""
    m = model(True)
    for blk in m.blocks:
        blk.act = "swiglu"
    assert not route(m, IDS)
    m = model(False)
    for blk in m.blocks:
        blk.mlp.act, blk.mlp.gated = "silu", True               # the layer goes by `gated`
    assert not route(m, IDS)


class _Wrapped(torch.nn.Module):
    def __init__(self, block):
        super().__init__()
        self.inner = block

    def forward(self, *a, **k):
        return self.inner(*a, **k)


@pytest.mark.parametrize("efla", [True, False])
def test_models_without_layers_or_with_other_ones(route, efla):
    assert not route(model(efla, layers=0), IDS)
    for i in (0, 1):
        m = model(efla)
        m.blocks[i] = _Wrapped(m.blocks[i])
        assert not route(m, IDS, fresh(model(efla), 2))
        m = model(efla)
        name = "efla" if efla else "mlp"
        setattr(m.blocks[i], name, _Wrapped(getattr(m.blocks[i], name)))
        assert not route(m, IDS)
    if efla:
        m = model(True)
        m.blocks[0].prism = _Wrapped(m.blocks[0].prism)
        assert not route(m, IDS)


def test_states_that_leave_things_out(route):
    """What the layers read with ``get`` may be absent, what they do not read may be too, and a layer without a state has ``None``."""
    m = model(False)
    assert route(m, IDS, {"pos": 0, "layers": [{}, {}]})
    assert not route(m, IDS, {"pos": 0, "layers": [None, None]}) and not route(m, IDS, {"pos": 0, "layers": [{}, None]})
    m = model(True, prism=False)
    states = [{"efla": s["efla"]} for s in fresh(m, 2)]
    assert route(m, IDS, states)
    assert not route(m, IDS, [None, None]) and not route(m, IDS, [states[0], None])
    m = model(True)
    states = [{"efla": s["efla"], "prism": s["prism"]} for s in fresh(m, 2)]
    assert route(m, IDS, states)


def test_a_table_that_is_not_the_configured_vocabulary(route):
    """Ids are checked against the configured vocabulary, the table may have more rows."""
    for efla in (True, False):
        m = model(efla)
        m.embed_tokens = torch.nn.Parameter(torch.zeros(80, 64, dtype=torch.bfloat16))
        m.lm_head = None
        assert not route(m, IDS)


def test_states_of_another_tensor_class(route):
    class Tagged(torch.Tensor):
        pass
    for efla in (True, False):
        m = model(efla)
        states = fresh(m, 2)
        if efla:
            states[1]["efla"] = states[1]["efla"].as_subclass(Tagged)
        else:
            states["pos"] = 1
            for c in states["layers"]:
                c["k"], c["v"] = (torch.zeros(1, 2, 2, 32, dtype=torch.bfloat16) for _ in range(2))
            assert route(m, IDS, {"pos": 1, "layers": [dict(c) for c in states["layers"]]})
            states["layers"][1]["v"] = states["layers"][1]["v"].as_subclass(Tagged)
        assert not route(m, IDS, states)


def test_modes_that_only_the_layers_know():
    def under(ctx):
        with torch.no_grad(), ctx:
            return streaming._plain_mode()
    assert under(contextlib.nullcontext())
    assert not streaming._plain_mode()                             # a gradient may be wanted
    assert not under(forward_ad.dual_level())
    assert not under(torch.utils._python_dispatch.TorchDispatchMode()) and not under(torch.overrides.TorchFunctionMode())
    seen = []
    with torch.no_grad():
        torch.func.vmap(lambda x: seen.append(streaming._plain_mode()) or x)(torch.zeros(2))
        torch.func.jvp(lambda x: seen.append(streaming._plain_mode()) or x, (torch.zeros(2),), (torch.ones(2),))
        torch.jit.trace(lambda x: seen.append(streaming._plain_mode()) or x, torch.zeros(2), check_trace=False)
        h = torch.nn.modules.module.register_module_forward_hook(lambda *a: None)
        seen.append(streaming._plain_mode())
        h.remove()
        assert len(seen) == 4 and not any(seen) and streaming._plain_mode()


@pytest.mark.parametrize("efla", [True, False])
def test_replaced_methods_are_called(route, monkeypatch, efla):
    m = model(efla)
    kinds = {type(x) for x in m.modules() if type(x).__module__.startswith("elfa_b200")}
    assert len(kinds) == 5
    for kind in kinds:
        names = ("hidden_states", "_embed", "_logits") if kind is EflaModel else ("hidden_states",) if kind is GPTModel else ("forward",)
        for name in names:
            with monkeypatch.context() as p:                       # on the class
                p.setattr(kind, name, lambda *a, **k: None)
                assert not route(m, IDS), (kind, name)
            x = next(x for x in reversed(list(m.modules())) if type(x) is kind)
            setattr(x, name, lambda *a, **k: None)                  # on one instance
            assert not route(m, IDS), (kind, name)
            delattr(x, name)
        with monkeypatch.context() as p:
            p.setattr(kind, "__call__", lambda *a, **k: None, raising=False)
            assert not route(m, IDS) or kind in (EflaModel, GPTModel), kind
    with monkeypatch.context() as p:
        p.setattr(torch.nn.Module, "__call__", lambda *a, **k: None)
        assert not route(m, IDS)
    m.blocks[1].ln1.compile(backend="eager")
    assert not route(m, IDS)
    assert route(model(efla), IDS)


@pytest.mark.parametrize("efla", [True, False])
def test_hooks_gradients_quantisers_and_parallel_layers(route, efla):
    def left(change):
        m = model(efla)
        change(m, m.blocks[1])
        return not route(m, IDS)
    assert not left(lambda m, b: None)
    assert left(lambda m, b: b.ln1.register_forward_hook(lambda *a: None)) and left(lambda m, b: b.register_forward_pre_hook(lambda *a: None))
    assert left(lambda m, b: m.final_norm.register_forward_hook(lambda *a, **k: None, with_kwargs=True))
    assert left(lambda m, b: setattr(b.ln2, "eps", 0.1)) and left(lambda m, b: setattr(m, "dtype", torch.float32))
    assert left(lambda m, b: setattr(b.ln2, "weight", torch.nn.Parameter(torch.ones(64))))
    w = "w_k" if efla else "w_o"
    layer = lambda b: b.efla if efla else b.attn
    assert left(lambda m, b: setattr(layer(b), w, torch.nn.Parameter(getattr(layer(b), w).t())))                # another layout
    assert left(lambda m, b: setattr(getattr(layer(b), w), "_gemm_gather", object()))                           # fetched on use
    two = ParallelContext(tp_size=2)
    assert left(lambda m, b: setattr(layer(b), "pc", two))
    if not efla:
        assert left(lambda m, b: setattr(b.attn, "quant", QuantSpec(fmt="mxfp8"))) and left(lambda m, b: setattr(b.mlp, "quant", QuantSpec(fmt="mxfp8")))
        assert left(lambda m, b: (setattr(b, "dropout", 0.1), b.train()))
    else:
        assert left(lambda m, b: setattr(m, "pc", two))
    m = model(efla)
    states = fresh(m, 2)
    if efla:
        states[1]["efla"].requires_grad_(True)
        assert not route(m, IDS, states)
        states = fresh(m, 2)
        states[1]["prism"] = states[1]["prism"].double()
        assert not route(m, IDS, states)
    else:
        kv = [torch.zeros(2, 2, 2, 32, dtype=torch.bfloat16) for _ in range(4)]
        layers = lambda: [dict(k=kv[0], v=kv[1]), dict(k=kv[2], v=kv[3])]
        assert route(m, IDS, {"pos": 2, "layers": layers()})
        kv[3] = kv[3].transpose(0, 1)
        assert not route(m, IDS, {"pos": 2, "layers": layers()})


def test_a_gated_mlp_is_refused_natively():
    """The EFLA block has none: rows of 2 F would leave a workspace of F. Refused before anything is issued."""
    dims = (ctypes.c_longlong * 14)(1, 1, 64, 2, 32, 64, 32, 1, 0, 1, streaming._ACTS["swiglu"], 0, 0, 0)
    p = (ctypes.c_uint64 * 26)()
    with pytest.raises(native.NativeError, match="not gated"):
        native.lib.call("elfa_efla_stream", ctypes.addressof(p), ctypes.addressof(dims), ctypes.addressof((ctypes.c_float * 1)()), 1e-5, 16, 0)
