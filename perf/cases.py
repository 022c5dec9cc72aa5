"""The workloads whose speed is watched: single layers and blocks of both model families, and one generation call of each.

``listed()`` names them, ``draw`` makes more of the same ranges, ``prepare`` builds what a program holds before the call, ``run`` is
one pass through the public entry points, ``exact`` the same result in 64-bit plain torch.
"""
from __future__ import annotations

import math

import torch
import torch.nn as nn
import torch.nn.functional as F

BF = torch.bfloat16


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one token per sequence of a batch that is being generated: the state is read, updated and handed back
        dict(name="efla_step", kind="efla", B=8, T=1, H=16, d=64, state=True, grad=False),
        # the token mixer of one layer of the 350M EFLA configuration, micro-batch of 8 x 2048, forward and backward
        dict(name="efla_train", kind="efla", B=8, T=2048, H=16, d=64, state=False, grad=True),
        # a ragged block of a long sequence that is trained with a carried state, wide heads
        dict(name="efla_ragged", kind="efla", B=2, T=1531, H=8, d=128, state=True, grad=True),
        # reading a long context without gradients, one sequence, continued from a state
        dict(name="efla_prefill", kind="efla", B=1, T=8192, H=16, d=64, state=True, grad=False),
        # PRISM with its ShortConv in the same 350M layer, forward and backward
        dict(name="prism_train", kind="prism", B=8, T=2048, G=16, d=64, L=2, W=16, grad=True),
        # attention of one 7B layer, one sequence of 4096 tokens, forward and backward
        dict(name="attn_train", kind="attn", B=1, S=4096, H=32, Hkv=32, hd=128, docs=0, grad=True),
        # grouped-query attention over packed documents, odd length
        dict(name="attn_packed", kind="attn", B=2, S=1777, H=16, Hkv=4, hd=64, docs=5, grad=True),
        # residual add, norm and gated MLP of the 1.3B width, forward and backward
        dict(name="mlp_swiglu", kind="mlp", B=2, S=2048, D=2048, F=8192, act="swiglu", norm="layernorm", grad=True),
        # the vocabulary projection with its loss, 350M configuration
        dict(name="head_loss", kind="head", rows=8192, D=1024, V=32000),
        # block-scaled product of the 7B QAT MLP: activations quantised on the way in, weights once
        dict(name="mxfp8_up", kind="mxfp8", M=4096, K=4096, N=11008),
        # prompt and cached decoding of the softmax-attention family (350M width, grouped keys, few layers)
        dict(name="gpt_generate", kind="gpt", B=4, prompt=512, steps=8, layers=4, H=16, Hkv=4, hd=64, Fd=4096, V=32000),
        # prompt and state-carried decoding of the EFLA family (350M width, few layers)
        dict(name="efla_generate", kind="eflam", B=2, prompt=64, steps=4, layers=2, H=16, hd=64, Fd=4096, V=32000, L=2, W=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["efla", "efla", "prism", "attn", "mlp", "head", "mxfp8", "gpt", "eflam"])
    if kind == "efla":
        d = rng.choice([32, 64, 64, 96, 128])
        H = rng.choice([4, 8, 16])
        T = _log(rng, 1, 8192)
        B = max(1, min(_log(rng, 1, 8), (8 * 2048 * 16 * 64) // (T * H * d)))
        return dict(kind=kind, B=B, T=T, H=H, d=d, state=rng.random() < 0.6, grad=rng.random() < 0.6)
    if kind == "prism":
        d = rng.choice([32, 64, 128])
        T = _log(rng, 16, 4096)
        G = rng.choice([2, 8, 16])
        B = max(1, min(_log(rng, 1, 8), (8 * 2048 * 1024) // (T * G * d)))
        return dict(kind=kind, B=B, T=T, G=G, d=d, L=rng.choice([1, 2, 3]), W=rng.choice([4, 16, 64]), grad=rng.random() < 0.7)
    if kind == "attn":
        S = _log(rng, 64, 4096)
        hd = rng.choice([64, 128])
        H = rng.choice([8, 16, 32])
        B = max(1, min(_log(rng, 1, 8), (4096 * 4096) // (S * S)))
        return dict(kind=kind, B=B, S=S, H=H, Hkv=rng.choice([H, H // 4]), hd=hd, docs=rng.choice([0, 0, 3, 7]), grad=rng.random() < 0.7)
    if kind == "mlp":
        D = rng.choice([512, 1024, 2048])
        return dict(kind=kind, B=rng.choice([1, 2]), S=_log(rng, 16, 2048), D=D, F=rng.choice([2 * D, 4 * D]),
                    act=rng.choice(["swiglu", "gelu", "silu"]), norm=rng.choice(["layernorm", "rmsnorm"]), grad=rng.random() < 0.7)
    if kind == "head":
        return dict(kind=kind, rows=_log(rng, 64, 8192), D=rng.choice([512, 1024]), V=rng.choice([4096, 8000, 32000]))
    if kind == "mxfp8":
        return dict(kind=kind, M=_log(rng, 32, 4096), K=rng.choice([1024, 2048, 4096]), N=rng.choice([3072, 4096, 11008]))
    if kind == "gpt":
        H = rng.choice([8, 16])
        return dict(kind=kind, B=rng.choice([1, 2, 4]), prompt=_log(rng, 16, 512), steps=rng.choice([1, 4, 8]), layers=rng.choice([1, 2, 4]),
                    H=H, Hkv=rng.choice([H, H // 4]), hd=rng.choice([64, 128]), Fd=4096, V=rng.choice([4096, 32000]))
    return dict(kind=kind, B=rng.choice([1, 2]), prompt=_log(rng, 8, 64), steps=rng.choice([1, 2, 4]), layers=rng.choice([1, 2]), H=rng.choice([8, 16]),
                hd=64, Fd=4096, V=rng.choice([4096, 32000]), L=rng.choice([1, 2, 3]), W=rng.choice([4, 16]))


# ------------------------------------------------------------------------------------------------ inputs
class _Draw:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape, std=1.0, dtype=BF):
        return (torch.randn(*shape, generator=self.g, device="cuda") * std).to(dtype)

    def ints(self, hi, *shape):
        return torch.randint(0, hi, shape, generator=self.g, device="cuda")


def _inputs(c, seed):
    """The tensors of a case, from the seed alone (also what ``exact`` starts from)."""
    r = _Draw(seed)
    k = c["kind"]
    if k == "efla":
        B, T, H, d = c["B"], c["T"], c["H"], c["d"]
        t = dict(k=r.normal(B, T, H, d, std=0.4), v=r.normal(B, T, H, d), beta=torch.full((1,), 0.3, device="cuda"),
                 do=r.normal(B, T, H, d), ds=r.normal(B, H, d, d, std=0.1, dtype=torch.float32))
        t["s0"] = r.normal(B, H, d, d, std=0.3, dtype=torch.float32) if c["state"] else None
        return t
    if k == "prism":
        D = c["G"] * c["d"]
        return dict(x=r.normal(c["B"], c["T"], D), v=r.normal(c["B"], c["T"], D, std=0.7), dy=r.normal(c["B"], c["T"], D),
                    cw=r.normal(D, c["W"], std=c["W"] ** -0.5), cb=r.normal(D, std=0.1), wp=[r.normal(D, c["d"], std=0.03) for _ in range(c["L"])])
    if k == "attn":
        B, S, H, Hkv, hd = c["B"], c["S"], c["H"], c["Hkv"], c["hd"]
        t = dict(qkv=r.normal(S, B, H + 2 * Hkv, hd), do=r.normal(S, B, H * hd), doc=None)
        if c["docs"]:
            first = r.ints(2 ** 30, B, S) % max(1, S // c["docs"]) == 0        # documents begin at random tokens
            first[:, 0] = True
            pos = torch.arange(S, device="cuda").expand(B, S)
            t["doc"] = torch.where(first, pos, torch.zeros_like(pos)).cummax(1).values.to(torch.int32)
        return t
    if k == "mlp":
        B, S, D, Fd = c["B"], c["S"], c["D"], c["F"]
        return dict(x=r.normal(S, B, D), res=r.normal(S, B, D), nw=r.normal(D, std=0.1) + 1, nb=r.normal(D, std=0.1),
                    up=r.normal(D, Fd * (2 if c["act"] == "swiglu" else 1), std=D ** -0.5), down=r.normal(Fd, D, std=Fd ** -0.5),
                    dy=r.normal(S, B, D), dr=r.normal(S, B, D))
    if k == "head":
        return dict(n=r.normal(c["rows"], c["D"]), w=r.normal(c["V"], c["D"], std=0.05), t=r.ints(c["V"], c["rows"]))
    if k == "mxfp8":
        return dict(x=r.normal(c["M"], c["K"]), w=r.normal(c["N"], c["K"], std=c["K"] ** -0.5))
    return dict(ids=r.ints(c["V"], c["B"], c["prompt"] + c["steps"]))


def _config(c):
    from elfa_b200.config import Config
    cfg = Config()
    m = cfg.model
    m.dtype, m.efla.enabled = "bf16", c["kind"] in ("eflam", "prism")
    m.prism.enabled = m.efla.enabled
    if c["kind"] == "mlp":
        m.hidden_dim, m.intermediate_dim, m.activation, m.norm_type = c["D"], c["F"], c["act"], c["norm"]
    elif c["kind"] == "prism":
        m.hidden_dim, m.head_dim, m.prism.num_iterations, m.prism.shortconv_window = c["G"] * c["d"], c["d"], c["L"], c["W"]
    else:
        m.num_heads, m.num_kv_heads, m.head_dim, m.hidden_dim = c["H"], c.get("Hkv", c["H"]), c["hd"], c["H"] * c["hd"]
        m.num_layers, m.intermediate_dim, m.vocab_size, m.activation = c["layers"], c["Fd"], c["V"], "gelu"
        m.max_seq_len = cfg.data.seq_len = c["prompt"] + c["steps"]
        m.norm_type, m.tie_embeddings = ("rmsnorm" if c["kind"] == "eflam" else "layernorm"), True
        m.efla.chunk_size, m.efla.initial_beta = 16, 0.5
        if c["kind"] == "eflam":
            m.prism.num_iterations, m.prism.shortconv_window = c["L"], c["W"]
        cfg.bench.init_std, cfg.bench.learned_positions = 0.02, True
    return cfg


def _model(c, seed):
    from elfa_b200.models.efla_model import EflaModel
    from elfa_b200.models.gpt import GPTModel
    cfg = _config(c)
    cfg.runtime.seed = seed
    return (EflaModel if c["kind"] == "eflam" else GPTModel)(cfg, device=torch.device("cuda")).eval()


def _set(p, t):
    with torch.no_grad():
        p.copy_(t)


def prepare(case, seed):
    t = _inputs(case, seed)
    st = dict(case=case, t=t)
    k = case["kind"]
    dev = torch.device("cuda")
    if k in ("efla", "attn", "head", "prism", "mlp"):
        grad = case.get("grad", True)
        for n in {"efla": ("k", "v", "beta", "s0"), "attn": ("qkv",), "head": ("n", "w"), "prism": ("x", "v"), "mlp": ("x", "res")}[k]:
            if t[n] is not None:
                t[n].requires_grad_(grad)
    if k == "prism":
        from elfa_b200.models.efla_model import PrismLayer
        p = PrismLayer(_config(case), BF, dev)
        _set(p.conv_weight, t["cw"])
        _set(p.conv_bias, t["cb"])
        for w, x in zip(p.w_p, t["wp"]):
            _set(w, x)
        st["mod"] = p
    if k == "mlp":
        from elfa_b200.models.gpt import MLP, Norm
        from elfa_b200.parallel.mesh import ParallelContext
        cfg = _config(case)
        st["norm"], st["mod"] = Norm(case["D"], case["norm"], BF, dev), MLP(cfg, ParallelContext(), BF, dev)
        _set(st["norm"].weight, t["nw"])
        if st["norm"].bias is not None:
            _set(st["norm"].bias, t["nb"])
        _set(st["mod"].up, t["up"])
        _set(st["mod"].down, t["down"])
    if k == "mxfp8":
        from elfa_b200.ops import gemm_mxfp8 as q8
        st["wq"], _ = q8.quantize_mxfp8(t["w"], right=True)
    if k in ("gpt", "eflam"):
        st["mod"] = _model(case, seed)
    return st


# ------------------------------------------------------------------------------------------------ one pass
def run(st):
    c, t = st["case"], st["t"]
    k = c["kind"]
    with torch.set_grad_enabled(bool(c.get("grad", k == "head"))):
        if k == "efla":
            from elfa_b200.ops.efla import efla_scan
            o, s = efla_scan(t["k"], t["v"], t["beta"], t["s0"])
            if not c["grad"]:
                return [o, s]
            ins = [t["k"], t["v"], t["beta"]] + ([t["s0"]] if c["state"] else [])
            return [o, s, *torch.autograd.grad([o, s], ins, [t["do"], t["ds"]])]
        if k == "prism":
            p = st["mod"]
            y, _, _ = p(t["x"], t["v"])
            if not c["grad"]:
                return [y]
            return [y, *torch.autograd.grad(y, [t["x"], t["v"], p.conv_weight, p.conv_bias, *p.w_p], t["dy"])]
        if k == "attn":
            from elfa_b200 import ops
            S, B, hd = c["S"], c["B"], c["hd"]
            qkv = t["qkv"].view(S, B, 3, c["H"], hd) if c["H"] == c["Hkv"] else t["qkv"]
            o = ops.attention(qkv, causal=True, seq_first=True, num_heads=c["H"], doc_start=t["doc"])
            if not c["grad"]:
                return [o]
            return [o, *torch.autograd.grad(o, [t["qkv"]], t["do"])]
        if k == "mlp":
            n, r = st["norm"](t["x"], t["res"])
            y = st["mod"](n)
            if not c["grad"]:
                return [y, r]
            ps = [st["norm"].weight] + ([st["norm"].bias] if st["norm"].bias is not None else []) + [st["mod"].up, st["mod"].down]
            return [y, r, *torch.autograd.grad([y, r], [t["x"], t["res"], *ps], [t["dy"], t["dr"]])]
        if k == "head":
            from elfa_b200 import ops
            loss = ops.cross_entropy(ops.linear_nt(t["n"], t["w"]), t["t"])
            return [loss.detach(), *torch.autograd.grad(loss, [t["n"], t["w"]])]
        if k == "mxfp8":
            from elfa_b200.ops import gemm_mxfp8 as q8
            xq, _ = q8.quantize_mxfp8(t["x"])
            return [q8.gemm_mxfp8(xq, st["wq"], gelu=True)]
        n0 = c["prompt"]
        logits, states = st["mod"].forward_with_states(t["ids"][:, :n0])
        out = [logits]
        for i in range(c["steps"]):
            logits, states = st["mod"].forward_with_states(t["ids"][:, n0 + i:n0 + i + 1], states)
            out.append(logits)
        if k == "eflam":
            out += [s[n] for s in states for n in ("efla", "prism")]
        else:
            out += [s[n] for s in states["layers"] for n in ("k", "v")]
        return out


# ------------------------------------------------------------------------------------------------ floors
def work(case):
    c = case
    k = c["kind"]
    bw = 3 if c.get("grad", True) else 1
    if k == "efla":
        n = c["B"] * c["T"] * c["H"] * c["d"]
        s = c["B"] * c["H"] * c["d"] ** 2 * 4
        by = n * 2 * 3 + s * (2 if c["state"] else 1)
        if c["grad"]:
            by += n * 2 * 3 + s * (2 if c["state"] else 1)               # do in, dk and dv out, ds in, ds0 out
        return dict(bytes=by, flops=4 * n * c["d"] * bw)
    if k == "prism":
        rows, D = c["B"] * c["T"], c["G"] * c["d"]
        return dict(bytes=rows * D * 2 * (7 if c["grad"] else 3), flops=bw * 2 * rows * D * (c["W"] + c["L"] * c["d"]))
    if k == "attn":
        n = c["B"] * c["S"] * c["hd"] * 2
        pairs = c["B"] * c["H"] * c["S"] * (c["S"] + 1) / 2 / (c["docs"] or 1)
        by = n * (2 * c["H"] + 2 * c["Hkv"])
        if c["grad"]:
            by += n * (2 * c["H"] + 2 * c["Hkv"])
        return dict(bytes=by, flops=pairs * c["hd"] * (14 if c["grad"] else 4))
    if k == "mlp":
        rows, up = c["B"] * c["S"], c["F"] * (2 if c["act"] == "swiglu" else 1)
        w = (c["D"] * up + c["F"] * c["D"]) * 2
        return dict(bytes=rows * c["D"] * 2 * (8 if c["grad"] else 4) + w * (2 if c["grad"] else 1), flops=bw * 2 * rows * c["D"] * (up + c["F"]))
    if k == "head":
        return dict(bytes=2 * (2 * c["rows"] * c["D"] + 2 * c["V"] * c["D"]) + 8 * c["rows"], flops=6 * c["rows"] * c["D"] * c["V"])
    if k == "mxfp8":
        return dict(bytes=c["M"] * c["K"] * 2 + c["N"] * c["K"] + c["M"] * c["N"] * 2, flops=2 * c["M"] * c["N"] * c["K"])
    D, T = c["H"] * c["hd"], c["prompt"] + c["steps"]
    if k == "gpt":
        per = D * (D + 2 * c["Hkv"] * c["hd"]) + D * D + 2 * D * c["Fd"]
    else:
        per = 3 * D * D + 2 * D * c["Fd"] + 3 * c["L"] * D * c["hd"]
    par = c["layers"] * per + c["V"] * D
    return dict(bytes=2 * par * (1 + c["steps"]) + 2 * c["B"] * T * c["V"], flops=2 * par * c["B"] * T)


def tolerance(case):
    return {"efla": {"rel": 1e-2}, "prism": {"rel": 1e-2}, "attn": {"rel": 1e-2}, "mlp": {"rel": 1.2e-2}, "head": {"rel": 1e-2},
            "mxfp8": {"rel": 1e-2}, "gpt": {"rel": 2e-2}, "eflam": {"rel": 2e-2}}[case["kind"]]


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _gelu(x):
    return F.gelu(x, approximate="tanh")


def _scan(k, v, beta, s0, C=64):
    """The delta-rule recurrence, 64 tokens at a time (a unit-lower-triangular solve inside, the state between)."""
    B, T, H, d = k.shape
    pad = (-T) % C
    k, v = (F.pad(x, (0, 0, 0, 0, 0, pad)).view(B, -1, C, H, d).permute(1, 0, 3, 2, 4) for x in (k, v))
    lam = (k * k).sum(-1)
    small = lam < 1e-6
    one = torch.where(small, torch.ones_like(lam), lam)
    cf = torch.where(small, beta - beta * beta * lam / 2 + beta ** 3 * lam * lam / 6, (1 - torch.exp(-beta * one)) / one)
    s = torch.zeros(B, H, d, d, dtype=k.dtype, device=k.device) if s0 is None else s0
    outs = []
    for kn, vn, cn in zip(k, v, cf):
        g = kn @ kn.transpose(-1, -2)
        a = torch.eye(C, dtype=k.dtype, device=k.device) + cn.unsqueeze(-1) * torch.tril(g, -1)
        u = torch.linalg.solve_triangular(a, cn.unsqueeze(-1) * (vn - kn @ s), upper=False, unitriangular=True)
        outs.append(kn @ s + torch.tril(g) @ u)
        s = s + kn.transpose(-1, -2) @ u
    return torch.stack(outs, 1).permute(0, 1, 3, 2, 4).reshape(B, T + pad, H, d)[:, :T], s


def _conv(x, w, b):
    W = w.shape[1]
    return F.conv1d(F.pad(x.transpose(1, 2), (W - 1, 0)), w.flip(1).unsqueeze(1), b, groups=x.shape[2]).transpose(1, 2)


def _refine(u, v, ps, d):
    r, deltas = (v - u).unflatten(-1, (-1, d)), []
    for p in ps:
        deltas.append(_gelu(p.unsqueeze(-2) * r))
        r = r - deltas[-1]
    return u + sum(deltas).flatten(-2), deltas


def _norm(x, w, b=None):
    if b is None:
        return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6) * w
    return F.layer_norm(x, x.shape[-1:], w, b, 1e-5)


def _softmax_attention(q, k, v, before=None):
    """``q, k, v [S, hd]`` of one head, causal; keys before ``before[i]`` are hidden from query ``i``."""
    S = q.shape[0]
    i = torch.arange(S, device=q.device)
    hide = i[None, :] > i[:, None]
    if before is not None:
        hide = hide | (i[None, :] < before[:, None])
    return torch.softmax((q @ k.t() / math.sqrt(q.shape[1])).masked_fill(hide, -math.inf), -1) @ v


def _leaf(t, grad):
    return None if t is None else t.detach().double().requires_grad_(grad)


def _exact_attn(c, t):
    S, B, H, Hkv, hd = c["S"], c["B"], c["H"], c["Hkv"], c["hd"]
    x, do = t["qkv"].detach().double(), t["do"].double().view(S, B, H, hd)
    out, dx = torch.empty(S, B, H, hd, dtype=x.dtype, device=x.device), torch.zeros_like(x)
    for b in range(B):
        for h in range(H):
            at = (h, H + h // (H // Hkv), H + Hkv + h // (H // Hkv))
            q = [_leaf(x[:, b, a], c["grad"]) for a in at]
            o = _softmax_attention(*q, None if t["doc"] is None else t["doc"][b])
            out[:, b, h] = o.detach()
            if c["grad"]:
                for a, g in zip(at, torch.autograd.grad(o, q, do[:, b, h])):
                    dx[:, b, a] += g
    return [out.view(S, B, H * hd)] + ([dx] if c["grad"] else [])


def _mx(x):
    """Values that the MXFP8 format (blocks of 32, power-of-two scale, e4m3) stands for."""
    b = x.float().unflatten(-1, (-1, 32))
    top = b.abs().amax(-1, keepdim=True)
    s = torch.exp2((torch.floor(torch.log2(top.clamp_min(2.0 ** -126))) - 8).clamp(-127, 127).double())
    q = (b.double() / s).clamp(-448, 448).float().to(torch.float8_e4m3fn).double()
    return torch.where(top > 0, q * s, torch.zeros_like(q)).flatten(-2)


def _exact_gpt(c, m, ids):
    f = lambda p: p.detach().double()
    B, T = ids.shape
    H, Hkv, hd = c["H"], c["Hkv"], c["hd"]
    x = f(m.embed_tokens)[ids] + f(m.pos_embed)[:T]
    kv = []
    for blk in m.blocks:
        qkv = (_norm(x, f(blk.ln1.weight), f(blk.ln1.bias)) @ f(blk.attn.w_qkv)).view(B, T, H + 2 * Hkv, hd)
        q, k, v = qkv[:, :, :H], qkv[:, :, H:H + Hkv], qkv[:, :, H + Hkv:]
        kv += [k.transpose(0, 1), v.transpose(0, 1)]
        o = torch.stack([torch.stack([_softmax_attention(q[b, :, h], k[b, :, h // (H // Hkv)], v[b, :, h // (H // Hkv)]) for h in range(H)], 1)
                         for b in range(B)])
        x = x + o.flatten(-2) @ f(blk.attn.w_o)
        x = x + _gelu(_norm(x, f(blk.ln2.weight), f(blk.ln2.bias)) @ f(blk.mlp.up)) @ f(blk.mlp.down)
    return _norm(x, f(m.final_norm.weight), f(m.final_norm.bias)) @ f(m.embed_tokens).t(), kv


def _exact_efla_model(c, m, ids):
    f = lambda p: p.detach().double()
    B, T = ids.shape
    H, d = c["H"], c["hd"]
    x = f(m.embed_tokens)[ids]
    states = []
    for blk in m.blocks:
        n = _norm(x, f(blk.ln1.weight))
        e, p = blk.efla, blk.prism
        o, s = _scan((n @ f(e.w_k)).view(B, T, H, d), (n @ f(e.w_v)).view(B, T, H, d), f(e.beta_param), None)
        v = o.flatten(-2) @ f(e.w_o)
        u = _conv(n, f(p.conv_weight), f(p.conv_bias))
        y, deltas = _refine(u, v, [torch.sigmoid(u @ f(w)) for w in p.w_p], d)
        betas = [torch.sigmoid((u @ f(w)).mean(-1)) for w in p.w_beta]
        ks = [F.normalize(u @ f(w), dim=-1) for w in p.w_k]
        S = torch.zeros(B, H, d, d, dtype=x.dtype, device=x.device)
        for i in range(T):
            for l in range(c["L"]):
                kk, bb = ks[l][:, i], betas[l][:, i].view(B, 1, 1, 1)
                if l == 0:
                    S = p.forget * (S - bb * torch.einsum("bgij,bj->bgi", S, kk).unsqueeze(-1) * kk[:, None, None, :])
                S = S + bb * deltas[l][:, i].unsqueeze(-1) * kk[:, None, None, :]
        states += [s, S]
        r = x + y
        x = r + _gelu(_norm(r, f(blk.ln2.weight)) @ f(blk.mlp_up)) @ f(blk.mlp_down)
    return _norm(x, f(m.final_norm.weight)) @ f(m.embed_tokens).t(), states


def exact(case, seed):
    c, t, k = case, _inputs(case, seed), case["kind"]
    grad = c.get("grad", k == "head")
    if k == "attn":
        return _exact_attn(c, t)
    if k == "mxfp8":
        return [_gelu(_mx(t["x"]) @ _mx(t["w"]).t())]
    if k in ("gpt", "eflam"):
        with torch.no_grad():
            logits, rest = (_exact_gpt if k == "gpt" else _exact_efla_model)(c, _model(c, seed), t["ids"])
        n0 = c["prompt"]
        return [logits[:, :n0]] + [logits[:, n0 + i:n0 + i + 1] for i in range(c["steps"])] + rest
    with torch.set_grad_enabled(grad):
        if k == "efla":
            ins = [_leaf(t[n], grad) for n in ("k", "v", "beta", "s0")]
            outs, gout = list(_scan(*ins)), [t["do"].double(), t["ds"].double()]
        elif k == "prism":
            ins = [_leaf(x, grad) for x in (t["x"], t["v"], t["cw"], t["cb"], *t["wp"])]
            u = _conv(ins[0], ins[2], ins[3])
            outs, gout = [_refine(u, ins[1], [torch.sigmoid(u @ w) for w in ins[4:]], c["d"])[0]], [t["dy"].double()]
        elif k == "mlp":
            ins = [_leaf(t[n], grad) for n in (("x", "res", "nw") + (("nb",) if c["norm"] == "layernorm" else ()) + ("up", "down"))]
            r = ins[0] + ins[1]
            h = _norm(r, ins[2], ins[3] if c["norm"] == "layernorm" else None) @ ins[-2]
            if c["act"] == "swiglu":
                g, h = h.chunk(2, -1)
                h = F.silu(g) * h
            else:
                h = _gelu(h) if c["act"] == "gelu" else F.silu(h)
            outs, gout = [h @ ins[-1], r], [t["dy"].double(), t["dr"].double()]
        else:
            ins = [_leaf(t[n], True) for n in ("n", "w")]
            outs, gout = [F.cross_entropy(ins[0] @ ins[1].t(), t["t"])], [None]
        ins = [x for x in ins if x is not None]
        return [o.detach() for o in outs] + (list(torch.autograd.grad(outs, ins, gout)) if grad else [])
