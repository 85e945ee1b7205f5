"""The work that users of this package have it do, as timed cases.

Training is most of that work, so most cases are the parts of a training step, forward and backward: decoder blocks
from the smallest model of the smoke test to the width of the 8B configuration, attention by itself (documents, long
context, sliding windows), the fused residual add + RMSNorm, the lm_head with its loss, routed experts, and one whole
optimizer step.  Two cases are whole inference calls: a prefill and one decode step.

Weights are laid out as the parameter store lays them out: bf16 matrices, each with an fp32 ``main_grad`` that the
backward kernels add into and that is cleared before each step; norm scales are fp32.
"""

import math

import torch

from research_b200.config import run_spec_from_mapping
from research_b200.config.specs import ModelSpec
from research_b200.infer import generation
from research_b200.models.build import build_model
from research_b200.models.execution import ExecutionContext
from research_b200.models.transformer import DecoderBlock, ForwardInputs
from research_b200.ops import functional as Fn
from research_b200.ops.grouped import RoutingPlan, routed_expert_ffn
from research_b200.runtime.trainer import Trainer

EPS = 1e-6
THETA = 10000.0


def listed():
    return [
        # the two-layer model of the smoke test: small kernels, launches and host work count
        dict(name="block_small", kind="block", B=2, S=512, H=512, hq=4, hkv=2, F=1024, docs=True),
        # one layer of the 1.3B configuration on two of its 4096-token rows with document masks
        dict(name="block_1p3b", kind="block", B=2, S=4096, H=2048, hq=16, hkv=8, F=5632, docs=True),
        # one layer of the 8B configuration on a sequence of no round length
        dict(name="block_8b_ragged", kind="block", B=1, S=2999, H=4096, hq=32, hkv=8, F=14336, docs=False),
        # attention of the 1.3B configuration at its micro-batch, packed documents
        dict(name="attn_docs", kind="attn", B=8, S=4096, hq=16, hkv=8, D=128, window=0, docs=True),
        # long-context training: one long causal sequence
        dict(name="attn_long", kind="attn", B=1, S=16384, hq=16, hkv=8, D=128, window=0, docs=False),
        # local layers of the Trinity recipe: head dimension 64, a sliding window, an odd length
        dict(name="attn_window", kind="attn", B=3, S=1111, hq=12, hkv=4, D=64, window=256, docs=True),
        # residual add + RMSNorm of the 1.3B configuration at its micro-batch
        dict(name="add_norm", kind="norm", rows=32768, H=2048),
        # lm_head and cross-entropy with z-loss of the 1.3B configuration
        dict(name="lm_head_loss", kind="head", T=8192, H=2048, V=50304),
        # routed experts of the MoE 7B configuration, one rank's tokens
        dict(name="experts", kind="moe", T=8192, H=2048, I=1024, E=64, k=8),
        # one optimizer step (Muon on the matrices, AdamW on the rest) over four layers of the 1.3B configuration
        dict(name="muon_step", kind="optim", layers=4, H=2048, hq=16, hkv=8, F=5632, V=8192),
        # a prompt of no round length into an empty cache, four layers of the 1.3B configuration
        dict(name="prefill", kind="prefill", layers=4, B=1, P=777, H=2048, hq=16, hkv=8, F=5632, V=50304),
        # one decode step of a serving batch behind 2k-token prompts, four layers of the 1.3B configuration
        dict(name="decode", kind="decode", layers=4, B=32, P=2100, H=2048, hq=16, hkv=8, F=5632, V=50304),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


_WIDTHS = ((512, 4, 2, 1024), (1024, 8, 8, 2816), (2048, 16, 8, 5632), (3072, 24, 8, 8192), (4096, 32, 8, 14336))


def draw(rng):
    kind = rng.choice(("block", "block", "block", "attn", "attn", "attn", "norm", "head", "moe", "optim", "prefill",
                       "prefill", "decode", "decode"))
    if kind == "block":
        H, hq, hkv, F = rng.choice(_WIDTHS)
        S = _log_int(rng, 128, 2048)
        most = max(1, min(8, int(8192 * 2048 / (S * H))))
        return dict(kind=kind, B=rng.randint(1, most), S=S, H=H, hq=hq, hkv=hkv, F=F, docs=rng.random() < 0.6)
    if kind == "attn":
        D = rng.choice((64, 128, 128))
        hkv = rng.choice((2, 4, 8))
        hq = hkv * rng.choice((1, 2, 4))
        S = _log_int(rng, 128, 8192)
        most = max(1, min(8, int(8 * 4096 * 4096 * 16 / (S * S * hq))))
        window = 0 if rng.random() < 0.6 else _log_int(rng, 64, 2048)
        return dict(kind=kind, B=rng.randint(1, most), S=S, hq=hq, hkv=hkv, D=D, window=min(window, S),
                    docs=rng.random() < 0.6)
    if kind == "norm":
        H = rng.choice((512, 768, 1024, 1536, 2048, 3072, 4096))
        return dict(kind=kind, rows=_log_int(rng, 256, 32768 * 2048 // H), H=H)
    if kind == "head":
        return dict(kind=kind, T=_log_int(rng, 256, 8192), H=rng.choice((512, 1024, 2048)),
                    V=rng.choice((4096, 32000, 50304)))
    if kind == "moe":
        E = rng.choice((8, 16, 32, 64))
        return dict(kind=kind, T=_log_int(rng, 256, 8192), H=rng.choice((1024, 2048)), I=rng.choice((512, 1024)), E=E,
                    k=rng.choice((2, 4, 8)))
    if kind == "optim":
        H, hq, hkv, F = rng.choice(_WIDTHS[:3])
        return dict(kind=kind, layers=rng.randint(1, 4), H=H, hq=hq, hkv=hkv, F=F, V=rng.choice((4096, 8192)))
    H, hq, hkv, F = rng.choice(_WIDTHS)
    layers = rng.randint(2, 4)
    if kind == "prefill":
        P = _log_int(rng, 64, 4000)
        return dict(kind=kind, layers=layers, B=rng.randint(1, max(1, min(4, 4000 // P))), P=P, H=H, hq=hq, hkv=hkv,
                    F=F, V=rng.choice((4096, 32000, 50304)))
    return dict(kind=kind, layers=layers, B=_log_int(rng, 1, 64), P=_log_int(rng, 32, 3500), H=H, hq=hq, hkv=hkv, F=F,
                V=rng.choice((4096, 32000, 50304)))


# ---- inputs: plain tensors from the seed, shared by prepare() and exact() ---------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape, scale=1.0, dtype=torch.bfloat16):
    return torch.randn(shape, generator=g, device="cuda").mul_(scale).to(dtype)


def _scales(g, n):
    return 1.0 + 0.1 * torch.randn(n, generator=g, device="cuda")


def _doc_starts(g, B, S, docs, window):
    """First visible position of every row: documents of geometric length and / or a sliding window; None if neither."""
    at = torch.arange(S, device="cuda", dtype=torch.int32).expand(B, S)
    lo = None
    if docs:
        cut = torch.rand(B, S, generator=g, device="cuda") < 3.0 / S
        cut[:, 0] = True
        lo = torch.cummax(torch.where(cut, at, torch.zeros_like(at)), dim=1).values
    if window:
        near = (at - (window - 1)).clamp_min(0)
        lo = near if lo is None else torch.maximum(lo, near)
    return None if lo is None else lo.to(torch.int32).contiguous()


def _layer_weights(g, c):
    H, F, D = c["H"], c["F"], c["H"] // c["hq"]
    return {
        "pre_norm.scale": _scales(g, H),
        "attn.wqkv": _randn(g, (c["hq"] + 2 * c["hkv"]) * D, H, scale=0.02),
        "attn.wo": _randn(g, H, c["hq"] * D, scale=0.02),
        "attn.q_norm": _scales(g, D),
        "attn.k_norm": _scales(g, D),
        "post_norm.scale": _scales(g, H),
        "mlp.w_gate_up": _randn(g, 2 * F, H, scale=0.02),
        "mlp.w_down": _randn(g, H, F, scale=0.02),
    }


def _model_weights(g, c):
    w = {"embed": _randn(g, c["V"], c["H"], scale=0.02), "norm.scale": _scales(g, c["H"]),
         "lm_head": _randn(g, c["V"], c["H"], scale=0.02)}
    for i in range(c["layers"]):
        w.update({f"layers.{i}.{k}": v for k, v in _layer_weights(g, c).items()})
    return w


def _draw_inputs(c, seed):
    g, kind = _gen(seed), c["kind"]
    if kind == "block":
        shape = (c["B"], c["S"], c["H"])
        t = {"w": _layer_weights(g, c), "x": _randn(g, *shape), "delta": _randn(g, *shape, scale=0.5)}
        t["lo"] = _doc_starts(g, c["B"], c["S"], c["docs"], 0)
        t["gx"], t["gm"] = _randn(g, *shape, scale=0.01), _randn(g, *shape, scale=0.01)
        return t
    if kind == "attn":
        T = c["B"] * c["S"]
        t = {"qkv": _randn(g, T, (c["hq"] + 2 * c["hkv"]) * c["D"]), "wq": _scales(g, c["D"]), "wk": _scales(g, c["D"])}
        t["lo"] = _doc_starts(g, c["B"], c["S"], c["docs"], c["window"])
        t["go"] = _randn(g, c["B"], c["S"], c["hq"] * c["D"], scale=0.01)
        return t
    if kind == "norm":
        shape = (c["rows"], c["H"])
        return {"x": _randn(g, *shape), "delta": _randn(g, *shape, scale=0.5), "w": _scales(g, c["H"]),
                "gy": _randn(g, *shape, scale=0.01), "gr": _randn(g, *shape, scale=0.01)}
    if kind == "head":
        return {"x": _randn(g, c["T"], c["H"]), "w": _randn(g, c["V"], c["H"], scale=0.02),
                "targets": torch.randint(0, c["V"], (c["T"],), generator=g, device="cuda", dtype=torch.int32),
                "mask": torch.rand(c["T"], generator=g, device="cuda") < 0.97}
    if kind == "moe":
        T, E, k = c["T"], c["E"], c["k"]
        popular = 0.5 * torch.randn(E, generator=g, device="cuda")          # a mildly uneven load
        scores = torch.randn(T, E, generator=g, device="cuda") + popular
        top = torch.topk(scores, min(k, E), dim=1)
        return {"x": _randn(g, T, c["H"]), "ids": top.indices, "p": torch.softmax(top.values, dim=1),
                "wgu": _randn(g, E, 2 * c["I"], c["H"], scale=0.02), "wd": _randn(g, E, c["H"], c["I"], scale=0.02),
                "gy": _randn(g, T, c["H"], scale=0.01)}
    if kind == "optim":
        w = {k: v.float() for k, v in _model_weights(g, c).items()}
        return {"w": w, "g": {k: _randn(g, *v.shape, scale=1e-3, dtype=torch.float32) for k, v in w.items()}}
    t = {"w": _model_weights(g, c)}
    n = c["P"] if kind == "prefill" else 1
    t["ids"] = torch.randint(0, c["V"], (c["B"], n), generator=g, device="cuda", dtype=torch.int32)
    if kind == "decode":                                                     # what a prefill left in the cache
        D = c["H"] // c["hq"]
        shape = (c["layers"], c["B"], c["P"], c["hkv"], D)
        t["k"], t["v"] = _randn(g, *shape), _randn(g, *shape)
    return t


# ---- states -------------------------------------------------------------------------------------------------------
def _install(module, weights, train):
    """Puts ``weights`` into a module's parameters; for training each gets its slice of one fp32 gradient arena."""
    params = dict(module.named_parameters())
    for name, p in params.items():
        p.data = weights[name]
    if not train:
        return None
    arena = torch.zeros(sum(p.numel() for p in params.values()), device="cuda")
    at = 0
    for p in params.values():
        p.main_grad = arena[at:at + p.numel()].view(p.shape)
        at += p.numel()
    return arena


def _param(t):
    p = torch.nn.Parameter(t)
    p.main_grad = torch.zeros(t.shape, dtype=torch.float32, device="cuda")
    return p


def _spec(c, layers):
    return ModelSpec(name="decoder", variant="case", vocab_size=c.get("V", 64), hidden_size=c["H"],
                     intermediate_size=c["F"], num_layers=layers, num_heads=c["hq"], n_kv_heads=c["hkv"],
                     max_seq_len=max(4096, c.get("S", 0)), rope_theta=THETA, norm_epsilon=EPS, attention_doc_mask=True)


def _positions(B, S):
    return torch.arange(S, device="cuda", dtype=torch.int32).repeat(B)


def prepare(case, seed):
    c, t, kind = case, _draw_inputs(case, seed), case["kind"]
    s = {"case": dict(c), "t": t}
    # a training program's backward thread is up and has the device's context
    torch.ones(1, device="cuda", requires_grad=True).sum().backward()
    if kind == "block":
        with torch.device("cuda"):
            s["block"] = DecoderBlock(_spec(c, 1), ExecutionContext())
        s["grads"] = _install(s["block"], t.pop("w"), train=True)
        s["ex"] = ExecutionContext()
        s["positions"] = _positions(c["B"], c["S"])
        t["x"].requires_grad_(True)
        t["delta"].requires_grad_(True)
    elif kind == "attn":
        s["wq"], s["wk"] = _param(t["wq"]), _param(t["wk"])
        s["positions"] = _positions(c["B"], c["S"])
        t["qkv"].requires_grad_(True)
    elif kind == "norm":
        s["w"] = _param(t["w"])
        t["x"].requires_grad_(True)
        t["delta"].requires_grad_(True)
    elif kind == "head":
        s["w"] = _param(t["w"])
        t["x"].requires_grad_(True)
    elif kind == "moe":
        s["wgu"], s["wd"] = _param(t["wgu"]), _param(t["wd"])
        t["x"].requires_grad_(True)
        t["p"].requires_grad_(True)
    elif kind == "optim":
        raw = {
            "run": {"id": "case"},
            "model": {"name": "decoder", "variant": "case", "vocab_size": c["V"], "hidden_size": c["H"],
                      "intermediate_size": c["F"], "num_layers": c["layers"], "num_heads": c["hq"],
                      "n_kv_heads": c["hkv"], "max_seq_len": 512, "rope_theta": THETA, "init": "normal_0.02"},
            "optimizer": {"name": "muon", "grad_clip_norm": 1.0, "weight_decay": 0.1,
                          "schedule": {"name": "constant", "peak_lr": 1e-2}},
            "data": {"train_manifest": "unused.json"},
            "training": {"seq_len": 512, "global_batch_size": 2, "target_tokens": 2 * 512 * 4, "precision": "bf16"},
        }
        s["trainer"] = tr = Trainer(run_spec_from_mapping(raw), build_data=False)
        for e in tr.store.entries:
            w, g = t["w"][e.name], t["g"][e.name]
            tr.store.master_view(tr.store.section_of(e), e).copy_(w)
            e.param.data.copy_(w)
            e.param.main_grad.copy_(g)
        del s["t"]
    else:
        s["model"] = m = build_model(_spec(c, c["layers"]), device="cuda", initialize=False).model
        _install(m, t.pop("w"), train=False)
        m.compute_dtype = torch.bfloat16
        m.eval()
        s["cache"] = cache = generation.init_kv_cache(m, c["B"], c["P"] + 64)
        if kind == "decode":
            with torch.no_grad():
                for i in range(c["layers"]):
                    pages = cache.k[i].view(c["B"], cache.pages_per_seq, c["hkv"], cache.page_size, -1)
                    at = torch.arange(c["P"], device="cuda")
                    pages[:, at // cache.page_size, :, at % cache.page_size] = t["k"][i].transpose(0, 1)
                    pages = cache.v[i].view(c["B"], cache.pages_per_seq, c["hkv"], cache.page_size, -1)
                    pages[:, at // cache.page_size, :, at % cache.page_size] = t["v"][i].transpose(0, 1)
            del t["k"], t["v"]
            s["token"] = t["ids"][:, 0].long()
            s["step"] = generation.GraphedDecodeStep(m, cache, s["token"], c["P"])
    return s


# ---- one pass -----------------------------------------------------------------------------------------------------
def run(state):
    c = state["case"]
    return _RUN[c["kind"]](state, c, state.get("t"))


def _run_block(s, c, t):
    s["grads"].zero_()
    inp = ForwardInputs(positions=s["positions"], B=c["B"], S=c["S"], lo_causal=t["lo"])
    x, m, _, _ = s["block"](t["x"], t["delta"], inp, s["ex"])
    dx, ddelta = torch.autograd.grad([x, m], [t["x"], t["delta"]], [t["gx"], t["gm"]])
    out = {"x": x.detach(), "m": m.detach(), "dx": dx, "ddelta": ddelta}
    out.update({"d_" + k: p.main_grad for k, p in s["block"].named_parameters()})
    return out


def _run_attn(s, c, t):
    s["wq"].main_grad.zero_()
    s["wk"].main_grad.zero_()
    o = Fn.attention_block(t["qkv"], s["wq"], s["wk"], s["positions"], B=c["B"], S=c["S"], hq=c["hq"], hkv=c["hkv"],
                           D=c["D"], eps=EPS, theta=THETA, rope=True, lo=t["lo"])
    (dqkv,) = torch.autograd.grad([o], [t["qkv"]], [t["go"]])
    return {"o": o.detach(), "dqkv": dqkv, "dwq": s["wq"].main_grad, "dwk": s["wk"].main_grad}


def _run_norm(s, c, t):
    s["w"].main_grad.zero_()
    y, res = Fn.add_rmsnorm(t["x"], t["delta"], s["w"], EPS)
    dx, ddelta = torch.autograd.grad([y, res], [t["x"], t["delta"]], [t["gy"], t["gr"]])
    return {"y": y.detach(), "res": res.detach(), "dx": dx, "ddelta": ddelta, "dw": s["w"].main_grad}


_Z = 1e-4


def _run_head(s, c, t):
    s["w"].main_grad.zero_()
    scale = 1.0 / c["T"]
    ce, z = Fn.lm_head_cross_entropy(t["x"], s["w"], t["targets"], t["mask"], grad_scale=scale, z_weight=_Z)
    objective = Fn.objective_from_sums(ce, z, grad_scale=scale, z_weight=_Z, native_path=Fn.use_native(t["x"]))
    (dx,) = torch.autograd.grad([objective], [t["x"]])
    return {"ce": ce.detach(), "z": z.detach(), "dx": dx, "dw": s["w"].main_grad}


def _run_moe(s, c, t):
    s["wgu"].main_grad.zero_()
    s["wd"].main_grad.zero_()
    plan = RoutingPlan(t["ids"], c["E"])
    y = routed_expert_ffn(t["x"], t["p"], plan, s["wgu"], s["wd"])
    dx, dp = torch.autograd.grad([y], [t["x"], t["p"]], [t["gy"]])
    return {"y": y.detach(), "dx": dx, "dp": dp, "dwgu": s["wgu"].main_grad, "dwd": s["wd"].main_grad}


def _run_optim(s, c, t):
    tr = s["trainer"]
    step = tr.optimizer.step()
    out = {e.name: tr.store.master_view(tr.store.section_of(e), e) for e in tr.store.entries}
    out["grad_norm"] = step["grad_norm"]
    return out


def _run_prefill(s, c, t):
    logits = generation.prefill(s["model"], t["ids"], s["cache"])
    return {"logits": logits, "k": s["cache"].k, "v": s["cache"].v}


def _run_decode(s, c, t):
    logits = s["step"](s["token"], c["P"])
    cache = s["cache"]
    page, row = c["P"] // cache.page_size, c["P"] % cache.page_size
    shape = (c["layers"], c["B"], cache.pages_per_seq, c["hkv"], cache.page_size, -1)
    return {"logits": logits, "k": cache.k.view(shape)[:, :, page, :, row], "v": cache.v.view(shape)[:, :, page, :, row]}


_RUN = {"block": _run_block, "attn": _run_attn, "norm": _run_norm, "head": _run_head, "moe": _run_moe,
        "optim": _run_optim, "prefill": _run_prefill, "decode": _run_decode}


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def _pairs(S, window, docs):
    """(query, key) pairs of one head on average: causal, in a window, and three documents of geometric length."""
    full = S * (S + 1) / 2
    if docs:                    # expected pairs of cuts at rate 3 / S
        n = S / 3.0
        full = n * S - n * n * (1 - math.exp(-S / n))
    if window and window < S:
        full = min(full, window * S - window * (window - 1) / 2)
    return full


def _layer_numel(c):
    D = c["H"] // c["hq"]
    return (c["hq"] + 2 * c["hkv"]) * D * c["H"] + c["H"] * c["H"] + 3 * c["F"] * c["H"]


def work(case):
    c, kind = case, case["kind"]
    if kind == "block":
        T, n = c["B"] * c["S"], _layer_numel(c)
        pairs = c["B"] * c["hq"] * _pairs(c["S"], 0, c["docs"])
        D = c["H"] // c["hq"]
        return {"bytes": 8 * T * c["H"] * 2 + n * (2 + 4), "flops": 6.0 * T * n + 14.0 * pairs * D}
    if kind == "attn":
        T = c["B"] * c["S"]
        pairs = c["B"] * c["hq"] * _pairs(c["S"], c["window"], c["docs"])
        return {"bytes": T * c["D"] * 2 * (2 * (c["hq"] + 2 * c["hkv"]) + 2 * c["hq"]), "flops": 14.0 * pairs * c["D"]}
    if kind == "norm":
        n = c["rows"] * c["H"]
        return {"bytes": 8 * n * 2, "flops": 20.0 * n}
    if kind == "head":
        return {"bytes": 4 * c["T"] * c["H"] + c["V"] * c["H"] * 6, "flops": 6.0 * c["T"] * c["H"] * c["V"]}
    if kind == "moe":
        rows, n = c["T"] * min(c["k"], c["E"]), 3 * c["H"] * c["I"]
        return {"bytes": 8 * c["T"] * c["H"] + c["E"] * n * 6, "flops": 6.0 * rows * n}
    if kind == "optim":
        H, F, D = c["H"], c["F"], c["H"] // c["hq"]
        flops = 0.0
        for m, n in ((H, H), (c["hkv"] * D, H), (c["hkv"] * D, H), (H, H), (F, H), (F, H), (H, F)):
            a, b = min(m, n), max(m, n)
            flops += 5 * (a * a * b * 2.0 + a * a * a * 2.0 + a * a * b * 2.0)      # a Gram is symmetric: half of it
        n, rest = c["layers"] * _layer_numel(c), 2 * c["V"] * H
        return {"bytes": n * (4 + 8 + 8 + 2) + rest * (4 + 8 + 16 + 2), "flops": flops * c["layers"]}
    n, head = c["layers"] * _layer_numel(c), c["V"] * c["H"]
    D = c["H"] // c["hq"]
    if kind == "prefill":
        T = c["B"] * c["P"]
        pairs = c["layers"] * c["B"] * c["hq"] * _pairs(c["P"], 0, False)
        return {"bytes": 2 * (n + head + T * c["H"]) + 4 * c["layers"] * T * c["hkv"] * D,
                "flops": 2.0 * (T * n + c["B"] * head) + 4.0 * pairs * D}
    cached = c["layers"] * c["B"] * (c["P"] + 1) * c["hkv"] * D
    return {"bytes": 2 * (n + head + c["B"] * c["V"]) + 4 * cached,
            "flops": 2.0 * c["B"] * (n + head) + 4.0 * cached * (c["hq"] // c["hkv"])}


def tolerance(case):
    # four times the distance from exact(): bf16 activations, and for the optimizer bf16 Newton-Schulz iterations whose
    # result is a small part of the updated weight
    return {"rel": {"block": 0.03, "attn": 0.016, "norm": 0.01, "head": 0.008, "moe": 0.016, "optim": 0.006,
                    "prefill": 0.05, "decode": 0.05}[case["kind"]]}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------
def _rms64(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS) * w


def _rope64(x, positions):
    """Rotates the (even, odd) pairs of ``x`` [..., T, heads, D] by its positions [T]."""
    D = x.shape[-1]
    inv = THETA ** (-torch.arange(0, D, 2, device="cuda", dtype=torch.float64) / D)
    ang = positions.double()[:, None, None] * inv
    c, s = ang.cos(), ang.sin()
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * c - b * s, a * s + b * c], dim=-1).flatten(-2)


def _attend64(q, k, v, lo, first=0):
    """q [S,hq,D] at positions first.. over k, v [Sk,hkv,D]; causal, from ``lo`` [S] on.  One head at a time."""
    S, hq, D = q.shape
    g = hq // k.shape[1]
    at = torch.arange(first, first + S, device="cuda")
    keys = torch.arange(k.shape[0], device="cuda")
    hidden = keys[None, :] > at[:, None]
    if lo is not None:
        hidden = hidden | (keys[None, :] < lo[:, None])
    heads = []
    for h in range(hq):
        p = (q[:, h] @ k[:, h // g].T * D ** -0.5).masked_fill_(hidden, float("-inf")).softmax(-1)
        heads.append(p @ v[:, h // g])
    return torch.stack(heads, dim=1)


def _attn64(qkv, wq, wk, lo, go, c):
    """Output of the attention block and the gradients of qkv, wq and wk, one sequence and one kv head at a time."""
    B, S, hq, hkv, D = c["B"], c["S"], c["hq"], c["hkv"], c["D"]
    g = hq // hkv
    qkv, go = qkv.view(B, S, hq + 2 * hkv, D), go.view(B, S, hq, D)
    o = torch.empty(B, S, hq, D, dtype=torch.float64, device="cuda")
    dqkv = torch.empty(B, S, hq + 2 * hkv, D, dtype=torch.float64, device="cuda")
    pos = torch.arange(S, device="cuda")
    wq, wk = wq.double().requires_grad_(True), wk.double().requires_grad_(True)
    dwq, dwk = torch.zeros_like(wq), torch.zeros_like(wk)
    for b in range(B):
        for h in range(hkv):
            for j in range(h * g, (h + 1) * g):
                with torch.enable_grad():
                    xs = [qkv[b, :, i:i + 1].double().requires_grad_(True) for i in (j, hq + h, hq + hkv + h)]
                    q, k = _rope64(_rms64(xs[0], wq), pos), _rope64(_rms64(xs[1], wk), pos)
                    out = _attend64(q, k, xs[2], None if lo is None else lo[b])
                    got = torch.autograd.grad([out], xs + [wq, wk], [go[b, :, j:j + 1].double()])
                o[b, :, j] = out[:, 0].detach()
                dqkv[b, :, j] = got[0][:, 0]
                for i, d in ((hq + h, got[1]), (hq + hkv + h, got[2])):
                    dqkv[b, :, i] = d[:, 0] if j == h * g else dqkv[b, :, i] + d[:, 0]
                dwq += got[3]
                dwk += got[4]
    return o.view(B, S, hq * D), dqkv.view(B * S, -1), dwq.detach(), dwk.detach()


def _swiglu64(gu):
    gate, up = gu.chunk(2, dim=-1)
    return gate * torch.sigmoid(gate) * up


def _block64(t, c):
    H, T = c["H"], c["B"] * c["S"]
    w = {k: v.double() for k, v in t["w"].items()}
    x0 = (t["x"].double() + t["delta"].double()).view(T, H)
    ac = dict(c, D=H // c["hq"])
    zero = torch.zeros(c["B"], c["S"], H, dtype=torch.bfloat16, device="cuda")

    def grads(outs, wanted, given):
        return torch.autograd.grad(outs, wanted, given, allow_unused=True)

    # forward up to the packed projection, attention by itself, then the rest; backward in the reverse order
    with torch.enable_grad():
        x0.requires_grad_(True)
        p1 = [w["pre_norm.scale"].requires_grad_(True), w["attn.wqkv"].requires_grad_(True)]
        qkv = _rms64(x0, p1[0]) @ p1[1].T
    q64 = qkv.detach()
    o = _attn64(q64, w["attn.q_norm"], w["attn.k_norm"], t["lo"], zero, ac)[0].view(T, H)
    with torch.enable_grad():
        o.requires_grad_(True)
        x1 = x0.detach().requires_grad_(True)
        p2 = [w[k].requires_grad_(True) for k in ("attn.wo", "post_norm.scale", "mlp.w_gate_up", "mlp.w_down")]
        x2 = x1 + o @ p2[0].T
        m = _swiglu64(_rms64(x2, p2[1]) @ p2[2].T) @ p2[3].T
        got = grads([x2, m], [o, x1] + p2, [t["gx"].double().view(T, H), t["gm"].double().view(T, H)])
    _, dqkv, dwq, dwk = _attn64(q64, w["attn.q_norm"], w["attn.k_norm"], t["lo"], got[0], ac)
    d1 = grads([qkv], [x0] + p1, [dqkv])
    dx = (got[1] + d1[0]).view(c["B"], c["S"], H)
    shape = (c["B"], c["S"], H)
    return {"x": x2.detach().view(shape), "m": m.detach().view(shape), "dx": dx, "ddelta": dx, "d_pre_norm.scale": d1[1],
            "d_attn.wqkv": d1[2], "d_attn.wo": got[2], "d_attn.q_norm": dwq, "d_attn.k_norm": dwk,
            "d_post_norm.scale": got[3], "d_mlp.w_gate_up": got[4], "d_mlp.w_down": got[5]}


def _head64(t, c):
    w, scale = t["w"].double(), 1.0 / c["T"]
    dw, dx = torch.zeros_like(w), []
    ce_sum = z_sum = 0.0
    for a in range(0, c["T"], 2048):
        x = t["x"][a:a + 2048].double()
        logits = x @ w.T
        lse = torch.logsumexp(logits, dim=1)
        mask, target = t["mask"][a:a + 2048].double(), t["targets"][a:a + 2048].long()
        ce_sum = ce_sum + ((lse - logits.gather(1, target[:, None])[:, 0]) * mask).sum()
        z_sum = z_sum + (lse.pow(2) * mask).sum()
        g = torch.exp(logits - lse[:, None]) * ((1.0 + 2.0 * _Z * lse) * mask * scale)[:, None]
        g.scatter_add_(1, target[:, None], -(mask * scale)[:, None])
        dx.append(g @ w)
        dw += g.T @ x
    return {"ce": ce_sum, "z": z_sum, "dx": torch.cat(dx), "dw": dw}


def _moe64(t, c):
    T, H = t["x"].shape
    x, p, gy = t["x"].double(), t["p"].double(), t["gy"].double()
    y, dx, dp = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(p)
    dwgu = torch.zeros(t["wgu"].shape, device="cuda")
    dwd = torch.zeros(t["wd"].shape, device="cuda")
    for e in range(c["E"]):
        rows, col = torch.nonzero(t["ids"] == e, as_tuple=True)
        if not len(rows):
            continue
        with torch.enable_grad():
            ins = [x[rows].requires_grad_(True), p[rows, col].requires_grad_(True),
                   t["wgu"][e].double().requires_grad_(True), t["wd"][e].double().requires_grad_(True)]
            out = (_swiglu64(ins[0] @ ins[2].T) @ ins[3].T) * ins[1][:, None]
            got = torch.autograd.grad([out], ins, [gy[rows]])
        y.index_add_(0, rows, out.detach())
        dx.index_add_(0, rows, got[0])
        dp[rows, col] = got[1]
        dwgu[e], dwd[e] = got[2].float(), got[3].float()
    return {"y": y, "dx": dx, "dp": dp, "dwgu": dwgu, "dwd": dwd}


def _optim64(t, c):
    H, D = c["H"], c["H"] // c["hq"]
    norm = torch.sqrt(sum(g.double().pow(2).sum() for g in t["g"].values()))
    clip, lr, decay = 1.0 / torch.clamp(norm, min=1.0), 1e-2, 0.1
    out = {"grad_norm": norm}
    for name, w in t["w"].items():
        w, g = w.double(), t["g"][name].double() * clip
        if "layers." not in name or "norm" in name:                # AdamW, first step
            mhat, vhat = g, g * g
            out[name] = (w - lr * (mhat / (vhat.sqrt() + 1e-8) + decay * w)).float()
            continue
        cuts = [w.shape[0]]
        if name.endswith("wqkv"):
            cuts = [c["hq"] * D, c["hkv"] * D, c["hkv"] * D]
        elif name.endswith("w_gate_up"):
            cuts = [c["F"], c["F"]]
        parts = []
        for gp in g.split(cuts):
            m = 0.05 * gp
            x = 0.05 * gp + 0.95 * m
            x = x / torch.clamp(x.norm(), min=1e-7)
            tall = x.shape[0] > x.shape[1]
            x = x.T if tall else x
            for _ in range(5):
                gram = x @ x.T
                x = 3.4445 * x + (-4.7750 * gram + 2.0315 * (gram @ gram)) @ x
            x = x.T if tall else x
            parts.append(0.2 * max(gp.shape) ** 0.5 * x)
        out[name] = (w * (1.0 - lr * decay) - lr * torch.cat(parts)).float()
    return out


def _model64(t, c, kind):
    B, H, hq, hkv = c["B"], c["H"], c["hq"], c["hkv"]
    D, n, first = H // hq, t["ids"].shape[1], 0 if kind == "prefill" else c["P"]
    pos = torch.arange(first, first + n, device="cuda")
    x = t["w"]["embed"][t["ids"].long()].double()
    ks, vs = [], []
    for i in range(c["layers"]):
        w = {k[len(f"layers.{i}."):]: v.double() for k, v in t["w"].items() if k.startswith(f"layers.{i}.")}
        qkv = (_rms64(x, w["pre_norm.scale"]) @ w["attn.wqkv"].T).view(B, n, hq + 2 * hkv, D)
        q = _rope64(_rms64(qkv[:, :, :hq], w["attn.q_norm"]), pos)
        k = _rope64(_rms64(qkv[:, :, hq:hq + hkv], w["attn.k_norm"]), pos)
        v = qkv[:, :, hq + hkv:]
        ks.append(k)
        vs.append(v)
        o = []
        for b in range(B):
            kb, vb = k[b], v[b]
            if kind == "decode":
                kb, vb = torch.cat([t["k"][i, b].double(), kb]), torch.cat([t["v"][i, b].double(), vb])
            o.append(_attend64(q[b], kb, vb, None, first))
        x = x + torch.stack(o).view(B, n, H) @ w["attn.wo"].T
        x = x + _swiglu64(_rms64(x, w["post_norm.scale"]) @ w["mlp.w_gate_up"].T) @ w["mlp.w_down"].T
    logits = _rms64(x[:, -1], t["w"]["norm.scale"].double()) @ t["w"]["lm_head"].double().T
    if kind == "decode":
        return {"logits": logits, "k": torch.stack([k[:, 0] for k in ks]), "v": torch.stack([v[:, 0] for v in vs])}
    pages = -(-(c["P"] + 64) // 128)
    out = {"logits": logits}
    for name, rows in (("k", ks), ("v", vs)):
        pool = torch.zeros(c["layers"], B, pages * 128, hkv, D, dtype=torch.float64, device="cuda")
        pool[:, :, :n] = torch.stack(rows)
        pool = pool.view(c["layers"], B, pages, 128, hkv, D).transpose(3, 4)
        out[name] = pool.reshape(c["layers"], B * pages, hkv, 128, D)
    return out


@torch.no_grad()
def exact(case, seed):
    c, t, kind = case, _draw_inputs(case, seed), case["kind"]
    if kind == "block":
        return _block64(t, c)
    if kind == "attn":
        o, dqkv, dwq, dwk = _attn64(t["qkv"], t["wq"], t["wk"], t["lo"], t["go"], c)
        return {"o": o, "dqkv": dqkv, "dwq": dwq, "dwk": dwk}
    if kind == "norm":
        with torch.enable_grad():
            ins = [t["x"].double().requires_grad_(True), t["delta"].double().requires_grad_(True),
                   t["w"].double().requires_grad_(True)]
            res = ins[0] + ins[1]
            y = _rms64(res, ins[2])
            got = torch.autograd.grad([y, res], ins, [t["gy"].double(), t["gr"].double()])
        return {"y": y.detach(), "res": res.detach(), "dx": got[0], "ddelta": got[1], "dw": got[2]}
    if kind == "head":
        return _head64(t, c)
    if kind == "moe":
        return _moe64(t, c)
    if kind == "optim":
        return _optim64(t, c)
    return _model64(t, c, kind)
