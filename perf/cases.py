"""Performance cases: the layers, operators and calls that a training or serving program spends its time in, each through a
public entry point of the framework.

Kinds of case (``case["kind"]``):

* ``block``      forward + backward of a Llama decoder layer and the model's closing norm (a small or a large model's training);
* ``attention``  forward + backward of causal attention on a fused QKV projection, up to long context;
* ``head``       forward + backward of the language-model head with its cross entropy;
* ``linear``     a projection at decode sizes, without gradients (one to a few hundred rows against a whole weight);
* ``paged``      attention of a ragged serving batch over the paged key/value cache: decode tokens, prompt portions, both mixed;
* ``moe``        the routed experts of a serving layer (router, dispatch, grouped products, combine);
* ``sink``       chunk-local or sliding-window attention with a sink logit and 32-bit weights (hybrid layer stacks);
* ``recurrence`` the linear recurrences of hybrid layer stacks over ragged prompts (delta rule, per-channel decay, state-space);
* ``engine``     requests through the ragged engine: prompts, then tokens one by one, then the pages are given back.

Widths come from the framework's model presets (``models/llama.py``, ``models/mixtral.py``) and from its serving benchmark's
sizes.
"""
from __future__ import annotations

import math

import torch

from shuffle_exchange_b200.inference.v2.config_v2 import RaggedInferenceEngineConfig
from shuffle_exchange_b200.inference.v2.engine_factory import build_engine_from_model
from shuffle_exchange_b200.inference.v2.inference_utils import ActivationType, DtypeEnum
from shuffle_exchange_b200.inference.v2.kernels import mixer_ops as M
from shuffle_exchange_b200.inference.v2.kernels import ragged_ops as R
from shuffle_exchange_b200.inference.v2.modules import heuristics
from shuffle_exchange_b200.inference.v2.modules.configs import DSMoEConfig
from shuffle_exchange_b200.inference.v2.ragged.ragged_manager import DSStateManagerConfig
from shuffle_exchange_b200.inference.v2.ragged.ragged_wrapper import RaggedBatchWrapper
from shuffle_exchange_b200.models.llama import LlamaDecoderLayer, LlamaForCausalLM, llama_config
from shuffle_exchange_b200.ops import functional as F

BF16 = torch.bfloat16
EPS = 1e-5
THETA = 500000.0

# width, query heads, key/value heads, feed-forward width
DIMS = {
    "llama-160m": (768, 12, 4, 2048),
    "w1024": (1024, 8, 2, 4096),
    "w2048": (2048, 16, 4, 8192),
    "llama2-7b": (4096, 32, 32, 11008),
    "llama3-8b": (4096, 32, 8, 14336),
}
PAGE = 64


def listed():
    return [
        # a training step of a small model on a ragged micro-batch: latency, launches and odd lengths count
        dict(name="block small ragged", kind="block", model="llama-160m", batch=2, seq=331),
        # a training step of the 8B model, half the headline micro-batch: tensor cores count
        dict(name="block 8b 4096", kind="block", model="llama3-8b", batch=1, seq=4096),
        # attention of the headline training configuration: 8192 tokens in one sequence
        dict(name="attention 8192", kind="attention", batch=1, seq=8192, heads=32, kv=8, dim=128),
        # the loss of a micro-batch over a 128k vocabulary
        dict(name="head 1999x128k", kind="head", rows=1999, width=4096, vocab=128256),
        # one token of one request through the largest projection of an 8B model: streams the weight
        dict(name="linear 1 row", kind="linear", rows=1, n=28672, k=4096),
        # a decode batch through a square projection
        dict(name="linear 48 rows", kind="linear", rows=48, n=4096, k=4096),
        # a decode step of 61 requests with contexts of all lengths around 2000 tokens
        dict(name="paged decode", kind="paged", decodes=61, context=2048, prompts=0, prompt=0, heads=32, kv=8, dim=128),
        # a scheduler's mixed step: two prompt portions behind some context, and decode tokens
        dict(name="paged mixed", kind="paged", decodes=24, context=1500, prompts=2, prompt=777, heads=32, kv=8, dim=128),
        # the experts of a Mixtral-sized layer for a decode batch with a short prompt in it
        dict(name="moe 200 tokens", kind="moe", tokens=200, width=4096, ff=14336, experts=8, k=2),
        # a prompt through a hybrid stack's attention layer (32-bit weights, chunks of 1024 positions)
        dict(name="sink prompt", kind="sink", seqs=1, rows=3000, context=0, heads=16, kv=4, dim=128, chunk=1024, window=0),
        # ragged prompts through a hybrid stack's delta-rule layer
        dict(name="delta prompts", kind="recurrence", rule="delta", seqs=3, rows=2300, heads=16, dim=128),
        # requests served from prompt to flush: four ragged prompts in one step, then six decode steps
        dict(name="engine requests", kind="engine", model="w2048", layers=4, requests=4, prompt=300, steps=6),
    ]


def _log(rng, lo, hi):
    """An integer between ``lo`` and ``hi``, spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["block", "attention", "head", "linear", "linear", "paged", "paged", "moe", "sink", "recurrence", "engine"])
    if kind == "block":
        seq = _log(rng, 64, 4096)
        return dict(kind=kind, model=rng.choice(["llama-160m", "w2048", "llama2-7b", "llama3-8b"]),
                    batch=rng.randint(1, max(1, min(4, 4096 // seq))), seq=seq)
    if kind == "attention":
        seq = _log(rng, 128, 8192)
        heads, kv, dim = rng.choice([(32, 8, 128), (16, 4, 128), (12, 4, 64), (32, 32, 128)])
        return dict(kind=kind, batch=rng.randint(1, max(1, min(4, 8192 // seq))), seq=seq, heads=heads, kv=kv, dim=dim)
    if kind == "head":
        width, vocab = rng.choice([(768, 32000), (2048, 32000), (4096, 32000), (4096, 128256)])
        return dict(kind=kind, rows=_log(rng, 64, 2048), width=width, vocab=vocab)
    if kind == "linear":
        w, hq, hk, ff = DIMS[rng.choice(list(DIMS))]
        d = w // hq
        n, k = rng.choice([((hq + 2 * hk) * d, w), (w, w), (2 * ff, w), (w, ff), (32000, w)])
        return dict(kind=kind, rows=_log(rng, 1, 256), n=n, k=k)
    if kind == "paged":
        heads, kv, dim = rng.choice([(32, 8, 128), (16, 4, 128), (12, 4, 64), (32, 32, 128)])
        prompts = rng.choice([0, 0, 1, 3])
        return dict(kind=kind, decodes=_log(rng, 1, 128) if prompts == 0 else rng.randint(0, 32), context=_log(rng, 64, 6000),
                    prompts=prompts, prompt=_log(rng, 17, 2048) if prompts else 0, heads=heads, kv=kv, dim=dim)
    if kind == "moe":
        width, ff, experts = rng.choice([(4096, 14336, 8), (2048, 8192, 8), (1024, 4096, 16)])
        return dict(kind=kind, tokens=_log(rng, 1, 2048), width=width, ff=ff, experts=experts, k=2)
    if kind == "sink":
        heads, kv = rng.choice([(8, 2), (16, 4), (32, 8)])
        chunk = rng.choice([1024, 4096, 0])
        shape = (dict(seqs=rng.randint(1, 4), rows=_log(rng, 100, 4096), context=rng.choice([0, 0, 700])) if rng.random() < 0.6
                 else dict(seqs=_log(rng, 1, 64), rows=0, context=_log(rng, 64, 4000)))
        return dict(kind=kind, heads=heads, kv=kv, dim=128, chunk=chunk, window=0 if chunk else 512, **shape)
    if kind == "recurrence":
        return dict(kind=kind, rule=rng.choice(["delta", "channel", "ssd"]), seqs=rng.randint(1, 8), rows=_log(rng, 64, 4096),
                    heads=rng.choice([8, 16, 32]), dim=128)
    return dict(kind=kind, model=rng.choice(["w1024", "w2048"]), layers=rng.randint(2, 4), requests=rng.randint(1, 8),
                prompt=_log(rng, 16, 400), steps=rng.randint(1, 6))


# ------------------------------------------------------------------------------------------------ sizes
def _spread(total, parts, seed=0):
    """``total`` rows split into ``parts`` uneven portions of at least one row."""
    parts = max(1, min(parts, total))
    w = [1.0 + 0.35 * ((7 * i + 3 + seed) % 5) for i in range(parts)]
    cut = [max(1, int(total * x / sum(w))) for x in w]
    cut[-1] += total - sum(cut)
    if cut[-1] < 1:
        cut = [total // parts + (1 if i < total % parts else 0) for i in range(parts)]
    return cut


def _plan(c):
    """``[(tokens seen before, tokens of this step)]`` per sequence of a ragged attention case."""
    if c["kind"] == "paged":
        plan = [(c["context"] * (2 + i % 3) // 6, c["prompt"] + 5 * i) for i in range(c["prompts"])]
        plan += [(max(1, c["context"] * (50 + (37 * i) % 101) // 100), 1) for i in range(c["decodes"])]
        return plan or [(c["context"], 1)]
    if c["rows"]:
        return [(c["context"], n) for n in _spread(c["rows"], c["seqs"])]
    return [(max(1, c["context"] * (50 + (37 * i) % 101) // 100), 1) for i in range(c["seqs"])]


def _first_key(c, pos):
    """First visible position of a query at ``pos`` of a ``sink`` case."""
    if c["chunk"] > 0:
        return pos // c["chunk"] * c["chunk"]
    return max(0, pos - c["window"] + 1) if c["window"] > 0 else 0


def _prompt_lengths(c):
    return [max(1, c["prompt"] * (60 + (53 * i) % 81) // 100) for i in range(c["requests"])]


def _params(model):
    w, hq, hk, ff = DIMS[model]
    return w * (hq + 2 * hk) * (w // hq) + w * w + 3 * w * ff


# ------------------------------------------------------------------------------------------------ states
class _Sequence:
    """What a ragged batch asks of a sequence: tokens already cached and the pages that hold it."""

    def __init__(self, seen, pages):
        self.seen_tokens, self._pages = seen, torch.tensor(pages, dtype=torch.int32)

    def kv_blocks(self):
        return self._pages


def _batch(plan, g):
    """A finalized ragged batch over pages in scattered order, and the number of pages."""
    need = [(seen + n + PAGE - 1) // PAGE for seen, n in plan]
    order = torch.randperm(sum(need), generator=g).tolist()
    batch = RaggedBatchWrapper(sum(n for _, n in plan), len(plan), max(need), device="cuda")
    at = 0
    for (seen, n), k in zip(plan, need):
        batch.insert_sequence(_Sequence(seen, order[at: at + k]), torch.zeros(n, dtype=torch.int64))
        at += k
    batch.finalize()
    return batch, sum(need)


def _engine(c, seed):
    w, hq, hk, ff = DIMS[c["model"]]
    cfg = llama_config("llama-tiny", hidden_size=w, num_hidden_layers=c["layers"], num_attention_heads=hq,
                       num_key_value_heads=hk, intermediate_size=ff, vocab_size=32000, rope_theta=THETA,
                       activation_checkpointing=False)
    torch.manual_seed(seed)
    model = LlamaForCausalLM(cfg, device="cuda", dtype=BF16).eval()
    pages = sum((n + c["steps"] + PAGE - 1) // PAGE for n in _prompt_lengths(c)) + 8
    sm = DSStateManagerConfig(max_tracked_sequences=16, max_ragged_sequence_count=16, max_ragged_batch_size=8192,
                              max_context=8192, num_kv_blocks=pages)
    return model, build_engine_from_model(model, RaggedInferenceEngineConfig(state_manager=sm, kv_block_size=PAGE))


def prepare(case, seed):
    c, kind = case, case["kind"]
    dev = "cuda"
    g = torch.Generator(device=dev).manual_seed(seed)
    gc = torch.Generator().manual_seed(seed)

    def rand(*shape, std=1.0, dtype=BF16):
        return (torch.randn(*shape, generator=g, device=dev) * std).to(dtype)

    if kind == "block":
        w, hq, hk, ff = DIMS[c["model"]]
        cfg = llama_config("llama3-8b", hidden_size=w, intermediate_size=ff, num_attention_heads=hq, num_key_value_heads=hk,
                           rope_theta=THETA, num_hidden_layers=1)
        layer = LlamaDecoderLayer(cfg, 0, device=dev, dtype=BF16)
        with torch.no_grad():
            for p in layer.parameters():
                p.copy_(rand(*p.shape, std=0.02) if p.dim() == 2 else 1.0 + rand(*p.shape, std=0.1))
        layer.norm = torch.nn.Parameter(1.0 + rand(w, std=0.1))
        B, S = c["batch"], c["seq"]
        cos, sin = F.rope_tables(8192, w // hq, THETA, torch.device(dev))
        return dict(c=c, layer=layer, h=rand(B, S, w, std=0.5).requires_grad_(), res=rand(B, S, w).requires_grad_(),
                    dy=rand(B, S, w, std=1e-3),
                    pos=torch.arange(S, device=dev).repeat(B), cos=cos, sin=sin)
    if kind == "attention":
        B, S, D = c["batch"], c["seq"], c["dim"]
        return dict(c=c, qkv=rand(B, S, (c["heads"] + 2 * c["kv"]) * D).requires_grad_(),
                    dout=rand(B, S, c["heads"], D, std=1e-2))
    if kind == "head":
        return dict(c=c, x=rand(c["rows"], c["width"]).requires_grad_(),
                    w=torch.nn.Parameter(rand(c["vocab"], c["width"], std=0.02)),
                    labels=torch.randint(0, c["vocab"], (c["rows"],), generator=g, device=dev))
    if kind == "linear":
        return dict(c=c, x=rand(c["rows"], c["k"]), w=rand(c["n"], c["k"], std=0.02))
    if kind == "paged":
        plan = _plan(c)
        batch, pages = _batch(plan, gc)
        T = sum(n for _, n in plan)
        return dict(c=c, batch=batch, cache=rand(pages, PAGE, 2, c["kv"], c["dim"]),
                    qkv=rand(T, c["heads"] + 2 * c["kv"], c["dim"]))
    if kind == "moe":
        W, Fw, E = c["width"], c["ff"], c["experts"]
        mod = heuristics.instantiate_moe(DSMoEConfig(
            max_tokens=4096, model_dim=W, intermediate_features=Fw, n_experts=E, top_k=c["k"], input_dtype=DtypeEnum.bf16,
            output_dtype=DtypeEnum.bf16, activation=ActivationType.SiGLU, normalize_scores=True,
            router_dtype=DtypeEnum.fp32), RaggedInferenceEngineConfig())
        return dict(c=c, mod=mod, x=rand(c["tokens"], W), gate=rand(E, W, std=W ** -0.5, dtype=torch.float32),
                    w1=rand(E, 2 * Fw, W, std=0.02), w2=rand(E, W, Fw, std=0.02))
    if kind == "sink":
        plan = _plan(c)
        batch, pages = _batch(plan, gc)
        T, d = sum(n for _, n in plan), c["dim"]
        unit = lambda t: t / t.square().mean(-1, keepdim=True).sqrt()  # noqa: E731
        return dict(c=c, batch=batch, q=unit(rand(T, c["heads"], d, dtype=torch.float32)),
                    kc=unit(rand(pages, PAGE, c["kv"], d, dtype=torch.float32)).to(BF16), vc=rand(pages, PAGE, c["kv"], d),
                    sink=rand(c["heads"], dtype=torch.float32))
    if kind == "recurrence":
        H, d, T = c["heads"], c["dim"], c["rows"]
        G = 1 if c["rule"] == "ssd" else H
        f32 = torch.float32
        rows = rand(T, 2 * G * d + H * d, dtype=f32)
        if c["rule"] != "ssd":                       # keys and queries of the delta rules are unit vectors
            kq = rows[:, : 2 * G * d].view(T, 2 * G, d)
            kq /= kq.square().sum(-1, keepdim=True).sqrt()
            rows[:, G * d: 2 * G * d] *= d ** -0.5
        else:
            rows[:, : 2 * G * d] *= d ** -0.5
        rate = torch.nn.functional.softplus(rand(T, H * (d if c["rule"] == "channel" else 1), dtype=f32))
        a = torch.exp(torch.rand(H, generator=g, device=dev) * 2.5 - 2.0)
        decay = torch.exp(-a.repeat_interleave(rate.shape[1] // H) * rate)
        beta = rate.clone() if c["rule"] == "ssd" else torch.sigmoid(rand(T, H, dtype=f32))
        cut = _spread(T, c["seqs"])
        info = torch.tensor([[sum(cut[:i]), n, 0, i] for i, n in enumerate(cut)], dtype=torch.int32, device=dev)
        return dict(c=c, rows=rows, decay=decay.contiguous(), beta=beta.contiguous(), info=info, G=G,
                    skip=rand(H, dtype=f32) if c["rule"] == "ssd" else None,
                    state=torch.zeros(len(cut), H, d, d, device=dev))
    if kind == "engine":
        model, eng = _engine(c, seed)
        toks = lambda n: torch.randint(0, 32000, (n,), generator=gc, dtype=torch.int32)  # noqa: E731
        return dict(c=c, model=model, engine=eng, prompts=[toks(n) for n in _prompt_lengths(c)],
                    steps=[[toks(1) for _ in range(c["requests"])] for _ in range(c["steps"])])
    raise ValueError(kind)


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    s, c = state, state["c"]
    kind = c["kind"]
    if kind == "block":
        layer = s["layer"]
        s["h"].grad = s["res"].grad = None
        layer.zero_grad(set_to_none=True)
        h, res = layer(s["h"], s["res"], s["pos"], s["cos"], s["sin"])
        y, res = F.rms_norm(h, layer.norm, EPS, res)
        y.backward(s["dy"])
        return dict(y=y.detach(), residual=res.detach(), dh=s["h"].grad, dresidual=s["res"].grad,
                    **{"d_" + n: p.grad for n, p in layer.named_parameters()})
    if kind == "attention":
        s["qkv"].grad = None
        out = F.flash_attention_qkv(s["qkv"], c["heads"], c["kv"], c["dim"], causal=True)
        out.backward(s["dout"])
        return dict(out=out.detach(), dqkv=s["qkv"].grad)
    if kind == "head":
        s["x"].grad = s["w"].grad = None
        loss = F.cross_entropy(F.linear(s["x"], s["w"]), s["labels"])
        loss.backward()
        return dict(loss=loss.detach(), dx=s["x"].grad, dw=s["w"].grad)
    with torch.no_grad():
        if kind == "linear":
            return F.linear(s["x"], s["w"])
        if kind == "paged":
            return R.ragged_attention(s["qkv"][:, : c["heads"]], s["cache"], s["batch"])
        if kind == "moe":
            return s["mod"](s["x"], s["gate"], s["w1"], s["w2"])
        if kind == "sink":
            b = s["batch"]
            return M.sink_attention(s["q"], s["kc"], s["vc"], s["sink"], b.token_to_seq(), b.token_positions(),
                                    b.block_tables(), c["dim"] ** -0.5, c["chunk"], BF16, b.atoms(),
                                    b.atoms_longer_than(M.SHORT_ATOM), window=c["window"])
        if kind == "recurrence":
            G, H, d = s["G"], c["heads"], c["dim"]
            rows = s["rows"]
            out = M.linear_recurrence(rows[:, : G * d], rows[:, G * d: 2 * G * d], rows[:, 2 * G * d:], s["decay"], s["beta"],
                                      s["skip"], s["state"], s["info"], H, G, d, d, c["rule"] != "ssd")
            return dict(out=out, state=s["state"])
        eng, uids = s["engine"], list(range(c["requests"]))
        logits = [eng.put(uids, s["prompts"])]
        for step in s["steps"]:
            logits.append(eng.put(uids, step))
        for u in uids:
            eng.flush(u)
        return dict(logits=logits)


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    c, kind = case, case["kind"]
    if kind == "block":
        w, hq, hk, ff = DIMS[c["model"]]
        T, P = c["batch"] * c["seq"], _params(c["model"])
        return dict(bytes=2.0 * (2 * P + 8 * T * w), flops=6.0 * P * T + 7.0 * c["batch"] * w * c["seq"] ** 2)
    if kind == "attention":
        T = c["batch"] * c["seq"]
        return dict(bytes=2.0 * T * c["dim"] * (4 * c["heads"] + 4 * c["kv"]),
                    flops=7.0 * c["batch"] * c["heads"] * c["dim"] * c["seq"] ** 2)
    if kind == "head":
        return dict(bytes=2.0 * (2 * c["vocab"] * c["width"] + 2 * c["rows"] * c["width"]),
                    flops=6.0 * c["rows"] * c["width"] * c["vocab"])
    if kind == "linear":
        return dict(bytes=2.0 * (c["n"] * c["k"] + c["rows"] * (c["n"] + c["k"])), flops=2.0 * c["rows"] * c["n"] * c["k"])
    if kind == "paged":
        plan = _plan(c)
        return dict(bytes=2.0 * c["dim"] * (sum(s + n for s, n in plan) * 2 * c["kv"] + sum(n for _, n in plan) * 2 * c["heads"]),
                    flops=4.0 * c["heads"] * c["dim"] * sum(n * s + n * (n + 1) / 2 for s, n in plan))
    if kind == "moe":
        used = min(c["experts"], c["tokens"] * c["k"])
        per = 3.0 * c["ff"] * c["width"]
        return dict(bytes=2.0 * (used * per + 2 * c["tokens"] * c["width"]), flops=2.0 * c["tokens"] * c["k"] * per)
    if kind == "sink":
        seen, keys, T = 0, 0, 0
        for s, n in _plan(c):
            seen += s + n - _first_key(c, s)
            keys += sum(p + 1 - _first_key(c, p) for p in range(s, s + n))
            T += n
        return dict(bytes=c["dim"] * (seen * 4.0 * c["kv"] + T * 6.0 * c["heads"]), flops=4.0 * c["heads"] * c["dim"] * keys)
    if kind == "recurrence":
        H, d, T = c["heads"], c["dim"], c["rows"]
        G = 1 if c["rule"] == "ssd" else H
        per = T * (2 * G * d + 2 * H * d + H * (d + 1 if c["rule"] == "channel" else 2))
        return dict(bytes=4.0 * (per + len(_spread(T, c["seqs"])) * H * d * d),
                    flops=(5.0 if c["rule"] == "ssd" else 7.0) * T * H * d * d)
    w, hq, hk, ff = DIMS[c["model"]]
    lens = _prompt_lengths(c)
    P, head = c["layers"] * _params(c["model"]), 32000 * w
    pairs = sum(n * (n + 1) / 2 + sum(n + j + 1 for j in range(c["steps"])) for n in lens)
    T = sum(lens) + c["steps"] * c["requests"]
    kv = c["layers"] * 2 * hk * (w // hq)
    return dict(bytes=2.0 * ((1 + c["steps"]) * (P + head + c["requests"] * 32000) + T * w
                             + kv * sum(n + sum(n + j + 1 for j in range(c["steps"])) for n in lens)),
                flops=2.0 * P * T + 2.0 * head * c["requests"] * (1 + c["steps"]) + 4.0 * c["layers"] * w * pairs)


# About four times the error against 64 bits that the kinds show (2-norm; largest single value): 16-bit outputs of 32-bit sums
# are off by half a unit of their last place (1.7e-3; 3.9e-3); 16-bit probabilities or activations in between add to that
# (attention 2.4e-3; 0.13 in a gradient near zero, experts 3.9e-3; 1.9e-2), and rounding travels on through a layer (1.1e-2; 0.10)
# and a stack (1.5e-2; 0.07).  The recurrences are 32-bit throughout (1.0e-7; 1.0e-6): their sums may be taken in another order.
_TOLERANCE = {
    "block": {"rel": 0.03, "max": 0.4},
    "attention": {"rel": 0.01, "max": 0.5},
    "head": {"rel": 0.012, "max": 0.03},
    "linear": {"rel": 0.007, "max": 0.016},
    "paged": {"rel": 0.01, "max": 0.06},
    "moe": {"rel": 0.016, "max": 0.08},
    "sink": {"rel": 0.007, "max": 0.016},
    "recurrence": {"rel": 2e-6, "max": 2e-5},
    "engine": {"rel": 0.03, "max": 0.3},
}


def tolerance(case):
    return dict(_TOLERANCE[case["kind"]])


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms64(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w


def _rotate64(x, pos):
    """Rotate-half on ``x`` ``[T, heads, d]`` at positions ``pos``."""
    d = x.shape[-1]
    inv = THETA ** (-torch.arange(0, d, 2, dtype=torch.float64, device=x.device) / d)
    ang = pos.double()[:, None] * inv
    cs, sn = ang.cos()[:, None], ang.sin()[:, None]
    a, b = x[..., : d // 2], x[..., d // 2:]
    return torch.cat([a * cs - b * sn, b * cs + a * sn], -1)


def _attend64(q, k, v, lo, hi, scale, sink=None):
    """``q`` ``[m, Hq, d]`` over ``k``, ``v`` ``[n, Hk, d]``; query ``i`` sees the keys ``lo[i] <= j < hi[i]``."""
    rep = q.shape[1] // k.shape[1]
    j = torch.arange(k.shape[0], device=q.device)
    seen = (j[None] >= lo[:, None]) & (j[None] < hi[:, None])
    out = []
    for h in range(q.shape[1]):
        s = (q[:, h] @ k[:, h // rep].t() * scale).masked_fill(~seen, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink[h].expand(s.shape[0], 1)], 1)
        out.append(s.softmax(-1)[:, : k.shape[0]] @ v[:, h // rep])
    return torch.stack(out, 1)


def _causal64(q, k, v):
    n = torch.arange(q.shape[0], device=q.device)
    return _attend64(q, k, v, torch.zeros_like(n), n + 1, q.shape[-1] ** -0.5)


def _layer64(p, x, res, pos, hq, hk, rows):
    """One decoder layer on ``x`` ``[T, w]``, ``rows`` the lengths of its sequences; the new ``x`` and residual."""
    d = x.shape[1] // hq
    res = x if res is None else x + res
    qkv = (_rms64(res, p["input_layernorm"]) @ p["wqkv"].t()).view(-1, hq + 2 * hk, d)
    qk = _rotate64(qkv[:, : hq + hk], pos)
    parts, at = [], 0
    for n in rows:
        parts.append(_causal64(qk[at: at + n, :hq], qk[at: at + n, hq:], qkv[at: at + n, hq + hk:]))
        at += n
    res = torch.cat(parts).reshape(x.shape[0], -1) @ p["wo"].t() + res
    gu = _rms64(res, p["post_attention_layernorm"]) @ p["w_gate_up"].t()
    f = gu.shape[1] // 2
    return (torch.nn.functional.silu(gu[:, :f]) * gu[:, f:]) @ p["w_down"].t(), res


def _gather64(cache, batch, i, n):
    """Positions ``0 .. n - 1`` of sequence ``i`` out of a paged tensor."""
    j = torch.arange(n, device=cache.device)
    return cache[batch.block_tables()[i, j // PAGE].long(), j % PAGE].double()


def exact(case, seed):
    c, kind = case, case["kind"]
    s = prepare(case, seed)
    if kind == "block":
        w, hq, hk, ff = DIMS[c["model"]]
        B, S = c["batch"], c["seq"]
        p = {n: t.detach().double().requires_grad_() for n, t in s["layer"].named_parameters()}
        x, r = (s[n].detach().double().view(B * S, w).requires_grad_() for n in ("h", "res"))
        h, res = _layer64(p, x, r, s["pos"], hq, hk, [S] * B)
        res = h + res
        y = _rms64(res, p["norm"])
        y.backward(s["dy"].double().view(B * S, w))
        shape = lambda t: t.detach().view(B, S, w)  # noqa: E731
        return dict(y=shape(y), residual=shape(res), dh=shape(x.grad), dresidual=shape(r.grad),
                    **{"d_" + n: t.grad for n, t in p.items()})
    if kind == "attention":
        B, S, D, Hq, Hk = c["batch"], c["seq"], c["dim"], c["heads"], c["kv"]
        out = torch.empty(B, S, Hq, D, dtype=torch.float64, device="cuda")
        grad = torch.zeros(B, S, Hq + 2 * Hk, D, dtype=torch.float64, device="cuda")
        hidden = torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1)
        for b in range(B):
            x, dy = s["qkv"].detach()[b].view(S, -1, D), s["dout"][b]
            for h in range(Hq):
                q, k, v, do = (t.double() for t in (x[:, h], x[:, Hq + h // (Hq // Hk)], x[:, Hq + Hk + h // (Hq // Hk)], dy[:, h]))
                pr = (q @ k.t() * D ** -0.5).masked_fill_(hidden, float("-inf")).softmax(-1)
                o = pr @ v
                out[b, :, h] = o
                grad[b, :, Hq + Hk + h // (Hq // Hk)] += pr.t() @ do
                ds = pr.mul_((do @ v.t()).sub_((do * o).sum(-1, keepdim=True))).mul_(D ** -0.5)
                grad[b, :, h] = ds @ k
                grad[b, :, Hq + h // (Hq // Hk)] += ds.t() @ q
        return dict(out=out, dqkv=grad.view(B, S, -1))
    if kind == "head":
        x, w = s["x"].detach().double().requires_grad_(), s["w"].detach().double().requires_grad_()
        loss = torch.nn.functional.cross_entropy(x @ w.t(), s["labels"])
        loss.backward()
        return dict(loss=loss.detach(), dx=x.grad, dw=w.grad)
    with torch.no_grad():
        if kind == "linear":
            return s["x"].double() @ s["w"].double().t()
        if kind in ("paged", "sink"):
            sink = kind == "sink"
            q = s["q"] if sink else s["qkv"][:, : c["heads"]]
            out, at = [], 0
            for i, (seen, n) in enumerate(_plan(c)):
                kv = None if sink else _gather64(s["cache"], s["batch"], i, seen + n)
                k, v = (_gather64(s[t], s["batch"], i, seen + n) for t in ("kc", "vc")) if sink else (kv[:, 0], kv[:, 1])
                pos = torch.arange(seen, seen + n, device=q.device)
                lo = torch.tensor([_first_key(c, int(t)) for t in range(seen, seen + n)], device=q.device) if sink \
                    else torch.zeros_like(pos)
                out.append(_attend64(q[at: at + n].double(), k, v, lo, pos + 1, c["dim"] ** -0.5,
                                     s["sink"].double() if sink else None))
                at += n
            out = torch.cat(out)
            return out.reshape(out.shape[0], -1) if sink else out
        if kind == "moe":
            x, E = s["x"].double(), c["experts"]
            top, who = (x @ s["gate"].double().t()).softmax(-1).topk(c["k"], -1)
            top = top / top.sum(-1, keepdim=True)
            y = torch.zeros_like(x)
            for e in range(E):
                t, j = (who == e).nonzero(as_tuple=True)
                if t.numel():
                    gu = x[t] @ s["w1"][e].double().t()
                    f = gu.shape[1] // 2
                    y[t] += top[t, j, None] * ((torch.nn.functional.silu(gu[:, :f]) * gu[:, f:]) @ s["w2"][e].double().t())
            return y
        if kind == "recurrence":
            G, H, d = s["G"], c["heads"], c["dim"]
            T, x = c["rows"], s["rows"].double()
            k, q = (x[:, i * G * d: (i + 1) * G * d].view(T, G, d).repeat_interleave(H // G, 1) for i in (0, 1))
            v, beta = x[:, 2 * G * d:].view(T, H, d), s["beta"].double().view(T, H, 1)
            decay = s["decay"].double().view(T, H, 1, -1)
            out, state = torch.empty(T, H, d, dtype=torch.float64, device="cuda"), torch.zeros_like(s["state"]).double()
            for first, n, _, slot in s["info"].tolist():
                S = state[slot]
                for t in range(first, first + n):
                    S = S * decay[t]
                    u = beta[t] * (v[t] if c["rule"] == "ssd" else v[t] - (S @ k[t][:, :, None]).squeeze(-1))
                    S = S + u[:, :, None] * k[t][:, None, :]
                    out[t] = (S @ q[t][:, :, None]).squeeze(-1)
                state[slot] = S
            if s["skip"] is not None:
                out += s["skip"].double()[:, None] * v
            return dict(out=out.reshape(T, -1), state=state)
        w, hq, hk, ff = DIMS[c["model"]]
        m = s["model"].model
        lens = _prompt_lengths(c)
        seqs = [torch.cat([p] + [step[i] for step in s["steps"]]).long().cuda() for i, p in enumerate(s["prompts"])]
        rows = [t.numel() for t in seqs]
        pos = torch.cat([torch.arange(n, device="cuda") for n in rows])
        h, res = m.embed_tokens.double()[torch.cat(seqs)], None
        for layer in m.layers:
            h, res = _layer64({n: t.double() for n, t in layer.named_parameters()}, h, res, pos, hq, hk, rows)
        x = _rms64(h + res, m.norm.double())
        starts = [sum(rows[:i]) for i in range(len(rows))]
        head = s["model"].lm_head.double()
        return dict(logits=[x[[a + n - 1 + j for a, n in zip(starts, lens)]] @ head.t() for j in range(c["steps"] + 1)])
