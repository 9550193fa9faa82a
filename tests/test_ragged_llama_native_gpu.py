"""The forward of a dense Llama issued by one native call: the same bits as operator by operator, and what it does not take goes
there."""

import pytest

pytestmark = pytest.mark.gpu


def _engine(hidden, heads, kv, ff, vocab, layers=2, page=64, tie=False):
    import torch
    from shuffle_exchange_b200.inference.v2.config_v2 import RaggedInferenceEngineConfig
    from shuffle_exchange_b200.inference.v2.engine_factory import build_engine_from_model
    from shuffle_exchange_b200.inference.v2.ragged.manager_configs import DSStateManagerConfig
    from shuffle_exchange_b200.models.llama import LlamaForCausalLM, llama_config
    torch.manual_seed(0)
    cfg = llama_config("llama-tiny", hidden_size=hidden, num_hidden_layers=layers, num_attention_heads=heads,
                       num_key_value_heads=kv, intermediate_size=ff, vocab_size=vocab, activation_checkpointing=False,
                       tie_word_embeddings=tie)
    model = LlamaForCausalLM(cfg, device="cuda", dtype=torch.bfloat16).eval()
    sm = DSStateManagerConfig(max_tracked_sequences=8, max_ragged_sequence_count=8, max_ragged_batch_size=2048, max_context=1024,
                              num_kv_blocks=64 * 64 // page)
    return model, build_engine_from_model(model, RaggedInferenceEngineConfig(state_manager=sm, kv_block_size=page))


STEPS = [[5], [1], [300, 1, 17, 130], [1, 1, 1, 1], [1, 64, 1]]


def _serve(eng, native, monkeypatch, **kw):
    import torch
    from shuffle_exchange_b200.inference.v2.model_implementations.llama_v2 import RaggedLlamaModel
    used = []
    if native:
        real = RaggedLlamaModel._native_forward
        monkeypatch.setattr(RaggedLlamaModel, "_native_forward", lambda s, b, p: used.append(1) or real(s, b, p))
    else:
        monkeypatch.setattr(RaggedLlamaModel, "_native_plan", lambda s, b: None)
    g = torch.Generator().manual_seed(1)
    out = []
    for lens in STEPS:
        toks = [torch.randint(0, 256, (n,), generator=g, dtype=torch.int32) for n in lens]
        out.append(eng.put(range(len(lens)), toks, **{k: v[: len(lens)] for k, v in kw.items()}).clone())
    for u in range(4):
        eng.flush(u)
    monkeypatch.undo()
    return out, len(used)


@pytest.mark.parametrize("hidden,heads,kv,ff,vocab,layers,page,tie", [
    (512, 4, 2, 1024, 1024, 2, 64, False), (512, 8, 8, 776, 512, 1, 16, True), (768, 6, 1, 2048, 1000, 3, 128, False)])
def test_same_bits_as_operator_by_operator(hidden, heads, kv, ff, vocab, layers, page, tie, monkeypatch):
    import torch
    model, eng = _engine(hidden, heads, kv, ff, vocab, layers, page, tie)
    got, n = _serve(eng, True, monkeypatch)
    want, _ = _serve(eng, False, monkeypatch)
    assert n == len(STEPS)
    for a, b in zip(got, want):
        assert torch.equal(a, b) and torch.isfinite(a).all()
    for _ in range(5):                       # its kernels overlap: as often as it runs
        again, _ = _serve(eng, True, monkeypatch)
        assert all(torch.equal(a, b) for a, b in zip(again, want))
    (a, _), (b, _) = (_serve(eng, x, monkeypatch, logit_positions=[[0], [], [0], [0]]) for x in (True, False))
    assert all(torch.equal(x, y) for x, y in zip(a, b))


def test_what_it_does_not_take(monkeypatch):
    """Odd vocabulary, head size of 32: operator by operator, as ever."""
    import torch
    for kw in (dict(vocab=1001, heads=4, kv=2), dict(vocab=1024, heads=16, kv=16)):
        model, eng = _engine(512, kw["heads"], kw["kv"], 1024, kw["vocab"])
        got, n = _serve(eng, True, monkeypatch)
        want, _ = _serve(eng, False, monkeypatch)
        assert n == 0 and all(torch.equal(a, b) for a, b in zip(got, want))


def test_replaced_weights_are_seen(monkeypatch):
    import torch
    model, eng = _engine(512, 4, 2, 1024, 1024)
    before, _ = _serve(eng, True, monkeypatch)
    layer = model.model.layers[1]
    layer.wqkv = torch.nn.Parameter(layer.wqkv.detach() * 0.5)
    layer.w_down.data = torch.cat([layer.w_down.data, layer.w_down.data], 1)[:, 512: 1536]       # another pitch
    got, n = _serve(eng, True, monkeypatch)
    want, _ = _serve(eng, False, monkeypatch)
    assert n == len(STEPS) and all(torch.equal(a, b) for a, b in zip(got, want))
    assert not torch.equal(got[0], before[0])


def test_a_feed_forward_of_its_own_is_called(monkeypatch):
    import torch
    from shuffle_exchange_b200.inference.v2.model_implementations.llama_v2 import RaggedLlamaModel
    model, eng = _engine(512, 4, 2, 1024, 1024)
    plain, n = _serve(eng, True, monkeypatch)
    assert n == len(STEPS)
    ragged = next(x for x in vars(eng).values() if isinstance(x, RaggedLlamaModel))

    class Halved(RaggedLlamaModel):
        def _mlp(self, layer_idx, layer, x):
            return super()._mlp(layer_idx, layer, x) * 0.5

    ragged.__class__ = Halved
    got, n = _serve(eng, True, monkeypatch)
    want, _ = _serve(eng, False, monkeypatch)
    assert n == 0 and all(torch.equal(a, b) for a, b in zip(got, want)) and not torch.equal(got[0], plain[0])
    ragged.__class__ = RaggedLlamaModel
    ragged._mlp = lambda layer_idx, layer, x: RaggedLlamaModel._mlp(ragged, layer_idx, layer, x) * 0.5
    again, n = _serve(eng, True, monkeypatch)
    assert n == 0 and all(torch.equal(a, b) for a, b in zip(again, want))


def test_operands_that_the_plan_refuses(monkeypatch):
    """Types, pitches, addresses, watchers and layouts that the native call has no check for are turned down before it."""
    import contextlib

    import torch
    from torch.utils._python_dispatch import TorchDispatchMode
    from shuffle_exchange_b200.inference.v2.model_implementations.llama_v2 import RaggedLlamaModel
    from shuffle_exchange_b200.ops import functional as F
    model, eng = _engine(512, 4, 2, 1024, 1024)
    m, layer, P = model.model, model.model.layers[1], torch.nn.Parameter

    @contextlib.contextmanager
    def put(obj, name, value):
        old = getattr(obj, name)
        setattr(obj, name, value)
        try:
            yield
        finally:
            setattr(obj, name, old)

    @contextlib.contextmanager
    def mark(w, name):
        setattr(w, name, None)
        try:
            yield
        finally:
            delattr(w, name)

    def pitched(w, pitch, shift=0):
        room = torch.zeros(w.shape[0] * pitch + 8, device="cuda", dtype=w.dtype)
        return P(torch.as_strided(room, w.shape, (pitch, 1), shift))

    class Watcher(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    ragged = eng._model
    cache = ragged.state_manager.get_cache(1)
    every = lambda c: lambda li: c if li == 1 else type(ragged.state_manager).get_cache(ragged.state_manager, li)  # noqa: E731
    cases = {}
    for name in ("wqkv", "wo", "w_gate_up", "w_down"):
        w = getattr(layer, name)
        cases.update({
            f"{name} fp32": put(layer, name, P(w.detach().float())),
            f"{name} fp16": put(layer, name, P(w.detach().half())),
            f"{name} pitch": put(layer, name, pitched(w, w.shape[1] + 4)),
            f"{name} base": put(layer, name, pitched(w, w.shape[1], 1)),
            f"{name} inner stride": put(layer, name, P(w.detach().t().contiguous().t())),
            f"{name} shape": put(layer, name, P(torch.zeros(0, device="cuda", dtype=w.dtype))),
            f"{name} device": put(layer, name, P(w.detach().cpu())),
            f"{name} gated": mark(w, "_sxb_gate"),
            f"{name} main gradient": mark(w, "_sxb_grad_ready")})
    norms = [(layer, "input_layernorm"), (layer, "post_attention_layernorm"), (m, "norm")]
    for obj, name in norms:
        w = getattr(obj, name)
        cases.update({
            f"{name} fp32": put(obj, name, P(w.detach().float())),
            f"{name} stride": put(obj, name, P(torch.as_strided(torch.ones(2 * 512, device="cuda", dtype=w.dtype), (512,), (2,)))),
            f"{name} shape": put(obj, name, P(torch.ones(256, device="cuda", dtype=w.dtype)))})
    cases.update({
        "embedding pitch": put(m, "embed_tokens", pitched(m.embed_tokens, 520)),
        "experts": put(ragged, "moe_layers", [{}, {}]),
        "flops counted": put(F, "flop_sink", lambda *a: None),
        "cache fp32": put(ragged.state_manager, "get_cache", every(cache.float())),
        "cache strided": put(ragged.state_manager, "get_cache", every(torch.cat([cache, cache], -1)[..., : cache.shape[-1]])),
        "cache elsewhere": put(ragged.state_manager, "get_cache", every(cache.cpu())),
        "cache in parts": put(ragged.state_manager, "get_cache", every((cache, cache))),
        "dispatch mode": Watcher()})
    taken, real = [], RaggedLlamaModel._native_plan

    def spy(self, batch):
        assert real(self, batch) is not None
        for what, change in cases.items():
            with change:
                if real(self, batch) is not None:
                    taken.append(what)
        plan = real(self, batch)
        assert plan is not None
        return plan

    monkeypatch.setattr(RaggedLlamaModel, "_native_plan", spy)
    eng.put([0, 1], [torch.arange(5, dtype=torch.int32), torch.arange(70, dtype=torch.int32)])
    assert not taken, taken


def test_counts_the_entry_points_it_stands_for(monkeypatch):
    import torch
    from shuffle_exchange_b200.inference.v2.model_implementations.llama_v2 import RaggedLlamaModel
    from shuffle_exchange_b200.native import lib
    model, eng = _engine(512, 4, 2, 1024, 1024, layers=3)
    real, counts = RaggedLlamaModel._native_forward, []

    def counting(s, b, p):
        before = lib.launch_count
        out = real(s, b, p)
        counts.append(lib.launch_count - before)
        return out
    monkeypatch.setattr(RaggedLlamaModel, "_native_forward", counting)
    for n in (1, 600):                       # one row: the gated product takes its activation along
        eng.put([n], [torch.ones(n, dtype=torch.int32)])
    assert counts == [8 * 3 + 4, 9 * 3 + 4]
