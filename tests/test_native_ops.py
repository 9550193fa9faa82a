"""The differentiable operators in C++ against the same operators as Python autograd functions: same bits in results and gradients,
and out of the way wherever something other than autograd watches."""
import pytest
import torch

from shuffle_exchange_b200.native import lib
from shuffle_exchange_b200.ops import functional as F

needs_ops = pytest.mark.skipif(lib.OPS is None, reason="_sxb_ops.so is not built here")


@needs_ops
def test_nothing_but_plain_gpu_tensors():
    x, w = torch.ones(4, 8, dtype=torch.bfloat16), torch.ones(16, 8, dtype=torch.bfloat16)
    one, cos = torch.ones(8, dtype=torch.bfloat16), torch.ones(4, 4)
    assert lib.OPS.linear(x, w) is None and lib.OPS.linear(None, 3) is None and lib.OPS.linear(x) is None
    assert lib.OPS.rms_norm(x, one, 1e-5, None) is None and lib.OPS.gated_act(x, 3) is None
    assert lib.OPS.rope(x, None, cos, cos, 1, 8) is None and lib.OPS.attention_qkv(x[None], 1, 1, 64, True, 1.0) is None
    assert F.linear(x, w).shape == (4, 16)


OPS = ["linear", "norm", "norm_residual", "gated", "rope", "rope_behind", "attention"]


def _make(op, shape=(2, 37), grad=True):
    g = torch.Generator(device="cuda").manual_seed(3)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16).requires_grad_(grad)  # noqa: E731
    if op == "linear":
        a = [mk(*shape, 64), mk(48, 64)]
        return a, lambda x, w: [F.linear(x, w)]
    if op.startswith("norm"):
        a = [mk(*shape, 72), mk(72)] + ([mk(*shape, 72)] if "res" in op else [])
        return a, lambda x, w, r=None: list(F.rms_norm(x, w, 1e-5, r))[: 1 if r is None else 2]
    if op == "gated":
        return [mk(*shape, 128)], lambda x: [F.gated_act(x, "silu")]
    cos, sin = F.rope_tables(64, 64, 10000.0, torch.device("cuda"))
    if op.startswith("rope"):                        # behind the heads: sixteen columns at a time, or some that are not
        pos = torch.arange(shape[1], device="cuda").repeat(shape[0])
        return [mk(*shape, 3 * 64 if op == "rope" else 2 * 64 + 8)], lambda x: [F.rope(x * 1, pos, cos, sin, 2, 64)]
    return [mk(*shape, 4 * 64)], lambda x: [F.flash_attention_qkv(x, 2, 1, 64)]


def _both(op, monkeypatch, step):
    res = []
    lib.load()                                      # which binds them
    for native in (True, False):
        with monkeypatch.context() as m:
            if not native:
                m.setattr(F, "_ops", None)
            args, f = _make(op)
            before = lib.OPS.calls()
            res.append(step(args, f))
            assert (lib.OPS.calls() > before) == native
    return res


def _step(args, f):
    out = f(*args)
    g = torch.Generator(device="cuda").manual_seed(5)
    torch.autograd.backward(out, [torch.randn(o.shape, generator=g, device="cuda").to(o.dtype) for o in out])
    return [o.detach() for o in out] + [a.grad for a in args]


@pytest.mark.gpu
def test_a_product_may_be_the_first_call_of_a_thread():
    import threading
    lib.load()
    (x, w), f = _make("linear", grad=False)
    want, rc = f(x, w)[0], []
    got = torch.full_like(want, float("nan"))
    t = threading.Thread(target=lambda: rc.append(lib.call(
        "sxb_gemm_bf16", x.data_ptr(), w.data_ptr(), got.data_ptr(), 74, 48, 64, 0, 64, 64, 48, lib.BF16, 0, 1.0, 0, 0)))
    torch.cuda.synchronize()
    t.start(), t.join()
    torch.cuda.synchronize()
    assert rc == [0] and torch.equal(got, want)


@needs_ops
@pytest.mark.gpu
@pytest.mark.parametrize("op", OPS)
def test_same_bits_as_python(op, monkeypatch):
    a, b = _both(op, monkeypatch, _step)
    assert len(a) == len(b) and all(torch.equal(x, y) for x, y in zip(a, b))


@needs_ops
@pytest.mark.gpu
@pytest.mark.parametrize("op", OPS)
def test_saved_tensors_go_through_hooks_and_checkpoints(op, monkeypatch):
    from torch.utils.checkpoint import checkpoint

    def hooked(args, f):
        seen = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: (seen.append(1), t.cpu())[1], lambda t: t.cuda()):
            r = _step(args, f)
        assert seen
        return r
    a, b = _both(op, monkeypatch, hooked)
    assert all(torch.equal(x, y) for x, y in zip(a, b))
    c, d = _both(op, monkeypatch, lambda args, f: _step(args, lambda *x: checkpoint(f, *x, use_reentrant=False)))
    assert all(torch.equal(x, y) for x, y in zip(a, c)) and all(torch.equal(x, y) for x, y in zip(a, d))


@needs_ops
@pytest.mark.gpu
@pytest.mark.parametrize("frozen", [0, 1])
def test_only_wanted_gradients_and_missing_ones(frozen):
    (x, w, r), f = _make("norm_residual")
    y, h = f(x, w, r)
    h.float().sum().backward()                      # nothing arrives at y
    assert torch.equal(x.grad, torch.ones_like(x)) and torch.equal(r.grad, x.grad) and not w.grad.any()
    args, f = _make("linear")
    args[frozen].requires_grad_(False)
    before = lib.OPS.calls()
    f(*args)[0].float().sum().backward()
    assert args[frozen].grad is None and args[1 - frozen].grad is not None and lib.OPS.calls() == before + 2


@needs_ops
@pytest.mark.gpu
def test_watched_calls_and_marked_weights_stay_in_python():
    (x, w), f = _make("linear", grad=False)
    calls = lib.OPS.calls
    f(x, w)
    n = calls()
    w._sxb_main_grad = None                         # a weight of the main-grad protocol, bound or not
    f(x, w)
    del w._sxb_main_grad
    f(x[..., 1:][..., :56], w[:, :56])              # rows that are not 16-byte aligned are copied first
    f(x[:0], w)                                     # no rows
    assert calls() == n and F.linear(x.float(), w.float()).dtype == torch.float32 and calls() == n
    import torch.autograd.forward_ad as fwAD
    with fwAD.dual_level():
        f(x, w)
    from torch.utils._python_dispatch import TorchDispatchMode

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))
    with Mode():
        f(x, w)
    assert calls() == n
    f(x, w)
    assert calls() == n + 1


@needs_ops
@pytest.mark.gpu
def test_changed_operands_are_noticed_and_refusals_are_the_bindings():
    (x, w), f = _make("linear")
    y = f(x, w)[0]
    with torch.no_grad():
        w.add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.float().sum().backward()
    (q,), f = _make("rope")
    z = q * 1
    v = z._version
    cos, sin = F.rope_tables(64, 64, 10000.0, torch.device("cuda"))
    out = F.rope(z, None, cos, sin, 2, 64)
    assert out is z and z._version == v + 1
    with pytest.raises(lib.NativeError):
        F.rope(z.detach().requires_grad_() * 1, None, cos, sin, 1, 33)


@needs_ops
@pytest.mark.gpu
def test_a_call_refused_in_backward_is_the_bindings_error():
    (x, w), f = _make("linear", shape=(1,))
    y = f(x, w)[0]
    calls = lib.OPS.calls()
    with pytest.raises(lib.NativeError, match="unsupported shape/alignment"):
        y.backward(torch.zeros(1, 56, dtype=torch.bfloat16, device="cuda")[:, 1:49])       # a row that starts two bytes off
    assert lib.OPS.calls() == calls + 1 and x.grad is None and w.grad is None


@needs_ops
@pytest.mark.gpu
@pytest.mark.parametrize("op", ["linear", "norm", "norm_residual"])
def test_a_weight_bound_after_the_forward_delivers_like_pythons(op, monkeypatch):
    def bound(args, f):
        w, ready = args[1], []
        out = f(*args)
        w._sxb_main_grad = torch.full(w.shape, 2.0, dtype=torch.float32 if op == "linear" else w.dtype, device="cuda")
        w._sxb_grad_ready, w._sxb_grad_written = lambda p: ready.append(p is w), True          # adds to what is there
        out[0].backward(torch.ones_like(out[0]))
        assert ready == [True] and w.grad is None
        return [w._sxb_main_grad] + [a.grad for a in args if a is not w]
    a, b = _both(op, monkeypatch, bound)
    assert all(torch.equal(x, y) for x, y in zip(a, b)) and bool((a[0] != 2).any())

    def refusing(p):
        raise KeyError("not now")
    args, f = _make(op)
    out = f(*args)[0]
    args[1]._sxb_main_grad, args[1]._sxb_grad_ready = torch.zeros_like(args[1]), refusing
    with pytest.raises(KeyError, match="not now"):
        out.backward(torch.ones_like(out))


@needs_ops
@pytest.mark.gpu
def test_attention_tells_its_ranks_in_both_directions():
    (x,), f = _make("attention")
    asked = []
    lib.OPS.backward_side(F._linear_bwd, F._rms_norm_bwd, lambda: asked.append(1))
    try:
        f(x)[0].float().sum().backward()
    finally:
        lib.OPS.backward_side(F._linear_bwd, F._rms_norm_bwd, lib.know_ranks)
    assert asked == [1] and x.grad is not None
