"""Operators that go straight to their kernel when nothing watches them: when that may happen (``native.lib.no_tape``), and
that they then give what the autograd function gives."""
import pytest
import torch
import torch.autograd.forward_ad as fwd_ad
from torch.utils._python_dispatch import TorchDispatchMode

from shuffle_exchange_b200.native import lib
from shuffle_exchange_b200.ops import functional as F


class _Quiet(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


def test_when_nothing_watches():
    x, w = torch.ones(3), torch.ones(3, requires_grad=True)
    assert lib.no_tape(x) and lib.no_tape(x, None) and not lib.no_tape(x, w)
    with torch.no_grad():
        assert lib.no_tape(x, w)
        with fwd_ad.dual_level():
            assert not lib.no_tape(x)
        with _Quiet():
            assert not lib.no_tape(x)
        seen = []
        torch.vmap(lambda t: (seen.append(lib.no_tape(t)), t)[1])(torch.ones(2, 3))
        torch.jit.trace(lambda t: (seen.append(lib.no_tape(t)), t + 1)[1], x, check_trace=False)
        assert seen == [False, False]
        assert lib.no_tape(x)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 64), (7, 64), (2, 3, 64), (64,)])
def test_same_bits_with_and_without_the_tape(shape):
    g = torch.Generator(device="cuda").manual_seed(1)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    x, r, w, b, gain = mk(*shape), mk(*shape), mk(40, 64), mk(40), mk(64)
    calls = [lambda t: F.linear(t, w), lambda t: F.linear(t, w, b), lambda t: F.rms_norm(t, gain, 1e-5)[0],
             lambda t: F.rms_norm(t, gain, 1e-5, r), lambda t: F.swiglu(t), lambda t: F.gated_act(t, "gelu")]
    for f in calls:
        with torch.no_grad():
            fast = f(x)
        taped = f(x.clone().requires_grad_())
        for a, c in zip(fast if isinstance(fast, tuple) else (fast,), taped if isinstance(taped, tuple) else (taped,)):
            assert a.shape == c.shape and a.stride() == c.stride() and torch.equal(a, c) and not a.requires_grad


@pytest.mark.gpu
def test_forward_mode_and_vmap_stay_refused():
    x, w = torch.randn(4, 64, device="cuda").bfloat16(), torch.randn(8, 64, device="cuda").bfloat16()
    with torch.no_grad(), fwd_ad.dual_level(), pytest.raises(Exception):
        F.linear(fwd_ad.make_dual(x, torch.ones_like(x)), w)
    with torch.no_grad(), pytest.raises(Exception):
        torch.vmap(lambda t: F.rms_norm(t, w[0], 1e-5)[0])(x[None])


@pytest.mark.gpu
def test_kernels_follow_the_current_stream():
    s = torch.cuda.Stream()
    assert lib.stream_ptr() == torch.cuda.current_stream().cuda_stream
    with torch.cuda.stream(s):
        assert lib.stream_ptr() == s.cuda_stream
