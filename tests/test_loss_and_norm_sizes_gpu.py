"""The scaled gradient of the loss, norm backward with its partial sums in registers, and the routed rows' activation: sizes
at the edges of their blocks, against 64-bit references."""
import pytest
import torch

from shuffle_exchange_b200.moe import fused_ep  # noqa: F401  (declares the routed rows' entry point)
from shuffle_exchange_b200.native import lib
from shuffle_exchange_b200.ops import functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [8, 1024, 32000, 128256])
@pytest.mark.parametrize("scale", [1.0, 0.37, 0.0])
def test_gradient_of_a_scaled_loss(V, scale):
    g = torch.Generator(device="cuda").manual_seed(V)
    x = (3 * torch.randn(5, V, generator=g, device="cuda")).bfloat16()
    labels = torch.tensor([V - 1, V // 2, 2, 0, -100], device="cuda")
    a = x.clone().requires_grad_()
    (F.cross_entropy(a * 1, labels) * scale).backward()       # the logits buffer is consumed
    b = x.double().requires_grad_()
    want = torch.nn.functional.cross_entropy(b, labels)
    (want * scale).backward()
    loss = F.cross_entropy(x.clone(), labels)
    assert abs(float(loss) - float(want)) < 1e-5 * max(1.0, abs(float(want)))
    f = float(torch.tensor(scale).bfloat16())                  # the loss's gradient is rounded to the logits' type first
    err = (a.grad.double() - (b.grad * (f / scale) if scale else 0 * b.grad)).abs()
    # two roundings to 16 bits, and a probability that is off by the exponential's relative 2^-20
    assert bool((err <= 2.0 ** -7 * b.grad.abs() + 2.0 ** -20).all())


def test_scale_that_is_not_a_number_reaches_the_gradient():
    x = torch.randn(3, 64, device="cuda").bfloat16().requires_grad_()
    (F.cross_entropy(x * 1, torch.tensor([1, 2, 3], device="cuda")) * float("nan")).backward()
    assert bool(x.grad.isnan().all())


@pytest.mark.parametrize("scale", [1.0, 0.5])
def test_second_pass_through_a_loss_is_refused(scale):
    """The first pass scales the gradient where it is saved; a second one would scale it again."""
    x = torch.randn(5, 1024, device="cuda").bfloat16().requires_grad_()
    labels = torch.arange(5, device="cuda")
    loss = F.cross_entropy(x * 1, labels) * scale
    loss.backward(retain_graph=True)
    first = x.grad.clone()
    with pytest.raises(RuntimeError, match="inplace"):
        loss.backward()
    assert torch.equal(x.grad, first)
    loss = F.cross_entropy(x * 1, labels) * scale
    torch.autograd.grad(loss, x, retain_graph=True)
    with pytest.raises(RuntimeError, match="inplace"):
        torch.autograd.grad(loss, x)


@pytest.mark.parametrize("rows", [1, 7, 296, 297, 1500])
@pytest.mark.parametrize("H", [8, 768, 2048, 2056, 4096, 5120, 8192, 16384])
@pytest.mark.parametrize("layer", [False, True])
def test_norm_backward(rows, H, layer):
    if rows > 300 and H > 4096:
        pytest.skip("covered by the narrower rows")
    g = torch.Generator(device="cuda").manual_seed(rows + H)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    x, r, w, b, dy, dh = mk(rows, H), mk(rows, H), mk(H), mk(H), mk(rows, H), mk(rows, H)
    ins = [t.clone().requires_grad_() for t in (x, r, w, b)]
    y, h = F.layer_norm(ins[0], ins[2], ins[3], 1e-5, ins[1]) if layer else F.rms_norm(ins[0], ins[2], 1e-5, ins[1])
    torch.autograd.backward([y, h], [dy, dh])
    ref = [t.double().requires_grad_() for t in (x, r, w, b)]
    s = ref[0] + ref[1]
    hd = s + ((x.float() + r.float()).bfloat16().double() - s).detach()        # the stream is stored in 16 bits
    if layer:
        yd = torch.nn.functional.layer_norm(hd, (H,), ref[2], ref[3], 1e-5)
    else:
        yd = hd * torch.rsqrt(hd.square().mean(-1, keepdim=True) + 1e-5) * ref[2]
    torch.autograd.backward([yd, hd], [dy.double(), dh.double()])
    for a, c in zip(ins[: 4 if layer else 3], ref):
        assert float((a.grad.double() - c.grad).norm() / c.grad.norm()) < 4e-3          # one rounding to 16 bits (1.7e-3)


@pytest.mark.parametrize("H", [768, 8192, 8200])
@pytest.mark.parametrize("layer", [False, True])
def test_norm_backward_with_scratch_that_starts_anywhere(H, layer):
    rows = 300
    mk = lambda *s: torch.randn(*s, device="cuda").bfloat16()  # noqa: E731
    dy, x, w = mk(rows, H), mk(rows, H), mk(H)
    mean, rstd = torch.zeros(rows, device="cuda"), torch.ones(rows, device="cuda")
    room = torch.empty(lib.call("sxb_norm_bwd_scratch_elems", rows, H, int(layer)) + 4, device="cuda")
    got = []
    for at in range(4):
        dx, dw, db = torch.empty_like(x), torch.empty_like(w), torch.empty_like(w)
        tail = (room[at:].data_ptr(), rows, H, lib.dtype_code(x.dtype), 0, lib.stream_ptr())
        if layer:
            lib.call("sxb_layernorm_bwd", dy.data_ptr(), x.data_ptr(), w.data_ptr(), mean.data_ptr(), rstd.data_ptr(), None,
                     dx.data_ptr(), dw.data_ptr(), db.data_ptr(), *tail)
        else:
            lib.call("sxb_rmsnorm_bwd", dy.data_ptr(), x.data_ptr(), w.data_ptr(), rstd.data_ptr(), None, dx.data_ptr(),
                     dw.data_ptr(), *tail)
        got.append((dx, dw, db) if layer else (dx, dw))
    for other in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], other))


@pytest.mark.parametrize("counts", [[3, 0, 5], [0, 0, 1], [1] * 40, [300, 2]])
@pytest.mark.parametrize("width", [16, 2056, 4096])
def test_routed_rows_activation(counts, width):
    offs, at = [], 0
    for c in counts:
        offs.append(at)
        at += (c + 255) // 256 * 256
    x = torch.randn(max(at, 256), 2 * width, device="cuda").bfloat16()
    out = torch.full((x.shape[0], width), 5.0, device="cuda", dtype=torch.bfloat16)
    o, c = (torch.tensor(t, dtype=torch.int32, device="cuda") for t in (offs, counts))
    lib.call("sxb_gated_act_groups", x.data_ptr(), out.data_ptr(), o.data_ptr(), c.data_ptr(), len(counts), sum(counts) + 2, width,
             3, lib.dtype_code(x.dtype), lib.stream_ptr())
    want = F.swiglu(x)
    used = torch.zeros(x.shape[0], dtype=torch.bool, device="cuda")
    for a, n in zip(offs, counts):
        used[a: a + n] = True
    assert torch.equal(out[used], want[used]) and bool((out[~used] == 5.0).all())
