"""The router's 32-bit product over tokens and rows at the edges of its CTAs, against 64 bits."""
import pytest
import torch

from shuffle_exchange_b200.inference.v2.kernels import mixer_ops as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [1, 2, 3, 4, 5, 33, 200, 1500])
@pytest.mark.parametrize("R,width", [(1, 4), (3, 1020), (8, 1024), (8, 4096), (9, 1028), (16, 2048)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_router(tokens, R, width, dtype):
    g = torch.Generator(device="cuda").manual_seed(tokens + R)
    x = torch.randn(tokens, width + 8, generator=g, device="cuda").to(dtype)[:, :width]
    w, b = torch.randn(R, width, generator=g, device="cuda") * width ** -0.5, torch.randn(R, generator=g, device="cuda")
    for bias in (b, None):
        got = M.router_logits(x, w, bias)
        want = x.double() @ w.double().t() + (0 if bias is None else bias.double())
        # 32-bit sums: of at most width / 256 + 13 additions one behind the other
        assert float((got.double() - want).abs().max()) < 2.0 ** -23 * (width / 256 + 16) * float((x.double().abs() @ w.double().abs().t()).max())
