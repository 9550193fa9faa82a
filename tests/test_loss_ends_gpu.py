"""The ends of the mean cross entropy (labels that count, mean of the rows' losses) against 64 bits."""
import pytest
import torch

from shuffle_exchange_b200.ops import functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 31, 1024, 1025, 5000])
@pytest.mark.parametrize("ignored", [0, 0.3, 1])
def test_mean_loss(rows, ignored):
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = (torch.randn(rows, 64, generator=g, device="cuda") * 2).to(torch.bfloat16).requires_grad_()
    labels = torch.randint(0, 64, (rows,), generator=g, device="cuda")
    labels[torch.rand(rows, generator=g, device="cuda") < ignored] = -7
    ref = x.detach().double().requires_grad_()
    want = torch.nn.functional.cross_entropy(ref, labels, ignore_index=-7, reduction="sum") / max(1, int((labels != -7).sum()))
    for lab in (labels, labels.int()):
        y = x.detach().clone().requires_grad_()
        loss = F.cross_entropy(y * 1, lab, ignore_index=-7)
        loss.backward()
        assert loss.shape == () and abs(float(loss) - float(want)) <= 1e-5 * max(1.0, float(want))
    want.backward()
    assert float((y.grad.double() - ref.grad).abs().max()) <= 2.0 ** -8 * float(ref.grad.abs().max()) + 1e-12
