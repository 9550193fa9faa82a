"""cross_entropy at the edges of its passes: runs of four words per thread, 256, 512 and 1024 threads."""
import pytest
import torch

from shuffle_exchange_b200.ops import functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [3, 300])
@pytest.mark.parametrize("vocab", [8, 2048, 8184, 8192, 8200, 24584, 32760, 32768, 32776, 49160, 65544, 98312])
def test_against_float64(rows, vocab):
    g = torch.Generator(device="cuda").manual_seed(vocab)
    x = (4 * torch.randn(rows, vocab, generator=g, device="cuda")).bfloat16()
    x[0, : vocab // 2] = -1e4                          # a row whose first half weighs nothing
    labels = torch.randint(0, vocab, (rows,), generator=g, device="cuda")
    labels[1] = -100
    y = x.double().requires_grad_()
    want = torch.nn.functional.cross_entropy(y, labels, reduction="sum", ignore_index=-100)
    want.backward()
    leaf = x.clone().requires_grad_()
    got = F.cross_entropy(leaf * 1, labels)          # (consumes its logits)
    got.backward()
    n = rows - 1                                       # the mean over rows with a label
    # a thread adds at most vocab / 256 + 8 terms one by one and the block eleven partial sums, each with 2^-24 of the sum, and
    # every exponential is within 2^-20 of itself here (arguments up to 40, 2^-23 of them, times the base's logarithm)
    eps = (vocab / 256 + 8 + 11) * 2.0 ** -24 + 2.0 ** -17
    # a row's loss (up to 1e4 where the label lies in the light half) and their mean are fp32: 2^-24 of themselves each
    assert abs(got.double() * n - want).item() <= n * (eps + 40 * 2.0 ** -22) + 3 * want.item() * 2.0 ** -24
    err = (leaf.grad.double() * n - y.grad).abs()
    assert (err <= y.grad.abs() * (2.0 ** -8 + 2 * eps) + 2 * eps + 2.0 ** -20).all()
