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


def _masked(rows, vocab, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = (4 * torch.randn(rows, vocab, generator=g, device="cuda")).bfloat16()
    lo, hi, inf = vocab // 2, vocab - vocab // 4, float("-inf")
    x[0, :lo], x[1, hi:], x[2, : vocab - 1], x[3, lo + 1:], x[3, :lo] = inf, inf, inf, inf, inf
    x[4, :lo] = torch.finfo(torch.bfloat16).min            # the lowest number there is
    x[5::7, ::2] = inf
    labels = torch.full((rows,), vocab - 1, device="cuda")
    labels[1], labels[3] = 0, lo
    return x, labels


def _check(grad, loss, x, labels, gs):
    y = x.double().requires_grad_()
    want = torch.nn.functional.cross_entropy(y, labels, reduction="none")
    want.sum().backward()
    eps = (x.shape[1] / 256 + 8 + 11) * 2.0 ** -24 + 2.0 ** -17         # as above
    assert ((loss.double() - want).abs() <= eps + 3 * want.abs() * 2.0 ** -24 + 40 * 2.0 ** -22).all()
    err = (grad.double() / gs - y.grad).abs()
    assert (err <= y.grad.abs() * (2.0 ** -8 + 2 * eps) + 2 * eps + 2.0 ** -20).all()


@pytest.mark.parametrize("rows", [6, 300])
@pytest.mark.parametrize("vocab", [8, 2048, 8192, 24584, 32768, 49160, 98312])
def test_masked_columns(rows, vocab):
    """Columns at -inf, whole words and whole threads of them, weigh nothing wherever they stand."""
    x, labels = _masked(rows, vocab, vocab)
    for r in range(rows):                                  # a label is one of the columns that count
        if not torch.isfinite(x[r, labels[r]]):
            labels[r] = int(torch.isfinite(x[r]).nonzero()[0])
    leaf = x.clone().requires_grad_()
    loss = F.cross_entropy(leaf * 1, labels)
    loss.backward()
    y = x.double()
    rows_loss = torch.logsumexp(y, 1) - y.gather(1, labels[:, None])[:, 0]
    assert abs(loss.double().item() - rows_loss.mean().item()) <= 2.0 ** -15 * max(1.0, rows_loss.mean().item())
    _check(leaf.grad, rows_loss, x, labels, 1.0 / rows)


@pytest.mark.parametrize("vocab", [5, 13, 2051, 32771])
def test_masked_columns_and_a_last_partial_word(vocab):
    from shuffle_exchange_b200.native import lib
    ld = (vocab + 7) // 8 * 8
    x, labels = _masked(6, vocab, vocab)
    wide = torch.zeros(6, ld, device="cuda", dtype=torch.bfloat16)
    wide[:, :vocab] = x
    loss = torch.empty(6, device="cuda")
    labels[5] = int(torch.isfinite(x[5]).nonzero()[0])
    lib.call("sxb_cross_entropy", wide.data_ptr(), labels.data_ptr(), loss.data_ptr(), None, 6, vocab, ld, -100, None, 1,
             lib.dtype_code(torch.bfloat16), lib.stream_ptr())
    _check(wide[:, :vocab], loss, x, labels, 1.0)
