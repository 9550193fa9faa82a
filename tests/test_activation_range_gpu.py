"""SiLU gates over the whole range of bf16: as accurate where the result is tiny as anywhere else."""
import pytest
import torch

from shuffle_exchange_b200.ops import functional as F

pytestmark = pytest.mark.gpu


def _gates(lo, hi):
    x = torch.arange(1 << 16, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    return x[(x >= lo) & (x <= hi) & (x.abs() > 1e-30)].cuda()


@pytest.mark.parametrize("lo,hi", [(-88.5, -80.0), (-80.0, -2.0), (-1.0, 80.0)])
def test_value_and_derivative(lo, hi):
    # e^88.5 is the last power of e below the largest fp32; around -1.28 the derivative's sum cancels
    x = _gates(lo, hi)
    pad = -x.numel() % 8
    g = torch.cat([x, x.new_zeros(pad)])
    row = torch.cat([g, torch.ones_like(g)])[None].requires_grad_()
    y = F.gated_act(row, "silu")
    y.backward(torch.ones_like(y))
    d = x.double()
    s = torch.sigmoid(d)
    # half a unit of the last of bf16's eight bits, and what e^x loses by its argument in 32 bits: |x| units
    tol = 2.0 ** -8 + 100 * 2.0 ** -23
    for got, want in ((y[0, : x.numel()], d * s), (row.grad[0, : x.numel()], s * (1 + d * (1 - s)))):
        assert bool(((got.double() - want).abs() <= tol * want.abs()).all())
