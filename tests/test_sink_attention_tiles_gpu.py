"""Tiles of the sink attention on the tensor cores: portions around the rows of a warp and of a tile, rings that wrap, keys that
begin anywhere in pages of any size."""
import pytest
import torch

from test_sink_attention_mma_gpu import _batch, _oracle
from shuffle_exchange_b200.inference.v2.kernels import mixer_ops as M
from shuffle_exchange_b200.native import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,dv", [(64, 64), (128, 128), (64, 128), (128, 64)])
@pytest.mark.parametrize("page,chunk,window", [(16, 0, 0), (48, 0, 129), (64, 128, 0), (7, 0, 64), (256, 100, 0)])
def test_edges(d, dv, page, chunk, window):
    plan = [(0, 31), (1, 32), (63, 33), (64, 64), (300, 65), (511, 127), (129, 128), (0, 256 + 17)]
    b, pages = _batch(plan, page)
    g = torch.Generator(device="cuda").manual_seed(page + d)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    T = sum(n for _, n in plan)
    q, kc, vc, sink = mk(T, 2, d), mk(pages, page, 1, d).bfloat16(), mk(pages, page, 1, dv).bfloat16(), mk(2)
    y = M.sink_attention(q, kc, vc, sink, b.token_to_seq(), b.token_positions(), b.block_tables(), d ** -0.5, chunk,
                         torch.bfloat16, b.atoms(), b.atoms_longer_than(M.SHORT_ATOM), window=window)
    want = _oracle(q, kc, vc, b, plan, page, d ** -0.5, chunk, window, sink, None, None)
    # half a unit of the 16-bit result, and scores that are 32-bit sums of d terms around 1
    assert bool(((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + (d ** 0.5 * 4 + 4) * 2.0 ** -20 * 6).all())
    assert lib.hang_info("seqmix") is None
