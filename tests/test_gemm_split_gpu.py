"""Products with few output tiles and a long K, which a cluster shares: every layout, ragged sizes, 16- and 32-bit results, accumulation,
against 64 bits and, bit for bit, against themselves."""
import pytest
import torch

from shuffle_exchange_b200.native import lib as _n
from shuffle_exchange_b200.ops import functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [F.GEMM_NT, F.GEMM_NN, F.GEMM_TN])
@pytest.mark.parametrize("M,N,K", [(8, 264, 8200), (128, 256, 4096), (136, 520, 16384), (200, 1000, 6400), (304, 4096, 7168), (520, 768, 32000)])
@pytest.mark.parametrize("dtype,accumulate", [(torch.bfloat16, False), (torch.float32, False), (torch.float32, True), (torch.bfloat16, True)])
def test_against_64_bits(layout, M, N, K, dtype, accumulate):
    g = torch.Generator(device="cuda").manual_seed(M + K)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    a = mk(K, M) if layout == F.GEMM_TN else mk(M, K)
    b = mk(N, K) if layout == F.GEMM_NT else mk(K, N)
    want = (a.double().t() if layout == F.GEMM_TN else a.double()) @ (b.double().t() if layout == F.GEMM_NT else b.double())
    room = torch.full((M + 1, N + 8), 3.0, device="cuda", dtype=dtype)
    out = room[:M, :N]
    F.gemm(a, b, layout, out=out, accumulate=accumulate, alpha=0.5)
    want = 0.5 * want + (3.0 if accumulate else 0.0)
    # 32-bit sums of K terms in chains of K / 16 S additions that cut off: far below 1e-4; half a unit of the last place of bf16
    bound = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-4
    assert float((out.double() - want).norm() / want.norm()) < bound
    assert float((out.double() - want).abs().max()) < 2 * bound * float(want.abs().max())
    assert bool((room[M:] == 3).all()) and bool((room[:, N:] == 3).all())
    again = torch.full_like(room, 3.0)
    F.gemm(a, b, layout, out=again[:M, :N], accumulate=accumulate, alpha=0.5)
    assert torch.equal(room, again)
    assert _n.hang_any() is None
