"""Products of few rows against a whole weight (csrc/gemm_skinny.cuh): edges of its token tiles, of the 128-row weight tiles,
of the 64-wide blocks of K and of the cluster splits, both output types, accumulation, padded pitches; the rule that
chooses it is checked by running the automatic route at the same sizes."""
import pytest
import torch

from shuffle_exchange_b200.native import lib
from shuffle_exchange_b200.ops import functional as F

pytestmark = pytest.mark.gpu

SIZES = [(1, 8, 8), (1, 128, 64), (15, 136, 72), (16, 768, 768), (17, 1000, 520), (32, 2048, 1536), (33, 3072, 2048), (64, 640, 4096),
         (65, 4096, 4096), (127, 2056, 8192), (128, 128, 64), (129, 768, 2048), (257, 520, 2048), (512, 2048, 2048), (3, 19072, 256)]


def _case(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N + K)
    x = torch.randn(M, K + 8, generator=g, device="cuda").bfloat16()[:, :K]          # a padded pitch
    w = torch.randn(N, K, generator=g, device="cuda").bfloat16()
    ref = x.double() @ w.double().t()
    # products of two bf16 are exact in fp32; a sum of K of them, in any order and with truncating adders, is off by at
    # most K units of the last place of the sum of magnitudes
    bound = (K + 8) * 2.0 ** -23 * (x.double().abs() @ w.double().abs().t())
    return x, w, ref, bound


@pytest.fixture(params=[3, 0], ids=["skinny", "auto"])
def mode(request):
    lib.load()
    lib.call("sxb_gemm_set_mode", request.param)
    yield request.param
    lib.call("sxb_gemm_set_mode", 0)
    assert lib.hang_info("gemm") is None


@pytest.mark.parametrize("M,N,K", SIZES)
def test_skinny_product(mode, M, N, K):
    x, w, ref, bound = _case(M, N, K)
    for dt in (torch.float32, torch.bfloat16):
        full = torch.full((M, N + 3), 7.0, dtype=dt, device="cuda")      # a pitch without alignment: scalar stores
        for out in (full[:, :N], torch.empty(M, N, dtype=dt, device="cuda")):
            F.gemm(x, w, F.GEMM_NT, out=out)
            assert bool(((out.double() - ref).abs() <= bound + (2.0 ** -8 * ref.abs() if dt == torch.bfloat16 else 0)).all())
        assert bool((full[:, N:] == 7.0).all())
    again = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    F.gemm(x, w, F.GEMM_NT, out=again)
    assert torch.equal(again, out)                                        # the same bits on every run
    acc = torch.randn(M, N, device="cuda")
    before = acc.clone()
    F.gemm(x, w, F.GEMM_NT, out=acc, accumulate=True, alpha=0.5)
    want = before.double() + 0.5 * ref
    assert bool(((acc.double() - want).abs() <= 0.5 * bound + 2.0 ** -23 * (want.abs() + before.abs())).all())


@pytest.mark.parametrize("M,N,K", SIZES + [(48, 4096, 4096), (5, 256, 14336)])
def test_partial_sums_keep_32_bits(mode, M, N, K):
    """Small integers: every partial sum stays below 2^24, so fp32 holds it exactly in any order and split, and 16 bits would
    not.  Over random numbers the error is that of fp32 additions (2^-23 each at most, the signs mixed: 1.6e-5 measured for
    one chain of 14336 in the tensor core); 16-bit partial sums would show 1e-3."""
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x, w = (torch.randint(-8, 9, s, generator=g, device="cuda").bfloat16() for s in ((M, K), (N, K)))
    want = x.double() @ w.double().t()
    assert float((x.double().abs() @ w.double().abs().t()).max()) < 2.0 ** 24
    y = F.gemm(x, w, F.GEMM_NT, out_dtype=torch.float32)
    assert torch.equal(y.double(), want)
    y = want.float() + 1.0
    F.gemm(x, w, F.GEMM_NT, out=y, accumulate=True, alpha=0.5)
    assert torch.equal(y.double(), 1.5 * want + 1.0)
    x, w, ref, _ = _case(M, N, K)
    y = F.gemm(x, w, F.GEMM_NT, out_dtype=torch.float32)
    assert float((y.double() - ref).norm() / ref.norm()) < 2e-5
    y = torch.randn(M, N, device="cuda")
    want = y.double() + ref
    F.gemm(x, w, F.GEMM_NT, out=y, accumulate=True)
    assert float((y.double() - want).norm() / want.norm()) < 2e-5


def test_not_finite_values_stay_in_their_rows():
    x, w, ref, bound = _case(20, 512, 1024)
    x = x.clone()
    x[3, 5] = float("inf")
    x[7, 9] = float("nan")
    y = F.gemm(x, w, F.GEMM_NT, out_dtype=torch.float32)
    keep = torch.ones(20, dtype=torch.bool, device="cuda")
    keep[3] = keep[7] = False
    assert not bool(torch.isfinite(y[3]).any()) and bool(torch.isnan(y[7]).all())
    assert bool(((y.double() - ref).abs() <= bound)[keep].all())
