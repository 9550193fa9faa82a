"""Products of few rows with the weights as the MMA's rows: groups at the edges of boxes of 32 rows, tiles and turns, with and
without the gated activation behind them, and the single product that ends in one."""
import pytest
import torch

from shuffle_exchange_b200.native import lib as _n
from shuffle_exchange_b200.ops import functional as F
from shuffle_exchange_b200.ops import gemm_ext

pytestmark = pytest.mark.gpu
ACTS = {0: lambda t: t, 1: torch.relu, 2: lambda t: torch.nn.functional.gelu(t, approximate="tanh"), 3: torch.nn.functional.silu}


def _groups(counts, K, seed=1):
    g = torch.Generator(device="cuda").manual_seed(seed)
    off = [0]
    for c in counts:
        off.append(off[-1] + (c + 255) // 256 * 256)
    x = torch.full((off[-1] + 256, K), float("nan"), device="cuda", dtype=torch.bfloat16)       # padding is not used
    for o, c in zip(off, counts):
        x[o:o + c] = torch.randn(c, K, generator=g, device="cuda").to(torch.bfloat16)
    return x, off, torch.tensor(off, dtype=torch.int32, device="cuda"), torch.tensor(counts, dtype=torch.int32, device="cuda"), g


@pytest.mark.parametrize("counts,N,K", [
    ([1, 31, 32, 33, 0, 64], 256, 128), ([127, 128, 129], 264, 200), ([0, 255, 1, 256, 257], 136, 64), ([513, 2], 72, 72),
    ([5, 0, 0, 7], 1000, 8), ([3, 20], 128, 4096), ([1], 64, 2048), ([40] * 8, 2048, 1024),
])
def test_groups(counts, N, K, monkeypatch):
    monkeypatch.setattr(gemm_ext, "FEW_ROWS", 1 << 20)
    x, off, offsets, cnt, g = _groups(counts, K)
    w = (torch.randn(len(counts), N, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    for routed in (sum(counts), sum(counts) + 300):          # an upper bound
        out = torch.full((x.shape[0], N), 7.0, device="cuda", dtype=torch.bfloat16)
        gemm_ext.grouped_gemm_nt_used(x, w, offsets, cnt, out=out, routed=routed)
        used = torch.zeros(x.shape[0], dtype=torch.bool, device="cuda")
        for e, (o, c) in enumerate(zip(off, counts)):
            if c:
                used[o:o + c] = True
                want = x[o:o + c].double() @ w[e].double().t()
                # half a unit of bf16's last place, and the 32-bit sums behind it
                assert float((out[o:o + c].double() - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max()) + 1e-5
        assert bool((out[~used] == 7).all())
    assert _n.hang_any() is None


@pytest.mark.parametrize("counts,Fw,K", [([1, 33, 0, 64], 64, 128), ([129, 300, 5], 136, 72), ([40] * 8, 1024, 512), ([2], 200, 2048)])
@pytest.mark.parametrize("act", [0, 1, 2, 3])
def test_groups_with_their_activation(counts, Fw, K, act, monkeypatch):
    monkeypatch.setattr(gemm_ext, "FEW_ROWS", 1 << 20)
    x, off, offsets, cnt, g = _groups(counts, K)
    w = (torch.randn(len(counts), 2 * Fw, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    got = gemm_ext.grouped_gated_nt_few(x, w, offsets, cnt, act, sum(counts))
    h = gemm_ext.grouped_gemm_nt_used(x, w, offsets, cnt, routed=sum(counts))
    for o, c in zip(off, counts):
        if c:
            one = F.gated_act(h[o:o + c].clone(), act)
            want = ACTS[act](h[o:o + c, :Fw].double()) * h[o:o + c, Fw:].double()
            assert float((got[o:o + c].double() - want).abs().max()) <= 2.0 ** -7 * float(want.abs().max()) + 1e-5
            if Fw % 64 == 0:                                  # the same tiles: the product's bits, then the activation's
                assert torch.equal(got[o:o + c], one)
    assert gemm_ext.grouped_gated_nt_few(x, w[:, :-8], offsets, cnt, act, sum(counts)) is None or (2 * Fw - 8) % 16 == 0


@pytest.mark.parametrize("M", [1, 16, 17, 32, 33, 64, 65, 128, 200])
@pytest.mark.parametrize("Fw,K", [(64, 1024), (2048, 4096), (704, 1536)])
def test_one_product_with_its_activation(M, Fw, K):
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(2 * Fw, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    out = torch.full((M + 1, Fw), 7.0, device="cuda", dtype=torch.bfloat16)
    rc = _n.load().sxb_gemm_gated(x.data_ptr(), w.data_ptr(), out.data_ptr(), M, Fw, K, K, K, Fw, 3, _n.stream_ptr())
    if rc == -2:                                              # too many rows: product and activation one after the other
        assert M > 32
        return
    assert rc == 0 and torch.equal(out[:M], F.gated_act(F.linear(x, w), "silu")) and bool((out[M:] == 7).all())


@pytest.mark.parametrize("longest,few", [(None, True), (256, True), (257, False)])
def test_long_groups_keep_to_the_kernel_that_reads_the_weights_once(longest, few, monkeypatch):
    counts = [250, 3, 0, 5, 7]                                # 53 a group on average
    x, off, offsets, cnt, g = _groups(counts, 64)
    w = torch.randn(5, 64, 64, generator=g, device="cuda").to(torch.bfloat16)
    names, real = [], _n.call
    monkeypatch.setattr(gemm_ext._n, "call", lambda name, *a: (names.append(name), real(name, *a))[1])
    y = gemm_ext.grouped_gemm_nt_used(x, w, offsets, cnt, routed=265, longest=longest)
    assert (names == ["sxb_gemm_grouped_few"]) == few and (names == ["sxb_gemm_grouped_used"]) != few
    gated = gemm_ext.grouped_gated_nt_few(x, w, offsets, cnt, 3, 265, longest)
    assert (gated is not None) == few and gemm_ext.grouped_gated_nt_few(x, w, offsets, cnt, 3, 321, longest) is None
    for e, (o, c) in enumerate(zip(off, counts)):
        want = x[o:o + c].double() @ w[e].double().t()
        assert not c or float((y[o:o + c].double() - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max()) + 1e-5


def test_refusals():
    x, _, offsets, cnt, g = _groups([3, 4], 64)
    w = torch.zeros(2, 64, 64, device="cuda", dtype=torch.bfloat16)
    out = torch.zeros(x.shape[0], 64, device="cuda", dtype=torch.bfloat16)
    call = lambda act=-1, ldc=64, shift=0: _n.load().sxb_gemm_grouped_few(  # noqa: E731
        x.data_ptr(), w.data_ptr(), out.data_ptr() + shift, 64, 64, 64, 64, ldc, 2, offsets.data_ptr(), cnt.data_ptr(), x.shape[0], 7,
        act, _n.stream_ptr())
    assert call() == 0 and call(act=4) == -1 and call(ldc=60) == -2 and call(shift=2) == -2
    torch.cuda.synchronize()
