"""Grouped product that leaves the padding of its groups out: the rows in use equal the product over the whole room, whatever
the padding holds, and where a group ends in a box of 64 rows, a half or a tile."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts,N,K", [
    ([1, 63, 64, 65], 256, 128), ([128, 129, 0, 191], 264, 192), ([193, 256, 257, 0, 300], 512, 64),
    ([0, 0, 7], 72, 8), ([513, 1], 1000, 1024),
])
def test_rows_in_use_equal_the_whole_product(counts, N, K):
    import torch
    from shuffle_exchange_b200.ops.gemm_ext import grouped_gemm_nt, grouped_gemm_nt_used
    torch.manual_seed(1)
    room = [(c + 255) // 256 * 256 for c in counts]
    off = [0]
    for r in room:
        off.append(off[-1] + r)
    R, G = off[-1] + 256, len(counts)
    used = torch.zeros(R, dtype=torch.bool, device="cuda")
    for o, c in zip(off, counts):
        used[o:o + c] = True
    x = torch.randn(R, K, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(G, N, K, device="cuda", dtype=torch.bfloat16)
    offsets = torch.tensor(off, dtype=torch.int32, device="cuda")
    cnt = torch.tensor(counts, dtype=torch.int32, device="cuda")
    want = grouped_gemm_nt(x, w, offsets)
    x[~used] = float("nan")
    got = grouped_gemm_nt_used(x, w, offsets, cnt, out=torch.full((R, N), 7.0, device="cuda", dtype=torch.bfloat16))
    assert torch.equal(got[used], want[used])            # same tiles and order of sums
    assert torch.equal(got[off[-1]:], torch.full_like(got[off[-1]:], 7.0))
    for o, r, c in zip(off, room, counts):               # whole boxes of 64 rows behind the last row in use: not written
        lo = o + (c + 63) // 64 * 64
        assert torch.equal(got[lo:o + r], torch.full_like(got[lo:o + r], 7.0))
