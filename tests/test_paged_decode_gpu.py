"""Attention of few queries per sequence over the paged cache (csrc/attention_decode.cu) against a 64-bit oracle: groups, head
sizes, pages, contexts at the edges of its 16-key steps, many and few sequences (cluster sizes), and beside prompt portions."""
import pytest
import torch

from shuffle_exchange_b200.inference.v2.kernels import ragged_ops as R
from shuffle_exchange_b200.inference.v2.ragged.ragged_wrapper import RaggedBatchWrapper
from shuffle_exchange_b200.native import lib

pytestmark = pytest.mark.gpu


class _Seq:
    def __init__(self, seen, pages):
        self.seen_tokens, self._pages = seen, torch.tensor(pages, dtype=torch.int32)

    def kv_blocks(self):
        return self._pages


CASES = [
    # (tokens seen, tokens of this step) per sequence, page, query heads, kv heads, head size
    ([(0, 1), (14, 1), (15, 1), (16, 1), (63, 1), (64, 1), (65, 1)], 16, 8, 2, 128),
    ([(2000, 1)], 64, 32, 8, 128),
    ([(700 + 37 * i, 1) for i in range(70)], 64, 16, 4, 128),
    ([(300, 1), (31, 1)], 128, 4, 4, 64),
    ([(129, 2), (0, 3), (500, 4)], 8, 8, 2, 64),
    ([(77, 1), (1, 5)], 192, 9, 3, 128),
    ([(1000, 1), (90, 1)], 32, 16, 1, 64),
    ([(250, 16), (17, 9)], 64, 2, 2, 128),
    ([(100, 300), (0, 77), (800, 1), (5, 1), (60, 20)], 64, 8, 2, 128),
    ([(64, 200), (333, 1)], 64, 6, 6, 64),
]


@pytest.mark.parametrize("plan,page,Hq,Hk,D", CASES)
def test_against_the_oracle(plan, page, Hq, Hk, D):
    need = [(s + n + page - 1) // page for s, n in plan]
    order = torch.randperm(sum(need), generator=torch.Generator().manual_seed(1)).tolist()
    b, at = RaggedBatchWrapper(sum(n for _, n in plan), len(plan), max(need), device="cuda"), 0
    for (s, n), k in zip(plan, need):
        b.insert_sequence(_Seq(s, order[at: at + k]), torch.zeros(n, dtype=torch.int64))
        at += k
    b.finalize()
    g = torch.Generator(device="cuda").manual_seed(2)
    T, few = sum(n for _, n in plan), 16 // (Hq // Hk)
    qkv = (2 * torch.randn(T, Hq + 2 * Hk, D, generator=g, device="cuda")).bfloat16()
    cache = torch.randn(sum(need), page, 2, Hk, D, generator=g, device="cuda").bfloat16()
    for i, (s, n) in enumerate(plan):             # what lies behind a sequence's last token is never looked at
        last = b.block_tables()[i, (s + n - 1) // page].long()
        cache[last, (s + n - 1) % page + 1:] = float("nan") if n <= few else 0.0
    q = qkv[:, :Hq]
    want, at = [], 0
    for i, (s, n) in enumerate(plan):
        j = torch.arange(s + n, device="cuda")
        kv = cache[b.block_tables()[i, j // page].long(), j % page].double().repeat_interleave(Hq // Hk, 2)
        sc = torch.einsum("mhd,nhd->hmn", q[at: at + n].double(), kv[:, 0]) * D ** -0.5
        sc = sc.masked_fill(j[None] > torch.arange(s, s + n, device="cuda")[:, None], float("-inf"))
        want.append(torch.einsum("hmn,nhd->mhd", sc.softmax(-1), kv[:, 1]))
        at += n
    want = torch.cat(want)
    for _ in range(2):
        y = R.ragged_attention(q, cache, b).clone()
        # 16-bit weights (2^-9 each of values of a few units) and a 16-bit result
        assert bool(((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 0.02).all())
        assert float((y.double() - want).norm() / want.norm()) < 4e-3
    assert lib.hang_info("attn") is None


def test_captured_step_keeps_its_order():
    """Prompt portions and decode tokens run side by side; what follows in the stream sees both results, captured too."""
    plan = [(0, 500), (300, 260)] + [(900, 1)] * 30
    need = [(s + n + 63) // 64 for s, n in plan]
    b, at = RaggedBatchWrapper(sum(n for _, n in plan), len(plan), max(need), device="cuda"), 0
    for (s, n), k in zip(plan, need):
        b.insert_sequence(_Seq(s, list(range(at, at + k))), torch.zeros(n, dtype=torch.int64))
        at += k
    b.finalize()
    g = torch.Generator(device="cuda").manual_seed(3)
    q = torch.randn(790, 32, 128, generator=g, device="cuda").bfloat16()
    cache = torch.randn(sum(need), 64, 2, 8, 128, generator=g, device="cuda").bfloat16()
    first = R.ragged_attention(q, cache, b).float() * 2
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        R.ragged_attention(q, cache, b)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            twice = R.ragged_attention(q, cache, b).float() * 2
    for _ in range(5):
        twice.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(twice, first)


PACKED = [
    # plan, page, query heads, kv heads, head size, atoms packed into the tile with their group, atoms of the decode kernel
    ([(40, 20), (0, 32), (300, 9)], 64, 8, 2, 128, 3, 0),
    ([(40, 20), (0, 32), (300, 9)], 64, 8, 2, 64, 3, 0),
    ([(40, 20), (0, 32), (700, 1), (300, 9), (5, 1)], 64, 8, 2, 128, 3, 2),
    ([(31, 17), (700, 1), (64, 64)], 32, 8, 4, 64, 2, 1),
    ([(0, 200)] + [(50 + 90 * i, 8 + i) for i in range(10)] + [(333, 1)], 64, 32, 8, 128, 10, 1),
    ([(0, 200)] + [(50 + 90 * i, 8 + i) for i in range(9)] + [(333, 1)], 64, 32, 8, 128, 0, 1),
    ([(100 + 61 * i, 1) for i in range(12)], 64, 32, 1, 128, 12, 0),
    ([(0, 150)] + [(100 + 61 * i, 1 + i % 4) for i in range(12)], 64, 32, 1, 64, 12, 0),
    ([(0, 150)] + [(100 + 61 * i, 1) for i in range(4)], 64, 32, 1, 128, 0, 0),
    ([(9 * i, 1) for i in range(8)], 64, 32, 2, 128, 0, 8),
    ([(30, 1)] * 20 + [(5000, 1), (2700, 1)], 64, 32, 8, 128, 0, 22),            # few long contexts beside short ones
    ([(11 * i, 1) for i in range(60)], 64, 32, 8, 64, 0, 60),
]


@pytest.mark.parametrize("plan,page,Hq,Hk,D,n_packed,n_few", PACKED)
def test_which_atoms_share_a_tile(plan, page, Hq, Hk, D, n_packed, n_few, monkeypatch):
    """Short atoms have a launch of their own when they are alone or many, run with the longer ones when they are few, and
    decode tokens have theirs in either case; all of it against the oracle."""
    seen, run = [], R.paged_attention_atoms
    monkeypatch.setattr(R, "paged_attention_atoms", lambda *a: (seen.append(a[5:7]), run(*a))[1])
    monkeypatch.setattr(R, "_sm_count", lambda device: 148)
    test_against_the_oracle(plan, page, Hq, Hk, D)
    assert set(seen) == {(n_packed, n_few)}
