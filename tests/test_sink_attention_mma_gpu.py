"""Prompt portions of sink attention over 16-bit caches (csrc/sink_attention_mma.cuh): head sizes, masks, portions of every
remainder, pages, biases, gates and values inside the key rows, against a 64-bit oracle."""
import pytest
import torch

from shuffle_exchange_b200.inference.v2.kernels import mixer_ops as M
from shuffle_exchange_b200.inference.v2.ragged.ragged_wrapper import RaggedBatchWrapper

pytestmark = pytest.mark.gpu


class _Seq:
    def __init__(self, seen, pages):
        self.seen_tokens, self._pages = seen, torch.tensor(pages, dtype=torch.int32)

    def kv_blocks(self):
        return self._pages


def _batch(plan, page):
    need = [(s + n + page - 1) // page for s, n in plan]
    order = torch.randperm(sum(need), generator=torch.Generator().manual_seed(3)).tolist()
    b, at = RaggedBatchWrapper(sum(n for _, n in plan), len(plan), max(need), device="cuda"), 0
    for (s, n), k in zip(plan, need):
        b.insert_sequence(_Seq(s, order[at: at + k]), torch.zeros(n, dtype=torch.int64))
        at += k
    b.finalize()
    return b, sum(need)


def _oracle(q, kc, vc, b, plan, page, scale, chunk, window, sink, bias, gate):
    out, rep, at = [], q.shape[1] // kc.shape[2], 0
    for i, (seen, n) in enumerate(plan):
        j = torch.arange(seen + n, device="cuda")
        rows = b.block_tables()[i, j // page].long(), j % page
        k, v = kc[rows].double().repeat_interleave(rep, 1), vc[rows].double().repeat_interleave(rep, 1)
        pos = torch.arange(seen, seen + n, device="cuda")
        lo = pos // chunk * chunk if chunk else ((pos - window + 1).clamp(min=0) if window else torch.zeros_like(pos))
        s = torch.einsum("mhd,nhd->hmn", q[at: at + n].double(), k) * scale
        dist = pos[:, None] - j[None]
        if bias is not None:
            s = s + bias.double()[:, dist.clamp(0, bias.shape[1] - 1)]
        s = s.masked_fill((dist < 0) | (j[None] < lo[:, None]), float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink.double()[:, None, None].expand(-1, n, 1)], -1)
        out.append(torch.einsum("hmn,nhd->mhd", s.softmax(-1)[..., : j.numel()], v))
        at += n
    out = torch.cat(out).reshape(q.shape[0], -1)
    if gate is not None:
        out = out * torch.sigmoid(gate.double()).repeat_interleave(out.shape[1] // gate.shape[1], 1)
    return out


CASES = [
    # plan, page, heads, kv heads, d, dv, chunk, window, sink, bias columns, gate, spread of the queries
    ([(0, 17)], 16, 2, 1, 64, 64, 0, 0, True, 0, "", 1.0),
    ([(0, 64), (5, 65), (130, 33)], 64, 4, 2, 128, 128, 0, 0, False, 0, "", 1.0),
    ([(0, 300), (700, 129)], 64, 8, 2, 128, 128, 256, 0, True, 0, "head", 4.0),
    ([(3, 500)], 128, 2, 2, 128, 64, 0, 100, True, 7, "", 1.0),
    ([(40, 128), (0, 31), (64, 1)], 16, 4, 1, 64, 128, 0, 0, True, 40, "channel", 30.0),
    ([(1, 191)], 64, 2, 1, 64, 64, 64, 0, False, 1, "", 1.0),
]


@pytest.mark.parametrize("plan,page,Hq,G,d,dv,chunk,window,with_sink,bias_cols,gated,spread", CASES)
def test_against_the_oracle(plan, page, Hq, G, d, dv, chunk, window, with_sink, bias_cols, gated, spread):
    g = torch.Generator(device="cuda").manual_seed(d + dv + Hq)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    b, pages = _batch(plan, page)
    T = sum(n for _, n in plan)
    q, kc, vc = mk(T, Hq, d) * spread, mk(pages, page, G, d).bfloat16(), mk(pages, page, G, dv).bfloat16()
    for i, (s, n) in enumerate(plan):          # what lies behind a sequence's last token is never looked at
        if (s + n) % page:
            last = b.block_tables()[i, (s + n) // page].long()
            kc[last, (s + n) % page:] = float("nan")
            vc[last, (s + n) % page:] = float("nan")
    sink = mk(Hq) if with_sink else None
    bias = mk(Hq, bias_cols) if bias_cols else None
    gate = {"": None, "head": mk(T, Hq).bfloat16(), "channel": mk(T, Hq * dv + 8).bfloat16()[:, : Hq * dv]}[gated]
    wide = torch.full((T, Hq * dv + 3), 9.0, device="cuda", dtype=torch.bfloat16)       # odd pitch: stores of single values
    args = (b.token_to_seq(), b.token_positions(), b.block_tables(), d ** -0.5, chunk, torch.bfloat16, b.atoms(),
            b.atoms_longer_than(M.SHORT_ATOM))
    want = _oracle(q, kc, vc, b, plan, page, d ** -0.5, chunk, window, sink, bias, gate)
    # half a unit of the 16-bit result; a score is a 32-bit sum of d terms (relative 2^-20 of their magnitudes), which the
    # exponential turns into a relative error of every weight
    size = (spread * d ** 0.5 * 4 + 4) * 2.0 ** -20
    bound = 2.0 ** -8 * want.abs() + size * 6
    for out in (None, wide[:, : Hq * dv]):
        y = M.sink_attention(q, kc, vc, sink, *args, window=window, dist_bias=bias, gate=gate, out=out, out_scale=0.5)
        assert bool(((y.double() - 0.5 * want).abs() <= bound).all())
    assert bool((wide[:, Hq * dv:] == 9.0).all())


def test_values_inside_the_key_rows():
    plan, page = [(0, 90), (33, 40)], 64
    b, pages = _batch(plan, page)
    g = torch.Generator(device="cuda").manual_seed(5)
    q = torch.randn(130, 4, 128, generator=g, device="cuda")
    kc = torch.randn(pages, page, 1, 128, generator=g, device="cuda").bfloat16()
    y = M.sink_attention(q, kc, None, None, b.token_to_seq(), b.token_positions(), b.block_tables(), 0.1, 0, torch.bfloat16,
                         b.atoms(), b.atoms_longer_than(M.SHORT_ATOM), value_cols=64, value_col0=8)
    want = _oracle(q, kc, kc[..., 8:72], b, plan, page, 0.1, 0, 0, None, None, None)
    assert bool(((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all())


def test_as_close_as_the_32_bit_form():
    """The three terms carry the 32-bit operands whole: against 64 bits the tensor-core form is no further off than fp32
    products (the cache as fp32 takes the FMA form)."""
    plan, page = [(0, 700)], 64
    b, pages = _batch(plan, page)
    g = torch.Generator(device="cuda").manual_seed(6)
    q = torch.randn(700, 4, 128, generator=g, device="cuda") * 3
    kc, vc = (torch.randn(pages, page, 2, 128, generator=g, device="cuda").bfloat16() for _ in range(2))
    args = (None, b.token_to_seq(), b.token_positions(), b.block_tables(), 128 ** -0.5, 0)
    rest = (b.atoms(), b.atoms_longer_than(M.SHORT_ATOM))
    want = _oracle(q, kc, vc, b, plan, page, 128 ** -0.5, 0, 0, None, None, None)
    y16 = M.sink_attention(q, kc, vc, *args, torch.bfloat16, *rest).double()
    y32 = M.sink_attention(q, kc.float(), vc.float(), *args, torch.float32, *rest)
    e16, e32 = ((t.double() - want).norm() / want.norm() for t in (y16, y32.bfloat16()))
    assert float(e16) <= 1.01 * float(e32)
    assert float((y16 != y32.bfloat16().double()).double().mean()) < 0.01      # they round differently at ties only


def test_infinite_keys_and_values():
    """What a plain softmax gives: an infinite value comes out infinite wherever its weight is not zero (the weight of the
    largest key is exactly one), a key whose score is minus infinity has no weight, and rows that do not see them are untouched."""
    plan, page, Hq, G, d = [(0, 150), (70, 40)], 64, 4, 2, 128
    b, pages = _batch(plan, page)
    g = torch.Generator(device="cuda").manual_seed(8)
    q = torch.randn(190, Hq, d, generator=g, device="cuda")
    kc, vc = (torch.randn(pages, page, G, d, generator=g, device="cuda").bfloat16() for _ in range(2))
    at = lambda i, j: (b.block_tables()[i, j // page].long(), j % page)  # noqa: E731
    q[3, 1], q[3, 1, 0] = 0.0, 64.0                    # row 3 of head 1: its own key takes weight one
    kc[at(0, 3)][0, 0] = 64.0
    vc[at(0, 3)][0, 5] = float("inf")
    vc[at(0, 90)][1, 7], vc[at(0, 91)][1, 8] = float("-inf"), float("inf")
    kc[at(1, 80)][0, 2] = float("inf")                 # a score of plus infinity (not a number) or minus infinity (no weight)
    vc[at(1, 100)][1, 9] = float("nan")
    args = lambda dev: (b.token_to_seq().to(dev), b.token_positions().to(dev), b.block_tables().to(dev), d ** -0.5, 0)  # noqa: E731
    y = M.sink_attention(q, kc, vc, None, *args("cuda"), torch.bfloat16, b.atoms(), b.atoms_longer_than(M.SHORT_ATOM)).cpu()
    want = M.sink_attention(q.cpu(), kc.cpu(), vc.cpu(), None, *args("cpu"), torch.float32)
    assert bool(want.isinf().any()) and bool(want.isnan().any()) and bool(want.view(190, Hq, d)[3, 1, 5].isinf())
    assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y.isinf(), want.isinf())
    assert torch.equal(y[want.isinf()].float(), want[want.isinf()])
    ok = want.isfinite()
    assert bool(((y.float() - want)[ok].abs() <= 2.0 ** -8 * want[ok].abs() + 1e-4).all())


@pytest.mark.parametrize("with_sink", [True, False])
def test_biases_of_the_lowest_value_leave_equal_weights(with_sink):
    """In 32 bits every score is the lowest value, the sink's too: all keys that a row sees weigh the same."""
    low, plan, page = torch.finfo(torch.float32).min, [(0, 90), (33, 40)], 64
    b, pages = _batch(plan, page)
    g = torch.Generator(device="cuda").manual_seed(9)
    q = torch.randn(130, 4, 128, generator=g, device="cuda")
    kc, vc = (torch.randn(pages, page, 2, 128, generator=g, device="cuda").bfloat16() for _ in range(2))
    sink = torch.zeros(4, device="cuda") if with_sink else None
    y = M.sink_attention(q, kc, vc, sink + low if with_sink else None, b.token_to_seq(), b.token_positions(), b.block_tables(), 0.1, 0,
                         torch.bfloat16, b.atoms(), b.atoms_longer_than(M.SHORT_ATOM), dist_bias=torch.full((4, 100), low, device="cuda"))
    want = _oracle(0 * q, kc, vc, b, plan, page, 0.1, 0, 0, sink, None, None)
    assert bool(((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all())
