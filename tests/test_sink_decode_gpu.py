"""Sink attention of single tokens over 16-bit caches against a 64-bit walk: keys at the edges of its steps of 16, warps and clusters, every
number of heads per key/value head, windows and chunks, biases, gates, slices, short portions, and infinities."""
import pytest
import torch

from shuffle_exchange_b200.inference.v2.kernels import mixer_ops as M

pytestmark = pytest.mark.gpu
PAGE = 64


def _case(contexts, Hq, G, d, seed=0, page=PAGE):
    g = torch.Generator(device="cuda").manual_seed(seed)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    need = [(c + page - 1) // page for c in contexts]
    order = torch.randperm(sum(need), generator=torch.Generator().manual_seed(seed)).tolist()
    tables = torch.zeros(len(contexts), max(need), dtype=torch.int32)
    at = 0
    for i, n in enumerate(need):
        tables[i, :n] = torch.tensor(order[at: at + n], dtype=torch.int32)
        at += n
    kc, vc = (mk(sum(need), page, G, d).to(torch.bfloat16) for _ in range(2))
    return mk(len(contexts), Hq, d), kc, vc, tables.cuda(), mk(Hq), g


def _walk(q, kc, vc, tables, seqs, poss, scale, chunk=0, window=0, sink=None, bias=None):
    T, Hq, d = q.shape
    rep, page, out = Hq // kc.shape[2], kc.shape[1], []
    for t in range(T):
        pos = poss[t]
        lo = pos // chunk * chunk if chunk else max(0, pos - window + 1) if window else 0
        j = torch.arange(lo, pos + 1, device="cuda")
        rows = tables[seqs[t], j // page].long(), j % page
        k, v = (c[rows].double().repeat_interleave(rep, 1) for c in (kc, vc))
        s = torch.einsum("hd,nhd->hn", q[t].double(), k) * scale
        if bias is not None:
            s = s + bias.double()[:, (pos - j).clamp(max=bias.shape[1] - 1)]
        if sink is not None:
            s = torch.cat([s, sink.double()[:, None]], 1)
        out.append(torch.einsum("hn,nhd->hd", s.softmax(-1)[:, : j.numel()], v))
    return torch.stack(out)


def _close(got, want):
    # half a unit of bf16's last place, and 32-bit sums behind it
    assert float((got.double() - want.reshape(got.shape)).norm() / want.norm()) < 2.0 ** -8
    assert float((got.double() - want.reshape(got.shape)).abs().max()) < 2.0 ** -8 * float(want.abs().max()) + 1e-5


@pytest.mark.parametrize("Hq,G,d", [(4, 1, 128), (16, 4, 128), (8, 8, 64), (6, 2, 128), (16, 2, 64), (5, 1, 128), (12, 6, 128)])
@pytest.mark.parametrize("reach", [{}, {"chunk": 100}, {"window": 37}])
def test_tokens(Hq, G, d, reach):
    contexts = [1, 15, 16, 17, 63, 64, 65, 128, 129, 200, 511, 513, 1100]
    q, kc, vc, tables, sink, g = _case(contexts, Hq, G, d, page=48)
    poss, n = [c - 1 for c in contexts], len(contexts)
    ts, tp = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in (list(range(n)), poss))
    for s in (sink, None):
        kw = dict(chunk=reach.get("chunk", 0), window=reach.get("window", 0))
        got = M.sink_attention(q, kc, vc, s, ts, tp, tables, d ** -0.5, kw["chunk"], torch.bfloat16, window=kw["window"])
        _close(got, _walk(q, kc, vc, tables, list(range(n)), poss, d ** -0.5, sink=s, **kw))


@pytest.mark.parametrize("n,context", [(1, 3000), (3, 700), (200, 130)])
def test_few_and_many_tokens(n, context):
    contexts = [context - i % 7 for i in range(n)]
    q, kc, vc, tables, sink, g = _case(contexts, 8, 2, 128, seed=n)
    poss = [c - 1 for c in contexts]
    ts, tp = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in (list(range(n)), poss))
    got = M.sink_attention(q, kc, vc, sink, ts, tp, tables, 0.1, 0, torch.bfloat16)
    _close(got, _walk(q, kc, vc, tables, list(range(n)), poss, 0.1, sink=sink))


@pytest.mark.parametrize("per_head", [True, False])
def test_bias_gate_and_slices(per_head):
    Hq, G, d = 8, 2, 128
    q, kc, vc, tables, sink, g = _case([70, 300, 5], Hq, G, d)
    ts, tp = torch.arange(3, dtype=torch.int32, device="cuda"), torch.tensor([69, 299, 4], dtype=torch.int32, device="cuda")
    bias = torch.randn(Hq, 40, generator=g, device="cuda")
    gate = torch.randn(3, Hq if per_head else Hq * d, generator=g, device="cuda").to(torch.bfloat16)
    room = torch.zeros(3, Hq * d + 3, dtype=torch.bfloat16, device="cuda")
    got = M.sink_attention(q, kc, vc, sink, ts, tp, tables, d ** -0.5, 0, torch.bfloat16, dist_bias=bias, gate=gate,
                           out=room[:, 3:], out_scale=0.5)
    want = _walk(q, kc, vc, tables, [0, 1, 2], [69, 299, 4], d ** -0.5, sink=sink, bias=bias)
    f = torch.sigmoid(gate.double()).view(3, Hq, -1) * 0.5
    _close(got, want * f)
    assert not room[:, :3].any()


def test_short_portions():
    # sequence 0: eleven rows from position 20; sequence 1: one row
    q, kc, vc, tables, sink, g = _case([31, 100], 8, 2, 128)
    q = torch.randn(12, 8, 128, generator=g, device="cuda")
    seqs, poss = [0] * 11 + [1], list(range(20, 31)) + [99]
    atoms = torch.tensor([[0, 0, 11, 20, 1, 31], [1, 11, 1, 99, 2, 100]], dtype=torch.int32, device="cuda")
    ts, tp = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in (seqs, poss))
    want = _walk(q, kc, vc, tables, seqs, poss, 0.1, sink=sink)
    a = M.sink_attention(q, kc, vc, sink, ts, tp, tables, 0.1, 0, torch.bfloat16, atoms, 0)
    _close(a, want)


def test_infinities_come_out_as_from_32_bit_products():
    Hq, d = 4, 128
    q, kc, vc, tables, sink, g = _case([50, 50, 50], Hq, 1, d)
    page = lambda i, j: (int(tables[i, j // PAGE]), j % PAGE)  # noqa: E731
    vc[page(0, 7)][0, 5] = float("inf")             # a value: that channel is infinite, the others are not
    kc[page(1, 9)][0] = float("inf")                # a key: scores of both signs, or not a number
    q[2, 1, 3] = float("inf")                       # a query: its head alone
    ts, tp = torch.arange(3, dtype=torch.int32, device="cuda"), torch.full((3,), 49, dtype=torch.int32, device="cuda")
    got = M.sink_attention(q, kc, vc, sink, ts, tp, tables, d ** -0.5, 0, torch.bfloat16).view(3, Hq, d)
    want = _walk(q, kc, vc, tables, [0, 1, 2], [49] * 3, d ** -0.5, sink=sink)
    assert bool((got[0, :, 5] == float("inf")).all()) and bool(got[0].isfinite().sum() == Hq * (d - 1))
    keep = torch.arange(d, device="cuda") != 5
    _close(got[0][:, keep], want[0][:, keep])
    assert bool((~got[1].isfinite()).all()) and bool((~got[2, 1].isfinite()).all())
    _close(got[2, [0, 2, 3]], want[2, [0, 2, 3]])


@pytest.mark.parametrize("with_sink", [True, False])
def test_biases_of_the_lowest_value_leave_equal_weights(with_sink):
    # in 32 bits every score is the lowest value, the sink's too: all keys weigh the same
    low = torch.finfo(torch.float32).min
    q, kc, vc, tables, sink, g = _case([50, 300], 8, 2, 128)
    poss = [49, 299]
    ts, tp = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in ([0, 1], poss))
    got = M.sink_attention(q, kc, vc, torch.full_like(sink, low) if with_sink else None, ts, tp, tables, 0.1, 0, torch.bfloat16,
                           dist_bias=torch.full((8, 400), low, device="cuda"))
    _close(got, _walk(0 * q, kc, vc, tables, [0, 1], poss, 0.1, sink=0 * sink if with_sink else None))
