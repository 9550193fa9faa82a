"""linear_recurrence over rows at the edges of its groups of eight tokens, in every form that the number of CTAs selects (one,
two or four columns per lane, operands read ahead or not): against a 64-bit walk, and bit for bit among the forms."""
import pytest
import torch

from shuffle_exchange_b200.inference.v2.kernels import mixer_ops as M
from test_recurrence_columns_gpu import _walk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rule", ["delta", "ssd", "channel"])
@pytest.mark.parametrize("n", [32, 64, 128, 72])
@pytest.mark.parametrize("with_beta", [True, False])
def test_edges_of_groups_in_every_form(rule, n, with_beta):
    rows, H, dv = [1, 7, 8, 9, 15, 16, 17, 41], 2, 64
    T, N = sum(rows), len(rows)
    g = torch.Generator(device="cuda").manual_seed(n)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    k, q, v = mk(T, H * n), mk(T, H * n) / n ** 0.5, mk(T, H * dv)
    k = torch.nn.functional.normalize(k.view(T, H, n), dim=-1).view(T, -1).contiguous()
    decay = torch.rand(T, H * (n if rule == "channel" else 1), generator=g, device="cuda")
    beta = torch.rand(T, H, generator=g, device="cuda") if with_beta else None
    state = mk(N, H, dv, n)
    base = [[sum(rows[:i]), r, i % 2, i] for i, r in enumerate(rows)]
    want, wst = _walk(k, q, v, decay, beta, None, state, torch.tensor(base), H, H, n, dv, rule != "ssd")
    first = None
    for copies in (1, 4, 30):               # 64, 128 and 960 CTAs of 16, 32 and 32 columns (or 480 of 64)
        info = torch.tensor([[f + T * c, r, seen, slot + N * c] for c in range(copies) for f, r, seen, slot in base],
                            dtype=torch.int32, device="cuda")
        st = state.repeat(copies, 1, 1, 1)
        rep = lambda t: None if t is None else t.repeat(copies, 1)  # noqa: E731
        out = M.linear_recurrence(rep(k), rep(q), rep(v), rep(decay), rep(beta), None, st, info, H, H, n, dv, rule != "ssd")
        if first is None:
            first = out, st
            for a, b in ((out, want), (st, wst)):   # sums of n terms over 41 rows, contracting: a few units of the last place
                assert float((a.double() - b).norm() / b.norm()) < 1e-6
        assert torch.equal(out.view(copies, T, -1), first[0][None].expand(copies, -1, -1))
        assert torch.equal(st.view(copies, N, H, dv, n), first[1][None].expand(copies, -1, -1, -1, -1))


@pytest.mark.parametrize("rule", ["delta", "ssd", "channel"])
@pytest.mark.parametrize("n,dv", [(64, 16), (128, 48), (256, 16), (100, 16)])
def test_many_sequences_long_and_short(rule, n, dv):
    """Beyond 32 sequences the rows they have decide on the read ahead; the bits are the same."""
    H, N = 2, 36
    g = torch.Generator(device="cuda").manual_seed(n + dv)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    rows = [70 + i % 5 for i in range(N)]
    T = sum(rows)
    k, q, v = mk(T, H * n), mk(T, H * n) / n ** 0.5, mk(T, H * dv)
    k = torch.nn.functional.normalize(k.view(T, H, n), dim=-1).view(T, -1).contiguous()
    decay = torch.rand(T, H * (n if rule == "channel" else 1), generator=g, device="cuda")
    beta, state = torch.rand(T, H, generator=g, device="cuda"), mk(N, H, dv, n)
    info = torch.tensor([[sum(rows[:i]), r, i % 2, i] for i, r in enumerate(rows)], dtype=torch.int32, device="cuda")
    st = state.clone()
    out = M.linear_recurrence(k, q, v, decay, beta, None, st, info, H, H, n, dv, rule != "ssd")
    want, wst = _walk(k, q, v, decay, beta, None, state, info, H, H, n, dv, rule != "ssd")
    for a, b in ((out, want), (st, wst)):           # sums of n terms over 74 rows, contracting: a few units of the last place
        assert float((a.double() - b).norm() / b.norm()) < 1e-6
    # with as many sequences again that have no rows they are short on average
    both = torch.cat([info, torch.tensor([[0, 0, 0, N + i] for i in range(N)], dtype=torch.int32, device="cuda")])
    st2 = torch.cat([state, state])
    assert torch.equal(M.linear_recurrence(k, q, v, decay, beta, None, st2, both, H, H, n, dv, rule != "ssd"), out)
    assert torch.equal(st2[:N], st)


@pytest.mark.parametrize("rule", ["delta", "channel"])
@pytest.mark.parametrize("n", [16, 40, 72, 96, 100, 200])
def test_padding_is_zero_before_its_first_reader(rule, n):
    """Keys that do not fill their rows of shared memory, behind a launch that leaves NaN in all of it on every SM."""
    rows, H, dv = [8, 9, 17, 41], 2, 64
    T, N, full = sum(rows), len(rows), next(p for p in (32, 64, 128, 256) if n <= p)
    g = torch.Generator(device="cuda").manual_seed(n)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    k, q, v = mk(T, H * n), mk(T, H * n) / n ** 0.5, mk(T, H * dv)
    k = torch.nn.functional.normalize(k.view(T, H, n), dim=-1).view(T, -1).contiguous()
    decay = torch.rand(T, H * (n if rule == "channel" else 1), generator=g, device="cuda")
    beta, state = torch.rand(T, H, generator=g, device="cuda"), mk(N, H, dv, n)
    info = torch.tensor([[sum(rows[:i]), r, i % 2, i] for i, r in enumerate(rows)], dtype=torch.int32, device="cuda")
    want, wst = _walk(k, q, v, decay, beta, None, state, info, H, H, n, dv, True)
    nan = lambda *s: torch.full(s, float("nan"), device="cuda")  # noqa: E731
    many = torch.tensor([[0, 32, 0, i] for i in range(32)], dtype=torch.int32, device="cuda")     # 32 sequences, 32 heads: 4096 CTAs at most
    fill = (nan(32, 32 * full), nan(32, 32 * full), nan(32, 32 * dv), nan(32, 32 * (full if rule == "channel" else 1)), nan(32, 32), None,
            nan(32, 32, dv, full), many, 32, 32, full, dv, True)
    first = None
    for _ in range(100):
        M.linear_recurrence(*fill)
        st = state.clone()
        out = M.linear_recurrence(k, q, v, decay, beta, None, st, info, H, H, n, dv, True)
        if first is None:
            first = out, st
            for a, b in ((out, want), (st, wst)):   # sums of n terms over 41 rows, contracting: a few units of the last place
                assert float((a.double() - b).norm() / b.norm()) < 1e-6
        assert torch.equal(out, first[0]) and torch.equal(st, first[1])
