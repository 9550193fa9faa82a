"""linear_recurrence with one and with two state columns per lane (chosen by the number of CTAs): both against the rows of a
64-bit walk, over sizes at the edges of the column blocks, and bit for bit against each other."""
import pytest
import torch

from shuffle_exchange_b200.inference.v2.kernels import mixer_ops as M

pytestmark = pytest.mark.gpu


def _walk(k, q, v, decay, beta, skip, state, info, H, G, n, dv, delta):
    out, T = torch.empty(v.shape[0], H, dv, dtype=torch.float64, device="cuda"), v.shape[0]
    ks, qs = (x.double().view(T, G, n).repeat_interleave(H // G, 1) for x in (k, q))
    vs, st = v.double().view(T, H, dv), state.double().clone()
    d = decay.double().view(T, H, 1, -1)
    for first, rows, seen, slot in info.tolist():
        S = st[slot] if seen else torch.zeros_like(st[slot])
        for t in range(first, first + rows):
            S = S * d[t]
            u = vs[t] - (S @ ks[t][:, :, None]).squeeze(-1) if delta else vs[t]
            if beta is not None:
                u = beta[t].double()[:, None] * u
            S = S + u[:, :, None] * ks[t][:, None, :]
            out[t] = (S @ qs[t][:, :, None]).squeeze(-1) + (0 if skip is None else skip.double()[:, None] * vs[t])
        st[slot] = S
    return out.view(T, -1), st


@pytest.mark.parametrize("n,dv", [(128, 128), (128, 33), (64, 48), (100, 17), (60, 31), (256, 64), (16, 129)])
@pytest.mark.parametrize("rule", ["delta", "ssd", "channel"])
def test_both_column_counts(n, dv, rule):
    g = torch.Generator(device="cuda").manual_seed(n + dv)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    rows = [1, 8, 21, 3]
    res = []
    for copies in (1, 40):                  # the same four sequences once and forty times over: few CTAs and many
        H, G, T = 2, 1, sum(rows)
        g.manual_seed(n + dv)
        k, q, v = mk(T, G * n) / n ** 0.5, mk(T, G * n), mk(T, H * dv)
        decay = torch.rand(T, H * (n if rule == "channel" else 1), generator=g, device="cuda")
        beta = torch.rand(T, H, generator=g, device="cuda") if rule != "ssd" else None
        skip = mk(H) if rule == "ssd" else None
        state = mk(4, H, dv, n)
        rep = lambda t, c=copies: None if t is None else t.repeat(c, *[1] * (t.dim() - 1))  # noqa: E731
        info, at = [], 0
        for c in range(copies):
            for i, r in enumerate(rows):
                info.append([at, r, 5 * (i % 2), 4 * c + i])
                at += r
        info = torch.tensor(info, dtype=torch.int32, device="cuda")
        st = rep(state)
        out = M.linear_recurrence(rep(k), rep(q), rep(v), rep(decay), rep(beta), skip, st, info, H, G, n, dv, rule != "ssd")
        assert torch.equal(out.view(copies, T, -1), out[None, :T].expand(copies, -1, -1))
        assert torch.equal(st.view(copies, 4, H, dv, n), st[None, :4].expand(copies, -1, -1, -1, -1))
        res.append((out[:T], st[:4]))
        if copies == 1:
            want, wst = _walk(k, q, v, decay, beta, skip, state, info, H, G, n, dv, rule != "ssd")
            for a, b in ((out, want), (st, wst)):       # sums of n terms over 21 rows: a few units of the last place
                assert float((a.double() - b).norm() / b.norm()) < 1e-6
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])
