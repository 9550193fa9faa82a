"""Backward attention of head dim 128 in blocks of 128: edges of blocks and of their halves, groups, packed sequences, key bias."""

import pytest

pytestmark = pytest.mark.gpu

# Each gradient is two products of bf16-rounded factors (P or dS against dO, K or Q) and is rounded itself; dS also carries the rounding
# of O through rowsum(dO * O).  A rounding to bf16 has a relative error of 2^-9 / sqrt(3) in the 2-norm: four of them at most add up to 4.5e-3.
REL = 4 * 2.0 ** -9 / 3 ** 0.5
# What is zero in exact arithmetic (one key: dP = rowsum(dO * O)) is the difference of two fp32 sums of 128 products of numbers around 1.
ABS = 128 * 2.0 ** -23


def _reference(q, k, v, do, causal, bias=None):
    import torch
    q, k, v = (t.detach().double().transpose(1, 2).requires_grad_() for t in (q, k, v))
    g, S = q.shape[1] // k.shape[1], q.shape[2]
    s = q @ k.repeat_interleave(g, 1).transpose(-1, -2) * q.shape[-1] ** -0.5
    if bias is not None:
        s = s + bias[:, None, None].double()
    if causal:
        s = s.masked_fill(~torch.ones(S, S, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    (s.softmax(-1) @ v.repeat_interleave(g, 1)).backward(do.double().transpose(1, 2))
    return [t.grad.transpose(1, 2) for t in (q, k, v)]


def _close(got, want):
    for a, b in zip(got, want):
        err = (a.double() - b).norm()
        assert err <= REL * b.norm() + ABS * b.numel() ** 0.5, (err, b.norm())


def _tensors(*shapes, seed=0):
    import torch
    torch.manual_seed(seed)
    return [torch.randn(*s, device="cuda", dtype=torch.bfloat16) for s in shapes]


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("B,S,Hq,Hk", [(2, 1, 4, 2), (1, 63, 2, 2), (1, 64, 4, 1), (2, 65, 3, 3), (1, 127, 4, 2), (2, 128, 4, 4),
                                       (1, 129, 6, 2), (1, 191, 2, 1), (1, 192, 2, 1), (1, 193, 4, 2), (3, 256, 4, 2),
                                       (1, 257, 4, 2), (1, 513, 8, 2), (1, 1100, 5, 1)])
def test_gradients(B, S, Hq, Hk, causal):
    from shuffle_exchange_b200.native import lib
    from shuffle_exchange_b200.ops import functional as F
    q, k, v, do = _tensors((B, S, Hq, 128), (B, S, Hk, 128), (B, S, Hk, 128), (B, S, Hq, 128))
    t = [x.clone().requires_grad_() for x in (q, k, v)]
    F.flash_attention(*t, causal=causal).backward(do)
    _close([x.grad for x in t], _reference(q, k, v, do, causal))
    assert lib.hang_info("attn") is None


@pytest.mark.parametrize("causal", [True, False])
def test_key_bias(causal):
    import torch
    from shuffle_exchange_b200.ops import functional as F
    q, k, v, do = _tensors((2, 196, 4, 128), (2, 196, 2, 128), (2, 196, 2, 128), (2, 196, 4, 128))
    bias = torch.randn(2, 196, device="cuda")
    bias[0, 150:] = float("-inf")
    t = [x.clone().requires_grad_() for x in (q, k, v)]
    F.flash_attention_key_bias(*t, bias, causal=causal).backward(do)
    _close([x.grad for x in t], _reference(q, k, v, do, causal, bias))


@pytest.mark.parametrize("causal", [True, False])
def test_packed_sequences_and_what_lies_behind_them(causal):
    """Sequences that end on a multiple of 64 rows are followed by NaN: their own results see none of it."""
    import torch
    from shuffle_exchange_b200.ops import functional as F
    lens = [64, 70, 192, 64, 128, 33, 320, 1]
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device="cuda")
    T = sum(lens)
    q, k, v, do = _tensors((T, 4, 128), (T, 2, 128), (T, 2, 128), (T, 4, 128))
    at = cu.tolist()
    for i in (1, 3, 5, 7):
        for x in (q, k, v, do):
            x[at[i]: at[i + 1]] = float("nan")
    t = [x.clone().requires_grad_() for x in (q, k, v)]
    F.flash_attention_varlen(*t, cu, max(lens), causal=causal).backward(do)
    for i in (0, 2, 4, 6):
        r = slice(at[i], at[i + 1])
        _close([x.grad[None, r] for x in t], _reference(q[None, r], k[None, r], v[None, r], do[None, r], causal))


@pytest.mark.parametrize("first", range(0, 15))
def test_sums_run_in_the_order_of_keys_and_queries(first):
    """Every weight is one, and 2^30 comes and goes in two neighbouring steps of 16 rows: ones that are added between them are lost
    to the 24 bits of a sum, those behind them are not."""
    import torch
    from shuffle_exchange_b200.ops import functional as F
    S = 256
    c = torch.zeros(S, device="cuda", dtype=torch.bfloat16)
    c[16 * first: 16 * first + 16], c[16 * first + 16: 16 * first + 32], c[16 * first + 32:] = 2.0 ** 30, -2.0 ** 30, 1.0
    want = float(max(0, S - 16 * first - 32))
    zero, unit = torch.zeros(1, S, 1, 128, device="cuda", dtype=torch.bfloat16), torch.zeros(1, S, 1, 128, device="cuda", dtype=torch.bfloat16)
    unit[..., 0] = 1.0
    rows = c[None, :, None, None].expand(1, S, 1, 128).contiguous()
    grad = rows.clone()
    grad[..., 0] = 1.0
    lse = torch.zeros(1, 1, S, device="cuda")
    dq, _, _ = F.attention_bwd_raw(zero, rows, unit, zero, unit, lse, False, 1.0)
    _, dk, dv = F.attention_bwd_raw(rows, zero, unit, zero, grad, lse, False, 1.0)
    assert (dq == want).all() and (dk == want).all() and (dv[..., 1:] == want).all()


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("S,Hq,Hk", [(1, 2, 1), (16, 2, 1), (33, 4, 2), (64, 4, 1), (130, 4, 1), (192, 6, 2), (193, 2, 1), (320, 4, 4)])
def test_infinite_last_row_stays_where_it_is(S, Hq, Hk, causal):
    """Blocks with at most 64 rows left have nothing behind those rows: an infinity of the last row of dO meets its own weights only,
    which are not zero, and is never read a second time with weight zero."""
    import torch
    from shuffle_exchange_b200.ops import functional as F
    q, k, v, do = _tensors((1, S, Hq, 128), (1, S, Hk, 128), (1, S, Hk, 128), (1, S, Hq, 128))
    do[0, -1, :, 5] = float("inf")
    t = [x.clone().requires_grad_() for x in (q, k, v)]
    F.flash_attention(*t, causal=causal).backward(do)
    dv = t[2].grad[0]
    assert (dv[:, :, 5] == float("inf")).all() and torch.isfinite(dv[:, :, :5]).all() and torch.isfinite(dv[:, :, 6:]).all()
