"""Attention backward whose dK / dV grid runs beside the dQ grid: what follows in the stream sees all three results, and results
that lie on the inputs (dK on K, dV on V) equal those that do not."""

import pytest

pytestmark = pytest.mark.gpu


def _backward(q, k, v, out, do, lse, dq, dk, dv):
    import torch
    from shuffle_exchange_b200.native import lib as _n
    B, S, Hq, D = q.shape
    delta = torch.empty((B, Hq, S), dtype=torch.float32, device=q.device)
    _n.call("sxb_attn_bwd", q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), do.data_ptr(), lse.data_ptr(),
            delta.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), B, S, Hq, k.shape[2], D, q.stride(1), k.stride(1),
            v.stride(1), out.stride(1), do.stride(1), dq.stride(1), dk.stride(1), dv.stride(1), 1, D ** -0.5, _n.stream_ptr())


@pytest.mark.parametrize("B,S,Hq,Hk,D", [(1, 1, 2, 1, 64), (2, 129, 12, 12, 64), (1, 777, 8, 2, 128), (2, 2048, 32, 8, 128),
                                         (1, 1500, 6, 3, 64)])
def test_results_on_the_inputs_and_readers_behind(B, S, Hq, Hk, D):
    import torch
    from shuffle_exchange_b200.ops import functional as F
    torch.manual_seed(0)
    mk = lambda h: torch.randn(B, S, h, D, device="cuda", dtype=torch.bfloat16)
    q, k, v, do = mk(Hq), mk(Hk), mk(Hk), mk(Hq)
    qg, kg, vg = (t.clone().requires_grad_() for t in (q, k, v))
    out = F.flash_attention(qg, kg, vg, causal=True)
    out.backward(do)
    lse = (q.float().transpose(1, 2) @ k.float().repeat_interleave(Hq // Hk, 2).permute(0, 2, 3, 1)) * D ** -0.5
    lse = lse.masked_fill(~torch.ones(S, S, dtype=torch.bool, device="cuda").tril(), float("-inf")).logsumexp(-1).contiguous()
    got = []
    for alias in (False, True):
        ks, vs = k.clone(), v.clone()
        dq, dk, dv = (torch.full_like(t, 9.0) for t in (q, k, v))
        if alias:
            dk, dv = ks, vs
        _backward(q, ks, vs, out.detach(), do, lse, dq, dk, dv)
        got.append([t.clone() for t in (dq, dk, dv)])      # on the stream, right behind
    for a, b in zip(*got):
        assert torch.equal(a, b)
    for a, g in zip(got[0], (qg.grad, kg.grad, vg.grad)):   # the same kernels with their own lse: bf16 rounding of either
        assert (a.float() - g.float()).norm() <= 2.0 ** -8 * g.float().norm() + 1e-6


def test_empty_first_sequence():
    """CTA 0 of the grid has no rows and still has to wait."""
    import torch
    from shuffle_exchange_b200.ops import functional as F
    torch.manual_seed(0)
    cu = torch.tensor([0, 0, 900, 1000], dtype=torch.int32, device="cuda")
    q, k, v, do = (torch.randn(1000, h, 64, device="cuda", dtype=torch.bfloat16) for h in (16, 4, 4, 16))
    grads = []
    for c in (cu, cu[1:].contiguous()):
        t = [x.clone().requires_grad_() for x in (q, k, v)]
        F.flash_attention_varlen(*t, c, 900, causal=True).backward(do)
        grads.append([x.grad.clone() for x in t])
    for a, b in zip(*grads):
        assert torch.equal(a, b)
