"""Expert exchange with a row dealt out over several warps: rows arrive unchanged, padding is zeroed or left as asked, and the
weighted sums equal those in 32 bits, at widths that end inside a piece and row counts on both sides of the rule."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,H", [(1, 512), (3, 520), (200, 4096), (74, 8200), (600, 1024), (2500, 768)])
@pytest.mark.parametrize("zero_pad", [True, False])
def test_push_and_pull(T, H, zero_pad):
    import torch
    from shuffle_exchange_b200.moe import fused_ep
    from shuffle_exchange_b200.ops import moe_ops
    torch.manual_seed(0)
    E, K, dev = 5, 2, "cuda"
    x = torch.randn(T, H, device=dev, dtype=torch.bfloat16)
    scores, assign, offsets, counts = moe_ops.top_k_gating(torch.randn(T, E, device=dev), K, renormalize=True)
    ep = fused_ep.FusedEP(None, H, E, T, K)
    plan = fused_ep.make_plan(ep, counts, assign, offsets)
    ep.recv_rows.fill_(3.0)
    ep.push(x, plan, zero_pad=zero_pad)
    group = plan.group_offsets.tolist()
    row = plan.group_offsets[assign.long()].long() + offsets.long()            # [T, K]
    assert torch.equal(ep.recv_rows[row], x[:, None].expand(T, K, H))
    for e, c in enumerate(counts.tolist()):
        pad = ep.recv_rows[group[e] + c: group[e + 1]]
        assert torch.equal(pad, torch.full_like(pad, 0.0 if zero_pad else 3.0))
    ep.ret_rows.copy_(torch.randn_like(ep.ret_rows))
    wts = scores.float().contiguous()
    y = torch.empty_like(x)
    keep = torch.empty(T * K, H, device=dev, dtype=torch.bfloat16)
    ep.pull(y, plan, weights=wts, keep=keep)
    assert torch.equal(keep.view(T, K, H), ep.ret_rows[row])
    want = (ep.ret_rows[row].float() * wts[..., None]).sum(1)
    # one rounding to bf16 (2^-9 relative) and two of 32 bits, whose products may cancel
    assert ((y.float() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -20).all()
    # scaled rows on the way in
    ep2 = fused_ep.make_plan(ep, counts, assign, offsets)
    ep.push(x, ep2, weights=wts, zero_pad=zero_pad)
    assert torch.equal(ep.recv_rows[row], (x[:, None].float() * wts[..., None]).to(torch.bfloat16))
