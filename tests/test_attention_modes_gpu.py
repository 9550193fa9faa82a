"""Packed-sequence (varlen) training attention and atom-scheduled paged attention on the tcgen05 kernels.

Oracles are plain PyTorch fp32 computations of the same op (``attention_varlen_ref``; the per-token paged attention
written out in ``ragged_ops.paged_attention``'s CPU branch)."""
import math

import pytest
import torch

from shuffle_exchange_b200.inference.v2.ragged.ragged_wrapper import RaggedBatchWrapper


class _Seq:
    def __init__(self, seen, blocks):
        self.seen_tokens, self._blocks = seen, torch.tensor(blocks, dtype=torch.int32)

    def kv_blocks(self):
        return self._blocks


def test_wrapper_cuts_atoms_on_cpu():
    w = RaggedBatchWrapper(1024, 8, 16, device="cpu")
    w.insert_sequence(_Seq(0, [3, 4, 5]), torch.arange(300))          # prefill: 3 atoms
    w.insert_sequence(_Seq(77, [1]), torch.arange(1))                 # decode: 1 atom
    w.insert_sequence(_Seq(100, [6, 7]), torch.arange(130))           # chunked prefill continuing at 100: 2 atoms
    w.finalize()
    atoms = w.atoms().tolist()
    # longest atoms first (stable), so the short tail can run with the GQA group packed into one tile
    assert atoms == [[0, 0, 128, 0, 2, 128], [0, 128, 128, 128, 4, 256], [2, 301, 128, 100, 4, 228],
                     [0, 256, 44, 256, 5, 300], [2, 429, 2, 228, 4, 230], [1, 300, 1, 77, 2, 78]]
    assert (w.atoms_longer_than(32), w.atoms_longer_than(64), w.atoms_longer_than(1), w.atoms_longer_than(0)) == (4, 3, 5, 6)
    w.clear()
    w.finalize()
    assert w.atoms().shape[0] == 0


def test_what_does_not_fit_a_batch_is_refused():
    one = torch.arange(1)
    for tokens, blocks in ((torch.zeros(3, 1, dtype=torch.int64), [0]), (torch.zeros(2, 2, dtype=torch.int64), [0]),
                           (one, list(range(5))), (torch.arange(9), [0])):
        w = RaggedBatchWrapper(8, 2, 4, device="cpu")
        with pytest.raises(RuntimeError):
            w.insert_sequence(_Seq(0, blocks), tokens, do_checks=False)
        w.insert_sequence(_Seq(4, [2]), one[None])                     # one row of tokens; nothing of the refused ones is left
        w.finalize()
        assert w.input_ids().tolist() == [0] and w.seq_info().tolist() == [[0, 1, 4, -1]]


def _rel_err(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-9)).item()


@pytest.mark.gpu
@pytest.mark.parametrize("D,Hq,Hk", [(128, 8, 2), (64, 4, 4), (128, 3, 1)])
@pytest.mark.parametrize("causal", [True, False])
def test_varlen_forward_backward_matches_reference(D, Hq, Hk, causal):
    from shuffle_exchange_b200.ops import functional as F
    torch.manual_seed(0)
    dev = "cuda"
    lens = [200, 1, 128, 333, 64, 70]
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=dev)
    T = sum(lens)
    qkv = torch.randn(T, (Hq + 2 * Hk) * D, device=dev, dtype=torch.bfloat16)
    qkv.requires_grad_(True)
    v3 = qkv.view(T, Hq + 2 * Hk, D)
    q, k, v = v3[:, :Hq], v3[:, Hq:Hq + Hk], v3[:, Hq + Hk:]
    out = F.flash_attention_varlen(q, k, v, cu, max(lens), causal=causal)
    dout = torch.randn_like(out)
    out.backward(dout)
    got_grad = qkv.grad.clone()

    ref_in = qkv.detach().float().requires_grad_(True)
    r3 = ref_in.view(T, Hq + 2 * Hk, D)
    ref = F.attention_varlen_ref(r3[:, :Hq], r3[:, Hq:Hq + Hk], r3[:, Hq + Hk:], cu.cpu(), causal)
    ref.backward(dout.float())
    assert _rel_err(out, ref) < 1e-2
    # per-sequence check: a leak across a boundary shows up as a large error on a SHORT sequence
    for a, b in zip(cu.tolist()[:-1], cu.tolist()[1:]):
        assert _rel_err(out[a:b], ref[a:b]) < 2e-2, (a, b)
        assert _rel_err(got_grad[a:b], ref_in.grad[a:b]) < 3e-2, (a, b)


@pytest.mark.gpu
def test_varlen_equals_dense_for_equal_lengths():
    from shuffle_exchange_b200.ops import functional as F
    torch.manual_seed(1)
    B, S, Hq, Hk, D = 3, 256, 8, 4, 128
    q = torch.randn(B, S, Hq, D, device="cuda", dtype=torch.bfloat16)
    k = torch.randn(B, S, Hk, D, device="cuda", dtype=torch.bfloat16)
    v = torch.randn(B, S, Hk, D, device="cuda", dtype=torch.bfloat16)
    dense = F.flash_attention(q, k, v, causal=True)
    cu = torch.arange(0, (B + 1) * S, S, dtype=torch.int32, device="cuda")
    packed = F.flash_attention_varlen(q.view(B * S, Hq, D), k.view(B * S, Hk, D), v.view(B * S, Hk, D), cu, S)
    assert torch.equal(packed.view(B, S, Hq, D), dense)          # same kernel, same tiles: bit-identical


@pytest.mark.gpu
@pytest.mark.parametrize("block_size", [16, 64, 128])
@pytest.mark.parametrize("D,Hq,Hk", [(128, 8, 2), (64, 4, 2)])
def test_atom_paged_attention_matches_per_token_oracle(block_size, D, Hq, Hk):
    from shuffle_exchange_b200.inference.v2.kernels import ragged_ops as R
    torch.manual_seed(2)
    dev = "cuda"
    # (seen, new tokens): long prefill, decode with history, chunked prefill continuing mid-block, tiny prefill
    plan = [(0, 300), (517, 1), (100, 130), (0, 5), (63, 1)]
    max_blocks = 16 * 128 // block_size
    n_blocks = 256 * 128 // block_size
    cache = torch.randn(n_blocks, block_size, 2, Hk, D, device=dev, dtype=torch.bfloat16)
    perm = torch.randperm(n_blocks).tolist()
    w = RaggedBatchWrapper(1024, 8, max_blocks, device=dev)
    for seen, n in plan:
        need = (seen + n + block_size - 1) // block_size
        blocks, perm = perm[:need], perm[need:]
        w.insert_sequence(_Seq(seen, blocks), torch.zeros(n, dtype=torch.int64))
    w.finalize()
    T = w.current_tokens
    q = torch.randn(T, Hq, D, device=dev, dtype=torch.bfloat16)
    assert R.atoms_supported(q, cache)
    got = R.ragged_attention(q, cache, w)
    want = R.paged_attention(q.cpu(), cache.cpu(), w.token_to_seq().cpu(), w.token_positions().cpu(),
                             w.block_tables().cpu())
    assert _rel_err(got.cpu(), want) < 1e-2
    for t in (0, 299, 300, 301, 430, 431, 435, 436):               # first / last rows of every atom
        assert _rel_err(got[t].cpu(), want[t]) < 2e-2, t
    simt = R.paged_attention(q, cache, w.token_to_seq(), w.token_positions(), w.block_tables())
    assert _rel_err(got, simt) < 1e-2


@pytest.mark.gpu
@pytest.mark.parametrize("Hq,Hk,D", [(32, 8, 128), (8, 1, 128), (16, 8, 64)])
def test_packed_decode_atoms_match_oracle(Hq, Hk, D):
    """Decode-only batch: every atom has one query, the whole GQA group shares a tile (one CTA per KV head)."""
    from shuffle_exchange_b200.inference.v2.kernels import ragged_ops as R
    torch.manual_seed(4)
    bs, ctx = 64, [1, 63, 64, 65, 700, 1023, 130, 5]
    cache = torch.randn(sum((c + bs) // bs for c in ctx) + 1, bs, 2, Hk, D, device="cuda", dtype=torch.bfloat16)
    w = RaggedBatchWrapper(64, len(ctx), 17, device="cuda")
    nxt = 0
    for c in ctx:
        need = (c + 1 + bs - 1) // bs
        w.insert_sequence(_Seq(c, list(range(nxt, nxt + need))), torch.zeros(1, dtype=torch.int64))
        nxt += need
    w.finalize()
    assert w.atoms_longer_than(128 // (Hq // Hk)) == 0
    q = torch.randn(len(ctx), Hq, D, device="cuda", dtype=torch.bfloat16)
    got = R.ragged_attention(q, cache, w)
    want = R.paged_attention(q.cpu(), cache.cpu(), w.token_to_seq().cpu(), w.token_positions().cpu(),
                             w.block_tables().cpu())
    for t in range(len(ctx)):
        assert _rel_err(got[t].cpu(), want[t]) < 2e-2, (t, ctx[t])


@pytest.mark.gpu
def test_atom_attention_on_fused_qkv_view():
    """q as a strided view of the fused QKV projection output (what the model passes)."""
    from shuffle_exchange_b200.inference.v2.kernels import ragged_ops as R
    torch.manual_seed(3)
    Hq, Hk, D, bs = 8, 2, 128, 64
    cache = torch.randn(32, bs, 2, Hk, D, device="cuda", dtype=torch.bfloat16)
    w = RaggedBatchWrapper(512, 4, 8, device="cuda")
    w.insert_sequence(_Seq(0, [5, 9, 2]), torch.zeros(150, dtype=torch.int64))
    w.finalize()
    qkv = torch.randn(150, (Hq + 2 * Hk) * D, device="cuda", dtype=torch.bfloat16)
    q = qkv.view(150, Hq + 2 * Hk, D)[:, :Hq]
    got = R.ragged_attention(q, cache, w, scale=1.0 / math.sqrt(D))
    want = R.paged_attention(q.contiguous(), cache, w.token_to_seq(), w.token_positions(), w.block_tables())
    assert _rel_err(got, want) < 1e-2


_VARIANT_SCRIPT = r"""
import torch, sys
from shuffle_exchange_b200.ops import functional as F
from shuffle_exchange_b200.native import lib
torch.manual_seed(0)
worst = 0.0
for (B, S, Hq, Hk, causal) in [(1, 512, 4, 2, True), (2, 300, 4, 1, True), (1, 1024, 2, 1, False), (1, 129, 8, 2, True)]:
    q = torch.randn(B, S, Hq, 128, device="cuda", dtype=torch.bfloat16)
    k = torch.randn(B, S, Hk, 128, device="cuda", dtype=torch.bfloat16)
    v = torch.randn(B, S, Hk, 128, device="cuda", dtype=torch.bfloat16)
    out, lse = F.attention_fwd_lse(q, k, v, causal, 128 ** -0.5)
    ref = F.attention_ref(q.float(), k.float(), v.float(), causal)
    worst = max(worst, ((out.float() - ref).norm() / ref.norm()).item())
    qf = q.float().permute(0, 2, 1, 3); kf = k.float().permute(0, 2, 1, 3).repeat_interleave(Hq // Hk, 1)
    s = qf @ kf.transpose(-1, -2) * 128 ** -0.5
    if causal:
        s = s.masked_fill(~torch.ones(S, S, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    worst = max(worst, (lse - torch.logsumexp(s, -1)).abs().max().item())
assert lib.hang_info("attn") is None
print("WORST", worst)
"""


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["1", "2"])
def test_forward_kernel_variants(mode):
    """SXB_ATTN_FWD128=1 (128-key blocks) and =2 (two heads of a GQA group per CTA) compute the same attention as the
    default kernel; the switch is read once per process, hence the subprocess."""
    import os
    import subprocess
    import sys
    env = dict(os.environ, SXB_ATTN_FWD128=mode)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _VARIANT_SCRIPT], capture_output=True, text=True, env=env, cwd=root,
                       timeout=200)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    worst = float(r.stdout.strip().split("WORST")[-1])
    assert worst < 1e-2, worst


@pytest.mark.gpu
@pytest.mark.parametrize("B,S,Hq,Hk,D,causal", [(2, 256, 4, 2, 128, False), (3, 300, 2, 2, 64, False), (2, 512, 4, 1, 128, True)])
def test_key_bias_attention_forward_backward(B, S, Hq, Hk, D, causal):
    """Additive per-key bias (key-padding mask with -inf / -1e4 entries) inside the flash kernels vs fp32 softmax."""
    from shuffle_exchange_b200.ops import functional as F
    torch.manual_seed(5)
    dev = "cuda"
    q, k, v = (torch.randn(B, S, h, D, device=dev, dtype=torch.bfloat16, requires_grad=True) for h in (Hq, Hk, Hk))
    bias = torch.zeros(B, S, device=dev)
    for b_ in range(B):                                   # a different padded tail per sample, never the whole row
        bias[b_, S - 17 * (b_ + 1):] = float("-inf") if b_ % 2 == 0 else -1e4
    bias[:, 5] = 0.7                                       # and a finite bias somewhere
    assert F.key_bias_supported(q, bias)
    out = F.flash_attention_key_bias(q, k, v, bias, causal=causal)
    g = torch.randn_like(out)
    out.backward(g)
    ref_in = [t.detach().float().requires_grad_(True) for t in (q, k, v)]
    qf = ref_in[0].permute(0, 2, 1, 3)
    kf = ref_in[1].permute(0, 2, 1, 3).repeat_interleave(Hq // Hk, dim=1)
    vf = ref_in[2].permute(0, 2, 1, 3).repeat_interleave(Hq // Hk, dim=1)
    sc = qf @ kf.transpose(-1, -2) * D ** -0.5 + bias[:, None, None, :]
    if causal:
        sc = sc.masked_fill(~torch.ones(S, S, dtype=torch.bool, device=dev).tril(), float("-inf"))
    ref = (sc.softmax(-1) @ vf).permute(0, 2, 1, 3)
    ref.backward(g.float())
    assert _rel_err(out, ref) < 1e-2
    for got, want in zip((q, k, v), ref_in):
        assert torch.isfinite(got.grad).all()
        assert _rel_err(got.grad, want.grad) < 3e-2
    # masked keys receive no gradient through the scores: dK of a -inf key is exactly zero
    assert float(k.grad[0, S - 1].abs().max()) == 0.0


@pytest.mark.gpu
def test_training_transformer_layer_uses_flash_kernels_for_padding_masks():
    from shuffle_exchange_b200.native import lib
    from shuffle_exchange_b200.ops import functional as F
    from shuffle_exchange_b200.ops.transformer import transformer as T
    torch.manual_seed(6)
    B, S, H, Dh = 2, 128, 4, 64

    class _Cfg:
        heads, hidden_size, attn_dropout_ratio = H, H * Dh, 0.0

    class _Layer:
        config, training = _Cfg, False
    qkv = torch.randn(B, S, 3 * H * Dh, device="cuda", dtype=torch.bfloat16)
    mask = torch.zeros(B, 1, 1, S, device="cuda")
    mask[1, ..., 100:] = -1e4
    before = lib.launch_count
    got = T._attention(_Layer, qkv, mask)
    assert lib.launch_count > before                      # went through the native library, not torch.matmul
    q, k, v = qkv.view(B, S, 3, H, Dh).unbind(2)
    want = F.flash_attention_key_bias(q.float().cpu(), k.float().cpu(), v.float().cpu(), mask.reshape(B, S).cpu())
    assert _rel_err(got.cpu().view(B, S, H, Dh), want) < 1e-2


@pytest.mark.gpu
def test_per_head_key_bias_alibi_style():
    """[B, Hq, S] bias (slope_h x key position, as BLOOM's alibi tensor) with GQA: every q head reads its own row in the
    forward, the dQ and the dK/dV kernels."""
    from shuffle_exchange_b200.ops import functional as F
    torch.manual_seed(7)
    B, S, Hq, Hk, D = 2, 384, 8, 2, 128
    dev = "cuda"
    q, k, v = (torch.randn(B, S, h, D, device=dev, dtype=torch.bfloat16, requires_grad=True) for h in (Hq, Hk, Hk))
    slopes = torch.tensor([2.0 ** (-(i + 1)) for i in range(Hq)], device=dev)
    bias = (slopes[None, :, None] * torch.arange(S, device=dev)[None, None, :] * 0.05).expand(B, Hq, S).contiguous()
    bias[1, :, S - 40:] = float("-inf")
    out = F.flash_attention_key_bias(q, k, v, bias, causal=True)
    g = torch.randn_like(out)
    out.backward(g)
    ref_in = [t.detach().float().requires_grad_(True) for t in (q, k, v)]
    qf = ref_in[0].permute(0, 2, 1, 3)
    kf = ref_in[1].permute(0, 2, 1, 3).repeat_interleave(Hq // Hk, dim=1)
    vf = ref_in[2].permute(0, 2, 1, 3).repeat_interleave(Hq // Hk, dim=1)
    sc = qf @ kf.transpose(-1, -2) * D ** -0.5 + bias[:, :, None, :]
    sc = sc.masked_fill(~torch.ones(S, S, dtype=torch.bool, device=dev).tril(), float("-inf"))
    ref = (sc.softmax(-1) @ vf).permute(0, 2, 1, 3)
    ref.backward(g.float())
    assert _rel_err(out, ref) < 1e-2
    for got, want in zip((q, k, v), ref_in):
        assert torch.isfinite(got.grad).all()
        assert _rel_err(got.grad, want.grad) < 3e-2


@pytest.mark.gpu
@pytest.mark.parametrize("D", [32, 80, 96])
def test_other_head_sizes_run_zero_padded(D):
    from shuffle_exchange_b200.ops import functional as F
    torch.manual_seed(8)
    B, S, Hq, Hk = 2, 200, 4, 2
    q, k, v = (torch.randn(B, S, h, D, device="cuda", dtype=torch.bfloat16, requires_grad=True) for h in (Hq, Hk, Hk))
    out = F.flash_attention(q, k, v, causal=True)
    assert out.shape == (B, S, Hq, D)
    g = torch.randn_like(out)
    out.backward(g)
    ref_in = [t.detach().float().requires_grad_(True) for t in (q, k, v)]
    ref = F.attention_ref(*ref_in, True)
    ref.backward(g.float())
    assert _rel_err(out, ref) < 1e-2
    for got, want in zip((q, k, v), ref_in):
        assert got.grad.shape == want.grad.shape and _rel_err(got.grad, want.grad) < 3e-2
