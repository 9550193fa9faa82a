// ragged_llama.cu — one forward of a dense Llama over a ragged batch, its kernels issued from here.
//
// The kernels are those of the operators' own entry points, in the same order and on the same operands (a product of few rows takes
// its activation along, with the same bits): this entry only takes the
// way from one launch to the next out of Python, which a decode step of a few requests spends its time on (4 layers of 2048, 4
// requests, prompts and six decode steps: 5.53 ms from Python, 2.88 this way, 2.4 of device work).  Nothing is kept between calls.
// The launches form a chain (sxb_common.cuh): a kernel comes onto the SMs while the one before it still runs, so that its launch, its
// set-up and a product's first weights are behind it when its operands are there: 2.88 -> 2.40 ms.
#include "sxb_common.cuh"
#include "sxb200.h"

SXB_API int sxb_ragged_llama_forward(struct sxb_ragged_llama* m, const struct sxb_ragged_llama_layer* layers, int n_layers,
                                     float eps, float theta, float scale, void* stream) {
  using namespace sxb;
  if (m == nullptr || (n_layers > 0 && layers == nullptr)) return SXB_ERR_BAD_ARG;
  const int T = (int)m->T, H = (int)m->H, F = (int)m->F, Hq = (int)m->Hq, Hk = (int)m->Hk, D = (int)m->D;
  const int C = (Hq + 2 * Hk) * D, Q = Hq * D;
  int rc;
  m->calls = 4;                // embedding, last norm, rows of the last tokens, head; eight or nine a layer
  auto product = [&](const void* x, const void* w, long long ldw, void* y, int rows, int n, int k) {
    return sxb_gemm_bf16(x, w, y, rows, n, k, 0, k, (int)ldw, n, kBF16, 0, 1.0f, 0, stream);
  };
  // h: what the last sublayer left; res: the stream before it (none at first).  A norm writes their sum over the third buffer.
  void *h = m->buf[0], *res = nullptr, *spare[2] = {m->buf[1], m->buf[2]};
  auto norm = [&](const void* w) -> int {
    void* sum = spare[0];
    if ((rc = sxb_rmsnorm_fwd(h, res, w, m->x, res ? sum : nullptr, nullptr, T, H, eps, kBF16, stream))) return rc;
    if (res == nullptr) {
      res = h; h = spare[0]; spare[0] = spare[1];
    } else {
      spare[0] = res; res = sum;
    }
    return SXB_OK;
  };
  if ((rc = sxb_ragged_embed(m->ids, nullptr, m->embed, nullptr, h, T, H, 0, stream))) return rc;
  const ChainScope chain;      // everything below reads only what kernels above wrote, the batch's tables and the weights
  for (int i = 0; i < n_layers; ++i) {
    const struct sxb_ragged_llama_layer& l = layers[i];
    if ((rc = norm(l.ln1))) return rc;
    if ((rc = product(m->x, l.wqkv, l.ld_qkv, m->qkv, T, C, H))) return rc;
    if ((rc = sxb_kv_rotary_blocked(m->qkv, l.cache, m->tok_seq, m->tok_pos, m->block_tables, T, (int)m->max_blocks,
                                    (int)m->block_size, Hq, Hk, D, D, theta, stream))) return rc;
    if ((rc = sxb_attn_fwd_atoms_keys(m->qkv, l.cache, m->ctx, m->atoms, (int)m->n_atoms, (int)m->n_packed, (int)m->n_few,
                                      m->few_keys, (int)m->few_most, m->block_tables, (int)m->max_blocks, (int)m->n_blocks,
                                      (int)m->block_size, T, Hq, Hk, D, C, Q, scale, stream))) return rc;
    if ((rc = product(m->ctx, l.wo, l.ld_o, h, T, H, Q))) return rc;
    if ((rc = norm(l.ln2))) return rc;
    m->calls += 8;
    rc = sxb_gemm_gated(m->x, l.w_gate_up, m->act, T, F, H, H, (int)l.ld_gate_up, F, 3, stream);
    if (rc == SXB_ERR_UNSUPPORTED) {      // many rows: the product and its activation one after the other, the same bits
      if ((rc = product(m->x, l.w_gate_up, l.ld_gate_up, m->gate_up, T, 2 * F, H))) return rc;
      rc = sxb_gated_act_fwd(m->gate_up, nullptr, m->act, T, F, 3, kBF16, stream);
      ++m->calls;
    }
    if (rc) return rc;
    if ((rc = product(m->act, l.w_down, l.ld_down, h, T, H, F))) return rc;
  }
  if ((rc = norm(m->norm))) return rc;
  if ((rc = sxb_logits_gather(m->x, m->last_token, m->rows, (int)m->n_rows, H, stream))) return rc;
  return product(m->rows, m->head, m->ld_head, m->logits, (int)m->n_rows, (int)m->vocab, H);
}
