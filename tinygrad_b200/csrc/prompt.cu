// A stretch of prompt rows through every block of a dense model, launched from native code: Transformer.forward for T > 1 tokens
// (tinygrad/llm/model.py:358-362) over one or several sequences of equal length.
// Per block: split (+ RMSNorm) and QKV GEMM, RoPE + cache append, causal attention, split and O GEMM (+ residual), split (+ RMSNorm) and
// gate/up GEMM (SwiGLU), split and down GEMM (+ residual); every launch programmatic, so the next kernel's prologue runs under the tail of
// the one before.  As one ctypes call per Linear the host took 35 us per block, as much as the device for a short prompt.
#include "common.cuh"

int b200q_embed_rows_seqs(const void* table_f16, const int32_t* tokens, int token_stride, int per_seq, int n_rows, int dim, int vocab, float* x, cudaStream_t st);

// kv_only: the last block only leaves its cache rows; x keeps what goes into it.  What else it would compute nobody reads when the last token's logits are all that is
// wanted: of a prompt of 1999 tokens on ten 7B-shaped blocks that was 2.3 ms, and the last token as a step of its own 0.7 (29.8 -> 26.8 ms; 45 tokens on 16 8B-shaped blocks
// 3.08 -> 2.41 ms; eight prompts of 128 and 32 answers on seven blocks 29.1 -> 27.4 ms).
static int prompt_rows(const b200q_rows_args* a, int first_seq, int n_seqs, int start_pos, int n_rows, bool kv_only, void* stream) {
  if (!a || !a->layers || !a->token_embd || !a->rope || !a->tokens || !a->x || !a->qkv || !a->q || !a->att || !a->act || !a->workspace) return B200Q_ERR_BAD_ARG;
  if (first_seq < 0 || n_seqs <= 0 || start_pos < 0 || n_rows <= 0 || a->n_layers < 0 || (long long)n_seqs * n_rows > a->rows_max) return B200Q_ERR_BAD_ARG;
  if (start_pos + n_rows > a->max_context) return B200Q_ERR_TOO_LARGE;
  cudaStream_t st = (cudaStream_t)stream;
  const int T = n_seqs * n_rows, q_dim = a->n_heads * a->head_dim, qkv_rows = q_dim + 2 * a->n_kv_heads * a->head_dim;
  const size_t seq_bytes = (size_t)a->n_kv_heads * a->max_context * a->head_dim * (a->kv_dtype == B200Q_F16 ? 2 : 4);
  const int stride = a->max_context + 1;
  int rc = b200q_embed_rows_seqs(a->token_embd, a->tokens + (size_t)first_seq * stride + start_pos, stride, n_rows, T, a->dim, a->vocab, a->x, st);
  for (int i = 0; i < a->n_layers && rc == B200Q_OK; i++) {
    const b200q_decode_layer& l = a->layers[i];
    const bool kv = kv_only && i == a->n_layers - 1;
    rc = b200q_qgemm_chain(a->qtype, l.qkv, a->x, B200Q_F32, l.attn_norm, a->norm_eps, l.qkv_bias, nullptr, B200Q_EPI_LINEAR, a->qkv, B200Q_F32, T, qkv_rows,
                             a->dim, a->workspace, a->workspace_bytes, st, true);
    if (rc == B200Q_OK)
      rc = b200q_attn_rows_chain(a->qkv, (char*)l.k_cache + first_seq * seq_bytes, (char*)l.v_cache + first_seq * seq_bytes, a->kv_dtype, a->rope, start_pos, n_rows,
                                   n_seqs, a->n_heads, a->n_kv_heads, a->head_dim, a->rope_dim, a->max_context, a->q, kv ? nullptr : a->att, B200Q_F32, st, true);
    if (kv) break;
    if (rc == B200Q_OK)
      rc = b200q_qgemm_chain(a->qtype, l.attn_output, a->att, B200Q_F32, nullptr, 0.f, nullptr, a->x, B200Q_EPI_LINEAR, a->x, B200Q_F32, T, a->dim, q_dim, a->workspace,
                          a->workspace_bytes, st, true);
    if (rc == B200Q_OK)
      rc = b200q_qgemm_chain(a->qtype, l.gate_up, a->x, B200Q_F32, l.ffn_norm, a->norm_eps, nullptr, nullptr, B200Q_EPI_SILU_MUL, a->act, B200Q_F32, T,
                               2 * a->hidden_dim, a->dim, a->workspace, a->workspace_bytes, st, true);
    if (rc == B200Q_OK)
      rc = b200q_qgemm_chain(a->qtype, l.ffn_down, a->act, B200Q_F32, nullptr, 0.f, nullptr, a->x, B200Q_EPI_LINEAR, a->x, B200Q_F32, T, a->dim, a->hidden_dim, a->workspace,
                          a->workspace_bytes, st, true);
  }
  return rc;
}
extern "C" int b200q_prompt_rows(const b200q_rows_args* a, int first_seq, int n_seqs, int start_pos, int n_rows, void* stream) {
  return prompt_rows(a, first_seq, n_seqs, start_pos, n_rows, false, stream);
}
extern "C" int b200q_prompt_rows_kv(const b200q_rows_args* a, int first_seq, int n_seqs, int start_pos, int n_rows, void* stream) {
  return prompt_rows(a, first_seq, n_seqs, start_pos, n_rows, true, stream);
}

// x += the shared expert's output on the normed rows xn (times its gate, where it has one)
static int shared_expert(const b200q_rows_args* a, const b200q_moe_block& b, int T, cudaStream_t st) {
  auto gemm = [&](const void* w, const float* x, int epilogue, float* y, int n_out, int n_in) {
    return b200q_qgemm_chain(a->qtype, w, x, B200Q_F32, nullptr, 0.f, nullptr, nullptr, epilogue, y, B200Q_F32, T, n_out, n_in, a->workspace, a->workspace_bytes, st, true, true);
  };
  int rc = gemm(b.sh_gate_up, b.xn, B200Q_EPI_SILU_MUL, b.sh_act, 2 * b.shared_dim, a->dim);
  if (rc == B200Q_OK) rc = gemm(b.sh_down, b.sh_act, B200Q_EPI_LINEAR, b.sh, a->dim, b.shared_dim);
  if (rc == B200Q_OK && b.sh_inp)
    rc = b200q_gemv_dense(b.sh_inp, b.sh_inp_dtype, 1, a->dim, T, b.xn, B200Q_F32, nullptr, 0.f, nullptr, nullptr, b.shg, B200Q_F32, B200Q_FLAG_PDL, st);
  return rc == B200Q_OK ? b200q_add_rows_gated_chain(a->x, b.sh, b.sh_inp ? b.shg : nullptr, T, a->dim, st) : rc;
}

// One token through the blocks of a mixture-of-experts model: nine launches a block where rows take 14, the same values bit for bit (8 tokens of a 1024-wide model of 4 blocks, 32
// experts top 4: with the narrow tiles of the expert GEMMs 2360 -> 1660 us, 480 of them these launches).  What stands between the GEMMs is one
// launch each (prepare_row_kernel, moe_router_kernel); a block's weighted sum of its experts is taken by the next block's first one.
static int moe_one_token(const b200q_rows_args* a, const b200q_moe_block* blocks, const int32_t* pos_dev, cudaStream_t st) {
  const int q_dim = a->n_heads * a->head_dim, qkv_rows = q_dim + 2 * a->n_kv_heads * a->head_dim;
  auto gemm = [&](const void* w, const float* x, const void* bias, const float* residual, int epilogue, float* y, int n_out, int n_in, const b200q_row_input* one) {
    return b200q_qgemm_chain(a->qtype, w, x, B200Q_F32, nullptr, 0.f, bias, residual, epilogue, y, B200Q_F32, 1, n_out, n_in, a->workspace, a->workspace_bytes, st, true, true, one);
  };
  int rc = B200Q_OK;
  for (int i = 0; i < a->n_layers && rc == B200Q_OK; i++) {
    const b200q_decode_layer& l = a->layers[i];
    const b200q_moe_block& b = blocks[i];
    const b200q_moe_args* before = i ? blocks[i - 1].moe : nullptr;
    const b200q_row_input in{a->x, before ? before->y : nullptr, before ? before->dest_row : nullptr, before ? before->weights : nullptr, before ? before->k : 0, l.attn_norm,
                             a->norm_eps}, att{a->att, nullptr, nullptr, nullptr, 0, nullptr, 0.f};
    rc = gemm(l.qkv, a->x, l.qkv_bias, nullptr, B200Q_EPI_LINEAR, a->qkv, qkv_rows, a->dim, &in);
    if (rc == B200Q_OK)
      rc = b200q_attn_rows_pos_chain(a->qkv, l.k_cache, l.v_cache, a->kv_dtype, a->rope, pos_dev, a->n_heads, a->n_kv_heads, a->head_dim, a->rope_dim, a->max_context, a->q,
                                     a->att, B200Q_F32, st);
    if (rc == B200Q_OK) rc = gemm(l.attn_output, a->att, nullptr, a->x, B200Q_EPI_LINEAR, a->x, a->dim, q_dim, &att);
    if (rc == B200Q_OK) rc = b200q_moe_router_one(b.moe, b.router, b.router_dtype, a->x, l.ffn_norm, a->norm_eps, b.shared_dim ? b.xn : nullptr, st);
    if (rc == B200Q_OK && b.shared_dim) rc = shared_expert(a, b, 1, st);
    if (rc == B200Q_OK) rc = b200q_moe_gemms_chain(b.moe, 1, st);
  }
  return rc == B200Q_OK && a->n_layers > 0 ? b200q_moe_combine_chain(blocks[a->n_layers - 1].moe, 1, a->x, st) : rc;
}

// The same for a mixture-of-experts model: the FFN of a block is the router, the expert layer and, where the model has one, the shared expert
// (tinygrad/llm/model.py:110-134).  The GEMMs' sums are not split (see b200q_qgemm_ws_norm), so a token's expert choice does not depend on the rows it
// came with.  pos_dev: one row of sequence 0 at the position kept on the device (graph replay).  As single calls, each fully ordered behind the one
// before, a one-token block took 19 launches and 95 us (1024-wide, 32 experts); here 14, programmatic.
extern "C" int b200q_moe_rows(const b200q_rows_args* a, const b200q_moe_block* blocks, int seq, int start_pos, const int32_t* pos_dev, int n_rows, void* stream) {
  if (!a || !blocks || !a->layers || !a->token_embd || !a->rope || !a->tokens || !a->x || !a->qkv || !a->q || !a->att || !a->workspace) return B200Q_ERR_BAD_ARG;
  if (seq < 0 || start_pos < 0 || n_rows <= 0 || a->n_layers < 0 || n_rows > a->rows_max || (pos_dev && (n_rows != 1 || seq != 0))) return B200Q_ERR_BAD_ARG;
  if (!pos_dev && start_pos + n_rows > a->max_context) return B200Q_ERR_TOO_LARGE;
  cudaStream_t st = (cudaStream_t)stream;
  const int T = n_rows, q_dim = a->n_heads * a->head_dim, qkv_rows = q_dim + 2 * a->n_kv_heads * a->head_dim;
  const size_t seq_bytes = (size_t)a->n_kv_heads * a->max_context * a->head_dim * (a->kv_dtype == B200Q_F16 ? 2 : 4);
  auto gemm = [&](const void* w, const float* x, const void* bias, const float* residual, int epilogue, float* y, int n_out, int n_in) {
    return b200q_qgemm_chain(a->qtype, w, x, B200Q_F32, nullptr, 0.f, bias, residual, epilogue, y, B200Q_F32, T, n_out, n_in, a->workspace, a->workspace_bytes, st, true, true);
  };
  int rc = pos_dev ? b200q_embed_rows(a->token_embd, a->tokens, 1, pos_dev, 1, a->dim, a->vocab, a->x, stream)
                   : b200q_embed_rows_seqs(a->token_embd, a->tokens + (size_t)seq * (a->max_context + 1) + start_pos, a->max_context + 1, T, T, a->dim, a->vocab, a->x, st);
  for (int i = 0; i < a->n_layers; i++) if (!blocks[i].moe || !blocks[i].router || !blocks[i].xn || !blocks[i].xb || !blocks[i].logits) return B200Q_ERR_BAD_ARG;
  bool one = pos_dev != nullptr && a->dim <= B200Q_ROW_INPUT_MAX && q_dim <= B200Q_ROW_INPUT_MAX;
  for (int i = 0; i < a->n_layers; i++) one = one && b200q_moe_router_one_takes(blocks[i].moe, blocks[i].router_dtype);
  if (one && rc == B200Q_OK) return moe_one_token(a, blocks, pos_dev, st);
  for (int i = 0; i < a->n_layers && rc == B200Q_OK; i++) {
    const b200q_decode_layer& l = a->layers[i];
    const b200q_moe_block& b = blocks[i];
    rc = b200q_rmsnorm_rows_chain(a->x, l.attn_norm, a->norm_eps, T, a->dim, b.xn, nullptr, st);
    if (rc == B200Q_OK) rc = gemm(l.qkv, b.xn, l.qkv_bias, nullptr, B200Q_EPI_LINEAR, a->qkv, qkv_rows, a->dim);
    if (rc == B200Q_OK)
      rc = pos_dev ? b200q_attn_rows_pos_chain(a->qkv, l.k_cache, l.v_cache, a->kv_dtype, a->rope, pos_dev, a->n_heads, a->n_kv_heads, a->head_dim, a->rope_dim, a->max_context,
                                               a->q, a->att, B200Q_F32, st)
                   : b200q_attn_rows_chain(a->qkv, (char*)l.k_cache + seq * seq_bytes, (char*)l.v_cache + seq * seq_bytes, a->kv_dtype, a->rope, start_pos, T, 1, a->n_heads,
                                           a->n_kv_heads, a->head_dim, a->rope_dim, a->max_context, a->q, a->att, B200Q_F32, st, true);
    if (rc == B200Q_OK) rc = gemm(l.attn_output, a->att, nullptr, a->x, B200Q_EPI_LINEAR, a->x, a->dim, q_dim);
    // router on the fp32 normed rows, experts on their bf16 rounding (the activation type of the MXFP8 path)
    if (rc == B200Q_OK) rc = b200q_rmsnorm_rows_chain(a->x, l.ffn_norm, a->norm_eps, T, a->dim, b.xn, b.xb, st);
    if (rc == B200Q_OK)
      rc = b200q_gemv_dense(b.router, b.router_dtype, b.moe->n_experts, a->dim, T, b.xn, B200Q_F32, nullptr, 0.f, nullptr, nullptr, b.logits, B200Q_F32, B200Q_FLAG_PDL, stream);
    if (rc == B200Q_OK && b.shared_dim) rc = shared_expert(a, b, T, st);
    if (rc == B200Q_OK) rc = b200q_moe_layer_chain(b.moe, b.xb, b.logits, T, a->x, st, true);
  }
  return rc;
}
