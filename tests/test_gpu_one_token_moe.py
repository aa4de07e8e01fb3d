"""One token through a block of a mixture-of-experts model: the launches made for it against the same block on rows of a prompt, bit for bit."""
import numpy as np
import pytest
from tinygrad_b200 import synth
from gpu_util import need_gpu

pytestmark = pytest.mark.gpu


# one expert; fewer than a cluster's warps, more than a warp's lanes (fp16 router), more than 64 and the most, more choices than rows loaded ahead; widths below and above
# a thread's first pieces; every gating but the default's, with a shared expert; attention rows of the most values that one CTA takes, and of more (the launches of rows then)
@pytest.mark.parametrize("dim,f,E,k,router,extra", [
  (256, 128, 1, 1, np.float32, {}), (768, 768, 8, 6, np.float32, {}), (1280, 1152, 40, 3, np.float16, dict(norm_topk_prob=True)),
  (512, 512, 130, 9, np.float32, dict(expert_gating_func="sigmoid", norm_topk_prob=True, routed_scaling_factor=2.0, shared_expert_dim=128)),
  (2304, 128, 256, 32, np.float32, dict(expert_gating_func="sqrt_softplus", expert_bias=True, shared_expert_dim=96, shared_expert_gate=False)),
  (256, 128, 8, 2, np.float32, dict(n_heads=96, n_kv_heads=8, head_dim=128, rope_dim=128)), (256, 128, 8, 2, np.float32, dict(n_heads=97, n_kv_heads=1, head_dim=128, rope_dim=128))])
def test_one_token_block_is_the_row_block(dim, f, E, k, router, extra):
  need_gpu()
  from tinygrad_b200 import _lib
  from tinygrad_b200.model import Transformer, TransformerConfig
  kw = dict(num_blocks=2, dim=dim, hidden_dim=f, n_heads=dim // 64, n_kv_heads=dim // 128, norm_eps=1e-5, vocab_size=64, head_dim=64, rope_theta=10000.0, rope_dim=64,
            max_context=64, num_experts=E, num_experts_per_tok=k) | extra
  cfg, rng = TransformerConfig(**kw), np.random.default_rng(dim + k)
  sd = {n: v for n, v in synth.dense_model_raw(cfg, 8, seed=7, embd_std=0.3, scale_std=0.0015).items() if ".ffn_gate." not in n and ".ffn_up." not in n and ".ffn_down." not in n}
  sh = cfg.shared_expert_dim
  for i in range(2):
    sd[f"blk.{i}.ffn_gate_inp.weight"] = (rng.standard_normal((E, dim)) / np.sqrt(dim)).astype(router)
    for n, shape in (("gate", (E, f, dim)), ("up", (E, f, dim)), ("down", (E, dim, f))):
      sd[f"blk.{i}.ffn_{n}_exps.weight"] = (rng.standard_normal(shape) / np.sqrt(shape[2])).astype(np.float32)
    if cfg.expert_bias: sd[f"blk.{i}.exp_probs_b.bias"] = (rng.standard_normal(E) * 0.3).astype(np.float32)
    if sh:
      for n, (o, ii) in (("ffn_gate_shexp", (sh, dim)), ("ffn_up_shexp", (sh, dim)), ("ffn_down_shexp", (dim, sh))):
        sd[f"blk.{i}.{n}.weight"] = synth.q8_0_blocks(o, ii, rng, scale_std=0.0015)
      if cfg.shared_expert_gate: sd[f"blk.{i}.ffn_gate_inp_shexp.weight"] = (rng.standard_normal(dim) * 0.1).astype(np.float32)
  m = Transformer(cfg, sd, ggml_type=8)
  m.set_state([int(t) for t in rng.integers(0, 64, 12)], 0)
  m.prefill(0, 12)
  out = []
  for pos in (None, m.pos):
    m.pos.copy_from(np.array([11], np.int32))
    _lib.check(_lib.load().b200q_moe_rows(m._row_arguments(), m._native_moe(1), 0, 11, pos.ptr if pos else None, 1, m.stream.ptr))
    m.stream.synchronize()
    tables = [[getattr(b.moe._workspace(1)["r"], n).numpy().copy() for n in ("topi", "weights", "dest_row", "off")] + [b.moe._workspace(1)["ends"].numpy().copy()] for b in m.blk]
    out.append([m._prefill_buffers()["x"].numpy()[0].copy(), m.blk[1].k_cache.numpy().copy(), m.blk[1].v_cache.numpy().copy(), *(t for b in tables for t in b)])
  for a, b in zip(*out): np.testing.assert_array_equal(a, b)
  assert np.isfinite(out[0][0]).all() and np.abs(out[0][0]).max() > 0
