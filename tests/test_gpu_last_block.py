"""A prompt's last token, which goes along with the others up to the last block: against one-token steps, at the edges of the passes."""
import numpy as np
import pytest
from tinygrad_b200 import synth
from gpu_util import need_gpu

pytestmark = pytest.mark.gpu

KW = dict(num_blocks=2, dim=256, hidden_dim=640, n_heads=4, n_kv_heads=2, norm_eps=1e-5, vocab_size=512, head_dim=64, rope_theta=500000.0, rope_dim=64, max_context=64)


def _model(**kw):
  from tinygrad_b200.model import Transformer, TransformerConfig
  opts = {k: kw.pop(k) for k in list(kw) if k in ("num_blocks", "kv_dtype", "head_dim", "rope_dim", "n_heads", "n_kv_heads")}
  cfg = TransformerConfig(**{**KW, **opts})
  return Transformer(cfg, synth.dense_model_raw(cfg, 8, seed=3, embd_std=0.3, scale_std=0.0015), ggml_type=8, **kw)


def _first(m, prompt, n=3):
  out, logits = [], None
  for tok in m.generate(list(prompt)):
    if logits is None: logits = m.read_logits().astype(np.float64)
    out.append(tok)
    if len(out) == n: return out, logits
  return out, logits


# a pass of 16 rows: all in one, one row behind it (steps), two rows behind it, one row behind two passes, a full context but one; one block only; fp32 cache; other
# heads; launches one by one; every hand-over between the block's kernels
@pytest.mark.parametrize("tokens,opts", [(12, {}), (16, {}), (17, {}), (18, {}), (33, {}), (63, {}), (18, dict(num_blocks=1)), (30, dict(kv_dtype="float32")),
                                         (20, dict(head_dim=32, rope_dim=32, n_heads=8, n_kv_heads=4)), (20, dict(use_graph=False)),
                                         (20, dict(head_dim=128, rope_dim=128, n_heads=2, n_kv_heads=1, handover=True))])
def test_last_token_goes_along(tokens, opts):
  """Greedy tokens as from one-token steps, and the first logits and the caches as near as the steps' 15-bit activation codes leave them."""
  need_gpu()
  prompt = [int(t) for t in np.random.default_rng(tokens).integers(0, 512, tokens)]
  n = min(3, 64 - tokens)
  rows, steps = _model(prefill_chunk=16, **dict(opts)), _model(prefill_rows=0, **dict(opts))
  got, lg = _first(rows, prompt, n)
  want, lw = _first(steps, prompt, n)
  assert got == want
  assert np.linalg.norm(lg - lw) <= 3e-3 * np.linalg.norm(lw)
  for a, b in zip(rows.blk, steps.blk):
    for x, y in ((a.k_cache, b.k_cache), (a.v_cache, b.v_cache)):
      x, y = x.numpy().astype(np.float64), y.numpy().astype(np.float64)
      assert np.linalg.norm(x - y) <= 3e-3 * np.linalg.norm(y)
  if tokens < 60 and opts == {}:      # the same once more on a conversation: part of the prompt is cached, the captured launches are replayed
    more = prompt + got + [int(t) for t in np.random.default_rng(0).integers(0, 512, 14)]
    assert _first(rows, more) [0] == _first(steps, more)[0]


# two sequences a pass (with a last pass of one), all in one pass, as many passes more as last tokens would cost (steps), one sequence a pass (steps); the GEMM instead of
# the few-row kernel
@pytest.mark.parametrize("batch,tokens,chunk", [(5, 8, 16), (3, 7, 32), (4, 9, 17), (2, 12, 16), (19, 10, 40)])
def test_last_tokens_of_a_batch_go_along(batch, tokens, chunk):
  need_gpu()
  rng = np.random.default_rng(batch)
  prompts = [[int(t) for t in rng.integers(0, 512, tokens)] for _ in range(batch)]
  m, got = _model(batch=batch, prefill_chunk=chunk), []
  for toks in m.generate_batch(prompts):
    got.append(toks)
    if len(got) == 3: break
  one = _model(prefill_rows=0)
  assert [list(t) for t in zip(*got)] == [_first(one, p)[0] for p in prompts]
  again = next(m.generate_batch([p[::-1] for p in prompts]))
  assert again == [_first(one, p[::-1], 1)[0][0] for p in prompts]


# prompts that go in one pass, and below `prefill_rows` in steps; a batch of one is the default model
@pytest.mark.parametrize("batch", [1, 3])
@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("order", ["one batch one batch", "batch one batch one", "short batch one short", "batch short one batch"])
def test_one_model_answers_prompts_and_batches(order, batch, use_graph):
  """What one model says to single prompts and to batches in turn, tokens, logits and all: as one that has done nothing else."""
  need_gpu()
  kw = dict(batch=batch, prefill_chunk=32, use_graph=use_graph)
  m = _model(**kw)
  for i, kind in enumerate(order.split()):
    rng, fresh = np.random.default_rng(i), _model(**kw)
    if kind == "batch":
      prompts = [[i] + [int(t) for t in rng.integers(0, 512, 9 + i)] for _ in range(batch)]
      got, want = ([t for t, _ in zip(x.generate_batch(prompts), range(4))] for x in (m, fresh))
      assert got == want
    else:
      prompt = [i] + [int(t) for t in rng.integers(0, 512, 20 if kind == "one" else 3)]
      (got, lg), (want, lw) = _first(m, prompt, 4), _first(fresh, prompt, 4)
      assert got == want
      np.testing.assert_array_equal(lg, lw)
    for a, b in zip(m.blk, fresh.blk):      # the rows that this call has written
      n = len(prompts[0] if kind == "batch" else prompt) + 3
      seqs = batch if kind == "batch" else 1
      for x, y in ((a.k_cache, b.k_cache), (a.v_cache, b.v_cache)):
        x, y = (t.numpy().reshape(batch, 2, 64, 64)[:seqs, :, :n] for t in (x, y))
        np.testing.assert_array_equal(x, y)


def test_a_conversation_goes_on_after_a_batch():
  """The batch has written over sequence 0's cache rows: none of them may be reused."""
  need_gpu()
  rng = np.random.default_rng(4)
  talk = [int(t) for t in rng.integers(0, 512, 20)]
  m, fresh = _model(batch=2), _model(batch=2)
  _first(m, talk, 2)
  next(m.generate_batch([[int(t) for t in rng.integers(0, 512, 15)] for _ in range(2)]))
  (got, lg), (want, lw) = _first(m, talk + [3, 1], 4), _first(fresh, talk + [3, 1], 4)
  assert got == want
  np.testing.assert_array_equal(lg, lw)
