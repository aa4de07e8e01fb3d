"""Tokens as `generate` sees them: polled from page-locked memory while the device may still be busy with other steps."""
import numpy as np
import pytest
from tinygrad_b200 import synth
from tinygrad_b200.model import Transformer, TransformerConfig
from gpu_util import need_gpu

pytestmark = pytest.mark.gpu
KW = dict(num_blocks=3, dim=512, hidden_dim=1408, n_heads=8, n_kv_heads=2, norm_eps=1e-5, vocab_size=2000, head_dim=64, rope_theta=500000.0, rope_dim=64,
          max_context=512, kv_dtype="float16")


def model(**kw):
  need_gpu()
  cfg = TransformerConfig(**{**KW, **kw.pop("cfg", {})})
  return Transformer(cfg, synth.dense_model_raw(cfg, synth.Q4_0, seed=5, embd_std=0.3), ggml_type=synth.Q4_0, **kw)


def test_queued_steps_do_not_pass_for_the_next_token():
  """`step` does not wait: its tokens may still be on their way when the next `generate` asks for its own."""
  m, prompt = model(), [int(t) for t in np.random.default_rng(1).integers(0, 2000, 40)]
  first = next(m.generate(prompt))
  for _ in range(3):
    for _ in range(300): m.step()                # about 15 ms of work
    assert next(m.generate(prompt)) == first     # all but the last prompt token are in the cache: one step


def test_generate_on_a_model_for_batches():
  """A model built for several sequences also answers one prompt, as one built for it does."""
  prompt = [int(t) for t in np.random.default_rng(2).integers(0, 2000, 9)]
  want, got = ([t for t, _ in zip(m.generate(prompt), range(6))] for m in (model(), model(batch=3)))
  assert got == want
