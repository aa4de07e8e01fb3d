"""Tokens as `generate` sees them: polled from page-locked memory while the device may still be busy with other steps."""
import numpy as np
import pytest
from tinygrad_b200 import _lib, synth
from tinygrad_b200.model import Transformer, TransformerConfig
from tinygrad_b200.runtime import PinnedBuffer, Stream
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


def test_a_step_without_a_token_is_called_that():
  """Words that nothing fills: an error of their own once the stream is done, not that of a bad argument."""
  need_gpu()
  words, st = PinnedBuffer((2,), np.int32), Stream()
  words.array[:] = (5, -1)
  assert _lib.load().b200q_wait_words(words.ptr, 2, -1, st.ptr) == -7 and b"no result" in _lib.load().b200q_strerror(-7)
