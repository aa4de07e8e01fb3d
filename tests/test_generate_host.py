"""What `generate` decides on the host, without a device."""
import random
import pytest
from tinygrad_b200.model import PREFILL_ROWS, Transformer


def test_reusable_prefix():
  """The cached tokens' common prefix with all of a prompt but its last token, found by halving: what a scan finds, for every length down to none."""
  m, rng = Transformer.__new__(Transformer), random.Random(0)
  for _ in range(2000):
    m._cached_tokens = [rng.randrange(2) for _ in range(rng.randrange(9))]
    prompt = m._cached_tokens[:rng.randrange(9)] + [rng.randrange(2) for _ in range(rng.randrange(4))]
    want = 0
    for a, b in zip(prompt[:-1], m._cached_tokens):
      if a != b: break
      want += 1
    assert m.get_start_pos(prompt) == want, (prompt, m._cached_tokens)


@pytest.mark.parametrize("rows,tokens,one_pass", [(64, 21, False), (64, 64, False), (64, 65, True), (20, 21, True), (PREFILL_ROWS, 6, False), (PREFILL_ROWS, 7, True), (1, 2, True), (0, 500, False)])
def test_prefill_rows_says_which_prompts_go_in_one_pass(monkeypatch, rows, tokens, one_pass):
  """`prefill_rows` uncached tokens (a prompt but its last) and more take one pass, fewer one step each; 0: always steps."""
  m, did = Transformer.__new__(Transformer), []
  m.prefill_rows, m.max_context, m._cached_tokens, m._step_args = rows, 1024, [], None
  for name, f in dict(_put_tokens=lambda t, p: None, prefill=lambda p, n: did.append(n), step=lambda with_head=True: did.append(1), _sampled=lambda step: [7]).items():
    monkeypatch.setattr(m, name, f)
  next(m.generate(list(range(tokens))))
  assert did == ([tokens - 1] if one_pass else [1] * (tokens - 1))
