"""What `generate` decides on the host, without a device."""
import random
from tinygrad_b200.model import Transformer


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
