"""Which launches `generate` and `generate_batch` make on one model object, without a device: the library, the buffers and the graphs are stand-ins that take notes."""
from types import SimpleNamespace
import pytest
from tinygrad_b200 import model
from tinygrad_b200.model import Transformer


class _Anything:
  """A buffer, a stream, a library: whatever is asked of it is there and answers 0."""
  ptr = 0
  def __getattr__(self, name): return lambda *a, **kw: 0


class _Library(_Anything):
  def __init__(self, log): self.log = log
  def __getattr__(self, name):
    def call(*a):
      if "wait" not in name: self.log.append((name, *a[1:5]))
      return 0
    return call


class _Graph:
  """Keeps what was noted while it was open, and notes it when it is launched."""
  def __init__(self, log): self.log = log
  def __enter__(self): self.kept, self.log[:] = list(self.log), []
  def __exit__(self, *exc): self.inside, self.log[:] = list(self.log), self.kept
  def launch(self): self.log.extend(self.inside)


@pytest.fixture
def made(monkeypatch):
  """made(batch, chunk) -> (model, notes)"""
  def make(batch, chunk=16, max_context=64):
    m, log = Transformer.__new__(Transformer), []
    m.config = SimpleNamespace(dim=32, max_context=max_context)
    m.batch, m.prefill_chunk, m.prefill_rows, m.max_context, m.use_graph, m.is_moe, m.engine = batch, chunk, 6, max_context, True, False, "chain"
    m._graphs, m._cached_tokens, m._step_args, m._host_pos, m._head_queued = {}, [], None, 0, False
    m.stream = m.tokens = m.pos = m.x = m._mirror = _Anything()
    m._pf, m._last_rows = {"x": _Anything()}, (_Anything(), _Anything())
    monkeypatch.setattr(model._lib, "load", lambda: _Library(log))
    monkeypatch.setattr(model, "Graph", lambda stream: _Graph(log))
    def sampled(step, n=1):
      step()
      return [7] * n
    for name, f in dict(_native_rows=lambda: m._prefill_buffers() and "rows", _prefill_buffers=lambda: m._pf, _batch_buffers=lambda: None, _sampled=sampled,
                        _enqueue_step=lambda with_head, last_block=False: log.append(("last block" if last_block else "step", "one", with_head)),
                        _enqueue_batch_step=lambda count=True, last_block=False: log.append(("last block" if last_block else "step", "batch", True))).items():
      monkeypatch.setattr(m, name, f)
    return m, log
  return make


def _steps(log):
  return [e[:2] for e in log if e[0] in ("step", "last block")]


ONE, BATCH = [("last block", "one"), ("step", "one"), ("step", "one")], [("last block", "batch"), ("step", "batch"), ("step", "batch")]


@pytest.mark.parametrize("batch", [2, 3])
@pytest.mark.parametrize("order", ["one batch one", "batch one batch", "one short batch short", "batch short one short"])
def test_one_model_for_a_prompt_and_for_a_batch(made, order, batch):
  """Each kind of call runs its own last block and its own steps, whichever came first on the model.  ("short": a prompt that goes in steps of one token.)"""
  m, log = made(batch)
  for i, kind in enumerate(order.split()):
    del log[:]
    prompt = [i + 1] * (7 if kind != "short" else 3)
    answers = m.generate_batch([prompt] * batch) if kind == "batch" else m.generate(prompt)
    for _ in range(3): next(answers)
    want = {"one": ONE, "batch": BATCH, "short": [("step", "one")] * 5}[kind]
    assert _steps(log) == want, (kind, i)


@pytest.mark.parametrize("batch,tokens", [(40, 8), (17, 7), (17, 1)])
def test_a_batch_of_more_sequences_than_rows_is_refused_before_its_first_launch(made, batch, tokens):
  """Their last rows are gathered in the row buffer: nothing may be on its way there when the number of sequences is looked at."""
  m, log = made(batch)
  with pytest.raises(AssertionError): next(m.generate_batch([list(range(tokens))] * batch))
  assert log == [] and m._graphs == {}


def test_prefill_is_the_same_call_after_a_prompt_that_failed(made, monkeypatch):
  """A prompt for whose buffers there is no memory leaves nothing behind that changes what `prefill` does: n tokens, waited for, the position moved."""
  m, log = made(1)
  def no_memory(): raise MemoryError
  with monkeypatch.context() as mp:
    mp.setattr(m, "_prefill_buffers", no_memory)
    with pytest.raises(MemoryError): next(m.generate(list(range(9))))
  del log[:]
  assert m.prefill(0, 20) is None
  assert log == [("b200q_prompt_rows", 0, 1, 0, 16), ("b200q_prompt_rows", 0, 1, 16, 4)]
  assert m._host_pos == 20


@pytest.mark.parametrize("between", ["batch", "failed", "full"])
def test_cache_rows_that_another_call_has_written_are_not_reused(made, monkeypatch, between):
  """A conversation goes on where its rows are still there.  They are not after a batch, after a prompt that failed on its way, or after one that fills the context (no token
  follows it): all three have written over them."""
  m, log = made(2)
  talk = [5, 6] + list(range(20))
  next(m.generate(talk))
  if between == "batch": next(m.generate_batch([[9] * 12] * 2))
  elif between == "full": assert list(m.generate([5] + [9] * 63)) == []
  else:
    with monkeypatch.context() as mp:
      mp.setattr(m, "_last_block", lambda *a: (_ for _ in ()).throw(MemoryError()))
      with pytest.raises(MemoryError): next(m.generate([5] + [9] * 19))
  assert m.get_start_pos(talk + [7, 1]) == {"batch": 0, "failed": 1, "full": 1}[between]
