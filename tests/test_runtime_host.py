"""Host memory of the runtime layer, on a library that is made up."""
import ctypes, gc
import numpy as np
from tinygrad_b200 import runtime


class Pages:
  """b200q_host_alloc / _free on ordinary memory that says what is still allocated."""
  def __init__(self): self.live = {}
  def b200q_host_alloc(self, out, nbytes):
    block = ctypes.create_string_buffer(nbytes)
    self.live[ctypes.addressof(block)] = block
    out._obj.value = ctypes.addressof(block)
    return 0
  def b200q_host_free(self, ptr): return 0 if self.live.pop(ptr, None) is not None else -1


def test_pinned_pages_live_as_long_as_a_view_of_them(monkeypatch):
  """A program may keep the array alone: the pages go back once the buffer and every view are gone, or at `free`."""
  pages = Pages()
  monkeypatch.setattr(runtime._lib, "load", lambda: pages)
  view = runtime.PinnedBuffer((4, 2), np.int32).array[1:]
  gc.collect()
  assert len(pages.live) == 1
  view[:] = 7
  part = view.reshape(-1)[2:]
  del view; gc.collect()
  assert len(pages.live) == 1 and (part == 7).all()
  del part; gc.collect()
  assert not pages.live
  b = runtime.PinnedBuffer(3, np.float32)
  assert b.array.shape == (3,) and b.nbytes == 12
  b.free(); b.free()
  assert not pages.live and b.array is None and b.ptr == 0
