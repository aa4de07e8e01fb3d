"""What the layers hand to the library, on a device that is made up."""
import ctypes
import numpy as np
import pytest
from tinygrad_b200 import fp8, moe, quant, runtime


class Device:
  """The C calls a layer makes: memory is a number, the one-call layers leave their argument block in `seen`."""
  def __init__(self): self.next, self.seen = 4096, None
  def __getattr__(self, name): return lambda *a: 4096 if name.endswith(("_bytes", "_bytes_for", "_max")) else 0
  def _alloc(self, out, nbytes, stream=None):
    self.next += 4096
    out._obj.value = self.next
    return 0
  b200q_malloc = b200q_pool_alloc = _alloc
  def _linear(self, desc, x, dtype, m, y, stream):
    self.seen = {f: getattr(desc._obj, f) for f, _ in desc._obj._fields_}
    return self._alloc(y, 0)
  b200q_linear = b200q_fp8_linear = _linear
  def b200q_moe_layer(self, args, *a):
    self.seen = {f: getattr(args._obj, f) for f, _ in args._obj._fields_}
    return 0


@pytest.fixture
def device(monkeypatch):
  d = Device()
  monkeypatch.setattr(runtime._lib, "load", lambda: d)
  return d


def test_layers_use_the_buffers_they_hold_now(device):
  """A weight or bias that a program puts into a layer is used from the next call on; nothing is read where the old one was."""
  buf = lambda *shape: runtime.DeviceBuffer.empty(shape, np.float32)
  lin = quant.QuantLinear(64, 32, 2, np.zeros(32 * 36, np.uint8), np.zeros(32))
  lin(buf(3, 64))
  assert device.seen["w"] == lin.weight.buf.ptr and device.seen["bias"] == lin.bias.ptr
  lin.weight, lin.bias = quant.PackedWeight(2, 32, 64, buf(1024), False), buf(32)
  lin(buf(3, 64))
  assert device.seen["w"] == lin.weight.buf.ptr and device.seen["bias"] == lin.bias.ptr
  lin.bias = None
  lin(buf(3, 64))
  assert not device.seen["bias"]
  f = fp8.FP8Linear(128, 256, np.zeros((256, 128), np.float32), np.zeros(256, np.float32))
  f(buf(5, 128))
  f.bias, f.weight = buf(256), buf(256, 128)
  f.requantize()
  f(buf(5, 128))
  assert device.seen["bias"] == f.bias.ptr and device.seen["w_q"] == f.w_q.ptr and device.seen["w_factor"] == f.w_factor.ptr
  layer = moe.MxMoE(*(np.zeros(s, np.float32) for s in ((2, 128, 256), (2, 128, 256), (2, 256, 128))), 1)
  layer(buf(4, 256), buf(4, 2), 4)
  layer.gu_q, layer.dn_e8 = buf(8), buf(8)
  layer(buf(4, 256), buf(4, 2), 4)
  assert device.seen["gu_q"] == layer.gu_q.ptr and device.seen["dn_e8"] == layer.dn_e8.ptr
