"""`FP8Linear` of extra/fp8/fp8_linear.py:43-63 on the B200 path: per-tensor E4M3 quantisation of weight and activations, the product on
the tcgen05 tensor cores with fp32 accumulation, the two scale factors and the bias applied afterwards.  Inference only: the weight is
quantised once (the reference re-quantises it on every call because it trains it); call `requantize()` after changing `weight`."""
import ctypes, math
import numpy as np
from . import _lib
from ._lib import check, F32, F16, BF16
from .runtime import DeviceBuffer, stream_ptr

_DT = {np.dtype(np.float32): F32, np.dtype(np.float16): F16}


def quantize_to_fp8(x: DeviceBuffer, n: int, x_dtype: int, stream=None):
  """-> (E4M3 codes [n] uint8, factor: one device float = 1 / scale); `quantize_to_fp8`, extra/fp8/fp8_linear.py:4-16."""
  lib, s = _lib.load(), stream_ptr(stream)
  q, amax, factor = DeviceBuffer.empty((n,), np.uint8), DeviceBuffer.empty((1,), np.float32), DeviceBuffer.empty((1,), np.float32)
  check(lib.b200q_fp8_absmax(x.ptr, x_dtype, n, amax.ptr, s))
  check(lib.b200q_fp8_quantize(x.ptr, x_dtype, n, amax.ptr, q.ptr, factor.ptr, s))
  return q, factor


class FP8Linear:
  """FP8Linear(in_features, out_features, weight [out, in] fp32, bias [out] or None); `__call__(x)` with x (..., in) fp32 / fp16 on the device
  returns (..., out) in x's dtype.  out_features must be a multiple of 256 and in_features of 128 (the tensor-core tile sizes)."""
  def __init__(self, in_features: int, out_features: int, weight: np.ndarray, bias=None):
    if out_features % 256 or in_features % 128: raise ValueError("out_features % 256 == in_features % 128 == 0 is required")
    self.in_features, self.out_features = in_features, out_features
    self.weight = DeviceBuffer.from_numpy(np.ascontiguousarray(weight, dtype=np.float32).reshape(out_features, in_features))
    self.bias = None if bias is None else DeviceBuffer.from_numpy(np.asarray(bias, dtype=np.float32).reshape(out_features))
    self._w_e8 = DeviceBuffer(out_features * in_features // 32)
    check(_lib.load().b200q_memset(self._w_e8.ptr, 127, self._w_e8.nbytes, None))       # E8M0 127 = 2^0: the codes as a block-scaled operand (`__call__` needs none)
    self._ws = {}
    self.requantize()

  def requantize(self) -> None:
    self.w_q, self.w_factor = quantize_to_fp8(self.weight, self.out_features * self.in_features, F32)

  def _workspace(self, m: int):
    mp = -(-m // 256) * 256
    w = self._ws.get(m)
    if w is None:
      lib = _lib.load()
      w = dict(x_q=DeviceBuffer.empty((mp, self.in_features), np.uint8, zero=True),
               off=DeviceBuffer.from_numpy(np.array([0, mp], np.int32)), parts=DeviceBuffer.empty((592,), np.float32), factor=DeviceBuffer.empty((1,), np.float32))
      check(lib.b200q_device_synchronize())
      w["desc"] = _lib.Fp8LinearDesc(self.out_features, self.in_features, mp, None, None, None, None, w["x_q"].ptr,
                                     None, w["off"].ptr, w["parts"].ptr, w["factor"].ptr)
      self._ws[m] = w
    return w["desc"]

  def __call__(self, x: DeviceBuffer, stream=None) -> DeviceBuffer:
    dt = _DT.get(x.dtype)
    if dt is None: raise TypeError(f"activations must be float16 or float32, got {x.dtype}")
    *lead, k = x.shape
    if k != self.in_features: raise ValueError(f"Input Tensor shapes {x.shape} cannot be multiplied with in_features={self.in_features}")
    m, shape = math.prod(lead), (*lead, self.out_features)
    if m == 0: return DeviceBuffer.empty(shape, x.dtype)
    d, y = self._workspace(m), ctypes.c_void_p()
    d.w_q, d.w_factor, d.bias = self.w_q.ptr, self.w_factor.ptr, self.bias and self.bias.ptr
    check(_lib.load().b200q_fp8_linear(ctypes.byref(d), x.ptr, dt, m, ctypes.byref(y), stream_ptr(stream)))
    return DeviceBuffer.adopt(y.value, m * self.out_features * x.dtype.itemsize, shape, x.dtype)
