"""What the kernels lose against exact arithmetic, held to what 32-bit arithmetic gives."""
import numpy as np
import pytest
from tinygrad_b200 import quant
from tinygrad_b200.runtime import DeviceBuffer
from gpu_util import need_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu(): need_gpu()


def test_activation_codes_are_the_rounded_quotients():
  """The codes of the activation blocks, read back through an identity matrix: the nearest integer to x * (16256 / max) for every value, for blocks of
  any magnitude."""
  rng = np.random.default_rng(0)
  n, m = 1024, 256
  raw = np.zeros((n, n // 32, 34), np.uint8)                          # Q8_0: scale 1, quant 1 on the diagonal
  raw[:, :, :2] = np.frombuffer(np.float16(1).tobytes(), np.uint8)
  raw[np.arange(n), np.arange(n) // 32, 2 + np.arange(n) % 32] = 1
  x = rng.standard_normal((m, n)).astype(np.float32)
  x[1] *= np.float32(7e37); x[2] *= np.float32(1e-33)
  pw, y = quant.repack(raw.reshape(-1), n, n, 8), DeviceBuffer.empty((m, n), np.float32)
  quant.gemv(pw.buf.ptr, 8, n, n, DeviceBuffer.from_numpy(x), y, m=m)
  blocks = x.reshape(m, n // 32, 32)
  amax = np.abs(blocks).max(-1, keepdims=True)
  codes = np.rint(blocks * (np.float32(16256) / amax))
  got = np.rint(y.numpy().reshape(blocks.shape).astype(np.float64) / (amax / np.float32(16256)).astype(np.float64))
  np.testing.assert_array_equal(got, codes)
