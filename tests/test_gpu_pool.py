"""Results from the pool: a block is not handed out again while queued work may still read it, sizes and dtypes mix, and the whole-call FP8 linear
matches its parts at the edges of its tiles."""
import ctypes
import numpy as np
import pytest
from tinygrad_b200 import _lib, fp8, quant, synth, runtime
from tinygrad_b200.runtime import DeviceBuffer
from gpu_util import need_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu(): need_gpu()


def test_a_result_keeps_its_values_while_later_calls_allocate():
  """Results are dropped right after a copy of them was queued on another stream, behind milliseconds of other copies: with blocks handed out too early a later
  result would be copied."""
  rng = np.random.default_rng(0)
  lin = quant.QuantLinear(512, 300, 2, synth.q4_0_blocks(300, 512, rng))
  xs = [DeviceBuffer.from_numpy(rng.standard_normal((8, 512)).astype(np.float32)) for _ in range(7)]
  want = [lin(x).numpy() for x in xs]
  st, copy = runtime.Stream(), runtime.Stream()
  out, lib = DeviceBuffer.empty((300, 8, 300), np.float32), _lib.load()
  far = [DeviceBuffer(256 << 20) for _ in range(2)]
  for i in range(300):
    if i % 30 == 0:
      for _ in range(40): _lib.check(lib.b200q_memcpy_d2d(far[0].ptr, far[1].ptr, far[0].nbytes, copy.ptr))
    y = lin(xs[i % 7], stream=st)
    st.synchronize()
    _lib.check(lib.b200q_memcpy_d2d(out.ptr + i * y.nbytes, y.ptr, y.nbytes, copy.ptr))
    del y
  got = out.numpy()
  for i in range(300): np.testing.assert_array_equal(got[i], want[i % 7])
  _lib.check(lib.b200q_pool_trim())
  np.testing.assert_array_equal(lin(xs[0]).numpy(), want[0])


@pytest.mark.parametrize("m,n_in,n_out,dt,bias", [(1, 128, 256, np.float32, True), (255, 256, 512, np.float16, True), (257, 384, 256, np.float32, False), (3, 128, 256, np.float16, False)])
def test_fp8_linear_equals_its_parts(m, n_in, n_out, dt, bias):
  """Quantise, product and scaling as one call against the three exported steps: bit for bit (same operations in the same order)."""
  rng = np.random.default_rng(m)
  w, b = rng.standard_normal((n_out, n_in)).astype(np.float32), rng.standard_normal(n_out).astype(np.float32) if bias else None
  lin = fp8.FP8Linear(n_in, n_out, w, b)
  x = DeviceBuffer.from_numpy(rng.standard_normal((m, n_in)).astype(dt))
  got = lin(x).numpy()
  lib, code, mp = _lib.load(), _lib.F32 if dt == np.float32 else _lib.F16, -(-m // 256) * 256
  q, factor = fp8.quantize_to_fp8(x, m * n_in, code)
  xq, e8, off = DeviceBuffer.empty((mp, n_in), np.uint8, zero=True), DeviceBuffer(mp * n_in // 32), DeviceBuffer.from_numpy(np.array([0, mp], np.int32))
  _lib.check(lib.b200q_memset(e8.ptr, 127, e8.nbytes, None)); _lib.check(lib.b200q_memcpy_d2d(xq.ptr, q.ptr, m * n_in, None))
  acc, y = DeviceBuffer.empty((mp, n_out), np.float32), DeviceBuffer.empty((m, n_out), dt)
  _lib.check(lib.b200q_grouped_mxfp8_gemm_f32(xq.ptr, e8.ptr, lin.w_q.ptr, lin._w_e8.ptr, off.ptr, 1, mp, n_out, n_in, acc.ptr, None))
  _lib.check(lib.b200q_fp8_scale_bias(acc.ptr, m, n_out, lin.w_factor.ptr, factor.ptr, lin.bias.ptr if bias else None, y.ptr, code, None))
  np.testing.assert_array_equal(got, y.numpy())


def test_results_of_captured_work_are_no_pool_blocks():
  """A graph writes its results whenever it is replayed: under capture the layers ask for memory of their own, which the capture mode of `Graph` refuses."""
  lin, x = quant.QuantLinear(512, 300, 2, synth.q4_0_blocks(300, 512, np.random.default_rng(0))), DeviceBuffer.empty((1, 512), np.float32, zero=True)
  for _ in range(70): lin(x)                  # blocks of that size are waiting in the pool
  st = runtime.Stream()
  with pytest.raises(_lib.B200QError):
    with runtime.Graph(st): lin(x, stream=st)
  assert not lin(x, stream=st).numpy().any()
