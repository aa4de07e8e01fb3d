"""The grouped FP8 GEMM's tiles of 64, 128 and 256 columns: a row's results are the same bits whatever the number of rows it comes with."""
import numpy as np
import pytest
from gpu_util import need_gpu

pytestmark = pytest.mark.gpu


# rows: one, the most of a narrow tile's short copies and one more, one and two row tiles and a row, as many as make tiles of 128 and 256 columns the shorter way
@pytest.mark.parametrize("n_in,n_out,dt", [(128, 256, np.float32), (640, 4096, np.float16), (1024, 2304, np.float32)])
def test_fp8_rows_do_not_depend_on_the_tile(n_in, n_out, dt):
  need_gpu()
  from tinygrad_b200.fp8 import FP8Linear
  from tinygrad_b200.runtime import DeviceBuffer
  rng = np.random.default_rng(n_in)
  lin = FP8Linear(n_in, n_out, rng.standard_normal((n_out, n_in)).astype(np.float32), rng.standard_normal(n_out).astype(np.float32))
  x = rng.standard_normal((2100, n_in)).astype(dt)
  x[0, 0] = 8                                   # the tensor's largest value is in every subset
  whole = lin(DeviceBuffer.from_numpy(x)).numpy()
  ref = x.astype(np.float64) @ lin.weight.numpy().astype(np.float64).T + lin.bias.numpy()
  assert np.linalg.norm(whole - ref) <= 0.06 * np.linalg.norm(ref)      # two E4M3 roundings of at most 2^-4 each, uniform: 2^-4 / sqrt(3) * sqrt(2) and less
  for m in (1, 31, 32, 33, 128, 129, 300, 500, 900, 1300):
    np.testing.assert_array_equal(lin(DeviceBuffer.from_numpy(x[:m].copy())).numpy(), whole[:m], err_msg=str(m))


@pytest.mark.parametrize("D,F,E,k", [(256, 128, 3, 2), (512, 384, 16, 4), (768, 1024, 40, 8)])
def test_expert_layer_rows_do_not_depend_on_the_tile(D, F, E, k):
  need_gpu()
  from tinygrad_b200 import moe
  from tinygrad_b200.runtime import DeviceBuffer
  rng = np.random.default_rng(E)
  layer = moe.MxMoE(*((rng.standard_normal(s) * 0.05).astype(np.float32) for s in ((E, F, D), (E, F, D), (E, D, F))), k)
  x, lg = moe.to_bf16_bits(rng.standard_normal((2500, D)).astype(np.float32)), rng.standard_normal((2500, E)).astype(np.float32)
  run = lambda T: layer(DeviceBuffer.from_numpy(x[:T].copy()), DeviceBuffer.from_numpy(lg[:T].copy()), T).numpy()
  whole = run(2500)
  for T in (1, 31, 32, 33, 128, 129, 400, 1200): np.testing.assert_array_equal(run(T), whole[:T], err_msg=str(T))


# one thread's piece, all of one CTA and a value more, the smallest and largest of one launch, and one past it; what is left of a thread's pieces; both kinds of rows
@pytest.mark.parametrize("rows,n_in,dt", [(1, 128, np.float32), (8, 1024, np.float16), (65, 128, np.float32), (4096, 256, np.float16), (1025, 1024, np.float32),
                                         (148 * 32, 1024, np.float32), (148 * 32 + 1, 1024, np.float16)])
def test_fp8_codes_in_one_launch(rows, n_in, dt):
  """Codes and factor of a call's activations are those of the separate entry points, the largest magnitude wherever it is."""
  need_gpu()
  from tinygrad_b200 import fp8, _lib
  from tinygrad_b200.runtime import DeviceBuffer
  rng = np.random.default_rng(rows)
  lin = fp8.FP8Linear(n_in, 256, rng.standard_normal((256, n_in)).astype(np.float32))
  for at in (0, rows * n_in // 2, rows * n_in - 1):
    x = rng.standard_normal((rows, n_in)).astype(dt)
    x.reshape(-1)[at] = -9.5
    d = DeviceBuffer.from_numpy(x)
    lin(d)
    q, f = fp8.quantize_to_fp8(d, x.size, _lib.F16 if dt == np.float16 else _lib.F32)
    w = lin._workspace(rows)
    got = DeviceBuffer.empty((rows, n_in), np.uint8)
    _lib.check(_lib.load().b200q_memcpy_d2d(got.ptr, w.x_q, rows * n_in, None))
    np.testing.assert_array_equal(got.numpy().reshape(-1), q.numpy().reshape(-1))
    factor = DeviceBuffer.empty((1,), np.float32)
    _lib.check(_lib.load().b200q_memcpy_d2d(factor.ptr, w.factor, 4, None))
    assert factor.numpy()[0] == f.numpy()[0]


@pytest.mark.parametrize("m", [1, 40, 300])
def test_fp8_linear_reads_no_block_scales(m):
  """The descriptor's block scales may be missing, or anything: per-tensor codes have none."""
  need_gpu()
  from tinygrad_b200.fp8 import FP8Linear
  from tinygrad_b200.runtime import DeviceBuffer
  rng = np.random.default_rng(m)
  lin = FP8Linear(256, 512, rng.standard_normal((512, 256)).astype(np.float32))
  x = DeviceBuffer.from_numpy(rng.standard_normal((m, 256)).astype(np.float32))
  want, d = lin(x).numpy(), lin._workspace(m)
  scales = DeviceBuffer.from_numpy(rng.integers(100, 150, (512, 8)).astype(np.uint8))
  d.w_e8 = d.x_e8 = scales.ptr
  np.testing.assert_array_equal(lin(x).numpy(), want)
  d.w_e8 = d.x_e8 = None
  np.testing.assert_array_equal(lin(x).numpy(), want)
