"""The K-quant GEMV that keeps full-precision activations, at the edges of its tiles, stages and grid, against fp64 sums over the fp16 weights."""
import numpy as np
import pytest
from oracle import ggml_quant as gq
from tinygrad_b200 import _lib, quant, synth
from tinygrad_b200.runtime import DeviceBuffer
from gpu_util import need_gpu

pytestmark = pytest.mark.gpu
TYPES = {12: _lib.Q4_K_WIDE, 14: _lib.Q6_K_WIDE}


def fp16_weight(raw, typ, n_out, n_in):
  return gq.dequantize(raw, n_out * n_in, typ).astype(np.float16).astype(np.float64).reshape(n_out, n_in)


def sum_bound(w, x):
  """The weights are the same fp16 values, an activation is off by 2^-23, products are exact, every addition and scaling is good to 2^-23 of the magnitudes that
  meet (tensor cores truncate): about 40 of them lie one behind the other (8 MMAs of 16 terms, warps, epilogue), and 8 per 2048 columns."""
  return 2.0 ** -23 * (40 + x.shape[1] / 256) * (np.abs(x) @ np.abs(w).T)


# one row / a partial row tile / one super-block (2 groups: most warps idle) / a stage remainder (18 groups) / one CTA per SM and the widest row
@pytest.mark.parametrize("typ", [12, 14])
@pytest.mark.parametrize("n_out,n_in,m", [(1, 256, 1), (16, 256, 3), (83, 2304, 1), (5000, 4096, 1), (40, 14336, 1), (24, 27648, 1)])
def test_kquant_wide(typ, n_out, n_in, m):
  need_gpu()
  rng = np.random.default_rng(n_in + n_out + typ)
  raw = synth.random_blocks(typ, n_out, n_in, rng)
  w = fp16_weight(raw, typ, n_out, n_in)
  x = (rng.standard_normal((m, n_in)) * 10.0 ** rng.uniform(-3, 3, (1, n_in))).astype(np.float32)      # six decades inside a block
  nw = (1 + 0.1 * rng.standard_normal(n_in)).astype(np.float16)
  bias, res = rng.standard_normal(n_out).astype(np.float16), rng.standard_normal((m, n_out)).astype(np.float32)
  pw = quant.repack(raw, n_out, n_in, TYPES[typ])
  y = DeviceBuffer.from_numpy(res.copy())
  quant.gemv(pw.buf.ptr, TYPES[typ], n_out, n_in, DeviceBuffer.from_numpy(x), y, m=m, norm_weight=DeviceBuffer.from_numpy(nw), norm_eps=1e-5,
             bias=DeviceBuffer.from_numpy(bias), residual=y)
  rs = 1 / np.sqrt((x.astype(np.float64) ** 2).mean(1, keepdims=True) + 1e-5)
  xn = x.astype(np.float64) * nw.astype(np.float64)
  ref = xn @ w.T * rs + bias + res
  bound = sum_bound(w, xn) * rs + 2.0 ** -22 * (np.abs(bias) + np.abs(res))
  err = np.abs(y.numpy((m, n_out), np.float32) - ref)
  assert (err <= bound).all(), (err / bound).max()
  # gate and up interleaved, the SwiGLU product in the epilogue, fp16 in and out
  up = synth.random_blocks(typ, n_out, n_in, rng)
  wu = fp16_weight(up, typ, n_out, n_in)
  pw = quant.repack(raw, n_out, n_in, TYPES[typ], raw_up=up)
  x16 = (x / np.abs(x).max(1, keepdims=True)).astype(np.float16)
  y16 = DeviceBuffer.empty((m, n_out), np.float16)
  quant.gemv(pw.buf.ptr, TYPES[typ], n_out, n_in, DeviceBuffer.from_numpy(x16), y16, m=m, x_dtype=quant.F16, y_dtype=quant.F16, epilogue=_lib.EPI_SILU_MUL)
  xd = x16.astype(np.float64)
  g, u = xd @ w.T, xd @ wu.T
  eg, eu = sum_bound(w, xd), sum_bound(wu, xd)
  sig = 1 / (1 + np.exp(-g))
  # |silu'| <= 1.1; __expf is good to 2 + 1.16 |g| units in the last place; fp16 rounds to 2^-11, below its normal range to 2^-25
  bound = 1.1 * eg * (np.abs(u) + eu) + np.abs(g * sig) * eu + 2.0 ** -22 * (4 + 1.2 * np.abs(g)) * np.abs(g * sig * u) + 2.0 ** -11 * np.abs(g * sig * u) * 1.01 + 2.0 ** -25
  err = np.abs(y16.numpy().astype(np.float64) - g * sig * u)
  assert (err <= bound).all(), (err / bound).max()


def test_kquant_two_matrices():
  """Q4_K rows with Q6_K rows behind them in one launch: the same bits as two launches."""
  need_gpu()
  rng = np.random.default_rng(7)
  n_in, rows = 1280, (48, 21)
  x, bias = DeviceBuffer.from_numpy(rng.standard_normal(n_in).astype(np.float32)), DeviceBuffer.from_numpy(rng.standard_normal(sum(rows)).astype(np.float16))
  p4, p6 = (quant.repack(synth.random_blocks(t, r, n_in, rng), r, n_in, TYPES[t]) for t, r in zip((12, 14), rows))
  y, z = DeviceBuffer.empty((sum(rows),), np.float32), DeviceBuffer.empty((sum(rows),), np.float32)
  quant.gemv(p4.buf.ptr, _lib.Q4_K_WIDE, sum(rows), n_in, x, y, bias=bias, w2_ptr=p6.buf.ptr, n_first=rows[0])
  quant.gemv(p4.buf.ptr, _lib.Q4_K_WIDE, rows[0], n_in, x, z, bias=bias)
  quant.gemv(p6.buf.ptr, _lib.Q6_K_WIDE, rows[1], n_in, x, z.ptr + 4 * rows[0], bias=bias.ptr + 2 * rows[0])
  np.testing.assert_array_equal(y.numpy(), z.numpy())
  with pytest.raises(_lib.B200QError): quant.gemv(p4.buf.ptr, _lib.Q4_K_WIDE, sum(rows), n_in, x, y, w2_ptr=p6.buf.ptr, n_first=40)      # not a whole row tile


def test_kquant_wide_refuses():
  need_gpu()
  raw = synth.random_blocks(12, 16, 512, np.random.default_rng(0))
  pw = quant.repack(raw, 16, 512, _lib.Q4_K_WIDE)
  x, y = DeviceBuffer.empty((27904,), np.float32, zero=True), DeviceBuffer.empty((16,), np.float32)
  for n_in in (384, 27904):      # not whole super-blocks; wider than the staged row may be
    with pytest.raises(_lib.B200QError): quant.gemv(pw.buf.ptr, _lib.Q4_K_WIDE, 16, n_in, x, y)
  with pytest.raises(_lib.B200QError): quant.gemv(pw.buf.ptr, _lib.Q4_K_WIDE, 16, 512, x, y, xq_in=x)
