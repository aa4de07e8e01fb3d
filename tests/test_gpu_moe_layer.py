"""The expert layer as one call, at the edges of its dispatch: routing in one CTA or in four launches, row tiles without a group's padding."""
import ctypes
import numpy as np
import pytest
from oracle import mxfp8 as mx
from gpu_util import need_gpu

pytestmark = pytest.mark.gpu


# one pair / both limits of the one-CTA routing (256 tokens, 1024 pairs) and one past each / more than 32 chunks of pairs to scan
@pytest.mark.parametrize("T,E,k", [(1, 1, 1), (1, 33, 8), (256, 256, 4), (257, 40, 1), (129, 16, 8), (4200, 12, 8)])
def test_route_edges(T, E, k):
  need_gpu()
  from tinygrad_b200 import moe
  from tinygrad_b200.runtime import DeviceBuffer
  logits = np.random.default_rng(T + E).standard_normal((T, E)).astype(np.float32)
  r = moe.Routing(T, E, k).run(DeviceBuffer.from_numpy(logits))
  w, topi, dest, off, _ = mx.route(logits, k, E)
  np.testing.assert_array_equal(r.topi.numpy(), topi)
  np.testing.assert_array_equal(r.dest_row.numpy(), dest)
  np.testing.assert_array_equal(r.off.numpy(), off)
  np.testing.assert_allclose(r.weights.numpy(), w, rtol=2e-6)


# group sizes that the logits choose: empty, 1, a whole row tile, one past it, a whole group, one past it
@pytest.mark.parametrize("sizes", [[3], [0, 1, 0, 128, 129], [255, 256, 257, 0], [128, 0, 384, 385]])
def test_layer_is_its_parts(sizes):
  """The same bits as the single entry points, whose GEMMs also run over the padding of the groups."""
  need_gpu()
  from tinygrad_b200 import _lib, moe
  from tinygrad_b200.runtime import DeviceBuffer
  rng = np.random.default_rng(len(sizes))
  E, T, D, F = len(sizes), sum(sizes), 256, 128
  logits = rng.standard_normal((T, E)).astype(np.float32)
  logits[np.arange(T), rng.permutation(np.repeat(np.arange(E), sizes))] += 100
  layer = moe.MxMoE(*((rng.standard_normal(s) * 0.1).astype(np.float32) for s in ((E, F, D), (E, F, D), (E, D, F))), 1, moe.ROUTE_SOFTMAX_TOPK)
  x, lg = DeviceBuffer.from_numpy(moe.to_bf16_bits(rng.standard_normal((T, D)).astype(np.float32))), DeviceBuffer.from_numpy(logits)
  got = layer(x, lg, T).numpy().copy()
  assert np.array_equal(np.bincount(layer.last_routing.topi.numpy().reshape(-1), minlength=E), sizes)
  res = rng.standard_normal((T, D)).astype(np.float32)
  acc = DeviceBuffer.from_numpy(res)
  _lib.check(_lib.load().b200q_moe_layer(ctypes.byref(layer.native_args(T)), x.ptr, lg.ptr, T, acc.ptr, None))
  np.testing.assert_array_equal(acc.numpy(), res + moe.from_bf16_bits(got))
  for f in layer.phases(x, lg, T).values(): f()
  np.testing.assert_array_equal(got, layer._workspace(T)["out"].numpy())


# one group / empty groups first, between and last / one K step, more K steps than the ring has stages / more tiles than SMs, several tiles of one group on a CTA
@pytest.mark.parametrize("sizes,n,k", [([256], 256, 128), ([0, 512, 0, 256, 0], 512, 640), ([256, 256, 256], 256, 2048), ([2560, 0, 768], 1536, 256)])
def test_grouped_gemm(sizes, n, k):
  """Every row of every group against the oracle (fp32 sums of at most k products, then one rounding to bf16); rows behind the last group are left alone."""
  need_gpu()
  from tinygrad_b200 import _lib, moe
  from tinygrad_b200.runtime import DeviceBuffer
  rng = np.random.default_rng(n + k)
  E, off = len(sizes), np.cumsum([0, *sizes]).astype(np.int32)
  m = int(off[-1]) + 256                                          # room behind the groups, as the routing leaves it
  aq, ae = mx.quantize_mxfp8(rng.standard_normal((m, k)).astype(np.float32))
  bq, be = mx.quantize_mxfp8((rng.standard_normal((E * n, k)) * np.exp(rng.uniform(-3, 3, (E * n, 1)))).astype(np.float32))
  c = DeviceBuffer.empty((m, n), np.uint16, zero=True)
  bufs = [DeviceBuffer.from_numpy(v) for v in (aq, ae, bq, be, off)]
  _lib.check(_lib.load().b200q_grouped_mxfp8_gemm(*(b.ptr for b in bufs), E, m, n, k, c.ptr, None))
  got = moe.from_bf16_bits(c.numpy())
  a, b = mx.dequantize_mxfp8(aq, ae).astype(np.float64), mx.dequantize_mxfp8(bq, be).astype(np.float64).reshape(E, n, k)
  for e in range(E):
    x = a[off[e]:off[e + 1]]
    want, mag = x @ b[e].T, np.abs(x) @ np.abs(b[e]).T
    err = np.abs(got[off[e]:off[e + 1]] - want)
    assert (err <= 2.0 ** -8 * np.abs(want) + 2.0 ** -23 * (k / 32 + 32) * mag).all(), (e, err.max())
  assert not got[off[E]:].any()
