"""One-row Linears on rows of more than 8192 values, which clusters of CTAs quantise together: parts that are not whole pairs of column groups, ragged ends, more row tiles than
CTAs, grids that are no multiple of the cluster, half-precision activations.  The codes and the order of the sums are those of a CTA that makes all of them itself: with
a limit on the CTAs, where each does, the result is the same bits."""
import ctypes
import numpy as np
import pytest
from tinygrad_b200 import _lib, quant, synth
from tinygrad_b200.runtime import DeviceBuffer, device_status
from gpu_util import need_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float32, np.float16])
@pytest.mark.parametrize("typ", [2, 8])
@pytest.mark.parametrize("n_out,n_in", [(16, 8224), (80, 8320), (4096, 14336), (3584, 18944), (5120, 18944), (2400, 11008), (1000, 28672)])
def test_shared_codes_are_the_same(typ, n_out, n_in, dt):
  need_gpu()
  rng, lib = np.random.default_rng(n_in + n_out), _lib.load()
  pw = quant.repack(synth.BLOCK_MAKERS[typ](n_out, n_in, rng), n_out, n_in, typ)
  x, b = DeviceBuffer.from_numpy(rng.standard_normal(n_in).astype(dt)), DeviceBuffer.from_numpy(rng.standard_normal(n_out).astype(np.float16))
  r = DeviceBuffer.from_numpy(rng.standard_normal(n_out).astype(np.float32))
  got = []
  for max_ctas in (0, 0, 100):
    y = DeviceBuffer.from_numpy(np.full(n_out, np.nan, np.float32))
    a = _lib.GemvArgs()
    a.qtype, a.n_out, a.n_in, a.m, a.w_packed, a.x, a.x_dtype, a.y_dtype, a.y, a.max_ctas = typ, n_out, n_in, 1, pw.buf.ptr, x.ptr, _lib.F16 if dt == np.float16 else _lib.F32, _lib.F32, y.ptr, max_ctas
    if typ == 2: a.bias = b.ptr          # one addend: where a tile is its CTA's first, the two are added to each other before the sum
    else: a.residual = r.ptr
    _lib.check(lib.b200q_gemv(ctypes.byref(a), None))
    got.append(y.numpy())
  assert np.isfinite(got[2]).all()
  np.testing.assert_array_equal(got[0], got[2])
  np.testing.assert_array_equal(got[1], got[2])
  assert device_status() == 0
