"""The many-row GEMM where every tile has a whole number of CTAs, each with an equal part of its K groups, and where CTAs have whole tiles."""
import numpy as np
import pytest
import test_gpu_qgemm_stream as stream
from tinygrad_b200 import quant, synth
from tinygrad_b200.runtime import DeviceBuffer
from gpu_util import need_gpu

pytestmark = pytest.mark.gpu

# 8 CTAs a tile with two K groups each and with a group more in one; 7, 3, 2 and 1; two tiles of activation rows; tiles of 256 weight rows; rows of either kind, through tensor
# memory and through shared memory; where the largest share is too large (equal shares of everything); two and more whole tiles a CTA;
# 16 CTAs a tile; wide tiles in many parts (equal shares of fp32 rows); one whole tile for little more than half of the SMs
SHAPES = [(2, 45, 2300, 2048, np.float32), (8, 16, 2300, 2176, np.float32), (2, 96, 2688, 1920, np.float32), (8, 130, 6200, 896, np.float32), (8, 64, 6200, 896, np.float16),
          (2, 45, 9472, 512, np.float32), (8, 13, 16600, 288, np.float32), (2, 128, 16600, 288, np.float16), (8, 300, 4700, 640, np.float16), (2, 512, 4600, 416, np.float32),
          (8, 200, 34000, 288, np.float32), (2, 512, 4096, 14336, np.float32), (2, 45, 37888, 416, np.float32), (8, 300, 20000, 224, np.float16), (2, 96, 30000, 96, np.float32), (2, 45, 1100, 4096, np.float32),
          (8, 13, 1100, 4064, np.float32), (8, 512, 1280, 3424, np.float32), (8, 512, 1280, 3424, np.float16), (2, 301, 5632, 1024, np.float16)]


@pytest.mark.parametrize("typ,m,n_out,n_in,dt", SHAPES)
def test_shares_against_the_exact_product(typ, m, n_out, n_in, dt):
  need_gpu()
  stream.test_rows_against_the_exact_product(typ, m, n_out, n_in, dt, True)


@pytest.mark.parametrize("typ,m,n_out,n_in", [(2, 45, 2300, 2176), (8, 96, 2688, 1920), (8, 130, 6200, 896)])
def test_shares_repeat_bit_for_bit(typ, m, n_out, n_in):
  """Whichever CTA of a tile counts last."""
  need_gpu()
  rng = np.random.default_rng(m)
  pw, x = quant.repack(synth.BLOCK_MAKERS[typ](n_out, n_in, rng), n_out, n_in, typ), DeviceBuffer.from_numpy(rng.standard_normal((m, n_in)).astype(np.float32))
  y, ws, first = DeviceBuffer.empty((m, n_out), np.float32), DeviceBuffer(quant.qgemm_workspace_bytes(m, n_in, n_out)), None
  for _ in range(20):
    quant.qgemm(pw.buf.ptr, typ, n_out, n_in, x, y, m, workspace=ws)
    if first is not None: np.testing.assert_array_equal(y.numpy(), first)
    first = y.numpy().copy()
