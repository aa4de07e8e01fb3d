"""Routing where its launches change (one CTA for up to 32 tokens, choices by a kernel of their own up to 1024 pairs, four kernels above; 32, 64 or 256 experts' worth of
registers) against the oracle, and the FP8 linear's rows at the edges of its 32-row stores."""
import numpy as np
import pytest
from tinygrad_b200 import moe
from tinygrad_b200.fp8 import FP8Linear
from tinygrad_b200.runtime import DeviceBuffer
from oracle import fp8_linear as f8, mxfp8 as mx
from gpu_util import need_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu(): need_gpu()


@pytest.mark.parametrize("T,E,k", [(32, 32, 8), (33, 32, 8), (33, 33, 3), (32, 64, 32), (64, 65, 16), (256, 64, 4), (257, 16, 3), (1024, 8, 1), (1025, 40, 1), (128, 8, 8), (129, 256, 8)])
def test_route_at_the_edges_of_its_launches(T, E, k):
  logits = np.random.default_rng(T + E).standard_normal((T, E)).astype(np.float32)
  logits[: T // 2, : E // 2] = np.round(logits[: T // 2, : E // 2])          # ties
  r = moe.Routing(T, E, k).run(DeviceBuffer.from_numpy(logits))
  w, topi, dest, off, _ = mx.route(logits, k, E)
  np.testing.assert_array_equal(r.topi.numpy(), topi)
  np.testing.assert_array_equal(r.dest_row.numpy(), dest)
  np.testing.assert_array_equal(r.off.numpy(), off)
  np.testing.assert_allclose(r.weights.numpy(), w, rtol=2e-6)      # expf and a sum of at most 32 terms: some units of 2^-24


@pytest.mark.parametrize("dt", [np.float32, np.float16])
@pytest.mark.parametrize("rows", [1, 31, 32, 33, 127, 129, 300])
def test_fp8_rows(rows, dt):
  """The rows a call has and no others (its result is a block that other results' neighbours share), against the product of the decoded codes."""
  rng = np.random.default_rng(rows)
  n_in, n_out = 256, 512
  lin = FP8Linear(n_in, n_out, rng.standard_normal((n_out, n_in)).astype(np.float32), rng.standard_normal(n_out).astype(np.float32))
  x = rng.standard_normal((rows, n_in)).astype(dt)
  y = lin(DeviceBuffer.from_numpy(x)).numpy()
  ref = f8.fp8_linear(x, lin.weight.numpy(), lin.bias.numpy())
  # fp32 sums of exact products, each rounded once per instruction of 32 and three times behind them: 11 units of 2^-23 of the sum of the magnitudes, which is some
  # 15 times the result's size here (256 terms of random sign); half precision: its rounding
  tol = 2.0 ** -10 if dt == np.float16 else 2e-5
  assert y.shape == ref.shape and (np.abs(y - ref) <= tol * (np.abs(ref) + np.sqrt(np.mean(ref.astype(np.float64) ** 2)))).all()
