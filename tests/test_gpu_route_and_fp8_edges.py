"""Routing where its launches change (one CTA for up to 32 tokens, choices by a kernel of their own up to 1024 pairs, four kernels above; 32, 64 or 256 experts' worth of
registers) against the oracle, and the FP8 linear's rows at the edges of its 32-row stores."""
import numpy as np
import pytest
from tinygrad_b200 import _lib, moe
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


MODES = [moe.ROUTE_TOPK_SOFTMAX, moe.ROUTE_SOFTMAX_TOPK, moe.Gating("softmax"), moe.Gating("sigmoid", True), moe.Gating("softmax", True), moe.Gating("sqrt_softplus")]


@pytest.mark.parametrize("mode", MODES, ids=lambda m: m if isinstance(m, int) else f"{m.func}-{m.norm_topk_prob}")
@pytest.mark.parametrize("T,E,k", [(9, 16, 4), (9, 64, 8), (9, 200, 8), (64, 8, 8), (300, 40, 4)])
def test_route_of_rows_that_are_not_finite(T, E, k, mode):
  """Each token has k different experts, ranked with NaN as -infinity, whatever its row holds, and their pairs are sorted by them."""
  rng = np.random.default_rng(E)
  logits = rng.standard_normal((T, E)).astype(np.float32)
  logits[0], logits[1] = np.nan, -np.inf
  logits[2], logits[2, E // 2] = np.nan, 0.5
  logits[3], logits[3, [E // 3, E - 1]] = -np.inf, (0.25, -0.5)
  logits[4, rng.permutation(E)[: E // 2]] = np.nan
  logits[5, rng.permutation(E)[: E - k // 2]] = -np.inf
  logits[6], logits[6, E - 2] = -np.finfo(np.float32).max, np.nan
  logits[-1, 1] = np.nan
  r = moe.Routing(T, E, k, mode).run(DeviceBuffer.from_numpy(logits))
  topi, w = r.topi.numpy(), r.weights.numpy()
  best = np.argsort(-np.where(np.isnan(logits), -np.inf, logits), axis=1, kind="stable")[:, :k]
  if mode != moe.ROUTE_TOPK_SOFTMAX: best = best[:, ::-1]
  whole = mode == moe.ROUTE_SOFTMAX_TOPK or getattr(mode, "func", "") == "softmax" and not mode.norm_topk_prob      # one NaN makes every score NaN
  for t in range(T):
    assert len(set(topi[t])) == k and (0 <= topi[t]).all() and (topi[t] < E).all(), t
    nan, low = np.isnan(logits[t]).any(), np.isneginf(logits[t])
    if not (whole and (nan or low.all())): np.testing.assert_array_equal(topi[t], best[t], str(t))
    if not nan and not low.all(): assert np.isfinite(w[t]).all(), t
    if whole and nan or np.isnan(logits[t, topi[t]]).any() and mode in MODES[:1] + MODES[4:5]: assert np.isnan(w[t]).all(), t
  flat = topi.reshape(-1)
  counts, dest, off = np.bincount(flat, minlength=E), r.dest_row.numpy(), r.off.numpy()
  np.testing.assert_array_equal(off, np.concatenate([[0], np.cumsum(-(-counts // 256) * 256)]))
  for e in range(E): np.testing.assert_array_equal(dest[flat == e], off[e] + np.arange(counts[e]))


@pytest.mark.parametrize("T,E,k", [(9, 16, 4), (300, 40, 4)])
def test_choices_that_are_no_experts_have_no_row(T, E, k):
  lib, rng = _lib.load(), np.random.default_rng(T)
  topi = rng.integers(0, E, (T, k)).astype(np.int32)
  topi[0], topi[T // 2, 1], topi[-1, -1] = -1, E, 0x7fffffff
  dest, off, scratch = DeviceBuffer.empty((T * k,), np.int32), DeviceBuffer.empty((E + 1,), np.int32), DeviceBuffer(lib.b200q_moe_route_scratch_bytes(T, E, k))
  sel = DeviceBuffer.from_numpy(topi)
  _lib.check(lib.b200q_moe_route_tables(sel.ptr, T, E, k, 256, dest.ptr, off.ptr, None, scratch.ptr, None))
  flat, d, o = topi.reshape(-1), dest.numpy(), off.numpy()
  there = (flat >= 0) & (flat < E)
  assert (d[~there] == -1).all()
  for e in range(E): np.testing.assert_array_equal(d[flat == e], o[e] + np.arange((flat == e).sum()))
  x, y, w = rng.standard_normal((T, 256)).astype(np.float32), rng.standard_normal((int(o[-1]), 64)).astype(np.float32), rng.standard_normal((T, k)).astype(np.float32)
  q = moe.quantize_mxfp8(DeviceBuffer.from_numpy(x), T, 256, _lib.F32, dest, k, int(o[-1]))[0].numpy()
  own = mx.quantize_mxfp8(x)[0]
  for i in np.flatnonzero(there): np.testing.assert_array_equal(q[d[i]], own[i // k])
  for D in (64, 60):                                # with and without 16-byte loads
    yb, out = moe.to_bf16_bits(np.ascontiguousarray(y[:, :D])), DeviceBuffer.empty((T, D), np.uint16)
    dy, dw = DeviceBuffer.from_numpy(yb), DeviceBuffer.from_numpy(w)
    _lib.check(lib.b200q_moe_combine(dy.ptr, dest.ptr, dw.ptr, T, k, D, out.ptr, None))
    ref = (np.where(there[:, None], moe.from_bf16_bits(yb)[np.maximum(d, 0)], 0).reshape(T, k, D) * w[..., None].astype(np.float64)).sum(1)
    assert (np.abs(moe.from_bf16_bits(out.numpy()) - ref) <= 2.0 ** -8 * np.abs(ref) + 1e-5).all()      # bf16; fp32 sums of four terms of size 1


def test_a_token_without_finite_logits_leaves_the_others_alone():
  T, D, F, E, k = 40, 256, 128, 16, 4
  rng = np.random.default_rng(3)
  layer = moe.MxMoE(*(rng.standard_normal(s).astype(np.float32) * 0.05 for s in ((E, F, D), (E, F, D), (E, D, F))), k)
  x, logits = DeviceBuffer.from_numpy(moe.to_bf16_bits(rng.standard_normal((T, D)).astype(np.float32))), rng.standard_normal((T, E)).astype(np.float32)
  clean = layer(x, DeviceBuffer.from_numpy(logits), T).numpy().reshape(T, D)
  logits[7], logits[30] = np.nan, -np.inf
  y, rest = layer(x, DeviceBuffer.from_numpy(logits), T).numpy().reshape(T, D), [t for t in range(T) if t not in (7, 30)]
  assert np.isnan(moe.from_bf16_bits(y[[7, 30]])).all()
  np.testing.assert_array_equal(y[rest], clean[rest])


@pytest.mark.parametrize("dt", [np.float32, np.float16])
@pytest.mark.parametrize("rows", [1, 31, 32, 33, 127, 129, 300])
def test_fp8_rows(rows, dt):
  """Every row of a call, against the product of the decoded codes."""
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


def _bytes(ptr, n):
  out = np.empty(n, np.uint8)
  _lib.check(_lib.load().b200q_memcpy_d2h(out.ctypes.data, ptr, n, None))
  return out


@pytest.mark.parametrize("with_bias", [True, False])
@pytest.mark.parametrize("dt", [np.float32, np.float16])
@pytest.mark.parametrize("rows", [1, 31, 33, 129])
def test_fp8_rows_and_nothing_behind_them(rows, dt, with_bias):
  """Results leave as boxes of 32 rows: what lies behind a result's last row, in its own pool block and in its neighbours, keeps its bytes."""
  lib, rng, n_in, n_out = _lib.load(), np.random.default_rng(rows), 128, 512
  lin = FP8Linear(n_in, n_out, rng.standard_normal((n_out, n_in)).astype(np.float32), rng.standard_normal(n_out).astype(np.float32) if with_bias else None)
  x = DeviceBuffer.from_numpy(rng.standard_normal((rows, n_in)).astype(dt))
  used, step = rows * n_out * np.dtype(dt).itemsize, 64
  while step * 16 < used: step *= 2
  block = max(512, -(-used // step) * step)             # what the pool hands out: an eighth of a power of two's steps
  held = [lin(x) for _ in range(12)]
  want = held[0].numpy()
  for y in held: _lib.check(lib.b200q_memset(y.ptr, 0xA5, block, None))
  _lib.check(lib.b200q_device_synchronize())
  mine = [y.ptr for y in held[::2]]
  held = held[1::2]
  seen = 0
  for _ in range(300):                                  # until the pool has handed out the blocks between the held ones again
    y = lin(x)
    if y.ptr in mine:
      mine.remove(y.ptr)
      seen += 1
      np.testing.assert_array_equal(y.numpy(), want)
      assert (_bytes(y.ptr + used, block - used) == 0xA5).all()
    for h in held: assert (_bytes(h.ptr, block) == 0xA5).all()
    if seen == 3: return
  pytest.fail("the pool did not hand its blocks out again")
