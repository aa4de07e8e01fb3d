"""One fp32 row times a small packed matrix: the kernel for it against 64 bits, and the calls of the GEMV that take it against the ones that do not."""
import numpy as np
import pytest
from oracle import ggml_quant as gq
from tinygrad_b200 import synth
from gpu_util import need_gpu

pytestmark = pytest.mark.gpu


def _blocks(typ, n_out, n_in, rng):
  return synth.q4_0_blocks(n_out, n_in, rng) if typ == 2 else synth.q8_0_blocks(n_out, n_in, rng)


# one block, one tile / a remainder of rows and of blocks / each warp count's K groups: 4, 5, 8, 9 / more groups than two per warp
@pytest.mark.parametrize("typ", [2, 8])
@pytest.mark.parametrize("n_out,n_in", [(1, 32), (16, 128), (40, 96), (768, 512), (33, 640), (256, 1024), (1000, 1056), (24, 4160), (17, 8192)])
def test_row_gemv(typ, n_out, n_in):
  """Every kind of call against 64 bits: fp32 sums of exact products, at most n_in additions deep but for the 32 partial sums of a block."""
  need_gpu()
  from tinygrad_b200 import _lib, quant
  from tinygrad_b200.runtime import DeviceBuffer
  rng = np.random.default_rng(n_out + n_in + typ)
  raw, up = _blocks(typ, n_out, n_in, rng), _blocks(typ, n_out, n_in, rng)
  w, wu = (gq.weight_matrix(r, n_out, n_in, typ).astype(np.float64) for r in (raw, up))
  x = (rng.standard_normal(n_in) * np.exp(rng.uniform(-2, 2, n_in))).astype(np.float32)
  nw, bias, res = rng.uniform(0.5, 1.5, n_in).astype(np.float16), rng.standard_normal(n_out).astype(np.float16), rng.standard_normal(n_out).astype(np.float32)
  dx, dn, db, dr = (DeviceBuffer.from_numpy(v) for v in (x, nw, bias, res))
  packed, both = quant.repack(raw, n_out, n_in, typ), quant.repack(raw, n_out, n_in, typ, raw_up=up)
  y = DeviceBuffer.empty((n_out + 1,), np.float32, zero=True)
  def run(p, norm=None, b=None, r=None, epi=0):
    _lib.check(_lib.load().b200q_row_gemv(typ, p.buf.ptr, dx.ptr, norm.ptr if norm else None, 1e-5, b.ptr if b else None, r.ptr if r else None, epi, y.ptr, n_out, n_in, 0, None))
    assert y.numpy()[n_out] == 0
    return y.numpy()[:n_out].astype(np.float64)
  eps = 2.0 ** -24 * (32 + n_in / 128)
  mag = np.abs(w) @ np.abs(x.astype(np.float64))
  assert (np.abs(run(packed) - w @ x.astype(np.float64)) <= eps * mag).all()
  xn = x.astype(np.float64) / np.sqrt((x.astype(np.float64) ** 2).mean() + 1e-5) * nw
  magn = np.abs(w) @ np.abs(xn)
  got, want = run(packed, norm=dn, b=db, r=dr), w @ xn + bias + res
  assert (np.abs(got - want) <= 2 * eps * (magn + np.abs(bias) + np.abs(res))).all()
  g, u = w @ xn, wu @ xn
  want = g / (1 + np.exp(-g)) * u
  gmag, umag = magn, np.abs(wu) @ np.abs(xn)
  assert (np.abs(run(both, norm=dn, epi=1) - want) <= 4 * eps * (np.abs(u) * gmag * 1.1 + np.abs(g) * umag + np.abs(want))).all()      # |silu'| <= 1.1


# the largest of the rule (16 K groups, 4096 tiles of 16 x 128) and the first sizes past it: those are the same kernel whichever way they are called
@pytest.mark.parametrize("typ,n_out,n_in,taken", [(2, 4096, 2048, True), (8, 4097, 2048, False), (2, 16, 2080, False), (8, 100, 32, True)])
@pytest.mark.parametrize("form", ["plain", "norm_bias_residual", "silu"])
def test_gemv_takes_the_row_kernel(typ, n_out, n_in, taken, form):
  """A grid limit keeps a call on the streaming kernel: the two differ by its 15-bit activation codes, half a step of a block's largest value per product.  Which one a call without
  a limit took shows on rows whose blocks have one large value beside small ones of less than half a step: codes lose those, fp32 does not."""
  need_gpu()
  from tinygrad_b200 import quant
  from tinygrad_b200.runtime import DeviceBuffer
  rng = np.random.default_rng(n_out + n_in)
  if form == "silu": n_out = -(-n_out // 2)
  raw, up = _blocks(typ, n_out, n_in, rng), _blocks(typ, n_out, n_in, rng)
  p = quant.repack(raw, n_out, n_in, typ, raw_up=up if form == "silu" else None)
  w, wu = (gq.weight_matrix(r, n_out, n_in, typ).astype(np.float64) for r in (raw, up))
  nw, bias, res = rng.uniform(0.5, 1.5, n_in).astype(np.float16), rng.standard_normal(n_out).astype(np.float16), rng.standard_normal(n_out).astype(np.float32)
  nw[::32] = 1
  kw = {}
  if form != "plain": kw.update(norm_weight=DeviceBuffer.from_numpy(nw), norm_eps=1e-5)
  if form == "norm_bias_residual": kw.update(bias=DeviceBuffer.from_numpy(bias), residual=DeviceBuffer.from_numpy(res))
  if form == "silu": kw.update(epilogue=quant.EPI_SILU_MUL)
  def run(x, limit):
    dx, y = DeviceBuffer.from_numpy(x), DeviceBuffer.empty((n_out,), np.float32, zero=True)
    quant.gemv(p.buf.ptr, typ, n_out, n_in, dx, y, max_ctas=limit, **kw)
    return y.numpy().astype(np.float64)
  def normed(x):
    return x.astype(np.float64) if form == "plain" else x / np.sqrt((x.astype(np.float64) ** 2).mean() + 1e-5) * nw
  def exact(xn):
    if form == "silu": return (w @ xn) / (1 + np.exp(-(w @ xn))) * (wu @ xn)
    return w @ xn + (bias.astype(np.float64) + res if form == "norm_bias_residual" else 0)
  def bound(xn, per_value):      # of the result, for an error per_value of each of the row's values (|silu'| <= 1.1)
    b = np.abs(w) @ per_value
    if form == "plain": return b
    if form == "norm_bias_residual": return b + 2.0 ** -22 * (np.abs(bias) + np.abs(res) + np.abs(exact(xn)))
    ub = np.abs(wu) @ per_value
    return 1.1 * np.abs(wu @ xn) * b + np.abs(w @ xn) * ub + b * ub + 2.0 ** -22 * np.abs(exact(xn))
  fp = 2.0 ** -24 * (64 + n_in / 64)
  x = rng.standard_normal(n_in).astype(np.float32)
  xn = normed(x)
  half = np.repeat(np.abs(xn.reshape(-1, 32)).max(1) / 16256 / 2, 32)
  assert (np.abs(run(x, 0) - run(x, 100000)) <= bound(xn, half + fp * np.abs(xn)) + fp * 8).all()
  x = (1.8e-5 * rng.choice([-1.0, 1.0], n_in)).astype(np.float32)      # (norm weights are 1.5 at most: 2.7e-5 of the block's largest; half a step is 3.1e-5)
  x[::32] = 1
  xn = normed(x)
  codes = np.where(np.arange(n_in) % 32 == 0, xn, 0)
  limit, lost = bound(xn, fp * np.abs(xn)), np.abs(exact(codes) - exact(xn))
  assert (lost > 2 * limit).any()      # so that a result without the small values, itself off by `limit`, is still off by more than that
  fp32 = lambda got: (np.abs(got - exact(xn)) <= limit).all()
  assert fp32(run(x, 0)) == taken and not fp32(run(x, 100000))
