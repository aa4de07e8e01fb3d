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
  """A grid limit keeps a call on the streaming kernel: the two differ by its 15-bit activation codes, half a step of a block's largest value per product."""
  need_gpu()
  from tinygrad_b200 import quant
  from tinygrad_b200.runtime import DeviceBuffer
  rng = np.random.default_rng(n_out + n_in)
  if form == "silu": n_out = -(-n_out // 2)
  raw, up = _blocks(typ, n_out, n_in, rng), _blocks(typ, n_out, n_in, rng)
  p = quant.repack(raw, n_out, n_in, typ, raw_up=up if form == "silu" else None)
  x = rng.standard_normal(n_in).astype(np.float32)
  dx, nw = DeviceBuffer.from_numpy(x), rng.uniform(0.5, 1.5, n_in).astype(np.float16)
  kw = {}
  if form != "plain": kw.update(norm_weight=DeviceBuffer.from_numpy(nw), norm_eps=1e-5)
  if form == "norm_bias_residual":
    kw.update(bias=DeviceBuffer.from_numpy(rng.standard_normal(n_out).astype(np.float16)), residual=DeviceBuffer.from_numpy(rng.standard_normal(n_out).astype(np.float32)))
  if form == "silu": kw.update(epilogue=quant.EPI_SILU_MUL)
  out = []
  for limit in (0, 100000):
    y = DeviceBuffer.empty((n_out,), np.float32, zero=True)
    quant.gemv(p.buf.ptr, typ, n_out, n_in, dx, y, max_ctas=limit, **kw)
    out.append(y.numpy().astype(np.float64))
  w, wu = (gq.weight_matrix(r, n_out, n_in, typ).astype(np.float64) for r in (raw, up))
  xn = x.astype(np.float64)
  if form != "plain": xn = xn / np.sqrt((xn ** 2).mean() + 1e-5) * nw
  half = np.repeat(np.abs(xn.reshape(-1, 32)).max(1) / 16256 / 2, 32)
  fp = 2.0 ** -24 * (64 + n_in / 64)
  bound = np.abs(w) @ (half + fp * np.abs(xn)) + fp * 8
  if form == "silu":
    g, u = w @ xn, wu @ xn
    ub = np.abs(wu) @ (half + fp * np.abs(xn))
    bound = 1.1 * np.abs(u) * bound + np.abs(g) * ub + bound * ub
  assert (np.abs(out[0] - out[1]) <= bound).all()
  assert taken == (np.abs(out[0] - out[1]).max() > 1e-6 * np.abs(out[0]).max())      # (the streaming kernel adds bias and residual in another order on another grid)
