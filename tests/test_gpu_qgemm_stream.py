"""The many-row GEMM with a workspace (csrc/qgemm_stream.cu) at the edges of its tiles and of its dispatch: activation tiles of 16 .. 256 rows,
weight tiles of 128 (up to 128 rows) and 256, one pass (fp16) and three (fp32), tiles split over CTAs or whole, remainders everywhere."""
import numpy as np
import pytest
from tinygrad_b200 import _lib, quant, synth
from tinygrad_b200.runtime import DeviceBuffer
from oracle import ggml_quant as gq
from gpu_util import need_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu(): need_gpu()


@pytest.mark.parametrize("split", [True, False])
@pytest.mark.parametrize("typ,m,n_out,n_in,dt", [(2, 1, 16, 32, np.float32), (8, 16, 130, 96, np.float32), (2, 17, 1000, 1184, np.float32), (8, 64, 128, 4096, np.float32),
                                                 (2, 65, 257, 4096, np.float32), (8, 128, 256, 160, np.float32), (2, 129, 300, 992, np.float32), (8, 256, 512, 512, np.float32),
                                                 (2, 257, 130, 1408, np.float32), (2, 301, 200, 640, np.float16), (8, 64, 300, 1184, np.float16), (8, 600, 72, 96, np.float16),
                                                 # enough row tiles for 256 weight rows each above 128 rows (the others take 128)
                                                 (2, 65, 19300, 96, np.float32), (8, 130, 30400, 160, np.float32), (2, 257, 15300, 96, np.float32),
                                                 (8, 300, 15300, 96, np.float16)])
def test_rows_against_the_exact_product(typ, m, n_out, n_in, dt, split):
  rng = np.random.default_rng(m + n_out)
  raw = synth.BLOCK_MAKERS[typ](n_out, n_in, rng)
  w = gq.weight_matrix(raw, n_out, n_in, typ).astype(np.float64)
  if dt == np.float16: w = w.astype(np.float16).astype(np.float64)          # fp16 activations take the fp16-rounded weight
  x, bias, res = rng.standard_normal((m, n_in)).astype(dt), rng.standard_normal(n_out).astype(np.float16), rng.standard_normal((m, n_out)).astype(dt)
  pw = quant.repack(raw, n_out, n_in, typ)
  dx, db, y = DeviceBuffer.from_numpy(x), DeviceBuffer.from_numpy(bias), DeviceBuffer.from_numpy(res)
  lib = _lib.load()
  ws = DeviceBuffer(lib.b200q_qgemm_workspace_bytes_for(m, n_out, n_in) if split else lib.b200q_qgemm_workspace_bytes(m, n_in))
  code = _lib.F32 if dt == np.float32 else _lib.F16
  quant.qgemm(pw.buf.ptr, typ, n_out, n_in, dx, y, m, x_dtype=code, y_dtype=code, bias=db, residual=y, workspace=ws)
  ref = x.astype(np.float64) @ w.T + bias + res
  # 2^-21: the dropped low x low product and the rounding of the low halves; then one rounding of the running sum (at most the sum of the
  # magnitudes) per tensor-core instruction, up to three per 16 columns; fp32 (fp16) rounding of the result
  size = np.abs(x).astype(np.float64) @ np.abs(w).T + np.abs(bias) + np.abs(res)
  bound = (2.0 ** -21 + 3 * np.ceil(n_in / 16) * 2.0 ** -23) * size + (2.0 ** -11 if dt == np.float16 else 2.0 ** -23) * np.abs(ref) + 1e-7
  assert (np.abs(y.numpy() - ref) <= bound).all(), f"worst {np.max(np.abs(y.numpy() - ref) / bound):.2f} of the bound"


# Weights through tensor memory: whole tiles between split ones, with and without room for them in shared memory (112 rows of Q4_0, Q8_0), tiles of one K group, the most
# rows of either type; and either side of the lines where shared memory takes over (32 rows; 4 K groups an SM up to 64, 10 above; 8 CTAs a tile).
@pytest.mark.parametrize("split", [True, False])
@pytest.mark.parametrize("typ,m,n_out,n_in,dt", [(2, 45, 51216, 416, np.float32), (8, 112, 38144, 640, np.float32), (2, 112, 64000, 416, np.float32), (8, 3, 57000, 96, np.float32),
                                                 (2, 128, 12800, 2080, np.float32), (2, 100, 40000, 288, np.float16), (8, 256, 1300, 992, np.float16), (2, 160, 2000, 2080, np.float16),
                                                 (2, 32, 1030, 2048, np.float32), (2, 33, 1030, 2048, np.float32), (8, 64, 18950, 512, np.float32), (8, 64, 18800, 512, np.float32),
                                                 (8, 65, 18950, 1280, np.float32), (8, 65, 18800, 1280, np.float32), (2, 33, 16, 18944, np.float32), (8, 16, 300, 6144, np.float32),
                                                 (8, 16, 300, 6400, np.float32), (2, 100, 100, 2048, np.float16), (2, 100, 100, 2176, np.float16)])
def test_weights_through_tensor_memory(typ, m, n_out, n_in, dt, split): test_rows_against_the_exact_product(typ, m, n_out, n_in, dt, split)


# more rows than m rounded up to 128: 3 x 224, 10 x 256
@pytest.mark.parametrize("split", [True, False])
@pytest.mark.parametrize("typ,m", [(8, 625), (2, 640), (2, 641), (8, 2401)])
def test_equal_tiles_of_more_rows(typ, m, split): test_rows_against_the_exact_product(typ, m, 300, 416, np.float32, split)


def test_more_rows_than_a_grid_has_along_y():
  m, n_out, n_in, rng = 8 * 65535 + 9, 16, 32, np.random.default_rng(1)
  lin = quant.QuantLinear(n_in, n_out, 8, synth.q8_0_blocks(n_out, n_in, rng))
  x = rng.standard_normal((m, n_in)).astype(np.float32)
  got, w = lin(DeviceBuffer.from_numpy(x)).numpy(), lin.weight.dequantize().numpy().astype(np.float64)
  assert (np.abs(got - x @ w.T) <= 2.0 ** -20 * (np.abs(x) @ np.abs(w).T)).all()      # six rounded sums and the rounding of the halves, as above


@pytest.mark.parametrize("typ,m,n_out,n_in", [(2, 1, 64, 32), (8, 1, 1536, 1024), (8, 52, 130, 128), (2, 200, 512, 992),
                                              # 65 to 128 rows: through tensor memory as well
                                              (8, 65, 300, 416), (2, 112, 1300, 992), (2, 128, 130, 2080), (8, 128, 1536, 1024)])
def test_unsplit_sums_have_the_bits_of_the_kernel_without_a_workspace(typ, m, n_out, n_in):
  rng = np.random.default_rng(m)
  pw, x = quant.repack(synth.BLOCK_MAKERS[typ](n_out, n_in, rng), n_out, n_in, typ), DeviceBuffer.from_numpy(rng.standard_normal((m, n_in)).astype(np.float32))
  a, b, ws = DeviceBuffer.empty((m, n_out), np.float32), DeviceBuffer.empty((m, n_out), np.float32), DeviceBuffer(quant.qgemm_workspace_bytes(m, n_in))
  quant.qgemm(pw.buf.ptr, typ, n_out, n_in, x, a, m)
  quant.qgemm(pw.buf.ptr, typ, n_out, n_in, x, b, m, workspace=ws, unsplit=True)
  np.testing.assert_array_equal(a.numpy(), b.numpy())


@pytest.mark.parametrize("typ,m,n_out,n_in", [(2, 45, 6144, 4096), (8, 45, 6144, 4096), (2, 80, 6144, 4096), (8, 80, 6144, 4096), (8, 33, 1024, 4096), (2, 128, 1000, 4096)])
def test_nothing_of_the_halves_is_lost(typ, m, n_out, n_in):
  """The whole result's error against 64 bits, which bounds on single values do not see: a lost wl xh or wh xl is some 2^-12.8 of the result (the fp16 rounding of one operand),
  all three products in one sum 7.3e-6 (a truncating addition to it per product and 16 columns), two sums 4.0e-6 measured; the last two shapes through shared memory."""
  rng = np.random.default_rng(n_out + m)
  raw = synth.BLOCK_MAKERS[typ](n_out, n_in, rng)
  x = rng.standard_normal((m, n_in)).astype(np.float32)
  pw, y, ws = quant.repack(raw, n_out, n_in, typ), DeviceBuffer.empty((m, n_out), np.float32), DeviceBuffer(quant.qgemm_workspace_bytes(m, n_in, n_out))
  quant.qgemm(pw.buf.ptr, typ, n_out, n_in, DeviceBuffer.from_numpy(x), y, m, workspace=ws)
  ref = x.astype(np.float64) @ gq.weight_matrix(raw, n_out, n_in, typ).astype(np.float64).T
  err = np.linalg.norm(y.numpy() - ref) / np.linalg.norm(ref)
  assert err < 6e-6, err


@pytest.mark.parametrize("epilogue", [_lib.EPI_LINEAR, _lib.EPI_SILU_MUL])
@pytest.mark.parametrize("typ,m,n_out,n_in,dt", [(2, 45, 4096, 4096, np.float32), (8, 128, 6144, 4096, np.float32), (8, 33, 1024, 2048, np.float32), (8, 301, 4608, 3584, np.float16)])
def test_split_sums_repeat(typ, m, n_out, n_in, dt, epilogue):
  """Whichever CTA comes last at a tile, and whether it still has its own part in tensor memory or stored it: the parts are added in the order of K."""
  rng = np.random.default_rng(m)
  pw, x = quant.repack(synth.BLOCK_MAKERS[typ](n_out, n_in, rng), n_out, n_in, typ), DeviceBuffer.from_numpy(rng.standard_normal((m, n_in)).astype(dt))
  code, ws = _lib.F32 if dt == np.float32 else _lib.F16, DeviceBuffer(quant.qgemm_workspace_bytes(m, n_in, n_out))
  ys = [DeviceBuffer.empty((m, n_out // (2 if epilogue else 1)), dt) for _ in range(40)]
  for y in ys: quant.qgemm(pw.buf.ptr, typ, n_out, n_in, x, y, m, x_dtype=code, y_dtype=code, epilogue=epilogue, workspace=ws)
  first = ys[0].numpy().view(np.uint8)
  for y in ys[1:]: np.testing.assert_array_equal(y.numpy().view(np.uint8), first)


@pytest.mark.parametrize("m", [45, 160])
def test_swiglu_of_half_precision_rows(m):
  hidden, dim, rng = 1408, 512, np.random.default_rng(m)
  gate, up = (synth.q8_0_blocks(hidden, dim, rng) for _ in range(2))
  x, pw = rng.standard_normal((m, dim)).astype(np.float16), quant.repack(gate, hidden, dim, 8, raw_up=up)
  y, ws = DeviceBuffer.empty((m, hidden), np.float16), DeviceBuffer(quant.qgemm_workspace_bytes(m, dim, 2 * hidden))
  quant.qgemm(pw.buf.ptr, 8, 2 * hidden, dim, DeviceBuffer.from_numpy(x), y, m, x_dtype=_lib.F16, y_dtype=_lib.F16, epilogue=_lib.EPI_SILU_MUL, workspace=ws)
  g, u = (x.astype(np.float64) @ gq.weight_matrix(b, hidden, dim, 8).astype(np.float16).astype(np.float64).T for b in (gate, up))
  ref = g / (1 + np.exp(-g)) * u
  # as below, sums of one product per 16 columns, and the result's rounding to half precision
  tol = 2.0 ** -18 * (1.1 * np.abs(g).max() * np.abs(u) + np.abs(g) * np.abs(u).max() + 1) + 2.0 ** -11 * np.abs(ref)
  assert (np.abs(y.numpy() - ref) <= tol).all()


def test_norm_in_front_and_swiglu_behind():
  m, hidden, dim = 45, 1408, 512
  rng = np.random.default_rng(4)
  gate, up = (synth.q4_0_blocks(hidden, dim, rng) for _ in range(2))
  nw, x = (1 + 0.1 * rng.standard_normal(dim)).astype(np.float16), rng.standard_normal((m, dim)).astype(np.float32)
  pw = quant.repack(gate, hidden, dim, 2, raw_up=up)
  y, ws = DeviceBuffer.empty((m, hidden), np.float32), DeviceBuffer(quant.qgemm_workspace_bytes(m, dim))
  quant.qgemm(pw.buf.ptr, 2, 2 * hidden, dim, DeviceBuffer.from_numpy(x), y, m, epilogue=_lib.EPI_SILU_MUL, workspace=ws, norm_weight=DeviceBuffer.from_numpy(nw), norm_eps=1e-5)
  xn = x.astype(np.float64) / np.sqrt((x.astype(np.float64) ** 2).mean(-1, keepdims=True) + 1e-5) * nw
  g, u = (xn @ gq.weight_matrix(b, hidden, dim, 2).astype(np.float64).T for b in (gate, up))
  ref = g / (1 + np.exp(-g)) * u
  # each factor is good to 2^-18 of its largest value (the bound above at 512 columns); |d silu| <= 1.1
  tol = 2.0 ** -18 * (1.1 * np.abs(g).max() * np.abs(u) + np.abs(g) * np.abs(u).max() + 1)
  assert (np.abs(y.numpy() - ref) <= tol).all()


@pytest.mark.parametrize("typ,m,n_out,n_in,split", [(2, 5, 300, 4096, True), (8, 70, 1000, 992, True), (8, 70, 300, 14336, True), (2, 300, 130, 512, False),
                                                    # through tensor memory: enough K groups an SM, or no split; with whole tiles that wait in shared memory and without
                                                    (2, 5, 2400, 4096, True), (8, 17, 19000, 512, True), (2, 45, 51216, 416, True), (8, 70, 19000, 1280, True), (2, 100, 300, 992, False)])
def test_rows_of_any_magnitude(typ, m, n_out, n_in, split):
  """Rows far outside fp16's range lose no more than others: the bound of the exact product for each row by itself; and the same behind a norm weight that leads
  out of it."""
  rng = np.random.default_rng(m)
  raw = synth.BLOCK_MAKERS[typ](n_out, n_in, rng)
  w, pw = gq.weight_matrix(raw, n_out, n_in, typ).astype(np.float64), quant.repack(raw, n_out, n_in, typ)
  mag = np.concatenate([[0, 1e-30, 3e4, 1e30], 10.0 ** rng.uniform(-20, 20, m - 4)])[:, None]
  if not split: mag = np.maximum(mag, 1)      # smaller rows keep the bits of the form without a workspace there
  x = (rng.standard_normal((m, n_in)) * mag).astype(np.float32)
  y, ws = DeviceBuffer.empty((m, n_out), np.float32), DeviceBuffer(quant.qgemm_workspace_bytes(m, n_in, n_out) if split else quant.qgemm_unsplit_workspace_bytes(m, n_in))
  quant.qgemm(pw.buf.ptr, typ, n_out, n_in, DeviceBuffer.from_numpy(x), y, m, workspace=ws, unsplit=not split)
  bound = (2.0 ** -21 + 3 * np.ceil(n_in / 16) * 2.0 ** -23) * (np.abs(x).astype(np.float64) @ np.abs(w).T)
  assert (np.abs(y.numpy() - x.astype(np.float64) @ w.T) <= bound).all()
  nw, x = (2e4 * (1 + 0.1 * rng.standard_normal(n_in))).astype(np.float16), rng.standard_normal((m, n_in)).astype(np.float32)
  quant.qgemm(pw.buf.ptr, typ, n_out, n_in, DeviceBuffer.from_numpy(x), y, m, workspace=ws, unsplit=not split, norm_weight=DeviceBuffer.from_numpy(nw), norm_eps=1e-5)
  xn = x.astype(np.float64) / np.sqrt((x.astype(np.float64) ** 2).mean(1, keepdims=True) + 1e-5) * nw.astype(np.float64)
  # ... the norm's own rounding: a few units of 2^-24
  bound = (2.0 ** -20 + 3 * np.ceil(n_in / 16) * 2.0 ** -23) * (np.abs(xn) @ np.abs(w).T)
  assert (np.abs(y.numpy() - xn @ w.T) <= bound).all()
