"""What the kernels lose against exact arithmetic, held to what 32-bit arithmetic gives."""
import ctypes
import numpy as np
import pytest
from oracle import ggml_quant as gq
from tinygrad_b200 import _lib, quant, synth
from tinygrad_b200.runtime import DeviceBuffer
from gpu_util import need_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu(): need_gpu()


def test_activation_codes_are_the_rounded_quotients():
  """The codes of the activation blocks, read back through an identity matrix: the nearest integer to x * (16256 / max) for every value, for blocks of
  any magnitude."""
  rng = np.random.default_rng(0)
  n, m = 1024, 256
  raw = np.zeros((n, n // 32, 34), np.uint8)                          # Q8_0: scale 1, quant 1 on the diagonal
  raw[:, :, :2] = np.frombuffer(np.float16(1).tobytes(), np.uint8)
  raw[np.arange(n), np.arange(n) // 32, 2 + np.arange(n) % 32] = 1
  x = rng.standard_normal((m, n)).astype(np.float32)
  x[1] *= np.float32(7e37); x[2] *= np.float32(1e-33)
  pw, y = quant.repack(raw.reshape(-1), n, n, 8), DeviceBuffer.empty((m, n), np.float32)
  quant.gemv(pw.buf.ptr, 8, n, n, DeviceBuffer.from_numpy(x), y, m=m)
  blocks = x.reshape(m, n // 32, 32)
  amax = np.abs(blocks).max(-1, keepdims=True)
  codes = np.rint(blocks * (np.float32(16256) / amax))
  got = np.rint(y.numpy().reshape(blocks.shape).astype(np.float64) / (amax / np.float32(16256)).astype(np.float64))
  np.testing.assert_array_equal(got, codes)


def decode_attention(qkv, kc, vc, n_heads, pos):
  """b200q_attn_decode at `pos` without rotation, and the exact result."""
  (n_kv, ctx, hd), kv, lib = kc.shape, kc.dtype, _lib.load()
  rope = np.concatenate([np.ones((ctx, hd // 2)), np.zeros((ctx, hd // 2))], 1).astype(np.float32)
  q, k, v = (a.astype(np.float64) for a in (qkv[:n_heads], qkv[n_heads:n_heads + n_kv].astype(kv), qkv[n_heads + n_kv:].astype(kv)))
  rep = lambda c, new: np.repeat(np.concatenate([c[:, :pos].astype(np.float64), new[:, None]], 1), n_heads // n_kv, 0)
  s = np.einsum("hd,hpd->hp", q, rep(kc, k)) / np.sqrt(hd)
  p = np.exp(s - s.max(-1, keepdims=True))
  want = np.einsum("hp,hpd->hd", p / p.sum(-1, keepdims=True), rep(vc, v))
  d = [DeviceBuffer.from_numpy(a) for a in (qkv, kc, vc, rope, np.array([pos], np.int32))]
  out, n_split = DeviceBuffer.empty((n_heads, hd), np.float32), lib.b200q_attn_min_split(ctx)
  scratch = DeviceBuffer(lib.b200q_attn_scratch_bytes(n_heads, n_kv, hd, n_split), zero=True)
  a = _lib.AttnArgs(d[0].ptr, d[1].ptr, d[2].ptr, _lib.F16 if kv == np.float16 else _lib.F32, d[3].ptr, d[4].ptr, out.ptr, scratch.ptr, n_heads, n_kv, hd, hd, ctx, n_split, 0, None)
  _lib.check(lib.b200q_attn_decode(ctypes.byref(a), None))
  return out.numpy(), want


@pytest.mark.parametrize("kv", [np.float16, np.float32])
@pytest.mark.parametrize("n_heads,n_kv,hd", [(8, 2, 128), (8, 2, 64)])
def test_decode_attention_rounds_to_nearest(n_heads, n_kv, hd, kv):
  """Far into a context, where a tensor core that truncates its running sums (always towards zero) is 4.6e-7 (fp16 cache) to 2.4e-6 (fp32 cache) off.  Sums
  rounded to nearest add up like a random walk: 55 chunks, 8 partial sums a score and 4 or 8 a chunk stay within 6 x 2^-24 of the output's norm."""
  rng = np.random.default_rng(hd)
  qkv = rng.standard_normal((n_heads + 2 * n_kv, hd)).astype(np.float32)
  got, want = decode_attention(qkv, *(rng.standard_normal((n_kv, 3520, hd)).astype(kv) for _ in range(2)), n_heads, 3507)
  assert np.linalg.norm(got - want) <= 6 * 2.0 ** -24 * np.linalg.norm(want)


@pytest.mark.parametrize("n_heads,n_kv,hd", [(8, 1, 128), (6, 2, 64)])
def test_decode_attention_takes_queries_of_any_magnitude(n_heads, n_kv, hd):
  """Heads from far below to far above fp16's range, each against keys that make scores of order one of it; a head that is not a number stays none."""
  rng, pos = np.random.default_rng(n_heads), 70
  qkv, kc, vc = rng.standard_normal((n_heads + 2 * n_kv, hd)).astype(np.float32), *(rng.standard_normal((n_kv, 128, hd)).astype(np.float16) for _ in range(2))
  for up, down in ((2.0 ** 17, 2.0 ** -12), (2.0 ** -18, 2.0 ** 12)):
    x = qkv.copy()
    x[:n_heads] *= np.float32(up); x[n_heads:n_heads + n_kv] *= np.float32(down)
    got, want = decode_attention(x, (kc.astype(np.float32) * np.float32(down)).astype(np.float16), vc, n_heads, pos)
    # the scores' error is 2^-22 of their size, which is up to 2^5 times that of the test above
    assert np.isfinite(got).all() and np.linalg.norm(got - want) <= 2.0 ** -17 * np.linalg.norm(want)
  qkv[1, 3] = np.nan
  got, _ = decode_attention(qkv, kc, vc, n_heads, pos)
  assert np.isnan(got[1]).all() and np.isfinite(np.delete(got, 1, 0)).all()


@pytest.mark.parametrize("typ", [12, 14])
def test_kquant_gemv_is_as_exact_as_the_dense_one(typ):
  """The same fp16 weights packed and dense: the packed form's tensor-core sums are no further from 64 bits than fp32 sums in the dense form (5.5e-7 against
  1.5e-7 with accumulators that run through the tensor core, which truncates)."""
  n_out, n_in, rng = 512, 14336, np.random.default_rng(typ)
  raw = synth.random_blocks(typ, n_out, n_in, rng)
  w = DeviceBuffer.from_numpy(gq.dequantize(raw, n_out * n_in, typ).astype(np.float16).reshape(n_out, n_in))
  pw, err = quant.repack(raw, n_out, n_in, quant.WIDE_QUANT[typ]), np.zeros(2)
  for _ in range(4):
    x = rng.standard_normal((1, n_in)).astype(np.float32)
    want, dx = w.numpy().astype(np.float64) @ x[0].astype(np.float64), DeviceBuffer.from_numpy(x)
    y, z = DeviceBuffer.empty((n_out,), np.float32), DeviceBuffer.empty((n_out,), np.float32)
    quant.gemv(pw.buf.ptr, pw.qtype, n_out, n_in, dx, y)
    quant.gemv_dense(w, _lib.F16, n_out, n_in, dx, z)
    err += [np.linalg.norm(b.numpy() - want) / np.linalg.norm(want) for b in (y, z)]
  assert err[0] <= 1.25 * err[1], err


def prompt_attention(q, k, v, kv, hd):
  """b200q_attn_prefill on rows [T, heads, hd] without rotation, and the exact result."""
  (T, H, _), K = q.shape, k.shape[1]
  ctx, lib = -(-T // 64) * 64, _lib.load()
  rope = np.concatenate([np.ones((ctx, hd // 2)), np.zeros((ctx, hd // 2))], 1).astype(np.float32)
  d = [DeviceBuffer.from_numpy(a) for a in (np.concatenate([q, k, v], 1).astype(np.float32), rope)]
  kc, vc = (DeviceBuffer.empty((K, ctx, hd), kv, zero=True) for _ in range(2))
  qs, out = DeviceBuffer.empty((T, H * hd), np.float32), DeviceBuffer.empty((T, H, hd), np.float32)
  _lib.check(lib.b200q_attn_prefill(d[0].ptr, kc.ptr, vc.ptr, _lib.F16 if kv == np.float16 else _lib.F32, d[1].ptr, 0, T, H, K, hd, hd, ctx, qs.ptr, out.ptr, _lib.F32, None))
  q64, k64, v64 = q.astype(np.float64), *(np.repeat(a.astype(kv).astype(np.float64), H // K, 1) for a in (k, v))
  s = np.einsum("thd,shd->hts", q64, k64) / np.sqrt(hd)
  s[:, np.triu(np.ones((T, T), bool), 1)] = -np.inf
  p = np.exp(s - s.max(-1, keepdims=True))
  return out.numpy(), np.einsum("hts,shd->thd", p / p.sum(-1, keepdims=True), v64)


@pytest.mark.parametrize("hd", [16, 32, 64, 128])
@pytest.mark.parametrize("T", [1, 17, 64, 201])
def test_prompt_attention_keeps_an_fp32_cache(hd, T):
  """Keys and values of an fp32 cache are not rounded on the way to the tensor cores (4e-4 when they were, as fp16): the one-token kernel's bound.  Rows of
  any magnitude, among them values beyond fp16's range and a query that only one row's values reach."""
  rng = np.random.default_rng(hd + T)
  q, k, v = (rng.standard_normal((T, n, hd)).astype(np.float32) for n in (4, 2, 2))
  got, want = prompt_attention(q, k, v, np.float32, hd)
  assert np.linalg.norm(got - want) <= 6 * 2.0 ** -24 * np.linalg.norm(want)
  # keys times queries of any magnitude give the same scores; a value row's magnitude shows in the rows that attend to it
  e = rng.integers(-60, 61, (2, 1, 1, 1)).astype(np.float32)
  big, size = prompt_attention(q * 2.0 ** e[0], k * 2.0 ** -e[0], v * np.float32(1e6), np.float32, hd), np.float32(1e6)
  assert np.linalg.norm(big[0] / size - want) <= 8 * 2.0 ** -24 * np.linalg.norm(want)
  mag = (10.0 ** rng.uniform(-6, 6, (T, 2, 1))).astype(np.float32)
  got, want = prompt_attention(q, k, v * mag, np.float32, hd)
  # each output against what its own sum is made of: |p v| summed
  reach = prompt_attention(q, k, np.abs(v * mag), np.float32, hd)[1]
  assert (np.abs(got - want) <= 2.0 ** -18 * reach).all()


def test_prompt_attention_takes_queries_of_any_magnitude():
  rng = np.random.default_rng(3)
  q, k, v = (rng.standard_normal((70, n, 64)).astype(np.float32) for n in (4, 2, 2))
  got, want = prompt_attention(q * np.float32(2.0 ** 17), k * np.float32(2.0 ** -12), v, np.float16, 64)       # queries past 65504
  assert np.isfinite(got).all() and np.linalg.norm(got - want) <= 2.0 ** -18 * np.linalg.norm(want)


@pytest.mark.parametrize("typ", [2, 8])
@pytest.mark.parametrize("tokens,chunk", [(37, 512), (37, 16), (3, 512)])
def test_a_small_model_is_as_exact_as_fp32_sums(typ, tokens, chunk):
  """Prompt (all in one pass, in passes of 16 with the last token along, in one-token steps) and three answers of a model whose Linears are small and whose cache is fp32: logits and the
  last block's cache rows against 64 bits.  No value is rounded to fewer than 32 bits on the way; sums of up to 1408 products through three blocks come to at most 2.4e-6, bound 5e-6.
  (Activation codes of 15 bits, in any one of the paths, leave 5e-5 to 1e-4.)"""
  from tinygrad_b200.model import Transformer, TransformerConfig, precompute_freqs_cis
  d, hid, H, KV, hd, vocab, nb = 512, 1408, 8, 2, 64, 2000, 3
  cfg = TransformerConfig(num_blocks=nb, dim=d, hidden_dim=hid, n_heads=H, n_kv_heads=KV, norm_eps=1e-5, vocab_size=vocab, head_dim=hd, rope_theta=500000.0, rope_dim=hd, max_context=64,
                          kv_dtype="float32")
  sd = synth.dense_model_raw(cfg, typ, seed=11, embd_std=0.3, scale_std=1 / ((4.61 if typ == 2 else 73.3) * d ** 0.5))
  m = Transformer(cfg, sd, ggml_type=typ, prefill_chunk=chunk)
  prompt = [int(t) for t in np.random.default_rng(tokens).integers(0, vocab, tokens)]
  first, ids = None, list(prompt)
  for _, tok in zip(range(3), m.generate(prompt)):
    if first is None: first = m.read_logits()
    ids.append(tok)
  last, T = m.read_logits(), len(ids) - 1
  table = precompute_freqs_cis(hd, T, 500000.0).astype(np.float64)
  cos, sin = table[:, None, :hd // 2], table[:, None, hd // 2:]
  w = lambda name, o, i: gq.weight_matrix(sd[name + ".weight"], o, i, typ).astype(np.float64)
  norm = lambda x, name: x / np.sqrt((x * x).mean(-1, keepdims=True) + 1e-5) * sd[name + ".weight"].astype(np.float64)
  def rope(x):
    a, b = x[..., :hd // 2], x[..., hd // 2:]
    return np.concatenate([a * cos - b * sin, b * cos + a * sin], -1)
  x = sd["token_embd.weight"].astype(np.float64)[ids[:T]]
  for i in range(nb):
    p = f"blk.{i}."
    h = norm(x, p + "attn_norm")
    q, k, v = rope((h @ w(p + "attn_q", H * hd, d).T).reshape(T, H, hd)), rope((h @ w(p + "attn_k", KV * hd, d).T).reshape(T, KV, hd)), (h @ w(p + "attn_v", KV * hd, d).T).reshape(T, KV, hd)
    s = np.einsum("qhd,khd->hqk", q, np.repeat(k, H // KV, 1)) / hd ** 0.5
    s = np.exp(np.where(np.tri(T, dtype=bool), s, -np.inf) - np.where(np.tri(T, dtype=bool), s, -np.inf).max(-1, keepdims=True))
    x = x + np.einsum("hqk,khd->qhd", s / s.sum(-1, keepdims=True), np.repeat(v, H // KV, 1)).reshape(T, H * hd) @ w(p + "attn_output", d, H * hd).T
    h = norm(x, p + "ffn_norm")
    g = h @ w(p + "ffn_gate", hid, d).T
    x = x + (g / (1 + np.exp(-g)) * (h @ w(p + "ffn_up", hid, d).T)) @ w(p + "ffn_down", d, hid).T
  logits = norm(x, "output_norm") @ w("output", vocab, d).T
  off = lambda got, want: np.linalg.norm(got - want) / np.linalg.norm(want)
  rows = lambda buf: buf.numpy().reshape(KV, 64, hd)[:, :T].transpose(1, 0, 2)
  got = [off(first, logits[tokens - 1]), off(last, logits[-1]), off(rows(m.blk[-1].k_cache), k), off(rows(m.blk[-1].v_cache), v)]
  assert max(got) <= 5e-6, got
