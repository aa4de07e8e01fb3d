"""Decode attention in thread-block clusters at the edges of its chunks (64 positions) and of its split over 8 or 16 CTAs: one position, whole and
ragged chunks, more chunks than CTAs, every group size of query heads, partial rotation, and the quantised hand-over record."""
import ctypes
import numpy as np
import pytest
from tinygrad_b200 import _lib
from tinygrad_b200.model import precompute_freqs_cis
from tinygrad_b200.runtime import DeviceBuffer, device_status
from oracle import llm
from gpu_util import need_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu(): need_gpu()


@pytest.mark.parametrize("kv", [np.float16, np.float32])
@pytest.mark.parametrize("n_heads,n_kv,hd,rope_dim,pos", [(8, 8, 64, 64, 0), (7, 1, 128, 128, 62), (6, 2, 64, 32, 63), (8, 1, 128, 128, 40), (5, 1, 128, 64, 64), (8, 1, 128, 128, 1023),
                                                          (32, 16, 64, 64, 511), (4, 2, 128, 0, 512), (30, 15, 128, 128, 1100), (4, 4, 64, 64, 2047)])
def test_cluster_attention(n_heads, n_kv, hd, rope_dim, pos, kv):
  rng = np.random.default_rng(pos + n_heads)
  ctx, lib = 2048 if pos > 63 else 64, _lib.load()                               # one chunk of positions at most: a single CTA
  qkv = (2 * rng.standard_normal((n_heads + 2 * n_kv) * hd)).astype(np.float32)
  kc = np.full((n_kv, ctx, hd), np.nan, kv); vc = kc.copy()              # rows from `pos` on hold no values yet
  kc[:, :pos], vc[:, :pos] = rng.standard_normal((n_kv, pos, hd)), rng.standard_normal((n_kv, pos, hd))
  fc = precompute_freqs_cis(max(rope_dim, 2), ctx, 10000.0)
  rope = lambda t: np.concatenate([llm.apply_rope(t[..., :rope_dim], fc[pos:pos + 1]), t[..., rope_dim:]], axis=-1) if rope_dim else t
  heads = qkv.reshape(-1, 1, hd)
  q, k, v = rope(heads[None, :n_heads])[0, :, 0].astype(np.float64), rope(heads[None, n_heads:n_heads + n_kv])[0, :, 0], heads[n_heads + n_kv:, 0]
  rep = lambda c, new: np.repeat(np.concatenate([c[:, :pos], new.astype(kv)[:, None]], 1).astype(np.float64), n_heads // n_kv, 0)
  s = np.einsum("hd,hpd->hp", q, rep(kc, k)) / np.sqrt(hd)
  p = np.exp(s - s.max(-1, keepdims=True))
  want = np.einsum("hp,hpd->hd", p / p.sum(-1, keepdims=True), rep(vc, v)).reshape(-1)
  d = [DeviceBuffer.from_numpy(a) for a in (qkv, kc, vc, fc, np.array([pos], np.int32))]
  out, n_split = DeviceBuffer.empty((n_heads * hd,), np.float32), lib.b200q_attn_min_split(ctx)
  scratch = DeviceBuffer(lib.b200q_attn_scratch_bytes(n_heads, n_kv, hd, n_split), zero=True)
  xq = DeviceBuffer(lib.b200q_xq_bytes(n_heads * hd), zero=True) if hd == 128 else None
  a = _lib.AttnArgs(d[0].ptr, d[1].ptr, d[2].ptr, _lib.F16 if kv == np.float16 else _lib.F32, d[3].ptr, d[4].ptr, out.ptr, scratch.ptr, n_heads, n_kv, hd, rope_dim, ctx, n_split, 0, xq.ptr if xq else None)
  _lib.check(lib.b200q_attn_decode(ctypes.byref(a), None))
  got = out.numpy()
  # scores are good to 2^-21 of sum |q k| (remainders of q to 2^-22, fp32 sums) and the approximate exponential to 2^-21 of its argument; values are
  # at most a few units: 1e-4 covers both at scores of tens
  assert np.abs(got - want).max() <= 1e-4 * max(1.0, np.abs(want).max())
  if rope_dim == 0: np.testing.assert_array_equal(d[1].numpy()[:, pos], k.astype(kv))
  np.testing.assert_array_equal(d[2].numpy()[:, pos], v.astype(kv))
  assert np.isnan(d[2].numpy()[:, pos + 1:].astype(np.float32)).all()               # nothing else written
  if xq is not None:                # the record: 15-bit digits with a scale per 32 (one group of 128 per head), within half a step of the output
    rec = xq.numpy((xq.nbytes,), np.uint8)
    words = rec[:n_heads * 256].view(np.int8).reshape(n_heads, 2, 8, 4, 4)          # [head][half of the words][slot][word][byte]
    scales = rec[n_heads * 256:].view(np.float32).reshape(n_heads, 2, 2, 2, 2)      # [head][digit][block pair][block][scale, offset]
    for h in range(n_heads):
      for b in range(4):
        digit = [np.concatenate([words[h, r >> 2, b + 4 * lo, r & 3] for r in (0, 2, 4, 6, 1, 3, 5, 7)]).astype(np.float64) for lo in (0, 1)]
        vals = digit[0] * scales[h, 0, b >> 1, b & 1, 0] + digit[1] * scales[h, 1, b >> 1, b & 1, 0]
        blk = got[h * hd + 32 * b:h * hd + 32 * b + 32]
        assert np.abs(vals - blk).max() <= 0.51 * np.abs(blk).max() / 16256 + 1e-12
  assert device_status() == 0
