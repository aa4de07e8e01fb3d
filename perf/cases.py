"""The work this package is used for, as cases that can be timed: greedy generation from quantised dense and mixture-of-experts
models, prompts, batches of sequences, one MXFP8 expert layer, and single quantised Linears.

A case is a dict of plain values.  `prepare` builds what a program holds before the call (the model with its conversation in the KV
cache, the layer with its weights), `run` is one call through the public interface.  Weights are random quant blocks whose scales give
every Linear unit gain; the embedding row of token t is the (scaled) head row of token t + 1, so that logits are peaked as a trained
model's are and the arg-max does not hang on the last bit of a sum."""
import zlib
import numpy as np
import torch
from tinygrad_b200 import moe, quant
from tinygrad_b200.fp8 import FP8Linear
from tinygrad_b200.model import Transformer, TransformerConfig
from tinygrad_b200.runtime import DeviceBuffer

Q4_0, Q8_0, Q4_K, Q6_K = 2, 8, 12, 14
QTYPES = {"q4_0": Q4_0, "q8_0": Q8_0, "q6_k": Q6_K}
# where the fp16 scales sit in a block, and the root mean square of the quants they multiply (random bytes)
F16_AT = {Q4_0: (0,), Q8_0: (0,), Q4_K: (0, 2), Q6_K: (208,)}
Q_RMS = {Q4_0: 4.61, Q8_0: 73.3, Q4_K: 323.0, Q6_K: 1367.0}
# a K-quant file as converters write it: value and down projections and the head in 6 bits, the rest in 4
K_MIX = {"attn_v": Q6_K, "ffn_down": Q6_K}

LLAMA_8B = dict(dim=4096, hidden=14336, heads=32, kv_heads=8, head_dim=128, vocab=128256, bias=False)
QWEN_7B = dict(dim=3584, hidden=18944, heads=28, kv_heads=4, head_dim=128, vocab=152064, bias=True)
SMALL = dict(dim=512, hidden=1408, heads=8, kv_heads=2, head_dim=64, vocab=2000, bias=False)


def listed():
  return [
    # a chat turn at batch 1: the package's headline workload (Llama-3-8B shape, Q4_0), 512 tokens of conversation
    dict(name="decode-8b-q4_0", kind="decode", quant="q4_0", **LLAMA_8B, blocks=32, context=512, new=8, kv="float16"),
    # the same far into a long conversation, where the KV cache counts (Qwen2-7B shape, Q8_0, q/k/v bias, a third of the depth)
    dict(name="decode-7b-q8_0-long", kind="decode", quant="q8_0", **QWEN_7B, blocks=10, context=3507, new=8, kv="float16"),
    # a small model with the reference's default fp32 cache: every launch is short, latency is everything
    dict(name="decode-small-q4_0", kind="decode", quant="q4_0", **SMALL, blocks=3, context=37, new=16, kv="float32"),
    # a file that mixes K-quants (the usual 4-bit download)
    dict(name="decode-8b-kquants", kind="decode", quant="k_mix", **LLAMA_8B, blocks=6, context=70, new=8, kv="float16"),
    # a short question to a model: time to the first token
    dict(name="prompt-45-8b-q4_0", kind="prompt", quant="q4_0", **LLAMA_8B, blocks=16, tokens=45, kv="float16"),
    # a document to a model: the prompt length of the 7B configuration, not a multiple of anything
    dict(name="prompt-1999-7b-q8_0", kind="prompt", quant="q8_0", **QWEN_7B, blocks=10, tokens=1999, kv="float16"),
    # serving a batch: eight prompts and their answers in lock-step
    dict(name="batch-8-7b-q8_0", kind="batch", quant="q8_0", **QWEN_7B, blocks=7, batch=8, tokens=128, new=32, kv="float16"),
    # one expert layer over a prompt (OLMoE shape)
    dict(name="moe-4096-olmoe", kind="moe", tokens=4096, dim=2048, ffn=1024, experts=64, topk=8, mode="softmax_topk"),
    # generation from a mixture-of-experts model at batch 1
    dict(name="decode-moe", kind="decode_moe", quant="q8_0", dim=1024, ffn=512, experts=32, topk=4, shared=0, heads=16, kv_heads=4, head_dim=64,
         vocab=32000, blocks=4, context=53, new=8),
    # the quantised Linear as an op: one activation row (the single-Linear configuration), and a ragged stack of half-precision rows
    dict(name="linear-1-q4_0", kind="linear", quant="q4_0", rows=1, n_in=4096, n_out=4096, x="float32", bias=False),
    dict(name="linear-301-q8_0-half", kind="linear", quant="q8_0", rows=301, n_in=3584, n_out=4608, x="float16", bias=True),
    # the per-tensor FP8 Linear
    dict(name="fp8-1000", kind="fp8", rows=1000, n_in=4096, n_out=4096, x="float32", bias=True),
  ]


# ---- drawn cases ----
def _log(rng, lo, hi):
  return int(round(lo * (hi / lo) ** rng.random()))


def _geometry(rng, quant_name, lo=384, hi=5120):
  step = 256 if quant_name == "k_mix" else 128
  dim = max(step, _log(rng, lo, hi) // step * step)
  head_dim = rng.choice([64, 128])
  heads = dim // head_dim
  hidden = max(step, int(dim * rng.uniform(2.5, 5.3)) // step * step) if quant_name == "k_mix" else int(dim * rng.uniform(2.5, 5.3)) // 32 * 32
  return dict(dim=dim, hidden=hidden, heads=heads, kv_heads=heads // rng.choice([r for r in (1, 2, 4, 7, 8) if heads % r == 0]), head_dim=head_dim,
              vocab=_log(rng, 2000, 152064), bias=rng.random() < 0.3)


def _block_bytes(c):
  q = c["heads"] * c["head_dim"]
  n = c["dim"] * (2 * q + 2 * c["kv_heads"] * c["head_dim"] + 3 * c["hidden"])
  return n * (2.0 if c["quant"] == "k_mix" else 34 / 32 if c["quant"] == "q8_0" else 18 / 32)


def draw(rng):
  kind = rng.choice(["decode"] * 3 + ["prompt"] * 3 + ["batch", "moe", "moe", "decode_moe", "linear", "linear", "fp8"])
  if kind in ("decode", "prompt", "batch"):
    c = dict(kind=kind, quant=rng.choice(["q4_0", "q8_0"] + (["k_mix"] if kind == "decode" else [])))
    c.update(_geometry(rng, c["quant"]))
    c["kv"] = rng.choice(["float16", "float16", "float32"])
    most = 1.5e9 if c["quant"] != "k_mix" else 2.0e9
    c["blocks"] = max(1, min(_log(rng, 1, 16), int(most / _block_bytes(c))))
    if kind == "decode": c.update(context=_log(rng, 8, 3500) if c["quant"] != "k_mix" else _log(rng, 8, 100), new=rng.choice([4, 8, 16]))
    elif kind == "prompt": c["tokens"] = _log(rng, 12, 2000)
    else: c.update(batch=_log(rng, 2, 40), tokens=_log(rng, 16, 200), new=rng.choice([8, 16, 32]))
    return c
  if kind == "moe":
    e = rng.choice([8, 16, 32, 64])
    return dict(kind=kind, tokens=_log(rng, 1, 4096), dim=256 * rng.randint(2, 8), ffn=128 * rng.randint(2, 8), experts=e, topk=rng.choice([1, 2, 4, 8]),
                mode=rng.choice(["topk_softmax", "softmax_topk"]))
  if kind == "decode_moe":
    dim = 256 * rng.randint(2, 6)
    return dict(kind=kind, quant=rng.choice(["q4_0", "q8_0"]), dim=dim, ffn=128 * rng.randint(2, 6), experts=rng.choice([8, 16, 32]), topk=rng.choice([2, 4, 6]),
                shared=rng.choice([0, 0, 512]), heads=dim // 64, kv_heads=dim // 64 // rng.choice([1, 2, 4]), head_dim=64, vocab=_log(rng, 2000, 50000),
                blocks=rng.randint(1, 4), context=_log(rng, 8, 400), new=8)
  if kind == "linear":
    q = rng.choice(["q4_0", "q8_0", "q6_k"])
    step = 256 if q == "q6_k" else 32
    return dict(kind=kind, quant=q, rows=_log(rng, 1, 600) if q != "q6_k" else _log(rng, 1, 8), n_in=max(step, _log(rng, 256, 8192) // step * step),
                n_out=_log(rng, 100, 16384), x=rng.choice(["float32", "float16"]), bias=rng.random() < 0.5)
  return dict(kind=kind, rows=_log(rng, 1, 2000), n_in=128 * rng.randint(2, 48), n_out=256 * rng.randint(1, 24), x=rng.choice(["float32", "float16"]),
              bias=rng.random() < 0.5)


# ---- inputs ----
def _gen(seed, name):
  return torch.Generator(device="cuda").manual_seed(zlib.crc32(name.encode()) + (int(seed) << 32))


def _host(t):
  """A device tensor as a numpy array in page-locked memory (torch keeps and reuses the pages)."""
  t = t.contiguous().reshape(-1)
  h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
  h.copy_(t)
  return h.numpy()


def _blocks(typ, n_out, n_in, seed, name):
  """Random quant blocks of a [n_out, n_in] weight with unit gain: zero-mean normal fp16 scales."""
  nel, nby = quant.GGML_QUANT[typ]
  nb, g = n_out * n_in // nel, _gen(seed, name)
  b = torch.randint(0, 256, (nb, nby), dtype=torch.uint8, device="cuda", generator=g)
  for at in F16_AT[typ]:
    d = torch.randn((nb, 1), device="cuda", generator=g) / (Q_RMS[typ] * n_in ** 0.5)
    b[:, at:at + 2] = d.half().view(torch.uint8)
  return b.reshape(-1)


class _Device:
  """A device buffer as torch sees it."""
  def __init__(self, buf, shape, typestr):
    self.buf = buf
    self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": typestr, "data": (buf.ptr, False), "version": 3}


def _view(buf, shape=None, typestr=None):
  shape = buf.shape if shape is None else shape
  return torch.as_tensor(_Device(buf, shape, typestr or {"float32": "<f4", "float16": "<f2", "uint16": "<i2"}[str(buf.dtype)]), device="cuda")


class _Weights:
  """The state dict of a random model: tensors are made when the constructor asks for them."""
  def __init__(self, c, seed):
    self.c, self.seed, self.biases = c, seed, c.get("bias", False)
    d, q, kv, h = c["dim"], c["heads"] * c["head_dim"], c["kv_heads"] * c["head_dim"], c.get("hidden", 0)
    self.shapes = {"attn_q": (q, d), "attn_k": (kv, d), "attn_v": (kv, d), "attn_output": (d, q), "ffn_gate": (h, d), "ffn_up": (h, d), "ffn_down": (d, h)}
    if c.get("shared"): self.shapes.update(ffn_gate_shexp=(c["shared"], d), ffn_up_shexp=(c["shared"], d), ffn_down_shexp=(d, c["shared"]))
    self.main = Q4_K if c["quant"] == "k_mix" else QTYPES[c["quant"]]
    self.head_type = Q6_K if c["quant"] == "k_mix" else self.main
    self.head = _blocks(self.head_type, c["vocab"], d, seed, "output")

  def type_of(self, short):
    return K_MIX.get(short, Q4_K) if self.c["quant"] == "k_mix" else self.main

  def types(self):
    return {f"blk.{i}.{n}.weight": self.type_of(n) for i in range(self.c["blocks"]) for n in self.shapes} if self.c["quant"] == "k_mix" else None

  def __contains__(self, key):
    return key != "output.bias" and not key.endswith("ffn_gate_inp_shexp.weight") and (not key.endswith(".bias") or self.biases)

  def __getitem__(self, key):
    c, short, kind = self.c, key.rsplit(".", 1)[0].split(".")[-1], key.rsplit(".", 1)[1]
    g, d = _gen(self.seed, key), c["dim"]
    if short == "token_embd":
      raw = DeviceBuffer.from_numpy(_host(self.head))
      e = _view(quant.dequantize(raw, c["vocab"] * d, self.head_type, np.float16)).reshape(c["vocab"], d)
      return _host(torch.roll(e, -1, 0) * d ** 0.5).reshape(c["vocab"], d)
    if short == "output": return _host(self.head)
    if short.endswith("_norm"): return _host((1 + 0.05 * torch.randn(d, device="cuda", generator=g)).half())
    if kind == "bias": return _host((0.02 * torch.randn(self.shapes[short][0], device="cuda", generator=g)).half())
    if short == "ffn_gate_inp": return _host(torch.randn((c["experts"], d), device="cuda", generator=g) / d ** 0.5).reshape(c["experts"], d)
    if short.endswith("_exps"):
      o, i = (d, c["ffn"]) if "down" in short else (c["ffn"], d)
      return _host(torch.randn((c["experts"], o, i), device="cuda", generator=g) / i ** 0.5).reshape(c["experts"], o, i)
    return _host(_blocks(self.type_of(short), *self.shapes[short], self.seed, key))


def _model(c, seed, room, **kw):
  w = _Weights(c, seed)
  extra = dict(num_experts=c["experts"], num_experts_per_tok=c["topk"], shared_expert_dim=c["shared"], norm_topk_prob=True) if c["kind"] == "decode_moe" else {}
  cfg = TransformerConfig(num_blocks=c["blocks"], dim=c["dim"], hidden_dim=c.get("hidden", c.get("ffn")), n_heads=c["heads"], n_kv_heads=c["kv_heads"],
                          norm_eps=1e-5, vocab_size=c["vocab"], head_dim=c["head_dim"], rope_theta=500000.0, rope_dim=c["head_dim"], v_head_dim=c["head_dim"],
                          max_context=-(-room // 64) * 64, qkv_bias=c.get("bias", False), kv_dtype=c.get("kv", "float16"), **extra)
  m = Transformer(cfg, w, ggml_type=w.main, output_type=w.head_type, linear_types=w.types(), **kw)
  return m


def _ids(seed, n, vocab):
  return [int(t) for t in np.random.default_rng([int(seed), 11]).integers(0, vocab, n)]


def _model_outputs(m):
  """What a step leaves behind besides the token: logits and the last block's KV cache."""
  return [_view(m.logits), _view(m.blk[-1].k_cache), _view(m.blk[-1].v_cache)]


def prepare(case, seed):
  c, kind = case, case["kind"]
  if kind in ("decode", "decode_moe"):
    # the conversation so far is in the cache; a pass writes the next answer (regenerated on every pass)
    m = _model(c, seed, c["context"] + c["new"] + 1)
    prompt = _ids(seed, c["context"], c["vocab"])
    next(m.generate(prompt))
    return dict(c=c, model=m, prompt=prompt, out=_model_outputs(m))
  if kind == "prompt":
    # two prompts in turn: nothing of the one can be reused for the other
    m = _model(c, seed, c["tokens"] + 1)
    ids = _ids(seed, 2 * c["tokens"], c["vocab"])
    a, b = ids[:c["tokens"]], ids[c["tokens"]:]
    b[0] = (a[0] + 1) % c["vocab"]
    return dict(c=c, model=m, prompts=[a, b], turn=0, out=_model_outputs(m))
  if kind == "batch":
    m = _model(c, seed, c["tokens"] + c["new"] + 1, batch=c["batch"])
    ids = _ids(seed, c["batch"] * c["tokens"], c["vocab"])
    return dict(c=c, model=m, prompts=[ids[i * c["tokens"]:(i + 1) * c["tokens"]] for i in range(c["batch"])],
                out=[_view(m.blk[-1].k_cache), _view(m.blk[-1].v_cache)])
  g = _gen(seed, kind)
  if kind == "moe":
    T, D, F, E = c["tokens"], c["dim"], c["ffn"], c["experts"]
    w = [_host(torch.randn(s, device="cuda", generator=g) * 0.02).reshape(s) for s in ((E, F, D), (E, F, D), (E, D, F))]
    layer = moe.MxMoE(*w, c["topk"], moe.ROUTE_SOFTMAX_TOPK if c["mode"] == "softmax_topk" else moe.ROUTE_TOPK_SOFTMAX)
    x = DeviceBuffer.from_numpy(_host(torch.randn((T, D), device="cuda", generator=g).bfloat16().view(torch.int16)).view(np.uint16).reshape(T, D))
    logits = DeviceBuffer.from_numpy(_host(torch.randn((T, E), device="cuda", generator=g)).reshape(T, E))
    return dict(c=c, layer=layer, x=x, logits=logits)
  x = torch.randn((c["rows"], c["n_in"]), device="cuda", generator=g)
  x = DeviceBuffer.from_numpy(_host(x.half() if c["x"] == "float16" else x).reshape(c["rows"], c["n_in"]))
  bias = _host(0.1 * torch.randn(c["n_out"], device="cuda", generator=g)) if c["bias"] else None
  if kind == "linear":
    typ = QTYPES[c["quant"]]
    return dict(c=c, layer=quant.QuantLinear(c["n_in"], c["n_out"], typ, _host(_blocks(typ, c["n_out"], c["n_in"], seed, "w")), bias), x=x)
  w = _host(torch.randn((c["n_out"], c["n_in"]), device="cuda", generator=g) / c["n_in"] ** 0.5).reshape(c["n_out"], c["n_in"])
  return dict(c=c, layer=FP8Linear(c["n_in"], c["n_out"], w, bias), x=x)


# ---- one pass ----
def run(s):
  c = s["c"]
  kind = c["kind"]
  if kind in ("decode", "decode_moe"):
    toks = []
    for t in s["model"].generate(s["prompt"]):
      toks.append(t)
      if len(toks) == c["new"]: break
    return [np.array(toks), *s["out"]]
  if kind == "prompt":
    prompt = s["prompts"][s["turn"]]
    s["turn"] ^= 1
    return [np.array([next(s["model"].generate(prompt))]), *s["out"]]
  if kind == "batch":
    toks = []
    for t in s["model"].generate_batch(s["prompts"]):
      toks.append(t)
      if len(toks) == c["new"]: break
    return [np.array(toks), *s["out"]]
  if kind == "moe":
    return _view(s["layer"](s["x"], s["logits"], c["tokens"])).view(torch.bfloat16)
  return _view(s["layer"](s["x"]))


# ---- what a pass cannot do without ----
def _raw_bytes(typ, n):
  nel, nby = quant.GGML_QUANT[typ]
  return n / nel * nby


def _llm_work(c):
  """(bytes of the block Linears, bytes of the head, weights of the block Linears, weights of the head) of a dense model."""
  d, q, kv, h = c["dim"], c["heads"] * c["head_dim"], c["kv_heads"] * c["head_dim"], c.get("hidden", 0)
  parts = {"attn_q": q * d, "attn_k": kv * d, "attn_v": kv * d, "attn_output": q * d, "ffn_gate": h * d, "ffn_up": h * d, "ffn_down": h * d}
  t = lambda n: K_MIX.get(n, Q4_K) if c["quant"] == "k_mix" else QTYPES[c["quant"]]
  per = sum(_raw_bytes(t(n), v) for n, v in parts.items() if v)
  head = c["vocab"] * d
  return c["blocks"] * per, _raw_bytes(Q6_K if c["quant"] == "k_mix" else QTYPES[c["quant"]], head), c["blocks"] * sum(parts.values()), head


def work(case):
  c, kind = case, case["kind"]
  if kind in ("decode", "prompt", "batch", "decode_moe"):
    wb, hb, wn, hn = _llm_work(c)
    kv_row = 2 * c["kv_heads"] * c["head_dim"] * (4 if c.get("kv") == "float32" else 2) * c["blocks"]
    att = 4 * c["heads"] * c["head_dim"] * c["blocks"]            # flops per query and cached position
    if kind == "prompt":
      n = c["tokens"]
      return {"bytes": wb + hb + n * (2 * c["dim"] + kv_row) + 4 * c["vocab"], "flops": 2.0 * wn * n + 2.0 * hn + att * n * n / 2}
    if kind == "batch":
      B, n, new = c["batch"], c["tokens"], c["new"]
      return {"bytes": (new + 1) * wb + new * hb + B * (n + new) * 2 * c["dim"] + B * kv_row * (n + new * (n + new / 2)) + 4.0 * B * new * c["vocab"],
              "flops": B * (2.0 * wn * (n + new) + 2.0 * hn * new + att * (n * n / 2 + new * (n + new / 2)))}
    if kind == "decode_moe":
      e = c["topk"] * 3 * c["dim"] * c["ffn"] * c["blocks"]       # the chosen experts' weights; MXFP8: 33 bytes per 32
      sh = 3 * c["dim"] * c["shared"] * c["blocks"]
      wb += e * 33 / 32 + _raw_bytes(QTYPES[c["quant"]], sh) + 4 * c["experts"] * c["dim"] * c["blocks"]
      wn += e + sh + c["experts"] * c["dim"] * c["blocks"]
    new, ctx = c["new"], c["context"] + c["new"] / 2
    return {"bytes": new * (wb + hb + ctx * kv_row + 2 * c["dim"] + 4 * c["vocab"]), "flops": new * (2.0 * (wn + hn) + att * ctx)}
  if kind == "moe":
    T, D, F, E, k = c["tokens"], c["dim"], c["ffn"], c["experts"], c["topk"]
    return {"bytes": min(E, T * k) * 3 * D * F * 33 / 32 + T * (4 * D + 4 * E), "flops": 6.0 * T * k * D * F}
  size = 2 if c["x"] == "float16" else 4
  w = c["n_in"] * c["n_out"]
  return {"bytes": (_raw_bytes(QTYPES[c["quant"]], w) if kind == "linear" else w) + size * c["rows"] * (c["n_in"] + c["n_out"]), "flops": 2.0 * c["rows"] * w}


def tolerance(case):
  kind = case["kind"]
  # token ids are exact; logits and cache rows carry the fp16 rounding of the cache (5e-4) and of quantised activations through the blocks
  if kind in ("decode", "prompt", "batch"): return {"rel": 3e-3, "max": 0.1}
  # a bf16 rounding that moves with the order of a sum can move an E4M3 code by one step (2^-4 of the value) before the second product
  if kind == "decode_moe": return {"rel": 1e-2, "max": 0.3}
  if kind == "moe": return {"rel": 5e-3, "max": 0.3}
  # half-precision results: their rounding; fp32: the 15-bit block quantisation of the activations in the one-row kernels, fp32 sums elsewhere
  if case["x"] == "float16": return {"rel": 1e-3, "max": 0.02}
  return {"rel": 1e-4, "max": 5e-3}
