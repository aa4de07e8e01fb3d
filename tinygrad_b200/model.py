"""The quantized-LLM decode path on one B200: host-side mirror of tinygrad/llm/model.py.

`TransformerConfig` carries the reference's field names (model.py:52-83);
`Transformer.generate(tokens)` yields greedy tokens like the reference's
`generate` at temperature 0 (model.py:464-484).  The forward pass of one token is
five fused launches per block (norm+QKV GEMV, attention, O GEMV+residual,
norm+gate/up GEMV+SwiGLU, down GEMV+residual) plus embedding, head GEMV and
arg-max, chained with programmatic dependent launch and replayed as one CUDA graph.
"""
from __future__ import annotations
from dataclasses import dataclass
import numpy as np
from . import _lib, quant
from ._lib import check, F32, F16, EPI_LINEAR, EPI_SILU_MUL, FLAG_PDL
from .runtime import DeviceBuffer, PinnedBuffer, Stream, Graph, Event, synchronize as runtime_sync
import ctypes, itertools, os

# batched decode with another head_dim than 64 or 128: attention of all sequences in one launch of the one-lane-per-position decode kernel instead of
# the prompt-pass kernels with one query row per CTA (measured 1.4 % slower at 8 sequences x 130 positions: off unless asked for)
SEQ_ATTENTION = os.environ.get("B200Q_SEQ_ATTENTION", "0") == "1"


# Prompts of at least this many uncached tokens take the GEMM path.  One pass over the weights for 3 to 12 tokens costs 1.02 ms on six 8B-shaped Q4_0 blocks (a
# one-token step 245 us), 0.90 on five 7B-shaped Q8_0 blocks (296 us), 0.22 on three 512-wide ones (47 us): it is the faster one from 4 or 5 tokens on.
PREFILL_ROWS = 6


@dataclass(frozen=True)
class TransformerConfig:           # field names of tinygrad/llm/model.py:52-83 (dense GQA subset)
  num_blocks: int
  dim: int
  hidden_dim: int
  n_heads: int
  n_kv_heads: int
  norm_eps: float
  vocab_size: int
  head_dim: int
  rope_theta: float
  rope_dim: int
  v_head_dim: int = 0
  max_context: int = 0
  qkv_bias: bool = False
  kv_dtype: str = "float16"        # the cache dtype; the reference takes it from DEFAULT_FLOAT (model.py:202-203)
  num_experts: int = 0             # > 0: every block's FFN is a routed mixture of experts (model.py:94-98,110-135) with MXFP8 expert weights
  num_experts_per_tok: int = 0
  norm_topk_prob: bool = False
  expert_gating_func: str = "softmax"   # "softmax" | "sigmoid" | "softmax_weight" | "sqrt_softplus" (ExpertGating, model.py:9-13)
  routed_scaling_factor: float = 1.0
  shared_expert_dim: int = 0            # > 0: a dense SwiGLU expert every token also goes through (model.py:99-103,131-134)
  shared_expert_gate: bool = True       # its output is scaled by sigmoid(x . ffn_gate_inp_shexp) when that tensor is present
  expert_bias: bool = False             # exp_probs_b: a bias added to the scores for the selection only (model.py:113,123)


def precompute_freqs_cis(dim: int, end: int, theta: float) -> np.ndarray:
  """cos || sin table of tinygrad/llm/model.py:15-19, fp32 [end, dim]."""
  f = (1.0 / (np.float32(theta) ** (np.arange(0, dim, 2, dtype=np.float32) / np.float32(dim)))).astype(np.float32)
  ang = np.arange(end, dtype=np.float32)[:, None] * f[None, :]
  return np.concatenate([np.cos(ang), np.sin(ang)], axis=-1).astype(np.float32)


class _Block:
  pass


class _BlockLinear:
  """A Linear of a block that keeps full-precision activations: a packed K-quant matrix, or an fp16 one (qtype None).  `row0`: where its rows
  start in the vector it writes."""
  def __init__(self, qtype, n_out: int, n_in: int, buf: DeviceBuffer, row0: int, swiglu: bool = False):
    self.qtype, self.n_out, self.n_in, self.buf, self.row0, self.swiglu = qtype, n_out, n_in, buf, row0, swiglu
    self.behind = None       # (Q6_K matrix, rows) of the rows behind a Q4_K one

  @property
  def algorithmic_bytes(self) -> int:
    if self.qtype is None: return 2 * self.n_out * self.n_in
    more = quant.PackedWeight(_lib.Q6_K_WIDE, self.behind[1], self.n_in, self.behind[0], False).algorithmic_bytes if self.behind else 0
    return quant.PackedWeight(self.qtype, self.n_out, self.n_in, self.buf, self.swiglu).algorithmic_bytes + more

  def run(self, x, y, bias=None, residual=None, flags=0, **kw) -> None:
    at = lambda buf, size: None if buf is None else buf.ptr + size * self.row0
    if self.qtype is None:
      quant.gemv_dense(self.buf, F16, self.n_out, self.n_in, x, at(y, 4), bias=at(bias, 2), residual=at(residual, 4), flags=flags, **kw)
    else:
      w2, rows2 = self.behind or (None, 0)
      quant.gemv(self.buf.ptr, self.qtype, self.n_out + rows2, self.n_in, x, at(y, 4), bias=at(bias, 2), residual=at(residual, 4), flags=flags,
                 epilogue=EPI_SILU_MUL if self.swiglu else quant.EPI_LINEAR, w2_ptr=w2.ptr if w2 else None, n_first=self.n_out if w2 else 0, **kw)


# hand-over edges used when the caller does not choose (see Transformer.__init__): the ones that measured faster
DEFAULT_HANDOVER = tuple(e for e in os.environ.get("B200Q_HANDOVER", "attn_o").split(",") if e)
STAGED_HANDOVER = os.environ.get("B200Q_STAGED_HANDOVER", "1") == "1"


class Transformer:
  engine = None        # "step" or "chain" once the constructor has chosen

  def __init__(self, config: TransformerConfig, state_dict: dict, ggml_type: int = _lib.Q4_0, n_split: int = 0, use_pdl: bool = True,
               use_graph: bool = True, gemv_max_ctas: int = 0, handover=None, tp=None, output_type: int = None, prefill_rows: int = PREFILL_ROWS,
               prefill_chunk: int = 512, batch: int = 1, engine: str = None, linear_types: dict = None, pipelined_gemm: bool = True):
    """state_dict: the reference's tensor names -> numpy arrays; Linear weights as raw
    GGUF block bytes (uint8), embeddings / norms / biases as fp16.
    tp: a tensor_parallel.TPGroup; `config` is then the FULL model and `state_dict` this rank's shard (shard_state_dict).
    output_type: GGML type of `output.weight` when it differs from the block Linears' (F16 / BF16 / F32 heads run the dense GEMV).
    prefill_rows: prompts with at least this many uncached tokens go through the tensor-core GEMM path, `prefill_chunk` rows at a time (0: always one
    token per step); shorter ones take decode steps.
    engine: how a one-token step runs.  "step": one persistent kernel for the whole step (b200q_decode_step); "chain": five launches per
    block chained with programmatic dependent launch and replayed as a CUDA graph (the default: at batch 1 it measured faster, the
    grid-wide waits inside one kernel costing more than kernel boundaries do).
    linear_types: state-dict name -> GGML type of block Linear weights whose type is not `ggml_type` (files that mix block formats, e.g.
    Q4_K with Q6_K).  Unless every block Linear is of one fused type (Q4_0 / Q8_0) the blocks keep their activations in full
    precision: Q4_K and Q6_K weights stay in their file form and run the K-quant GEMV, the others are dequantised once to fp16 on the device (the
    cast the reference applies to every loaded tensor, model.py:376) and run the dense-weight GEMV.
    batch: sequences decoded in lock-step (`generate_batch`): one KV cache per sequence, every Linear a tensor-core GEMM over the
    batch rows (the reference's forward on tokens [B, T], model.py:358-364; its cache is sized by the first call's batch, model.py:200-203)."""
    self.tp, self.full_config = tp, config
    if tp is not None:
      from .tensor_parallel import local_config
      config = local_config(config, tp.size)
    c = self.config = config
    vocab_full = self.full_config.vocab_size
    assert c.max_context > 0 and c.n_heads % c.n_kv_heads == 0
    self.qtype, self.flags, self.use_graph = ggml_type, (FLAG_PDL if use_pdl else 0), use_graph
    self.q_dim, self.kv_dim = c.n_heads * c.head_dim, c.n_kv_heads * c.head_dim
    self.pipelined_gemm = pipelined_gemm      # prompt GEMMs on the pipelined kernel (False: the single-buffered one)
    self.gemv_max_ctas = gemv_max_ctas if isinstance(gemv_max_ctas, dict) else {"*": gemv_max_ctas}   # per Linear ("qkv", "o", "gate_up", "down", "head") or one for all
    self.n_split = n_split or _lib.load().b200q_attn_min_split(c.max_context)
    self.max_context = c.max_context
    self.stream = Stream(tp.stream_ptr()) if (tp is not None and tp.stream_ptr() is not None) else Stream()
    self.tp_peer = tp is not None and tp.kind_id == "peer"
    sd = state_dict
    qkv_rows = self.q_dim + 2 * self.kv_dim
    assert self.q_dim % 16 == 0 and self.kv_dim % 16 == 0, "q/k/v are packed back to back in whole 16-row tiles"
    self.blk = []
    self.weight_bytes = 0
    lt = dict(linear_types or {})
    names7 = ("attn_q", "attn_k", "attn_v", "attn_output", "ffn_gate", "ffn_up", "ffn_down")
    self.dense_blocks = ggml_type not in (_lib.Q4_0, _lib.Q8_0) or any(lt.get(f"blk.{i}.{n}.weight", ggml_type) != ggml_type
                                                                      for i in range(c.num_blocks) for n in names7)
    if self.dense_blocks:
      assert tp is None and batch == 1 and not c.num_experts, "the dense-weight path serves single-sequence dense models on one GPU"
      def dense16(name, n_out, n_in):       # -> fp16 [n_out, n_in] on the device, whatever the tensor's type
        raw, typ = sd[name], lt.get(name, ggml_type)
        if typ in quant.GGML_QUANT: return quant.dequantize(np.ascontiguousarray(raw).view(np.uint8).reshape(-1), n_out * n_in, typ, np.float16)
        return DeviceBuffer.from_numpy(np.asarray(raw).astype(np.float16).reshape(n_out, n_in))
      def wide(name, n_in):                 # the packed type of a Linear the K-quant GEMV takes, else None
        return quant.WIDE_QUANT.get(lt.get(name, ggml_type)) if n_in % 256 == 0 and n_in <= _lib.WIDE_MAX_IN else None
      def stacked(names, rows, n_in):       # Linears that read the same vector: neighbours of one type become one matrix
        out, at = [], 0
        for typ, run in itertools.groupby(zip(names, rows), key=lambda nr: wide(nr[0], n_in)):
          run = list(run)
          n_out = sum(r for _, r in run)
          buf, off = DeviceBuffer(quant.packed_bytes(typ, n_out, n_in) if typ else 2 * n_out * n_in), 0
          for name, r in run:
            if typ:
              quant.repack(sd[name], r, n_in, typ, out=buf, out_offset=off)
              off += quant.packed_bytes(typ, r, n_in)
            else:
              part = dense16(name, r, n_in)
              check(_lib.load().b200q_memcpy_d2d(buf.ptr + off, part.ptr, part.nbytes, None)); off += part.nbytes
              runtime_sync()
          if out and out[-1].qtype == _lib.Q4_K_WIDE and typ == _lib.Q6_K_WIDE: out[-1].behind = buf, n_out      # one launch for both
          else: out.append(_BlockLinear(typ, n_out, n_in, buf, at))
          at += n_out
        return out
    for i in range(c.num_blocks if self.dense_blocks else 0):
      b = _Block()
      blk = lambda *names: [f"blk.{i}.{n}.weight" for n in names]
      b.qkv = stacked(blk("attn_q", "attn_k", "attn_v"), (self.q_dim, self.kv_dim, self.kv_dim), c.dim)
      b.qkv_bias = DeviceBuffer.from_numpy(np.concatenate([np.asarray(sd[f"blk.{i}.attn_{n}.bias"], dtype=np.float16) for n in "qkv"])) if c.qkv_bias else None
      b.o_w, = stacked(blk("attn_output"), (c.dim,), self.q_dim)
      gate, up = blk("ffn_gate", "ffn_up")
      if wide(gate, c.dim) and wide(gate, c.dim) == wide(up, c.dim):          # interleaved: the SwiGLU product comes out of one launch
        pw = quant.repack(sd[gate], c.hidden_dim, c.dim, wide(gate, c.dim), raw_up=sd[up])
        b.gate_up = [_BlockLinear(pw.qtype, c.hidden_dim, c.dim, pw.buf, 0, swiglu=True)]
      else: b.gate_up = [stacked([n], (c.hidden_dim,), c.dim)[0] for n in (gate, up)]
      b.down_w, = stacked(blk("ffn_down"), (c.dim,), c.hidden_dim)
      b.moe = b.router = None
      b.attn_norm = DeviceBuffer.from_numpy(np.asarray(sd[f"blk.{i}.attn_norm.weight"], dtype=np.float16))
      b.ffn_norm = DeviceBuffer.from_numpy(np.asarray(sd[f"blk.{i}.ffn_norm.weight"], dtype=np.float16))
      kvdt = np.float16 if c.kv_dtype == "float16" else np.float32
      b.k_cache = DeviceBuffer.empty((batch, c.n_kv_heads, c.max_context, c.head_dim), kvdt, zero=True)
      b.v_cache = DeviceBuffer.empty((batch, c.n_kv_heads, c.max_context, c.head_dim), kvdt, zero=True)
      self.blk.append(b)
      self.weight_bytes += sum(w.algorithmic_bytes for w in b.qkv + [b.o_w] + b.gate_up + [b.down_w])
    for i in range(0 if self.dense_blocks else c.num_blocks):
      b = _Block()
      b.qkv = DeviceBuffer(quant.packed_bytes(ggml_type, qkv_rows, c.dim))
      off = 0
      for name, rows in (("attn_q", self.q_dim), ("attn_k", self.kv_dim), ("attn_v", self.kv_dim)):
        quant.repack(sd[f"blk.{i}.{name}.weight"], rows, c.dim, ggml_type, out=b.qkv, out_offset=off)
        off += quant.packed_bytes(ggml_type, rows, c.dim)
      b.qkv_bias = None
      if c.qkv_bias:
        b.qkv_bias = DeviceBuffer.from_numpy(np.concatenate([np.asarray(sd[f"blk.{i}.attn_{n}.bias"], dtype=np.float16) for n in "qkv"]))
      b.attn_output = quant.repack(sd[f"blk.{i}.attn_output.weight"], c.dim, self.q_dim, ggml_type)
      b.moe = b.router = None
      if c.num_experts:
        # routed experts: fp32 (E, out, in) weights quantised to MXFP8 on the device; the router stays a dense Linear (model.py:94-98)
        from . import moe
        if c.expert_gating_func not in moe.GATING: raise ValueError(f"unknown expert gating function {c.expert_gating_func!r}")
        gating = moe.Gating(c.expert_gating_func, c.norm_topk_prob, c.routed_scaling_factor,
                            np.asarray(sd[f"blk.{i}.exp_probs_b.bias"], dtype=np.float32) if c.expert_bias else None)
        b.moe = moe.MxMoE(*(np.asarray(sd[f"blk.{i}.ffn_{n}_exps.weight"], dtype=np.float32) for n in ("gate", "up", "down")), c.num_experts_per_tok, gating)
        r = np.asarray(sd[f"blk.{i}.ffn_gate_inp.weight"])
        b.router = quant.DenseWeight(r, c.num_experts, c.dim, quant.GGML_F16 if r.dtype == np.float16 else quant.GGML_F32)
        b.sh_gate_up = b.sh_down = b.sh_inp = None
        if c.shared_expert_dim:      # the shared expert is an ordinary quantised SwiGLU FFN; its optional gate a [dim] vector
          b.sh_gate_up = quant.repack(sd[f"blk.{i}.ffn_gate_shexp.weight"], c.shared_expert_dim, c.dim, ggml_type, raw_up=sd[f"blk.{i}.ffn_up_shexp.weight"])
          b.sh_down = quant.repack(sd[f"blk.{i}.ffn_down_shexp.weight"], c.dim, c.shared_expert_dim, ggml_type)
          if c.shared_expert_gate and f"blk.{i}.ffn_gate_inp_shexp.weight" in sd:
            gw = np.asarray(sd[f"blk.{i}.ffn_gate_inp_shexp.weight"])
            b.sh_inp = quant.DenseWeight(gw.reshape(1, c.dim), 1, c.dim, quant.GGML_F16 if gw.dtype == np.float16 else quant.GGML_F32)
      else:
        b.gate_up = quant.repack(sd[f"blk.{i}.ffn_gate.weight"], c.hidden_dim, c.dim, ggml_type, raw_up=sd[f"blk.{i}.ffn_up.weight"])
        b.ffn_down = quant.repack(sd[f"blk.{i}.ffn_down.weight"], c.dim, c.hidden_dim, ggml_type)
      b.attn_norm = DeviceBuffer.from_numpy(np.asarray(sd[f"blk.{i}.attn_norm.weight"], dtype=np.float16))
      b.ffn_norm = DeviceBuffer.from_numpy(np.asarray(sd[f"blk.{i}.ffn_norm.weight"], dtype=np.float16))
      kvdt = np.float16 if c.kv_dtype == "float16" else np.float32
      b.k_cache = DeviceBuffer.empty((batch, c.n_kv_heads, c.max_context, c.head_dim), kvdt, zero=True)
      b.v_cache = DeviceBuffer.empty((batch, c.n_kv_heads, c.max_context, c.head_dim), kvdt, zero=True)
      self.blk.append(b)
      nel, nby = quant.GGML_QUANT[ggml_type]
      self.weight_bytes += (qkv_rows * c.dim + c.dim * self.q_dim + (0 if c.num_experts else 3 * c.hidden_dim * c.dim)) // nel * nby
    if self.dense_blocks: self.up_buf = DeviceBuffer.empty((c.hidden_dim,), np.float32, zero=True)
    self.output_type = ggml_type if output_type is None else output_type
    # a Q6_K head (the usual companion of K-quant blocks) runs the fused GEMV too; several sequences at once go through the dense GEMV
    if self.output_type in (_lib.Q4_0, _lib.Q8_0) or (self.output_type == _lib.Q6_K and batch == 1 and c.dim % 256 == 0):
      self.output = quant.repack(sd["output.weight"], c.vocab_size, c.dim, self.output_type)
      self.weight_bytes += c.vocab_size * c.dim // quant.GGML_QUANT[self.output_type][0] * quant.GGML_QUANT[self.output_type][1]
    else:
      self.output = quant.DenseWeight(sd["output.weight"], c.vocab_size, c.dim, self.output_type)
      self.weight_bytes += self.output.algorithmic_bytes
    self.output_norm = DeviceBuffer.from_numpy(np.asarray(sd["output_norm.weight"], dtype=np.float16))
    self.token_embd = DeviceBuffer.from_numpy(np.asarray(sd["token_embd.weight"], dtype=np.float16))
    self.rope = DeviceBuffer.from_numpy(precompute_freqs_cis(c.rope_dim, c.max_context, c.rope_theta))
    # activations of one token (fp32 residual stream, model.py:359)
    self.x = tp.empty_f32(c.dim) if tp is not None else DeviceBuffer.empty((c.dim,), np.float32, zero=True)   # NCCL reduces it in place
    self.qkv = DeviceBuffer.empty((qkv_rows,), np.float32, zero=True)
    self.attn = DeviceBuffer.empty((self.q_dim,), np.float32, zero=True)
    self.act = DeviceBuffer.empty((c.hidden_dim,), np.float32, zero=True)
    if tp is not None: self.logits_part, self.logits = tp.empty_f32(c.vocab_size), tp.empty_f32(vocab_full)
    else: self.logits = self.logits_part = DeviceBuffer.empty((c.vocab_size,), np.float32, zero=True)
    if self.tp_peer and isinstance(self.output, quant.DenseWeight): raise NotImplementedError("sharded models need a Q4_0 / Q8_0 head")
    if self.tp_peer:      # two alternating mailboxes for the row-split linears (O, down), one for the vocabulary slices of the head
      from .tensor_parallel import PeerMailbox
      self.mb_o, self.mb_down = PeerMailbox(tp, tp.size, c.dim), PeerMailbox(tp, tp.size, c.dim)
      self.mb_logits = PeerMailbox(tp, 1, vocab_full)
    self.batch = batch
    assert batch >= 1 and (batch == 1 or tp is None), "batched decode runs on one GPU"
    self.tokens = DeviceBuffer.empty((batch, c.max_context + 1), np.int32, zero=True)     # sequence 0 is the single-sequence state
    self.pos = DeviceBuffer.empty((batch,), np.int32, zero=True)
    self.seq_cache_bytes = c.n_kv_heads * c.max_context * c.head_dim * np.dtype(kvdt).itemsize
    self.attn_scratch = DeviceBuffer(_lib.load().b200q_attn_scratch_bytes(c.n_heads, c.n_kv_heads, c.head_dim, self.n_split), zero=True)
    self._mirror = PinnedBuffer((batch,), np.int32)      # the sampled tokens as the arg-max kernel leaves them for the host
    self._head_queued = False                            # a step with the head may not have written its token there yet
    self.argmax_scratch = DeviceBuffer(batch * _lib.load().b200q_argmax_scratch_bytes(), zero=True)
    # Quantised activation hand-over between consecutive kernels (needs whole 128-wide groups everywhere).  Each edge of
    # the chain can be switched on its own: attn_o (attention -> output projection), o_gateup, gateup_down, down_qkv.
    can = c.head_dim == 128 and c.dim % 128 == 0 and c.hidden_dim % 128 == 0 and self.q_dim % 128 == 0 and not self.dense_blocks
    all_edges = ("attn_o", "o_gateup", "gateup_down", "down_qkv")
    if handover is None: edges = DEFAULT_HANDOVER
    elif isinstance(handover, str): edges = tuple(e for e in handover.split(",") if e)
    else: edges = all_edges if handover else ()
    assert all(e in all_edges for e in edges), f"unknown hand-over edge in {edges}"
    if tp is not None: edges = tuple(e for e in edges if e in ("attn_o", "gateup_down"))   # records of all-reduced vectors would hold partial sums
    self.edges = frozenset(edges) if can else frozenset()
    self.handover = bool(self.edges)
    xqb = _lib.load().b200q_xq_bytes
    if "down_qkv" in self.edges: self.xq_a, self.ss_a = DeviceBuffer(xqb(c.dim), zero=True), DeviceBuffer.empty((c.dim // 32,), np.float32, zero=True)
    if "o_gateup" in self.edges: self.xq_b, self.ss_b = DeviceBuffer(xqb(c.dim), zero=True), DeviceBuffer.empty((c.dim // 32,), np.float32, zero=True)
    if "attn_o" in self.edges: self.xq_attn = DeviceBuffer(xqb(self.q_dim), zero=True)
    if "gateup_down" in self.edges: self.xq_act = DeviceBuffer(xqb(c.hidden_dim), zero=True)
    # staging row of the producing GEMVs (32-bit words, all-ones = empty; the kernels leave it empty): row tiles stay dealt to CTAs
    # one by one.  Without it a producing CTA takes runs of 2 / 4 consecutive tiles, which leaves the grid unevenly loaded.
    self.ho_stage = None
    if self.edges and STAGED_HANDOVER:
      self.ho_stage = {n: DeviceBuffer.from_numpy(np.concatenate([np.full(n, 0xFFFFFFFF, np.uint32), np.zeros(n // 32, np.uint32)]))
                       for n in {c.dim, c.hidden_dim}}      # [n_out words | n_out / 32 counters] per producing width
    self._graphs = {}
    self._cached_tokens: list = []
    self.prefill_rows = prefill_rows if (tp is None and not self.dense_blocks and c.hidden_dim % 8 == 0 and c.head_dim in (16, 32, 64, 128)) else 0
    self.prefill_chunk, self._pf, self._batch_logits, self._rows_ws = max(1, prefill_chunk), None, None, None
    self._rows_args, self._moe_blocks = None, {}
    self._seq_attn_scratch = self._last_rows = None
    self.is_moe, self._host_pos, self._rows_warm = c.num_experts > 0, 0, False
    if self.is_moe:
      assert tp is None and c.head_dim in (16, 32, 64, 128), "the mixture-of-experts model runs on the row path of one GPU"
      self.prefill_rows = 1
    self.launches_per_step = 3 + (sum(3 + len(b.qkv) + len(b.gate_up) + (not b.gate_up[0].swiglu) for b in self.blk) if self.dense_blocks else 5 * c.num_blocks)
    # ---- the whole-step kernel: a device table of the blocks' pointers, its workspace, and the two argument blocks (with / without head)
    self._step_args = None
    if engine not in (None, "step", "chain"): raise ValueError(f"unknown engine {engine!r}")
    if engine == "step" and tp is None and not self.is_moe and not self.dense_blocks and batch == 1 and not isinstance(self.output, quant.DenseWeight) and self.output_type == ggml_type:
      lib = _lib.load()
      table = (_lib.DecodeLayer * c.num_blocks)(*[_lib.DecodeLayer(b.qkv.ptr, b.qkv_bias.ptr if b.qkv_bias else None, b.attn_output.buf.ptr, b.gate_up.buf.ptr,
                                                                  b.ffn_down.buf.ptr, b.attn_norm.ptr, b.ffn_norm.ptr, b.k_cache.ptr, b.v_cache.ptr) for b in self.blk])
      self._layer_table = DeviceBuffer.from_numpy(np.frombuffer(bytes(table), dtype=np.uint8))
      def mk(with_head):
        return _lib.DecodeStepArgs(self._layer_table.ptr, c.num_blocks, ggml_type, c.dim, c.hidden_dim, c.n_heads, c.n_kv_heads, c.head_dim, c.rope_dim,
                                   c.max_context, c.vocab_size, c.vocab_size, F16 if c.kv_dtype == "float16" else F32, c.norm_eps, self.token_embd.ptr,
                                   self.output_norm.ptr, self.output.buf.ptr, self.rope.ptr, self.tokens.ptr, self.pos.ptr, self.x.ptr, self.qkv.ptr,
                                   self.attn.ptr, self.act.ptr, self.logits.ptr, None, 0, with_head, 0, None)
      probe = mk(1)
      rc = lib.b200q_decode_step_supported(ctypes.byref(probe))
      if rc == 0:
        self._step_ws = DeviceBuffer(lib.b200q_decode_step_workspace_bytes(ctypes.byref(probe)), zero=True)
        self._step_args = {}
        for wh in (0, 1):
          a = mk(wh)
          a.workspace, a.workspace_bytes = self._step_ws.ptr, self._step_ws.nbytes
          self._step_args[bool(wh)] = a
        self.launches_per_step = 1
      elif engine == "step":
        check(rc)
    elif engine == "step":
      raise ValueError("the whole-step kernel takes dense single-GPU models whose head has the block Linears' quant type")
    self.engine = "step" if self._step_args else "chain"

  # ---- one token through the network (launch sequence; captured into a graph) ----
  def _enqueue_step(self, with_head: bool, attention: bool = True, tail: bool = True, last_block: bool = False) -> None:
    """last_block: the last block and what follows it, on the row in `x` (a prompt's last row, behind the pass over the prompt)."""
    c, lib, s, fl = self.config, _lib.load(), self.stream.ptr, self.flags
    kvdt = F16 if c.kv_dtype == "float16" else F32
    grid = lambda name: self.gemv_max_ctas.get(name, self.gemv_max_ctas.get("*", 0))
    kw = dict(flags=fl, stream=s)
    tp = self.tp
    # A launch that follows an NCCL call is fully stream-ordered: the programmatic-launch attribute right behind the
    # event waits NCCL leaves in the stream was measured to let the kernel start before the reduced vector is there.
    peer = self.tp_peer
    kw_after_coll = dict(kw, flags=0) if (tp is not None and not peer) else kw
    rkw = dict(residual=self.x, residual_scale=1.0 / tp.size) if tp is not None else dict(residual=self.x)   # row-split shards add residual / n_ranks
    # peer-memory collectives: the row-split GEMV stores its partial row into every rank's mailbox; the reducer adds the residual once
    rkw_o = dict(peers=self.mb_o.targets, peer_rank=tp.rank) if peer else rkw
    rkw_d = dict(peers=self.mb_down.targets, peer_rank=tp.rank) if peer else rkw
    vocab_full = self.full_config.vocab_size
    e, nss = self.edges - {"down_qkv"} if last_block else self.edges, c.dim // 32
    qkv_rows = self.q_dim + 2 * self.kv_dim
    # the four hand-over edges: kwargs of the consuming (xq_in...) and of the producing (xq_out...) launch
    in_a = dict(xq_in=self.xq_a, ss_in=self.ss_a, ss_count=nss) if "down_qkv" in e else {}
    in_b = dict(xq_in=self.xq_b, ss_in=self.ss_b, ss_count=nss) if "o_gateup" in e else {}
    in_attn = dict(xq_in=self.xq_attn) if "attn_o" in e else {}
    in_act = dict(xq_in=self.xq_act) if "gateup_down" in e else {}
    if (attention or tail) and not last_block:
      ho = "down_qkv" in e
      check(lib.b200q_embed(self.token_embd.ptr, self.tokens.ptr, self.pos.ptr, self.x.ptr, c.dim, vocab_full, c.max_context,
                            self.xq_a.ptr if ho else None, self.blk[0].attn_norm.ptr if ho else None, self.ss_a.ptr if ho else None, fl, s))
    for i, b in enumerate(self.blk if self.dense_blocks else ()):
      # K-quant and fp16 blocks: the same step with the row between the launches in fp32 (norm / bias / residual / SwiGLU fused)
      for w in b.qkv: w.run(self.x, self.qkv, norm_weight=b.attn_norm, norm_eps=c.norm_eps, bias=b.qkv_bias, flags=fl, stream=s)
      a = _lib.AttnArgs(self.qkv.ptr, b.k_cache.ptr, b.v_cache.ptr, kvdt, self.rope.ptr, self.pos.ptr, self.attn.ptr, self.attn_scratch.ptr,
                        c.n_heads, c.n_kv_heads, c.head_dim, c.rope_dim, c.max_context, self.n_split, fl, None)
      check(lib.b200q_attn_decode(ctypes.byref(a), s))
      b.o_w.run(self.attn, self.x, residual=self.x, flags=fl, stream=s)
      for w, y in zip(b.gate_up, (self.act, self.up_buf)): w.run(self.x, y, norm_weight=b.ffn_norm, norm_eps=c.norm_eps, flags=fl, stream=s)
      if not b.gate_up[0].swiglu: check(lib.b200q_silu_mul(self.act.ptr, self.up_buf.ptr, self.act.ptr, c.hidden_dim, fl, s))
      b.down_w.run(self.act, self.x, residual=self.x, flags=fl, stream=s)
    for i, b in () if self.dense_blocks else list(enumerate(self.blk))[-1 if last_block else 0:]:
      nxt_norm = self.blk[i + 1].attn_norm if i + 1 < len(self.blk) else self.output_norm
      st = (lambda n: dict(xq_out_stage=self.ho_stage[n])) if self.ho_stage is not None else (lambda n: {})
      out_b = dict(xq_out=self.xq_b, xq_out_norm_weight=b.ffn_norm, ss_out=self.ss_b, **st(c.dim)) if "o_gateup" in e else {}
      out_act = dict(xq_out=self.xq_act, **st(c.hidden_dim)) if "gateup_down" in e else {}
      out_a = dict(xq_out=self.xq_a, xq_out_norm_weight=nxt_norm, ss_out=self.ss_a, **st(c.dim)) if "down_qkv" in e else {}
      quant.gemv(b.qkv.ptr, self.qtype, qkv_rows, c.dim, None if in_a else self.x, self.qkv, norm_weight=b.attn_norm, norm_eps=c.norm_eps,
                 bias=b.qkv_bias, max_ctas=grid("qkv"), **in_a, **(kw_after_coll if i > 0 else kw))      # (last_block: a graph's first node, or behind a copy: fully ordered)
      if attention:
        a = _lib.AttnArgs(self.qkv.ptr, b.k_cache.ptr, b.v_cache.ptr, kvdt, self.rope.ptr, self.pos.ptr, self.attn.ptr, self.attn_scratch.ptr,
                          c.n_heads, c.n_kv_heads, c.head_dim, c.rope_dim, c.max_context, self.n_split, fl,
                          self.xq_attn.ptr if "attn_o" in e else None)
        check(lib.b200q_attn_decode(ctypes.byref(a), s))
      quant.gemv(b.attn_output.buf.ptr, self.qtype, c.dim, self.q_dim, None if in_attn else self.attn, None if peer else self.x, **rkw_o,
                 **in_attn, **out_b, max_ctas=grid("o"), **kw)
      if peer: self.mb_o.reduce(self.x, residual=self.x, flags=fl, stream=s)
      elif tp is not None: tp.all_reduce(self.x)
      quant.gemv(b.gate_up.buf.ptr, self.qtype, c.hidden_dim, c.dim, None if in_b else self.x, None if out_act else self.act,
                 norm_weight=b.ffn_norm, norm_eps=c.norm_eps, epilogue=EPI_SILU_MUL, max_ctas=grid("gate_up"), **in_b, **out_act, **kw_after_coll)
      quant.gemv(b.ffn_down.buf.ptr, self.qtype, c.dim, c.hidden_dim, None if in_act else self.act, None if peer else self.x, **rkw_d,
                 **in_act, **out_a, max_ctas=grid("down"), **kw)
      if peer: self.mb_down.reduce(self.x, residual=self.x, flags=fl, stream=s)
      elif tp is not None: tp.all_reduce(self.x)
    if with_head:
      if isinstance(self.output, quant.DenseWeight):
        quant.gemv_dense(self.output.buf, self.output.dtype, c.vocab_size, c.dim, self.x, self.logits_part, norm_weight=self.output_norm,
                         norm_eps=c.norm_eps, flags=kw_after_coll["flags"], stream=s)
      else:
        in_h = {} if self.output_type == _lib.Q6_K else in_a       # the Q6_K kernel quantises the row itself
        quant.gemv(self.output.buf.ptr, self.output_type, c.vocab_size, c.dim, None if in_h else self.x, self.logits_part,
                   norm_weight=self.output_norm, norm_eps=c.norm_eps, max_ctas=grid("head"), **in_h, **kw_after_coll,
                   **(dict(peers=self.mb_logits.targets, peer_rank=tp.rank) if peer else {}))
      if peer: self.mb_logits.reduce(self.logits, flags=fl, stream=s)          # every rank's vocabulary slice, handed over
      elif tp is not None: tp.all_gather(self.logits, self.logits_part)
      if tail: check(lib.b200q_argmax_advance_seqs(self.logits.ptr, vocab_full, self.tokens.ptr, 0, self.pos.ptr, c.max_context, self.argmax_scratch.ptr, 1,
                                                   self._mirror.ptr, 0 if (tp is not None and not peer) else fl, s))
    elif tail:
      check(lib.b200q_advance(self.pos.ptr, c.max_context, 0 if (tp is not None and not peer) else fl, s))

  # ---- several prompt tokens at once: tcgen05 dequant GEMMs + batched causal attention ----
  def _rows_workspace_bytes(self, T: int) -> int:
    """The GEMMs' workspace for chunks of up to T rows (partial sums grow with a tile's rows, and fewer rows may be in larger tiles: 640 are 3 x 224, 512
    2 x 256)."""
    c, qkv_rows = self.config, self.q_dim + 2 * self.kv_dim
    if self.is_moe: return quant.qgemm_unsplit_workspace_bytes(T, max(c.dim, self.q_dim, c.shared_expert_dim))
    shapes = ((qkv_rows, c.dim), (c.dim, self.q_dim), (2 * c.hidden_dim, c.dim), (c.dim, c.hidden_dim))
    return max(quant.qgemm_workspace_bytes(m, i, o) for o, i in shapes for m in {T, *range(16, T, 16)})      # tiles are whole 16 rows

  def _prefill_buffers(self):
    if self._pf is None:
      c, T = self.config, self.prefill_chunk
      self._pf = dict(x=DeviceBuffer.empty((T, c.dim), np.float32), xn=DeviceBuffer.empty((T, c.dim), np.float32),
                      qkv=DeviceBuffer.empty((T, self.q_dim + 2 * self.kv_dim), np.float32), q16=DeviceBuffer.empty((T, self.q_dim), np.float32),
                      att=DeviceBuffer.empty((T, self.q_dim), np.float32),
                      act=DeviceBuffer.empty((T, max(c.hidden_dim, c.shared_expert_dim, 1)), np.float32),
                      # Activation tiles and partial sums of the GEMMs.  Mixture-of-experts models take sums that are not split: their expert
                      # choice and E4M3 codes turn a last-bit difference into a visible one, and a token's result must not depend on how
                      # many rows it was computed with.
                      ws=DeviceBuffer(self._rows_workspace_bytes(T)) if self.pipelined_gemm else None)
      if self.is_moe:
        self._pf.update(xb=DeviceBuffer.empty((T, c.dim), np.uint16), logits=DeviceBuffer.empty((T, c.num_experts), np.float32))
        if c.shared_expert_dim: self._pf.update(sh=DeviceBuffer.empty((T, c.dim), np.float32), shg=DeviceBuffer.empty((T,), np.float32))
    return self._pf

  def prefill(self, start_pos: int, n: int, sync: bool = True, seq: int = 0) -> None:
    """Run tokens[start_pos : start_pos + n] (already on the device) through every block and fill the KV cache; no logits.
    The forward of tinygrad/llm/model.py:358-362 for T = n, in chunks: per block rmsnorm -> QKV GEMM -> RoPE + cache append +
    causal attention -> O GEMM (+residual) -> rmsnorm -> gate/up GEMM with SwiGLU epilogue -> down GEMM (+residual).
    Activations stay fp32 between the kernels; the GEMMs split them into fp16 hi + lo halves for the tensor core."""
    c, lib, s, f = self.config, _lib.load(), self.stream.ptr, self._prefill_buffers()
    native = self._native_rows()
    for p0 in range(start_pos, start_pos + n, self.prefill_chunk) if native else ():
      check(lib.b200q_prompt_rows(native, seq, 1, p0, min(self.prefill_chunk, start_pos + n - p0), s))
    for p0 in () if native else range(start_pos, start_pos + n, self.prefill_chunk):
      T = min(self.prefill_chunk, start_pos + n - p0)
      if (blocks := self._native_moe(T)) is not None:
        check(lib.b200q_moe_rows(self._rows_args[1], blocks, seq, p0, None, T, s))
        continue
      check(lib.b200q_embed_rows(self.token_embd.ptr, self.tokens.ptr + 4 * (seq * (c.max_context + 1) + p0), 1, None, T, c.dim,
                                 self.full_config.vocab_size, f["x"].ptr, s))
      for b in self.blk: self._enqueue_rows_block(b, T, f, p0, seq)
    if sync:
      self.stream.synchronize()
      self.pos.copy_from(np.array([start_pos + n], dtype=np.int32), offset=4 * seq)
      self._host_pos = start_pos + n

  def _prompt_rows(self, native, start_pos: int, n: int, seq: int = 0) -> int:
    """Prompt tokens of one sequence, of which only the cache rows are wanted and what goes into the last block: the rows of the last pass, whose number is returned, are
    in the row buffer then."""
    for p0 in range(start_pos, start_pos + n, self.prefill_chunk):
      rows = min(self.prefill_chunk, start_pos + n - p0)
      check(_lib.load().b200q_prompt_rows_kv(native, seq, 1, p0, rows, self.stream.ptr))
    return rows

  def _captured(self, key: tuple, enqueue) -> Graph:
    """The graph of a launch sequence.  key: what `enqueue` enqueues, in full: one model serves single prompts and batches, with sequences of their own."""
    g = self._graphs.get(key)
    if g is None:
      g = Graph(self.stream)
      with g: enqueue()
      self._graphs[key] = g
    return g

  def _last_block(self, kind: str, enqueue, step) -> None:
    """Replays the last block, the head and the arg-max on rows that a prompt pass has left (captured on first use).  The steps that will follow, `step`, are captured here
    too: the device still has the prompt to do.  kind: "one" sequence or a "batch"."""
    self._head_queued = True
    if not self.use_graph: return enqueue()
    self._captured((kind, "last block"), enqueue).launch()
    self._captured((kind, "step", True), step)

  def _last_goes_along(self, n: int) -> bool:
    """Whether the token behind n prompt tokens goes through the blocks with them (a last pass of one row would cost what a step does)."""
    return self.engine == "chain" and n % self.prefill_chunk != 0 and self._native_rows() is not None

  def _prompt_to_last_block(self, native, start_pos: int, n: int):
    """tokens[start_pos : start_pos + n] as rows up to the last block -> what takes the last one of them through that and samples the token behind it."""
    self.pos.copy_from(np.array([start_pos + n - 1], dtype=np.int32), stream=self.stream)
    rows, size = self._prompt_rows(native, start_pos, n), 4 * self.config.dim
    check(_lib.load().b200q_memcpy_d2d(self.x.ptr, self._pf["x"].ptr + (rows - 1) * size, size, self.stream.ptr))
    self._host_pos = start_pos + n - 1
    def finish():
      self._check_room()
      self._host_pos += 1
      self._last_block("one", lambda: self._enqueue_step(True, last_block=True), lambda: self._enqueue_step(True))
    return finish

  def _enqueue_rows_block(self, b, T: int, f: dict, p0, seq: int) -> None:
    """One block for T rows in f["x"]: positions p0 .. of sequence `seq`, or (p0 None) one row at the position kept on the device."""
    c, lib, s = self.config, _lib.load(), self.stream.ptr
    kvdt = F16 if c.kv_dtype == "float16" else F32
    qkv_rows = self.q_dim + 2 * self.kv_dim
    def normed(norm):       # the GEMM with a workspace applies the RMSNorm while it splits its activations
      if f["ws"] is not None and quant.PIPELINED_GEMM and not self.is_moe: return f["x"], {"norm_weight": norm, "norm_eps": c.norm_eps}
      check(lib.b200q_rmsnorm_rows(f["x"].ptr, norm.ptr, c.norm_eps, T, c.dim, f["xn"].ptr, F32, s))
      return f["xn"], {}
    xin, kw = normed(b.attn_norm)
    quant.qgemm(b.qkv.ptr, self.qtype, qkv_rows, c.dim, xin, f["qkv"], T, x_dtype=F32, y_dtype=F32, bias=b.qkv_bias, stream=s, workspace=f["ws"], unsplit=self.is_moe, **kw)
    if p0 is None:       # position on the device
      check(lib.b200q_attn_decode_batch(f["qkv"].ptr, b.k_cache.ptr, b.v_cache.ptr, kvdt, self.rope.ptr, 0, self.pos.ptr, T, c.n_heads, c.n_kv_heads, c.head_dim,
                                        c.rope_dim, c.max_context, f["q16"].ptr, f["att"].ptr, F32, s))
    else:
      check(lib.b200q_attn_prefill(f["qkv"].ptr, b.k_cache.ptr + seq * self.seq_cache_bytes, b.v_cache.ptr + seq * self.seq_cache_bytes, kvdt,
                                   self.rope.ptr, p0, T, c.n_heads, c.n_kv_heads, c.head_dim,
                                   c.rope_dim, c.max_context, f["q16"].ptr, f["att"].ptr, F32, s))
    quant.qgemm(b.attn_output.buf.ptr, self.qtype, c.dim, self.q_dim, f["att"], f["x"], T, x_dtype=F32, y_dtype=F32, residual=f["x"], stream=s, workspace=f["ws"], unsplit=self.is_moe)
    if b.moe is not None:
      check(lib.b200q_rmsnorm_rows(f["x"].ptr, b.ffn_norm.ptr, c.norm_eps, T, c.dim, f["xn"].ptr, F32, s))
      # router on the fp32 normed rows, experts on their bf16 rounding (the activation dtype of the MXFP8 path); bf16 result + residual
      quant.gemv_dense(b.router.buf, b.router.dtype, c.num_experts, c.dim, f["xn"], f["logits"], m=T, stream=s)
      check(lib.b200q_rmsnorm_rows(f["x"].ptr, b.ffn_norm.ptr, c.norm_eps, T, c.dim, f["xb"].ptr, _lib.BF16, s))
      y = b.moe(f["xb"], f["logits"], T, stream=s)
      if b.sh_gate_up is not None:      # shared expert on the fp32 normed rows (model.py:131-134), added before x moves
        quant.qgemm(b.sh_gate_up.buf.ptr, self.qtype, 2 * c.shared_expert_dim, c.dim, f["xn"], f["act"], T, x_dtype=F32, y_dtype=F32,
                    epilogue=EPI_SILU_MUL, stream=s, workspace=f["ws"], unsplit=self.is_moe)
        quant.qgemm(b.sh_down.buf.ptr, self.qtype, c.dim, c.shared_expert_dim, f["act"], f["sh"], T, x_dtype=F32, y_dtype=F32, stream=s, workspace=f["ws"], unsplit=self.is_moe)
        if b.sh_inp is not None: quant.gemv_dense(b.sh_inp.buf, b.sh_inp.dtype, 1, c.dim, f["xn"], f["shg"], m=T, stream=s)
        check(lib.b200q_add_rows_gated(f["x"].ptr, f["sh"].ptr, f["shg"].ptr if b.sh_inp is not None else None, T, c.dim, s))
      check(lib.b200q_add_rows_bf16(f["x"].ptr, y.ptr, T * c.dim, s))
      return
    xin, kw = normed(b.ffn_norm)
    quant.qgemm(b.gate_up.buf.ptr, self.qtype, 2 * c.hidden_dim, c.dim, xin, f["act"], T, x_dtype=F32, y_dtype=F32, epilogue=EPI_SILU_MUL,
                stream=s, workspace=f["ws"], unsplit=self.is_moe, **kw)
    quant.qgemm(b.ffn_down.buf.ptr, self.qtype, c.dim, c.hidden_dim, f["act"], f["x"], T, x_dtype=F32, y_dtype=F32, residual=f["x"], stream=s, workspace=f["ws"], unsplit=self.is_moe)

  def _native_rows(self):
    """The argument block of b200q_prompt_rows (every launch of a chunk from one call), or None where the model does not run on it."""
    if self.is_moe or self.dense_blocks or self.tp is not None or not self.pipelined_gemm or not quant.PIPELINED_GEMM: return None
    return self._row_arguments()

  def _native_moe(self, T: int):
    """The expert FFNs' argument blocks of b200q_moe_rows for T rows (self._rows_args is its first argument then), or None where it does not run."""
    if not self.is_moe or not self.pipelined_gemm or not quant.PIPELINED_GEMM: return None
    if T not in self._moe_blocks:
      c, f = self.config, self._prefill_buffers()
      self._row_arguments()
      args = [b.moe.native_args(T) for b in self.blk]
      ptr = lambda o: o.ptr if o is not None else None
      def block(b, a):
        sh = b.sh_gate_up is not None
        return _lib.MoeBlock(ctypes.pointer(a), b.router.buf.ptr, b.sh_gate_up.buf.ptr if sh else None, b.sh_down.buf.ptr if sh else None,
                             b.sh_inp.buf.ptr if sh and b.sh_inp is not None else None, b.router.dtype, b.sh_inp.dtype if sh and b.sh_inp is not None else 0,
                             c.shared_expert_dim if sh else 0, f["xn"].ptr, f["xb"].ptr, f["logits"].ptr, f["act"].ptr, ptr(f.get("sh")), ptr(f.get("shg")))
      self._moe_blocks[T] = None if any(a is None for a in args) else (_lib.MoeBlock * len(args))(*[block(b, a) for b, a in zip(self.blk, args)])
    return self._moe_blocks[T]

  def _row_arguments(self):
    if self._rows_args is None:
      c, f = self.config, self._prefill_buffers()
      self._layer_host = (_lib.DecodeLayer * c.num_blocks)(*[_lib.DecodeLayer(b.qkv.ptr, b.qkv_bias.ptr if b.qkv_bias else None, b.attn_output.buf.ptr,
                                                                             *((None, None) if self.is_moe else (b.gate_up.buf.ptr, b.ffn_down.buf.ptr)),
                                                                             b.attn_norm.ptr, b.ffn_norm.ptr, b.k_cache.ptr, b.v_cache.ptr) for b in self.blk])
      a = _lib.RowsArgs(self._layer_host, c.num_blocks, self.qtype, c.dim, c.hidden_dim, c.n_heads, c.n_kv_heads, c.head_dim, c.rope_dim, c.max_context,
                        self.full_config.vocab_size, F16 if c.kv_dtype == "float16" else F32, self.prefill_chunk, c.norm_eps, self.token_embd.ptr, self.rope.ptr,
                        self.tokens.ptr, f["x"].ptr, f["qkv"].ptr, f["q16"].ptr, f["att"].ptr, f["act"].ptr, f["ws"].ptr, f["ws"].nbytes)
      self._rows_args = (a, ctypes.byref(a))
    return self._rows_args[1]

  # ---- several sequences in lock-step ----
  def decode_batch_step(self) -> None:
    """One new token for each of the `batch` sequences, all at the same position: every Linear is one GEMM over the batch rows
    (weights streamed once per step), attention runs per sequence on its own cache, the arg-max per sequence.  Captured once into a
    CUDA graph (positions and tokens live on the device) and replayed."""
    self._check_room()
    self._head_queued = True
    if not self.use_graph: return self._enqueue_batch_step()
    self._prefill_buffers()
    self._batch_buffers()                              # (a capture allocates nothing)
    self._captured(("batch", "step", True), lambda: self._enqueue_batch_step(count=False)).launch()
    self._host_pos += 1

  def _batch_buffers(self):
    """What a step of the batch needs besides the row buffers (allocated on first use) -> (quantised head, few-row kernel, attention in one launch)."""
    c, lib, B = self.config, _lib.load(), self.batch
    qkv_rows, head_q = self.q_dim + 2 * self.kv_dim, not isinstance(self.output, quant.DenseWeight)
    few = B <= quant.FEW_ROW_MAX and quant.FEW_ROW_FUSED     # 8 rows per pass on the int8 tensor cores at the one-row GEMV's arithmetic; else one pass of the GEMM
    if self._rows_ws is None:
      shapes = [(qkv_rows, c.dim), (c.dim, self.q_dim), (2 * c.hidden_dim, c.dim), (c.dim, c.hidden_dim)] + ([(c.vocab_size, c.dim)] if head_q else [])
      need = quant.qgemv_rows_workspace_bytes if few else (lambda m, o, i: quant.qgemm_workspace_bytes(m, i, o))
      self._rows_ws = DeviceBuffer(max(need(B, o, i) for o, i in shapes))
    # head_dim 64 or 128: one launch of the cluster kernel, a cluster per (KV head, sequence)
    seq_attn = (SEQ_ATTENTION or c.head_dim in (64, 128)) and c.n_heads // c.n_kv_heads <= 8 and c.head_dim % 8 == 0 and c.head_dim <= 128
    if seq_attn and self._seq_attn_scratch is None:
      stride = lib.b200q_attn_seq_scratch_stride(c.n_heads, c.n_kv_heads, c.head_dim, self.n_split)
      self._seq_attn_scratch = DeviceBuffer(B * stride, zero=True)
    if self._batch_logits is None: self._batch_logits = DeviceBuffer.empty((B, c.vocab_size), np.float32)
    return head_q, few, seq_attn

  def _enqueue_batch_step(self, count: bool = True, last_block: bool = False) -> None:
    c, lib, s, f, B = self.config, _lib.load(), self.stream.ptr, self._prefill_buffers(), self.batch
    assert B <= self.prefill_chunk and not self.is_moe
    kvdt = F16 if c.kv_dtype == "float16" else F32
    qkv_rows = self.q_dim + 2 * self.kv_dim
    head_q, few, seq_attn = self._batch_buffers()
    if few:
      def gemm(w, qt, n_out, n_in, x, y, **kw): quant.qgemv_rows(w, qt, n_out, n_in, x, y, B, self._rows_ws, x_dtype=F32, y_dtype=F32, stream=s, **kw)
    else:
      def gemm(w, qt, n_out, n_in, x, y, **kw): quant.qgemm(w, qt, n_out, n_in, x, y, B, x_dtype=F32, y_dtype=F32, stream=s, workspace=self._rows_ws, **kw)
    # the position comes from the device (sequence 0's counter; all sequences move together), so the launch sequence can be replayed as a graph
    if not last_block: check(lib.b200q_embed_rows(self.token_embd.ptr, self.tokens.ptr, c.max_context + 1, self.pos.ptr, B, c.dim, c.vocab_size, f["x"].ptr, s))
    fold = few or quant.PIPELINED_GEMM     # both apply the RMSNorm in their pre-pass: no norm launches
    def normed(norm):
      if fold: return f["x"], {"norm_weight": norm, "norm_eps": c.norm_eps}
      check(lib.b200q_rmsnorm_rows(f["x"].ptr, norm.ptr, c.norm_eps, B, c.dim, f["xn"].ptr, F32, s))
      return f["xn"], {}
    for b in self.blk[-1:] if last_block else self.blk:
      xin, kw = normed(b.attn_norm)
      gemm(b.qkv.ptr, self.qtype, qkv_rows, c.dim, xin, f["qkv"], bias=b.qkv_bias, **kw)
      if seq_attn:     # the one-token kernel over (KV head, slice, sequence): RoPE, cache append and attention in one launch
        a = _lib.AttnArgs(f["qkv"].ptr, b.k_cache.ptr, b.v_cache.ptr, kvdt, self.rope.ptr, self.pos.ptr, f["att"].ptr, self._seq_attn_scratch.ptr,
                          c.n_heads, c.n_kv_heads, c.head_dim, c.rope_dim, c.max_context, self.n_split, _lib.FLAG_PDL, None)
        check(lib.b200q_attn_decode_seqs(ctypes.byref(a), B, s))
      else:
        check(lib.b200q_attn_decode_batch(f["qkv"].ptr, b.k_cache.ptr, b.v_cache.ptr, kvdt, self.rope.ptr, 0, self.pos.ptr, B, c.n_heads, c.n_kv_heads,
                                          c.head_dim, c.rope_dim, c.max_context, f["q16"].ptr, f["att"].ptr, F32, s))
      gemm(b.attn_output.buf.ptr, self.qtype, c.dim, self.q_dim, f["att"], f["x"], residual=f["x"])
      xin, kw = normed(b.ffn_norm)
      gemm(b.gate_up.buf.ptr, self.qtype, 2 * c.hidden_dim, c.dim, xin, f["act"], epilogue=EPI_SILU_MUL, **kw)
      gemm(b.ffn_down.buf.ptr, self.qtype, c.dim, c.hidden_dim, f["act"], f["x"], residual=f["x"])
    if head_q and fold:
      gemm(self.output.buf.ptr, self.output_type, c.vocab_size, c.dim, f["x"], self._batch_logits, norm_weight=self.output_norm, norm_eps=c.norm_eps)
    else:
      check(lib.b200q_rmsnorm_rows(f["x"].ptr, self.output_norm.ptr, c.norm_eps, B, c.dim, f["xn"].ptr, F32, s))
      if head_q: gemm(self.output.buf.ptr, self.output_type, c.vocab_size, c.dim, f["xn"], self._batch_logits)
      else: quant.gemv_dense(self.output.buf, self.output.dtype, c.vocab_size, c.dim, f["xn"], self._batch_logits, m=B, stream=s)
    check(lib.b200q_argmax_advance_seqs(self._batch_logits.ptr, c.vocab_size, self.tokens.ptr, c.max_context + 1, self.pos.ptr, c.max_context,
                                        self.argmax_scratch.ptr, B, self._mirror.ptr, FLAG_PDL, s))
    if count: self._host_pos += 1

  def _prefill_batch(self, n: int) -> None:
    """tokens[:n] of every sequence: as many whole sequences per pass as fit prefill_chunk rows (the weights are streamed once per pass)."""
    native, per = self._native_rows(), self.prefill_chunk // n
    if native is None or per < 2:
      for i in range(self.batch):
        if native is None: self.prefill(0, n, seq=i)
        else: self._prompt_rows(native, 0, n, seq=i)
    else:
      for i in range(0, self.batch, per):
        check(_lib.load().b200q_prompt_rows_kv(native, i, min(per, self.batch - i), 0, n, self.stream.ptr))
    self.stream.synchronize()

  def _prompt_tokens(self, native, per: int, n: int) -> None:
    """The first n tokens of every sequence, `per` sequences in a pass, and the tokens behind them: the passes' last rows are gathered for the last block."""
    B, f, lib, s, size = self.batch, self._pf, _lib.load(), self.stream.ptr, 4 * self.config.dim
    self._batch_buffers()      # (a capture allocates nothing)
    self.pos.copy_from(np.full((B,), n - 1, dtype=np.int32), stream=self.stream)
    if self._last_rows is None: self._last_rows = DeviceBuffer.empty((B, self.config.dim), np.float32), DeviceBuffer.empty((B,), np.int32)
    last, at = self._last_rows
    at.copy_from(np.arange(n - 1, n * per, n, dtype=np.int32), stream=self.stream)
    for i in range(0, B, per):
      seqs = min(per, B - i)
      check(lib.b200q_prompt_rows_kv(native, i, seqs, 0, n, s))
      check(lib.b200q_permute_rows(f["x"].ptr, at.ptr, seqs, size, last.ptr + i * size, 1, s))
    check(lib.b200q_memcpy_d2d(f["x"].ptr, last.ptr, B * size, s))
    self._host_pos = n
    self._last_block("batch", lambda: self._enqueue_batch_step(count=False, last_block=True), lambda: self._enqueue_batch_step(count=False))

  def generate_batch(self, prompts: list):
    """Greedy generation for `batch` prompts of equal length; yields the list of the sequences' next tokens per step."""
    c, B = self.config, self.batch
    assert len(prompts) == B and len({len(p) for p in prompts}) == 1 and len(prompts[0]) >= 1
    L = len(prompts[0])
    assert L >= c.max_context or B <= self.prefill_chunk and not self.is_moe, "a step takes a row of the row buffers per sequence"
    self._cached_tokens = []      # sequence 0's rows are the ones that `generate` reuses
    self.stream.synchronize()
    tok = np.zeros((B, c.max_context + 1), np.int32)
    for i, p in enumerate(prompts): tok[i, :L] = p
    self.tokens.copy_from(tok)
    step, n = self.decode_batch_step, L
    native, per = self._native_rows() if 1 < L < c.max_context else None, min(self.prefill_chunk // L, B)
    # several sequences in a pass, and no more passes than without their last tokens
    if native is not None and per >= 2 and -(-B // per) == -(-B // min(self.prefill_chunk // (L - 1), B)): step = lambda: self._prompt_tokens(native, per, L)
    else:
      if L > 1: self._prefill_batch(L - 1)
      self.pos.copy_from(np.full((B,), L - 1, dtype=np.int32))
      self._host_pos = L - 1
    while n < c.max_context:
      yield self._sampled(step, B)
      step, n = self.decode_batch_step, n + 1

  def _step_rows(self, with_head: bool) -> None:
    """One token through the row path (mixture-of-experts models: their FFN is not part of the fused one-token chain).  Positions come
    from the device, so the launches are captured once (behind a first step that allocates) and replayed as a CUDA graph."""
    if not self.use_graph: self._enqueue_step_rows(with_head)
    elif not self._rows_warm:
      self._enqueue_step_rows(with_head)
      self._rows_warm = True
    else: self._captured(("rows", "step", bool(with_head)), lambda: self._enqueue_step_rows(with_head)).launch()
    self._host_pos += 1

  def _enqueue_step_rows(self, with_head: bool) -> None:
    c, lib, s, f = self.config, _lib.load(), self.stream.ptr, self._prefill_buffers()
    fl = 0
    if (blocks := self._native_moe(1)) is not None:
      check(lib.b200q_moe_rows(self._rows_args[1], blocks, 0, 0, self.pos.ptr, 1, s))
      fl = self.flags
    else:
      check(lib.b200q_embed_rows(self.token_embd.ptr, self.tokens.ptr, 1, self.pos.ptr, 1, c.dim, self.full_config.vocab_size, f["x"].ptr, s))
      for b in self.blk: self._enqueue_rows_block(b, 1, f, None, 0)
    if with_head:
      x_last = self._pf["x"]
      if isinstance(self.output, quant.DenseWeight):
        quant.gemv_dense(self.output.buf, self.output.dtype, c.vocab_size, c.dim, x_last, self.logits, norm_weight=self.output_norm, norm_eps=c.norm_eps,
                         flags=fl, stream=s)
      else:
        quant.gemv(self.output.buf.ptr, self.output_type, c.vocab_size, c.dim, x_last, self.logits, norm_weight=self.output_norm, norm_eps=c.norm_eps,
                   flags=fl, stream=s)
      check(lib.b200q_argmax_advance_seqs(self.logits.ptr, c.vocab_size, self.tokens.ptr, 0, self.pos.ptr, c.max_context, self.argmax_scratch.ptr, 1,
                                          self._mirror.ptr, fl, s))
    else:
      check(lib.b200q_advance(self.pos.ptr, c.max_context, 0, s))

  def _check_room(self) -> None:
    if self._host_pos >= self.max_context:
      raise RuntimeError(f"context full: position {self._host_pos} has no KV-cache row (max_context {self.max_context})")

  def gemv_launches(self) -> list:
    """(n_out rows streamed, n_in) of every GEMV launch of one step with the head, in launch order."""
    c = self.config
    per_block = [(self.q_dim + 2 * self.kv_dim, c.dim), (c.dim, self.q_dim), (2 * c.hidden_dim, c.dim), (c.dim, c.hidden_dim)]
    return per_block * c.num_blocks + [(c.vocab_size, c.dim)]

  def gemv_only_graph(self) -> Graph:
    """The GEMV launches of one step alone, in order, for timing the weight stream by itself
    (it overwrites the activation buffers: use it after the real steps)."""
    g = Graph(self.stream)
    with g: self._enqueue_step(with_head=True, attention=False, tail=False)
    return g

  def step(self, with_head: bool = True) -> None:
    """Advance by one token on the device: reads tokens[pos]; with the head, writes tokens[pos+1].
    The host mirrors the device position and refuses a step that has no KV-cache row left (nothing is launched then)."""
    self._check_room()
    if with_head: self._head_queued = True
    if self.is_moe: return self._step_rows(with_head)
    self._host_pos += 1
    if self._step_args: return check(_lib.load().b200q_decode_step(ctypes.byref(self._step_args[bool(with_head)]), self.stream.ptr))
    if not self.use_graph: return self._enqueue_step(with_head)
    self._captured(("one", "step", bool(with_head)), lambda: self._enqueue_step(with_head)).launch()

  # ---- host-visible state ----
  def set_state(self, tokens: list, pos: int) -> None:
    self.stream.synchronize()
    if tokens: self.tokens.copy_from(np.asarray(tokens, dtype=np.int32))
    self.pos.copy_from(np.array([pos], dtype=np.int32))
    self._host_pos = pos

  def _put_tokens(self, tokens: list, pos: int) -> None:
    """set_state for a prompt whose first `pos` tokens are in the cache: only the others are copied, in stream order (no waiting)."""
    self.tokens.copy_from(np.asarray(tokens[pos:], dtype=np.int32), stream=self.stream, offset=4 * pos)
    self.pos.copy_from(np.array([pos], dtype=np.int32), stream=self.stream)
    self._host_pos = pos

  def read_token(self, index: int) -> int:
    self.stream.synchronize()
    return int(self.tokens.numpy((1,), np.int32, offset=4 * index)[0])

  def _sampled(self, step, n: int = 1) -> list:
    """Run `step` and wait for the `n` tokens it samples: the arg-max kernel also writes them to page-locked memory, which is polled.  Steps that a caller has
    queued must have left theirs first: one that comes after the words are cleared would pass for this step's."""
    if self._head_queued: self.stream.synchronize()
    m = self._mirror.array[:n]
    m[:] = -1
    step()
    check(_lib.load().b200q_wait_words(self._mirror.ptr, n, -1, self.stream.ptr))
    self._head_queued = False
    return m.tolist()

  def read_logits(self) -> np.ndarray:
    self.stream.synchronize()
    return self.logits.numpy()

  def get_start_pos(self, tokens: list) -> int:
    """How much of the KV cache the new prompt can reuse (model.py:456-462)."""
    n, old = max(0, min(len(tokens) - 1, len(self._cached_tokens))), self._cached_tokens
    if tokens[:n] == old[:n]: return n
    lo = 0                                    # tokens[:lo] agree, tokens[:n] do not
    while n - lo > 1:
      mid = (lo + n) // 2
      if tokens[lo:mid] == old[lo:mid]: lo = mid
      else: n = mid
    return lo

  def generate(self, tokens: list, temperature: float = 0.0):
    """Greedy generation (model.py:464-484 at temperature 0).  Yields one token id at a time; a prompt is consumed in chunks (`prefill_rows`), its last token with them
    up to the last block, or one position per step."""
    if temperature != 0.0: raise NotImplementedError("only greedy decoding (temperature 0) is implemented")
    tokens = list(tokens)
    start_pos = self.get_start_pos(tokens)
    del self._cached_tokens[start_pos:]      # the rows behind them are about to be written, whether or not a token comes of it
    self._put_tokens(tokens, start_pos)
    n_pre, step = len(tokens) - 1 - start_pos, self.step
    if self.prefill_rows and n_pre >= self.prefill_rows:
      if len(tokens) < self.max_context and self._last_goes_along(n_pre): step = self._prompt_to_last_block(self._native_rows(), start_pos, n_pre + 1)
      else: self.prefill(start_pos, n_pre)
    else:
      for _ in range(n_pre): self.step(with_head=False)
    while len(tokens) < self.max_context:
      if self._step_args:
        self.step(with_head=True)
        tok = self.read_token(len(tokens))
      else: tok, step = self._sampled(step)[0], self.step
      tokens.append(tok)
      self._cached_tokens = tokens[:-1]
      yield tok
