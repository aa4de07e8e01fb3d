"""The many-row GEMM's workspace sizes, on the CPU: what the size functions promise holds the kernel's activation tiles at every row count."""
import numpy as np
import pytest
from tinygrad_b200 import _lib, build, quant
from tinygrad_b200.model import Transformer, TransformerConfig


@pytest.fixture(scope="module")
def lib():
  build.build_lib()
  return _lib.load()


def tile_rows(m):
  """Equal tiles of at most 256 rows, each a whole number of 16."""
  tiles = -(-m // 256)
  return tiles * (-(-(-(-m // tiles)) // 16) * 16)


def test_the_promised_size_holds_the_tiles(lib):
  n_in, last = 96, 0                                    # one group of 128 columns, 4 bytes each
  for m in range(1, 9001):
    size = lib.b200q_qgemm_workspace_bytes(m, n_in)
    assert size >= tile_rows(m) * 128 * 4 and size >= last, m
    assert lib.b200q_qgemm_workspace_bytes_for(m, 4096, n_in) > size
    # one byte less is refused, without asking for a device
    assert lib.b200q_qgemm_ws(_lib.Q4_0, 16, 16, _lib.F32, None, None, 0, 16, _lib.F32, m, 16, n_in, 16, size - 1, None) == -6, m
    last = size


@pytest.mark.parametrize("chunk,experts", [(640, 0), (640, 8), (512, 0), (1100, 0)])
def test_a_model_has_room_for_every_chunk(lib, chunk, experts):
  m = Transformer.__new__(Transformer)
  m.config = TransformerConfig(num_blocks=1, dim=1024, hidden_dim=2816, n_heads=16, n_kv_heads=4, norm_eps=1e-5, vocab_size=1000, head_dim=64, rope_theta=1e4, rope_dim=64)
  m.is_moe, m.q_dim, m.kv_dim = bool(experts), 1024, 256
  room = m._rows_workspace_bytes(chunk)
  for rows in range(1, chunk + 1):
    if experts: assert room >= quant.qgemm_unsplit_workspace_bytes(rows, 1024)
    else: assert room >= max(quant.qgemm_workspace_bytes(rows, i, o) for o, i in ((1536, 1024), (1024, 1024), (5632, 1024), (1024, 2816))), rows
