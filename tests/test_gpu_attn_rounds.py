"""Decode attention in clusters of 8 CTAs where a CTA has 2 to 4 chunks of 64 positions, which it takes two at a time: last rounds of one and of two chunks, of one position and
full, the new position first, in the middle and last in its chunk."""
import numpy as np
import pytest
import test_gpu_attn_cluster as cluster
from gpu_util import need_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kv", [np.float16, np.float32])
@pytest.mark.parametrize("hd,rope_dim", [(64, 64), (128, 96)])
@pytest.mark.parametrize("pos", [1022, 1024, 1151, 1216, 1279, 1535, 1536, 1663, 1730, 1791, 2046])
def test_rounds_of_chunks(pos, hd, rope_dim, kv):
  need_gpu()
  cluster.test_cluster_attention(30, 15, hd, rope_dim, pos, kv)
