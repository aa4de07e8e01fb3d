"""The order of tensor-core additions, on the CPU: two tcgen05.mma are promised to run in the order of issue only if they have the same accumulator and the same shape.
Products that are added to one accumulator without a commit between them therefore share one instruction descriptor in each kernel that issues them."""
import pathlib
import re
import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "tinygrad_b200" / "csrc"


def issued(text):
  """The (accumulator, instruction descriptor) operands of every mma( / mma_ts( call: mma(d, a, b, hi, idesc, acc)."""
  calls = re.findall(r"(?<![\w.])mma(?:_ts)?\(((?:[^()]|\([^()]*\))*)\);", text)
  out = []
  for c in calls:
    args = re.split(r",(?![^()]*\))", c)
    if len(args) == 6: out.append((args[0].strip(), args[4].strip()))
  return out


@pytest.mark.parametrize("name", ["qgemm_tmem.cuh", "qgemm_stream.cu"])
def test_products_of_one_accumulator_have_one_shape(name):
  text = (CSRC / name).read_text()
  got = issued(text)
  assert len(got) >= 3                                  # wh xh, wh xl, wl xh
  shapes = {i for _, i in got}
  assert len(shapes) == 1, f"instructions of several shapes: {got}"
  assert re.search(rf"\b{shapes.pop()} = make_idesc\(128, nt\)", text)
