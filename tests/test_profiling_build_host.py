"""The build with time stamps (-DB200Q_GEMV_PROF) measures the launches of the plain one: nothing is launched in a branch of its own, where cluster sizes and attributes could be
missing (a kernel made for a cluster of four that runs in one of one addresses shared memory that does not exist)."""
import pathlib
import re
import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "tinygrad_b200" / "csrc"


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cu*") if "B200Q_GEMV_PROF" in p.read_text()))
def test_time_stamps_add_no_launches(name):
  parts = re.findall(r"^#ifdef B200Q_GEMV_PROF$(.*?)^#(?:else|endif)", (CSRC / name).read_text(), re.S | re.M)
  assert parts
  for part in parts: assert not re.search(r"launch_k|cudaLaunch|<<<", part), part
