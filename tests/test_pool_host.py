"""The result pool's rules on a made-up device (pool_host.cpp): no block is handed out again before the device has been waited for, and the waits and locks
of one device leave the others alone."""
import pathlib, shutil, subprocess
import pytest
from tinygrad_b200 import build

HERE = pathlib.Path(__file__).resolve().parent


def test_pool_on_a_made_up_device(tmp_path):
  cxx = shutil.which("g++")
  if not cxx: pytest.skip("no host C++ compiler")
  nvcc = pathlib.Path(build.nvcc_path()).resolve()
  cuda = nvcc.parent.parent
  subprocess.run([str(nvcc), *build.NVCC_FLAGS[:2], "-std=c++17", "-c", "-o", str(tmp_path / "pool.o"), str(build.CSRC / "pool.cu")], check=True)
  subprocess.run([cxx, "-std=c++17", f"-I{cuda}/include", str(HERE / "pool_host.cpp"), str(tmp_path / "pool.o"), "-o", str(tmp_path / "pool_host"), f"-L{cuda}/lib64",
                  "-lcudart", "-lpthread", f"-Wl,-rpath,{cuda}/lib64"], check=True)
  r = subprocess.run([str(tmp_path / "pool_host")], capture_output=True, text=True, timeout=60)
  assert r.returncode == 0, r.stdout + r.stderr
