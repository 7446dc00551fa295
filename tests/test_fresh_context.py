"""What a kernel has to be granted on each device (csrc/smem_grant.h, the shared
memory above 48 KB): on the CPU against a fake runtime with two devices, and on
the GPU after the process's CUDA context was reset between two
cases, which then have to give the same fields (in a child process, whose own
context it is; every object of the library is closed before)."""
import pathlib
import shutil
import subprocess
import sys

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]

CHILD = """
import ctypes, sys
import numpy as np
from simplenavierstokessolver_gb300 import Case

nx, ny, form = int(sys.argv[1]), int(sys.argv[2]), sys.argv[3]

def fields():
    rng = np.random.default_rng(7)
    su, sc = (ny + 2, nx + 1), (ny + 2, nx + 2)
    state = [0.1 * rng.uniform(-1, 1, su), 0.1 * rng.uniform(-1, 1, sc), np.zeros(sc), rng.uniform(-0.5, 0.5, sc)]
    with Case(nx, ny, ly=1.0, Ra=1e6, Pr=1.0, costs=[1e6, 1e6, 1e6, 1.0]) as c:
        c.set_form(form == "parallel")
        c.set_fused(form == "fused")
        c.set_state(*state)
        c.run(1)
        return c.get_state()

a = fields()
rt = ctypes.CDLL("libcudart.so.13")
assert rt.cudaDeviceReset() == 0
b = fields()
for k in ("ux", "uy", "p", "temp"):
    assert np.array_equal(a[k], b[k]), k
print("same")
"""


def test_every_device_is_asked(tmp_path):
    cxx, cuda = shutil.which("g++"), pathlib.Path("/usr/local/cuda/include")
    if cxx is None or not cuda.exists():
        pytest.skip("no g++ or CUDA headers")
    exe = tmp_path / "smem_grant_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", str(ROOT / "simplenavierstokessolver_gb300" / "csrc"),
                    "-I", str(cuda), str(ROOT / "tests" / "c" / "smem_grant_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["0:204800", "1:204800"] * 2


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["fused", "separate", "parallel"])
def test_second_context_runs_like_the_first(form):
    """long lines along x, implicit in both directions"""
    r = subprocess.run([sys.executable, "-c", CHILD, "8192", "16", form], capture_output=True, text=True, timeout=300,
                       cwd=ROOT)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stdout + r.stderr
