"""The fixed-point DFT's passes of radix 4 (csrc/fft_fixed.cuh; four values per
thread, which mid-size grids take): tests/c/fft_radix4_check.cpp runs the
kernels' arithmetic beside an FP64 transform, both against a long double DFT."""
import pathlib
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]


def test_error_is_below_the_fp64_transform(tmp_path):
    """forward and inverse, jtot 16 to 4096; noise, smooth, single-mode, delta,
    wide-range and mean-dominated columns of sizes from 2^-960 to 2^100"""
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = tmp_path / "fft_radix4_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    str(ROOT / "simplenavierstokessolver_gb300" / "csrc"),
                    str(ROOT / "tests" / "c" / "fft_radix4_check.cpp"), "-o", str(exe)], check=True)
    rows = [line.split() for line in
            subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()]
    assert len(rows) == 9 * 6
    for jtot, kind, fwd, fwd64, inv, inv64 in rows:
        assert float(fwd) <= float(fwd64) and float(inv) <= float(inv64), (jtot, kind, fwd, fwd64, inv, inv64)
