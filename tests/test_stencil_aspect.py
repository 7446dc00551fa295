"""The integer advective and diffusive terms (csrc/stencil_fixed.cuh) on cells
that are not square: tests/c/stencil_aspect_check.cpp runs the kernels'
arithmetic beside the FP64 expressions, both against long double, at cell
aspects dy / dx from 1/512 to 512, for the four schemes, with ux and uy of one
size and a thousand times apart, and fields that vary along one direction."""
import pathlib
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
ASPECTS = ["0.001953125", "0.015625", "0.03125", "0.125", "0.25", "0.75", "1", "1.5", "4", "8", "32", "64", "512"]


def test_error_is_below_the_fp64_expressions_on_any_cell(tmp_path):
    """Where the FP64 expression is the exact value rounded once (diffusion along
    one direction, spacings that are powers of two) nothing can be below it: the
    integers are off by the roundings of two coefficients and two products, 2^-59
    each, before their rounding. Hence the 2^-57."""
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = tmp_path / "stencil_aspect_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    str(ROOT / "simplenavierstokessolver_gb300" / "csrc"),
                    str(ROOT / "tests" / "c" / "stencil_aspect_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), *ASPECTS], check=True, capture_output=True, text=True).stdout
    rows = [line.split() for line in out.splitlines()]
    assert len(rows) == len(ASPECTS) * 2 * 6 * (3 + 3 * 6)
    for *which, fixed, fp64 in rows:
        assert float(fixed) <= float(fp64) + 2.0**-57, (which, fixed, fp64)
