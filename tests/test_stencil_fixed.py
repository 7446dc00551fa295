"""The advective and diffusive terms of the parallel form in 64-bit integers
(csrc/stencil_fixed.cuh). On the CPU tests/c/stencil_fixed_check.cpp runs the
kernels' arithmetic beside the FP64 expressions, both against long double. On
the GPU the velocity and temperature updates against the oracle."""
import pathlib
import shutil
import subprocess

import numpy as np
import pytest

from oracle.bindings import Config, OracleCase

ROOT = pathlib.Path(__file__).resolve().parents[1]


def test_error_is_below_the_fp64_expressions(tmp_path):
    """grids of 64 to 8192 columns, equal and nearly equal spacings, walls;
    smooth, noise and wide-range fields; advection-diffusion of ux, uy, T and
    the diffusion of T alone"""
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = tmp_path / "stencil_fixed_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    str(ROOT / "simplenavierstokessolver_gb300" / "csrc"),
                    str(ROOT / "tests" / "c" / "stencil_fixed_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), "64", "8192"], check=True, capture_output=True, text=True).stdout
    rows = [line.split() for line in out.splitlines()]
    assert len(rows) == 2 * 8 * 4 * 4
    for *which, fixed, fp64 in rows:
        assert float(fixed) <= float(fp64), (which, fixed, fp64)


@pytest.mark.gpu
@pytest.mark.parametrize("field", ["noise", "rest", "negative_zero", "huge", "tiny"])
@pytest.mark.parametrize("nx,ny", [(64, 8), (64, 128), (128, 256), (1152, 32), (2048, 16)])
@pytest.mark.parametrize("scheme", [(0, 0), (1, 0), (0, 1), (1, 1)], ids=["exp", "imp_x", "imp_y", "imp_imp"])
def test_updates_match_the_oracle(nx, ny, scheme, field):
    """one thread's rows from 1 to 8, columns at both walls and a block's edge,
    spacings equal to the bit and (1152) not;
    fields at rest (also of negative zeros) and cells whose values lie outside
    the integers' range (1e70, 1e-70), which take FP64. Source terms: each side
    is within a few round-offs of the sum of its terms' magnitudes, which for
    noise is the size of the result: 16 * 2^-53 relative to the rows' norm."""
    from simplenavierstokessolver_gb300 import Case

    cfg = Config(nx, ny, ly=1.0, Ra=1e6, Pr=0.7)
    rng = np.random.default_rng(3)
    su, sc = (ny + 2, nx + 1), (ny + 2, nx + 2)
    scale = 1e-70 if field == "tiny" else 1.0
    state = [scale * 0.1 * rng.uniform(-1, 1, su), scale * 0.1 * rng.uniform(-1, 1, sc),
             0.1 * rng.uniform(-1, 1, sc), rng.uniform(-0.5, 0.5, sc)]
    if field == "rest":
        state[0][:], state[1][:] = 0.0, 0.0
    if field == "negative_zero":
        state[0][:], state[1][:] = -0.0, -0.0
    if field == "huge":
        for a in (state[0], state[1], state[3]):
            a[ny // 2, nx // 3] = 1e70
    src = {"srcuxa": rng.uniform(-1, 1, (ny, nx - 1)), "srcuya": rng.uniform(-1, 1, (ny, nx)),
           "srctempa": rng.uniform(-1, 1, (ny, nx))}
    o = OracleCase(cfg)
    o.set_state(*state)
    o.set_sources(src["srcuxa"], src["srcuya"], src["srctempa"])
    o.call("update_boundaries")
    with Case(nx, ny, ly=1.0, Ra=1e6, Pr=0.7) as c:
        c.set_form(True)
        c.set_state(*state, sources=src)
        for x in (c, o):
            x.set_dt(1e-4, *scheme)
        c.temperature_compute_force()
        c.temperature_update_temp(1)
        o.call("temperature_force_and_update", 1)
        c.fluid_update_velocity(1)
        o.call("fluid_update_velocity", 1)
        got, want = c.get_sources(), o.get_sources()
        for k in want:
            for g, w in zip(got[k], want[k]):
                # a row's huge cells and the others apart
                for part in (np.abs(w) > 1e30, np.abs(w) <= 1e30):
                    d, n = np.linalg.norm((g - w)[part]), np.linalg.norm(w[part])
                    assert d <= 16 * 2.0**-53 * n, (k, d, n)
