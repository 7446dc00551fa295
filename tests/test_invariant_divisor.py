"""The two-instruction division by the grid spacings (csrc/host_common.h,
invariant_divisor): on the CPU against the division itself, and on the GPU
through the kernels that use it, on grids whose spacings are no powers of two,
bit for bit against the oracle (whose C code divides)."""
import pathlib
import shutil
import subprocess

import numpy as np
import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]


def test_pairs_divide_like_the_division(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = tmp_path / "divisor_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    str(ROOT / "simplenavierstokessolver_gb300" / "csrc"),
                    str(ROOT / "tests" / "c" / "divisor_check.cpp"), "-o", str(exe)], check=True)
    total, none, wrong, naive = map(int, subprocess.run([str(exe)], check=True, capture_output=True,
                                                        text=True).stdout.split())
    assert wrong == 0
    assert none <= total // 500  # such divisors keep their division
    assert naive > 100000  # the check tells a wrong rounding


@pytest.mark.gpu
@pytest.mark.parametrize("scheme", [(0, 0), (1, 0), (0, 1), (1, 1)], ids=["exp", "imp_x", "imp_y", "imp_xy"])
@pytest.mark.parametrize("nx,ny,ly,stretch", [(2, 2, 1.0, 1e9), (33, 8, 0.3, 1e9), (70, 32, 2.0, 3), (100, 64, 1.7, 1e9),
                                              (640, 512, 3.0, 5)])
def test_calls_divide_bitwise(scheme, nx, ny, ly, stretch):
    """every call of two substages from fields with exact zeros, subnormals and
    values on both sides of the pair's range (2^-723, 2^877)"""
    from oracle.bindings import Config, OracleCase
    from simplenavierstokessolver_gb300 import Case

    cfg = Config(nx, ny, ly=ly, Ra=2e5, Pr=0.8, stretch=stretch)
    rng = np.random.default_rng(21)
    su, sc = (ny + 2, nx + 1), (ny + 2, nx + 2)

    def field(shape, scale, edge):
        a = scale * rng.uniform(-1, 1, shape)
        pick = rng.uniform(size=shape)
        for k, v in enumerate(edge):
            a[(pick >= 0.01 * k) & (pick < 0.01 * (k + 1))] = v
        return a

    small = (0.0, 5e-320, -3e-218, 2e-218, 1e-217)
    state = (field(su, 0.2, small), field(sc, 0.2, small), field(sc, 0.05, small + (1e200, -3e263)),
             field(sc, 0.5, small))
    o = OracleCase(cfg)
    o.set_state(*state)
    o.call("update_boundaries")
    with Case(nx, ny, ly=ly, stretch=stretch, Ra=cfg.Ra, Pr=cfg.Pr) as c:
        c.set_state(*state)
        for x in (c, o):
            x.set_dt(1e-3, *scheme)
        for rk in range(2):
            c.temperature_compute_force()
            c.temperature_update_temp(rk)
            o.call("temperature_force_and_update", rk)
            for name in ("fluid_update_velocity", "fluid_compute_potential", "fluid_correct_velocity",
                         "fluid_update_pressure"):
                getattr(c, name)(rk)
                o.call(name, rk)
                got, want = c.get_state(), o.get_state()
                for k in ("ux", "uy", "p", "psi", "temp"):
                    if k == "psi" and name == "fluid_update_velocity":
                        continue
                    assert np.array_equal(got[k], want[k], equal_nan=True), (name, k, rk)
