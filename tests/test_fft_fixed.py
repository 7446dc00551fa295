"""The real DFTs of the tolerance-held forms in 64-bit block fixed point
(csrc/fft_fixed.cuh). On the CPU tests/c/fft_fixed_check.cpp runs the kernels'
arithmetic beside the same passes in double, both against a long double DFT.
On the GPU one Poisson solve of the parallel form against the exact form's
(another DFT and another line solver, both FP64)."""
import pathlib
import shutil
import subprocess

import numpy as np
import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]


@pytest.mark.parametrize("args,lengths", [([], 10), (["2"], 5)], ids=["radix8", "radix2"])
def test_error_is_below_the_fp64_transforms(tmp_path, args, lengths):
    """forward and inverse, jtot 16 to 8192 (256 with radix 2), noise, smooth,
    single-mode, delta, wide-range and mean-dominated columns of sizes from
    2^-960 to 2^100"""
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = tmp_path / "fft_fixed_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    str(ROOT / "simplenavierstokessolver_gb300" / "csrc"),
                    str(ROOT / "tests" / "c" / "fft_fixed_check.cpp"), "-o", str(exe)], check=True)
    rows = [line.split() for line in
            subprocess.run([str(exe), *args], check=True, capture_output=True, text=True).stdout.splitlines()]
    assert len(rows) == lengths * 6
    for jtot, kind, fwd, fwd64, inv, inv64 in rows:
        assert float(fwd) <= float(fwd64) and float(inv) <= float(inv64), (jtot, kind, fwd, fwd64, inv, inv64)


def _solve(nx, ny, parallel, ux, uy, dt):
    from simplenavierstokessolver_gb300 import Case

    zero = np.zeros((ny + 2, nx + 2))
    with Case(nx, ny, ly=2.0, Ra=1e7, Pr=1.0) as c:
        if parallel:
            c.set_form(True)
        c.set_state(ux, uy, zero, zero)
        c.set_dt(dt, 0, 0)
        c.fluid_compute_potential(1)
        return c.get_state()["psi"][1:-1, 1:-1]


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(64, 16), (64, 32), (64, 64), (128, 128), (64, 256), (64, 512), (1024, 512),
                                   (64, 1024), (512, 2048), (64, 4096), (128, 8192)])
@pytest.mark.parametrize("size", [1.0, 1e-300], ids=["1", "1e-300"])
def test_poisson_solve_matches_the_exact_form(nx, ny, size):
    """radix 8 and 4 with a last pass of 8, 4 and 2, one to sixteen columns per
    block; the two solvers differ by round-off times the condition of the mean
    mode (nx^2), as in the other Poisson tests: 1e-10"""
    rng = np.random.default_rng(8)
    ux, uy = size * rng.uniform(-1, 1, (ny + 2, nx + 1)), size * rng.uniform(-1, 1, (ny + 2, nx + 2))
    want, got = (_solve(nx, ny, p, ux, uy, 1e-3) for p in (False, True))
    err = np.linalg.norm((got - want) / size) / np.linalg.norm(want / size)
    assert err < 1e-10, err


@pytest.mark.gpu
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_a_non_finite_column_makes_the_potential_non_finite(value):
    nx, ny = 64, 64
    ux, uy = np.zeros((ny + 2, nx + 1)), np.ones((ny + 2, nx + 2))
    uy[10, 20] = value
    assert not np.isfinite(_solve(nx, ny, True, ux, uy, 1e-3)).any()


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,stretch", [(64, 8, 1e9), (64, 16, 1e9), (96, 32, 1e9), (64, 64, 3), (64, 2048, 1e9),
                                           (64, 8192, 1e9)])
@pytest.mark.parametrize("compensated", [False, True], ids=["fp32", "compensated"])
def test_batched_steps_match_the_plain_path(nx, ny, stretch, compensated):
    """the batched form's column groups of 1 to 16, its FP64 stages (jtot 8) and
    its divergences as pairs and as doubles (grids of no powers of two): three
    steps of a fixed dt against the exact form from the same start, within the
    forms' stated errors (1e-5 and 1e-10)"""
    from simplenavierstokessolver_gb300 import Case
    from simplenavierstokessolver_gb300.batch import Batch, Desc, initial_temperature

    d = Desc(nx, ny, ly=2.0, stretch=stretch, Ra=1e6, Pr=1.0, seed=3, fixed_dt=1e-4, compensated=compensated)
    with Batch(1 << 30, max_cases=2) as b:
        s = b.add(d)
        b.step(3)
        got = b.state(s)
    z = np.zeros((ny + 2, nx + 2))
    with Case(nx, ny, ly=2.0, stretch=stretch, Ra=1e6, Pr=1.0) as c:
        c.set_state(np.zeros((ny + 2, nx + 1)), z, z, initial_temperature(d))
        c.set_dt(1e-4, 0, 0)
        for _ in range(3):
            c.integrate()
        want = c.get_state()
    for k in ("ux", "uy", "temp"):
        w = want[k][1:-1, 1:-1]
        err = np.linalg.norm(got[k][1:-1, 1:-1] - w) / np.linalg.norm(w)
        assert err < (1e-10 if compensated else 1e-5), (k, err)


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,stretch", [(64, 8, 1e9), (96, 32, 3), (256, 128, 1e9)])
@pytest.mark.parametrize("given", [False, True], ids=["seeded", "given"])
def test_admitted_temperature_is_the_hosts(nx, ny, stretch, given):
    """the device's seeded (or split) initial field against the host's, as the
    pair of floats that holds it"""
    from simplenavierstokessolver_gb300.batch import Batch, Desc, initial_temperature

    d = Desc(nx, ny, ly=2.0, stretch=stretch, Ra=1e6, Pr=1.0, seed=11)
    t = initial_temperature(d)
    with Batch(256 << 20, max_cases=2) as b:
        got = b.state(b.add(d, t if given else None))["temp"]
    hi = t.astype(np.float32)
    assert np.array_equal(got, hi.astype(np.float64) + (t - hi).astype(np.float32))
