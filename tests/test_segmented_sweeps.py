"""The exact form's Crank-Nicolson solves by segments (csrc/plain_fp64.cu,
k_solve_seg): bit for bit the serial sweeps of the oracle (src/linalg.c:9-108),
from steps whose sweeps forget their start within a few rows to steps that
take the serial kernel, and on lines that a spike, still far above the field's
size after the rows that a sweep needs to forget it, makes fail the check."""
import numpy as np
import pytest

from oracle.bindings import Config, OracleCase

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spike", [False, True], ids=["plain", "spike"])
@pytest.mark.parametrize("dt", [1e-6, 2e-3, 0.1, 20.0])
@pytest.mark.parametrize("nx,ny,stretch", [(31, 32, 1e9), (32, 64, 1e9), (65, 32, 1e9), (130, 128, 3), (260, 512, 1e9),
                                           (1030, 64, 1e9), (64, 2048, 1e9)])
def test_implicit_updates_are_the_serial_sweeps(nx, ny, stretch, dt, spike):
    from simplenavierstokessolver_gb300 import Case

    cfg = Config(nx, ny, ly=1.0, Ra=1e6, Pr=0.7, stretch=stretch)
    rng = np.random.default_rng(13)
    su, sc = (ny + 2, nx + 1), (ny + 2, nx + 2)
    state = [0.1 * rng.uniform(-1, 1, su), 0.1 * rng.uniform(-1, 1, sc), 0.1 * rng.uniform(-1, 1, sc),
             rng.uniform(-0.5, 0.5, sc)]
    if spike:
        state[3][ny // 2, nx // 3] = 1e200
    o = OracleCase(cfg)
    o.set_state(*state)
    o.call("update_boundaries")
    with Case(nx, ny, ly=1.0, stretch=stretch, Ra=1e6, Pr=0.7) as c:
        c.set_state(*state)
        for scheme in ((1, 0), (0, 1), (1, 1)):
            for x in (c, o):
                x.set_dt(dt, *scheme)
            c.temperature_compute_force()
            c.temperature_update_temp(1)
            o.call("temperature_force_and_update", 1)
            c.fluid_update_velocity(1)
            o.call("fluid_update_velocity", 1)
            got, want = c.get_state(), o.get_state()
            for k in ("ux", "uy", "temp"):
                assert np.array_equal(got[k][1:-1], want[k][1:-1], equal_nan=True), (scheme, k)
