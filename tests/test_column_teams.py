"""The fused Poisson launch of the exact form with its worker blocks split into
teams (csrc/plain_fp64.cu, kFusedTeams): bit for bit the oracle, at one, two and
four teams, with fewer columns than teams and with a remainder in the last round;
and with DFT stages of 1 to 64 butterflies (csrc/fft_dev.cuh, butterfly4)."""
import numpy as np
import pytest

from oracle.bindings import Config, OracleCase

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,stretch", [(32, 1024, 1e9), (8, 2048, 1e9), (130, 2048, 3), (512, 2048, 1e9),
                                           (601, 2048, 1e9), (1025, 2048, 1e9), (33, 4096, 1e9), (24, 8192, 3),
                                           (16, 16384, 1e9), (8, 8, 1e9), (9, 16, 3),
                                           (16, 32, 1e9), (33, 64, 3), (64, 128, 1e9), (31, 256, 1e9), (40, 512, 3)])
def test_teams_give_the_oracles_step(nx, ny, stretch):
    from simplenavierstokessolver_gb300 import Case

    costs = (1.0, 1e6, 1e6, 1e6)
    cfg = Config(nx, ny, ly=2.0, Ra=1e7, Pr=1.0, stretch=stretch)
    rng = np.random.default_rng(5)
    su, sc = (ny + 2, nx + 1), (ny + 2, nx + 2)
    state = [0.1 * rng.uniform(-1, 1, su), 0.1 * rng.uniform(-1, 1, sc), 0.1 * rng.uniform(-1, 1, sc),
             rng.uniform(-0.5, 0.5, sc)]
    o = OracleCase(cfg, threads=4)
    o.set_costs(costs)
    o.set_state(*state)
    o.call("update_boundaries")
    with Case(nx, ny, ly=2.0, stretch=stretch, Ra=1e7, Pr=1.0, costs=costs) as c:
        c.set_state(*state)
        c.run(1)
        o.run(1)
        got, want = c.get_state(), o.get_state()
        for k in ("ux", "uy", "p", "psi", "temp"):
            assert np.array_equal(got[k][1:-1], want[k][1:-1]), k
