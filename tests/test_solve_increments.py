"""The implicit step's last solves add the fields' increments as they write them
(csrc/plain_fp64.cu, k_solve_seg and the serial sweeps; csrc/plain_parallel.cu,
k_par_cn and k_par_cn_cols): the exact form's step against the oracle's, bit for
bit, also on lines that fail the segments' check (a spike far above the field)
and with sweeps that take the serial kernels; the parallel form's against the
exact form's."""
import numpy as np
import pytest

from oracle.bindings import Config, OracleCase

pytestmark = pytest.mark.gpu
# the cost of (explicit, implicit x, implicit y, both): each makes its scheme win
COSTS = {"imp_x": (1e6, 1.0, 1e6, 1e6), "imp_y": (1e6, 1e6, 1.0, 1e6), "imp_imp": (1e6, 1e6, 1e6, 1.0)}
FIELDS = ("ux", "uy", "p", "temp")


def _state(nx, ny):
    rng = np.random.default_rng(23)
    su, sc = (ny + 2, nx + 1), (ny + 2, nx + 2)
    return [0.1 * rng.uniform(-1, 1, su), 0.1 * rng.uniform(-1, 1, sc), 0.1 * rng.uniform(-1, 1, sc),
            rng.uniform(-0.5, 0.5, sc)]


@pytest.mark.parametrize("spike", [False, True], ids=["plain", "spike"])
@pytest.mark.parametrize("scheme", sorted(COSTS))
@pytest.mark.parametrize("nx,ny,Ra,stretch", [(31, 32, 1e6, 1e9), (130, 128, 1e6, 3), (260, 512, 1e8, 1e9),
                                              (1030, 64, 1e6, 1e9), (64, 2048, 1e6, 1e9), (64, 64, 1.0, 1e9)])
def test_exact_step_is_the_oracles(nx, ny, Ra, stretch, scheme, spike):
    from simplenavierstokessolver_gb300 import Case

    cfg = Config(nx, ny, ly=1.0, Ra=Ra, Pr=0.7, stretch=stretch)
    state = _state(nx, ny)
    if spike:
        state[3][ny // 2, nx // 3] = 1e30
    o = OracleCase(cfg, threads=4)
    o.set_costs(COSTS[scheme])
    o.set_state(*state)
    o.call("update_boundaries")
    with Case(nx, ny, ly=1.0, stretch=stretch, Ra=Ra, Pr=0.7, costs=COSTS[scheme]) as c:
        c.set_state(*state)
        c.run(1)
        o.run(1)
        assert c.get_dt() == o.get_dt()
        got, want = c.get_state(), o.get_state()
        for k in FIELDS:
            assert np.array_equal(got[k][1:-1], want[k][1:-1], equal_nan=True), k


@pytest.mark.parametrize("scheme", sorted(COSTS))
@pytest.mark.parametrize("nx,ny,Ra", [(64, 64, 1e6), (64, 64, 1.0), (128, 1024, 1e8), (1152, 64, 1e6), (2048, 32, 1e9),
                                      (64, 4096, 1e6)])
def test_parallel_step_matches_the_exact_one(nx, ny, Ra, scheme):
    """segments of 2 to 128 rows, interface values that reach all of them (Ra 1)
    and few; the fields that take increments (the pressure of noise differs
    between the two forms by their Poisson solves). The solves' round-off passes
    through the Poisson solve, whose mean mode has the condition nx^2: 1e-10
    relative, as for the solve alone."""
    from simplenavierstokessolver_gb300 import Case

    out = []
    for parallel in (False, True):
        with Case(nx, ny, ly=1.0, Ra=Ra, Pr=0.7, costs=COSTS[scheme]) as c:
            if parallel:
                c.set_form(True)
            c.set_state(*_state(nx, ny))
            c.run(1)
            out.append(c.get_state())
    for k in ("ux", "uy", "temp"):
        a, b = (s[k][1:-1, 1:-1] for s in out)
        assert np.linalg.norm(a - b) <= 1e-10 * np.linalg.norm(a), k
