"""The max-|u| reduction's way to the host (csrc/plain_fp64.cu, k_publish): the dt
decided after any order of calls is the one of the same state set anew. The words
are nx + 1, 256 to a block; two fluids of one param keep reductions of their own."""
import pytest

pytestmark = pytest.mark.gpu


def _fresh(nx, state):
    from simplenavierstokessolver_gb300 import Case

    with Case(nx, 16, Ra=1e7) as c:
        c.set_state(*(state[k] for k in ("ux", "uy", "p", "temp")))
        c.param_decide_dt()
        return c.get_dt()["dt"]


@pytest.mark.parametrize("nx,parallel", [(4, False), (254, False), (255, False), (256, False), (257, False),
                                         (513, False), (64, True), (256, True), (512, True)])
def test_dt_after_any_order_of_calls(nx, parallel):
    from simplenavierstokessolver_gb300 import Case

    with Case(nx, 16, Ra=1e7) as c:
        c.set_form(parallel)
        c.run(3)
        for call in (lambda: c.run(2), lambda: c.run_calls(2), c.integrate, c.integrate, lambda: c.run(1)):
            call()
            got = []
            for _ in range(2):
                c.param_decide_dt()
                got.append(c.get_dt()["dt"])
            assert got == [_fresh(nx, c.get_state())] * 2


def test_two_fluids_of_one_param():
    from simplenavierstokessolver_gb300 import Case

    nx = 64
    with Case(nx, 16, Ra=1e7) as c:
        c.run(4)
        want = _fresh(nx, c.get_state())
        first = c.fluid
        c.fluid = c.lib.fluid_init(c.param, c.parallel)
        assert c.fluid
        try:
            c.integrate()  # the other fluid
        finally:
            c.lib.fluid_finalise(c.fluid)
            c.fluid = first
        c.param_decide_dt()
        assert c.get_dt()["dt"] == want
