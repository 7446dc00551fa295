"""sns_diagnostics called by several host threads at once on one case: its first
call allocates the case's partials, once, and every caller gets its own
results, those of a call alone."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stepped", [False, True], ids=["fresh", "update_pending"])
def test_first_calls_of_several_threads(stepped):
    from simplenavierstokessolver_gb300 import Case
    from simplenavierstokessolver_gb300 import _native as N

    for seed in range(12):
        with Case(64, 128, ly=2.0, Ra=1e6, Pr=1.0) as c:
            rng = np.random.default_rng(seed)
            su, sc = (130, 65), (130, 66)
            c.set_state(0.1 * rng.uniform(-1, 1, su), 0.1 * rng.uniform(-1, 1, sc), np.zeros(sc),
                        rng.uniform(-0.5, 0.5, sc))
            if stepped:  # leaves the temperature's update to the next call that needs it
                c.set_dt(1e-3, 0, 0)
                c.temperature_compute_force()
                c.temperature_update_temp(0)
            out = np.full((8, 11), np.nan)
            codes, gate = [None] * 8, threading.Barrier(8)

            def call(k):
                gate.wait()
                codes[k] = c.lib.sns_diagnostics(c.param, c.fluid, c.temperature,
                                                 out[k].ctypes.data_as(ctypes.POINTER(ctypes.c_double)))

            before = c.lib.sns_allocations()
            threads = [threading.Thread(target=call, args=(k,)) for k in range(8)]
            for t in threads:
                t.start()
            for t in threads:
                t.join()
            assert codes == [N.SNS_OK] * 8
            assert c.lib.sns_allocations() == before + 1
            alone = c.diagnostics()
        assert np.isfinite(alone).all()
        assert (out == alone).all()
