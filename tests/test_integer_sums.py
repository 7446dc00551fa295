"""The exact form's additions in the integer unit (csrc/plain_fp64.cu, num_sum):
velocity, temperature, correction and pressure kernels bit for bit the oracle's
on operands at which a rounding can go wrong: ties and near ties (few and many
trailing ones and zeros), neighbours that cancel, exponents from equal to 2^120
apart, zeros of both signs, and values outside the range, whose rows take FP64."""
import numpy as np
import pytest

from oracle.bindings import Config, OracleCase

pytestmark = pytest.mark.gpu


def _values(rng, shape, kind):
    n = int(np.prod(shape))
    frac = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    low = rng.integers(0, 53, n).astype(np.uint64)
    ones = (np.uint64(1) << low) - np.uint64(1)
    pick = rng.integers(0, 3, n)
    frac = np.where(pick == 1, frac & ~ones, np.where(pick == 2, frac | ones, frac)) & np.uint64((1 << 52) - 1)
    spread = {"near": 2, "apart": 120, "edges": 20}[kind]
    e = (1023 - spread // 2 + rng.integers(0, spread, n)).astype(np.uint64)
    v = (frac | e << np.uint64(52) | rng.integers(0, 2, n, dtype=np.uint64) << np.uint64(63)).view(np.float64)
    # the next cell's value again, or the next number to it, of either sign
    same = rng.integers(0, 4, n)
    prev = np.roll(v, 1)
    v = np.where(same == 1, -prev, np.where(same == 2, np.nextafter(prev, 0.0), v))
    if kind == "edges":
        special = np.array([0.0, -0.0, 5e-324, -1e-310, 2.3e-308, 1e-290, -1e-200, 1e30])
        v = np.where(rng.integers(0, 6, n) == 0, special[rng.integers(0, len(special), n)], v)
    return v.reshape(shape)


@pytest.mark.parametrize("kind", ["near", "apart", "edges"])
@pytest.mark.parametrize("scheme", [(0, 0), (1, 0), (0, 1), (1, 1)], ids=["exp", "imp_x", "imp_y", "imp_imp"])
@pytest.mark.parametrize("nx,ny,stretch", [(32, 16, 1e9), (33, 32, 1e9), (65, 64, 3), (256, 512, 1e9), (200, 512, 1e9)])
def test_updates_round_like_the_oracle(nx, ny, stretch, scheme, kind):
    """spacings that are powers of two, others with their division pairs"""
    from simplenavierstokessolver_gb300 import Case

    cfg = Config(nx, ny, ly=2.0, Ra=1e6, Pr=0.7, stretch=stretch)
    rng = np.random.default_rng(29)
    su, sc = (ny + 2, nx + 1), (ny + 2, nx + 2)
    state = [_values(rng, s, kind) for s in (su, sc, sc, sc)]
    o = OracleCase(cfg)
    o.set_state(*state)
    o.call("update_boundaries")
    with Case(nx, ny, ly=2.0, stretch=stretch, Ra=1e6, Pr=0.7) as c:
        c.set_state(*state)
        for x in (c, o):
            x.set_dt(1e-3, *scheme)
        c.temperature_compute_force()
        c.temperature_update_temp(1)
        o.call("temperature_force_and_update", 1)
        c.fluid_update_velocity(1)
        o.call("fluid_update_velocity", 1)
        got, want = c.get_sources(), o.get_sources()
        for k in want:
            assert np.array_equal(got[k], want[k]), k
        for name in ("fluid_compute_potential", "fluid_correct_velocity", "fluid_update_pressure"):
            getattr(c, name)(1)
            o.call(name, 1)
        got, want = c.get_state(), o.get_state()
        for k in ("ux", "uy", "temp", "psi", "p"):
            assert np.array_equal(got[k][1:-1], want[k][1:-1]), k
