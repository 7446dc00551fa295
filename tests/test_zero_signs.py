"""The exact form on fields that hold zeros of both signs (csrc/plain_fp64.cu):
compared as bits, which np.array_equal of floats does not."""
import numpy as np
import pytest

from oracle.bindings import Config, OracleCase

pytestmark = pytest.mark.gpu
STATE = ("ux", "uy", "p", "psi", "temp")


def _state(nx, ny, kind, seed):
    """negative: -0 everywhere; zeros: of either sign; mixed: mostly these, beside
    numbers of which some are neighbours' negatives"""
    rng = np.random.default_rng(seed)
    out = []
    for shape in ((ny + 2, nx + 1), (ny + 2, nx + 2), (ny + 2, nx + 2), (ny + 2, nx + 2)):
        a = np.full(shape, -0.0) if kind == "negative" else rng.choice([0.0, -0.0], shape)
        if kind == "mixed":
            a = np.where(rng.integers(0, 3, shape) == 0, 0.25 * rng.integers(-1, 2, shape), a)
        out.append(a)
    return out


def _same_bits(got, want, where):
    for k in want:
        for g, w in zip(np.atleast_1d(got[k]), np.atleast_1d(want[k])):
            diff = np.ascontiguousarray(g).view(np.uint64) != np.ascontiguousarray(w).view(np.uint64)
            assert not diff.any(), (where, k, int(diff.sum()), g[diff][0], w[diff][0])


def _compare(nx, ny, stretch, scheme, kind, rkstep=1):
    """every call of a substage that integrates these fields"""
    from simplenavierstokessolver_gb300 import Case

    cfg = Config(nx, ny, ly=2.0, Ra=1e6, Pr=0.7, stretch=stretch)
    state = _state(nx, ny, kind, 41)
    o = OracleCase(cfg)
    o.set_state(*state)
    o.call("update_boundaries")
    with Case(nx, ny, ly=2.0, stretch=stretch, Ra=1e6, Pr=0.7) as c:
        c.set_state(*state)
        for x in (c, o):
            x.set_dt(1e-3, *scheme)

        def state_of(x):
            return {k: v[1:-1] for k, v in x.get_state().items() if k in STATE}

        c.temperature_compute_force()
        c.temperature_update_temp(rkstep)
        o.call("temperature_force_and_update", rkstep)
        c.fluid_update_velocity(rkstep)
        o.call("fluid_update_velocity", rkstep)
        _same_bits(c.get_sources(), o.get_sources(), "sources")
        _same_bits(state_of(c), state_of(o), "updated fields")
        for name in ("fluid_compute_potential", "fluid_correct_velocity", "fluid_update_pressure"):
            getattr(c, name)(rkstep)
            o.call(name, rkstep)
            _same_bits(state_of(c), state_of(o), name)


@pytest.mark.parametrize("kind", ["negative", "mixed"])
@pytest.mark.parametrize("nx,ny", [(32, 16), (256, 512)])
def test_sums_keep_the_sign_of_zero(nx, ny, kind):
    """spacings that are powers of two; one and two rows a thread (the velocity's
    integer sums start at two)"""
    _compare(nx, ny, 1e9, (0, 0), kind)


@pytest.mark.parametrize("scheme", [(1, 0), (0, 1), (1, 1)], ids=["imp_x", "imp_y", "imp_xy"])
@pytest.mark.parametrize("nx,ny,stretch", [(64, 64, 1e9), (130, 128, 3), (260, 512, 1e9), (1024, 64, 1e9), (64, 2048, 1e9)])
def test_implicit_substages_keep_the_sign_of_zero(nx, ny, stretch, scheme):
    """-0 everywhere but at the walls; lines cut into segments. (Zeros of both
    signs are left out: the reference adds an implicit direction's diffusion to
    the explicit terms with weight zero, the kernels leave it out, and where
    every other term is -0 the sum is +0 there and -0 here.)"""
    _compare(nx, ny, stretch, scheme, "negative")


@pytest.mark.parametrize("kind", ["negative", "zeros", "mixed"])
@pytest.mark.parametrize("nx,ny,stretch", [(33, 8, 1e9), (100, 64, 1e9), (70, 32, 3), (400, 256, 1e9)])
def test_divisions_keep_the_sign_of_zero(nx, ny, stretch, kind):
    """spacings that divide by their pair"""
    _compare(nx, ny, stretch, (0, 0), kind)
