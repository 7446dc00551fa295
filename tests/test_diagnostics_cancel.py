"""Sums of sns_diagnostics whose large terms cancel (csrc/diagnostics.cu, Sum128):
what is left is what a compensated FP64 sum of a thread's terms holds, down to
2^-98 of the largest one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [0, 36, 60, 88, 97])
def test_small_terms_survive_the_large_ones(k):
    """three values in one thread's rows (a thread takes 32 of them here), the
    large ones first, last and around the small one; spacings that are powers of
    two, so that the expected momenta are exact"""
    from simplenavierstokessolver_gb300 import Case

    nx, ny, big = 1024, 2048, 2.0**k
    ux, uy = np.zeros((ny + 2, nx + 1)), np.zeros((ny + 2, nx + 2))
    for column, values in ((5, (big, 1.5, -big)), (70, (1.5, big, -big)), (900, (big, -big, 1.5))):
        for row, v in enumerate(values):
            ux[1 + 40 + row, column] = v
            uy[1 + 40 + row, column] = -v
    z = np.zeros_like(uy)
    with Case(nx, ny, ly=2.0, Ra=1e6, Pr=1.0) as c:
        c.set_state(ux, uy, z, z)
        got = c.diagnostics()
    cell = 1.0 / nx * (2.0 / ny)
    assert got[2] == 4.5 * cell and got[3] == -4.5 * cell, (got[2] / cell, got[3] / cell)
