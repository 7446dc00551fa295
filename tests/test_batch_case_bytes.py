"""Arena bytes of a batched case (csrc/batch_api.cpp, layout_for): per Fourier
mode 4 itot + 352 doubles of factors; per cell five FP32 fields' words (two sets
of ux, uy, T with their low words, the three explicit terms, in compensated
cases with low words too), p and psi; the spectrum; small arrays of itot or jtot
words; every array from a multiple of 256 bytes. Host code only: no device is needed."""
import pytest


def expected(nx, ny, compensated):
    def up(v):
        return (v + 255) // 256 * 256

    nh, cells, f, d = ny // 2 + 1, nx * ny, 4, 8
    sizes = [f * nx, f * nx, f * (nx + 1)] + [f * nx] * 4
    sizes += [d * nx, d * (nx + 1), d * (nx + 1), d * nx, d * (nx + 1), d * 2 * ny, d * nx, d * nx]
    sizes += [d * (4 * nx + 352) * nh] + [d * nx] * 4
    sizes += [f * cells] * (12 + (6 if compensated else 3)) + [d * cells] * 2 + [2 * d * nh * nx]
    return sum(up(v) for v in sizes)


@pytest.mark.parametrize("compensated", [False, True])
@pytest.mark.parametrize("nx,ny", [(64, 8), (64, 16), (64, 64), (128, 256), (640, 1024), (1024, 4096)])
def test_case_bytes(nx, ny, compensated):
    from simplenavierstokessolver_gb300.batch import Desc, case_bytes
    from simplenavierstokessolver_gb300.build import build

    build()
    assert case_bytes(Desc(nx, ny, compensated=compensated)) == expected(nx, ny, compensated)
