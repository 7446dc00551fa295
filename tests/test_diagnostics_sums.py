"""sns_diagnostics (csrc/diagnostics.cu: 128-bit integer sums per thread) against
long double sums of the same terms: grids of a few cells, of one to 32 rows per
thread and of columns beyond a block, equal and stretched spacings; a wide range
of magnitudes, and infinities and NaN, which make the sums that they enter NaN."""
import numpy as np
import pytest

from oracle.bindings import Config, OracleCase

pytestmark = pytest.mark.gpu
L = np.longdouble


def _terms(cfg, ux, uy, T):
    """per log quantity from the second on (divergence sum, ...): its terms"""
    g = OracleCase(cfg).get_grid()
    dxf, dxc, dy = g["dxf"].astype(L), g["dxc"].astype(L), L(g["dy"])
    q = np.sqrt(L(cfg.Pr)) * np.sqrt(L(cfg.Ra))
    nu, kappa = np.sqrt(L(cfg.Pr)) / np.sqrt(L(cfg.Ra)), 1 / np.sqrt(L(cfg.Pr)) / np.sqrt(L(cfg.Ra))
    u, v, t = (a[1:-1].astype(L) for a in (ux, uy, T))
    u = u.copy()
    u[:, 0] = u[:, -1] = 0
    v, t = v.copy(), t.copy()
    v[:, 0] = v[:, -1] = 0
    t[:, 0], t[:, -1] = 0.5, -0.5
    un, vn, tn = (np.roll(a, -1, axis=0) for a in (u, v, t))
    vc, tc = v[:, 1:-1], t[:, 1:-1]
    lxly = L(1) * L(cfg.ly)
    dissipation = [np.diff(u, axis=1) ** 2 * dy / dxf, (un - u)[:, 1:-1] ** 2 * dxc[1:-1] / dy,
                   np.diff(v, axis=1) ** 2 * dy / dxc, (vn - v)[:, 1:-1] ** 2 * dxf / dy]
    thermal = [np.diff(t, axis=1) ** 2 * dy / dxc, (tn - t)[:, 1:-1] ** 2 * dxf / dy]
    flux = [-(t[:, 1] - t[:, 0]) / dxc[0] * dy / 2, -(t[:, -1] - t[:, -2]) / dxc[-1] * dy / 2]
    return {1: [np.diff(u, axis=1) / dxf, (vn - v)[:, 1:-1] / dy], 2: [u * dxc * dy], 3: [vc * dxf * dy],
            4: [u**2 * dxc * dy / 2], 5: [vc**2 * dxf * dy / 2], 6: [tc**2 * dxf * dy / 2],
            7: [f / L(cfg.ly) for f in flux],
            8: [u * (t[:, :-1] + t[:, 1:]) / 2 * dxc * dy * q / lxly, [L(1)]],
            9: [d * q * nu / lxly for d in dissipation] + [[L(1)]], 10: [d * q * kappa / lxly for d in thermal]}


@pytest.mark.parametrize("kind", ["noise", "wide", "not_finite"])
@pytest.mark.parametrize("nx,ny,stretch", [(2, 2, 1e9), (5, 4, 3), (31, 8, 1e9), (64, 128, 1e9), (65, 32, 3),
                                           (128, 256, 1e9), (513, 64, 1e9), (200, 2048, 3), (1024, 2048, 1e9)])
def test_sums_are_those_of_their_terms(nx, ny, stretch, kind):
    """a term takes at most 8 roundings: 8 * 2^-53 of the terms' magnitudes"""
    from simplenavierstokessolver_gb300 import Case

    cfg = Config(nx, ny, ly=2.0, Ra=1e6, Pr=0.7, stretch=stretch)
    rng = np.random.default_rng(17)
    size = 10.0 ** rng.uniform(-30, 30, (ny + 2, nx + 2)) if kind == "wide" else np.ones((ny + 2, nx + 2))
    ux, uy, t = (s * rng.uniform(-0.5, 0.5, s.shape) for s in (size[:, :-1], size, size))
    if kind == "not_finite":
        ux[ny // 2 + 1, nx // 2 or 1], t[1, 1] = np.inf, np.nan
    with Case(nx, ny, ly=2.0, stretch=stretch, Ra=1e6, Pr=0.7) as c:
        c.set_state(ux, uy, np.zeros_like(uy), t)
        got = c.diagnostics()
    with np.errstate(invalid="ignore"):
        for k, parts in _terms(cfg, ux, uy, t).items():
            want = sum(np.sum(p, dtype=L) for p in parts)
            magnitude = sum(np.sum(np.abs(p), dtype=L) for p in parts)
            if np.isfinite(magnitude):
                assert abs(L(got[k]) - want) <= 8 * 2.0**-53 * magnitude, (k, got[k], want, magnitude)
            else:
                assert np.isnan(got[k]), k
