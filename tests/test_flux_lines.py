"""FLUXES by lines (k_flux_x: 58 faces to a warp; k_flux_y: strips of a
column) against the TMA-staged tiles (k_flux_tma), which evaluate the limiter
and the face states per face: the same bits at the widths and heights where
the lines' lanes and strips end, over water, dry land and still water."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(5, 4), (54, 9), (57, 33), (58, 65), (59, 64), (113, 31), (116, 40), (117, 130), (300, 71)]


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("precision", ["MIXED", "FP64"])
@pytest.mark.parametrize("size", SIZES)
def test_line_fluxes_equal_staged_tiles(fw, size, precision, periodic):
    M, N = size
    rng = np.random.default_rng(M + 1000 * N)
    depth = np.asfortranarray(np.linspace(2.0, -0.6, M)[:, None] + 0.3 * rng.normal(size=(M, N)))
    eta = 0.2 * rng.normal(size=(M, N))
    u, v = 0.3 * rng.normal(size=(M, N)), 0.3 * rng.normal(size=(M, N))
    still = slice(N // 3, max(N // 3 + 1, 2 * N // 3))
    for a in (eta, u, v):
        a[:, still] = 0.0
    p = fw.with_defaults({"Mglob": M, "Nglob": N, "DX": 1.0, "DY": 1.5, "PERIODIC": periodic, "WAVEMAKER": "NONE",
                          "MinDepth": 0.01, "MinDepthFrc": 0.1})
    got = []
    for tma, fy in ((0, 8), (1, 8), (0, 16)):
        s = fw.Solver(p, precision=precision)
        s.init(depth, eta, u, v)
        t = s.tuning()
        t.update({"flux_x_tma": tma, "flux_y_tma": tma, "flux_x": fy, "flux_y": fy})
        s.set_tuning(t)
        s.begin_step()
        s.cal_dispersion()
        s.fluxes()
        got.append({n: s.get(n) for n in ("P", "Fx", "Gx", "Q", "Fy", "Gy")})
        s.close()
    for other in got[1:]:
        for n, a in got[0].items():
            assert np.array_equal(a, other[n]), n
    assert np.abs(got[0]["P"]).max() > 0
