"""FLUXES by lines against the TMA-staged tiles, bit for bit, over states with
signed zeros, tiny values, infinities and NaN (test_flux_lines.py has the
sizes, over finite states and by value)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bits(a):
    """The bits, every NaN the same."""
    return np.where(np.isnan(a), np.uint64(0x7ff8000000000000), a.view(np.uint64))


@pytest.mark.parametrize("special", ["zeros", "tiny", "inf", "nan"])
@pytest.mark.parametrize("precision", ["MIXED", "FP64"])
@pytest.mark.parametrize("size", [(61, 40), (117, 33)])
def test_line_fluxes_have_the_tiles_bits(fw, size, precision, special):
    M, N = size
    rng = np.random.default_rng(M + N)
    depth = np.asfortranarray(np.linspace(2.0, -0.4, M)[:, None] + 0.2 * rng.normal(size=(M, N)))
    p = fw.with_defaults({"Mglob": M, "Nglob": N, "DX": 1.0, "DY": 1.5, "WAVEMAKER": "NONE", "MinDepth": 0.01,
                          "MinDepthFrc": 0.1})
    st = [np.asfortranarray(a * rng.normal(size=(M, N))) for a in (0.1, 0.3, 0.3)]
    fields = ("U", "V", "HU", "HV", "Eta", "U4", "V4")
    got = []
    for tma in (0, 1):
        s = fw.Solver(p, precision=precision)
        s.init(depth, *st)
        t = s.tuning()
        t.update({"flux_x_tma": tma, "flux_y_tma": tma, "flux_x": 8, "flux_y": 8})
        s.set_tuning(t)
        s.begin_step()
        s.cal_dispersion()
        r = np.random.default_rng(11)
        for n in fields:
            a = s.get(n)
            pick = r.uniform(size=a.shape)
            if special == "zeros":
                a[pick < 0.3] = 0.0
                a[pick > 0.6] = -0.0
            elif special == "tiny":
                # below float's smallest normal, above it, and at double's
                scale = r.choice([1e-36, 1e-30, 1e-7] if precision == "MIXED" else [1e-310, 1e-300, 1e-160, 1e-9],
                                 size=a.shape)
                a = np.asfortranarray(np.where(pick < 0.7, a * scale, a))
            else:
                a[pick < 0.02] = np.inf if special == "inf" else np.nan
                if special == "inf":
                    a[pick > 0.98] = -np.inf
            s.set(n, a)
        s.fluxes()
        got.append({n: s.get(n) for n in ("P", "Fx", "Gx", "Q", "Fy", "Gy")})
        s.close()
    for n, a in got[0].items():
        assert np.array_equal(_bits(a), _bits(got[1][n])), n
