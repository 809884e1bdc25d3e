"""Captured steps put independent launches on two branches of the graph (the
time step's end, the factorisation, the y fluxes, the y solve); the single
parts of a step run in line on one stream.  Both must leave the same bits: over
wetting and drying, with and without dispersion, viscosity breaking (without
it MASK9 moves and the factorisation runs) and a periodic y."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("Eta", "U", "V", "Ubar", "Vbar", "HU", "HV", "H", "MASK", "MASK9", "AGE", "nu_break")
MODES = {"plain": {}, "nodisp": {"DISPERSION": False}, "novisc": {"VISCOSITY_BREAKING": False},
         "periodic": {"PERIODIC": True}}


@pytest.mark.parametrize("mode", sorted(MODES))
@pytest.mark.parametrize("precision", ["MIXED", "FP64"])
@pytest.mark.parametrize("size", [(64, 32), (130, 70), (530, 45)])
def test_branches_equal_one_stream(fw, size, precision, mode):
    M, N = size
    rng = np.random.default_rng(7 * M + N)
    depth = np.asfortranarray(np.linspace(3.0, -0.5, M)[:, None] + 0.1 * rng.normal(size=(M, N)))
    x = np.arange(M)[:, None]
    eta = 0.5 * np.exp(-((x - 0.4 * M) / 6.0) ** 2) + 0.02 * rng.normal(size=(M, N))
    u, v = 0.2 * eta, 0.05 * rng.normal(size=(M, N))
    p = fw.with_defaults(dict({"Mglob": M, "Nglob": N, "DX": 1.0, "DY": 1.5, "WAVEMAKER": "NONE", "MinDepth": 0.01,
                               "MinDepthFrc": 0.1}, **MODES[mode]))
    got = []
    for captured in (True, False):
        s = fw.Solver(p, precision=precision)
        s.init(depth, eta, u, v)
        if captured:
            assert s.step(9) == 0
        else:
            for _ in range(9):
                s.begin_step()
                for k in (1, 2, 3):
                    s.stage(k)
                s.end_step()
        got.append({n: s.get(n) for n in FIELDS})
        got[-1]["TIME"] = np.float64(s.scalar("TIME"))
        s.close()
    for n, a in got[0].items():
        assert np.array_equal(a, got[1][n]), n
    assert np.isfinite(got[0]["Eta"]).all()


@pytest.mark.parametrize("precision", ["MIXED", "FP64"])
@pytest.mark.parametrize("shape", [(200, 24, 60.0), (331, 67, 90.0)])
def test_wavemaker_band_equals_inline(fw, shape, precision):
    """JON_2D: whole steps take the wavemaker's mass from a kernel of its own
    over the band, single parts sum it in each cell."""
    M, N, shore = shape
    p, depth, phases, _ = fw.cases.barred_beach(M, N, 1.0, seed=3, wk_from_shore=shore)
    p = fw.with_defaults(p)
    got = []
    for captured in (True, False):
        s = fw.Solver(p, precision=precision)
        s.init(depth, phases=phases)
        if captured:
            assert s.step(7) == 0
        else:
            for _ in range(7):
                s.begin_step()
                for k in (1, 2, 3):
                    s.stage(k)
                s.end_step()
        got.append({n: s.get(n) for n in FIELDS})
        s.close()
    for n, a in got[0].items():
        assert np.array_equal(a, got[1][n]), n
    assert np.abs(got[0]["Eta"]).max() > 0
