"""JON_2D: whole steps take the wavemaker's mass from a kernel of its own over
the band (k_wm_band), single parts sum it in each cell; both leave the same
bits, from still water on and after a restart in the middle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("Eta", "U", "V", "Ubar", "Vbar", "HU", "HV", "H", "MASK", "AGE", "nu_break")


@pytest.mark.parametrize("precision", ["MIXED", "FP64"])
@pytest.mark.parametrize("size", [(200, 24), (331, 67)])
def test_band_mass_equals_the_sum_in_each_cell(fw, size, precision, tmp_path):
    M, N = size
    p, depth, phases, _ = fw.cases.barred_beach(M, N, 1.0, seed=3, wk_from_shore=120.0, shore_from_east=40.0, nfreq=16,
                                                ntheta=3, Hmo=0.5, Sponge_west_width=20.0)
    p = fw.with_defaults(p)

    def parts(s):
        s.begin_step()
        for k in (1, 2, 3):
            s.stage(k)
        s.end_step()

    got = []
    for way in ("step", "parts", "restart"):
        s = fw.Solver(p, precision=precision)
        s.init(depth, phases=phases)
        assert 0 <= s.scalar("ilo") < s.scalar("ihi") < M
        if way == "parts":
            for _ in range(60):
                parts(s)
        else:
            s.step(29)
            if way == "restart":
                s.checkpoint(str(tmp_path / "ck"))
                s.close()
                s = fw.Solver(p, precision=precision)
                s.restore(str(tmp_path / "ck"))
                parts(s)
                s.step(30)
            else:
                s.step(31)
        got.append({n: s.get(n) for n in FIELDS})
        s.close()
    for n, a in got[0].items():
        assert np.array_equal(a, got[1][n]), n
        assert np.array_equal(a, got[2][n]), n
    assert np.abs(got[0]["Eta"]).max() > 1e-4  # the wavemaker has made waves
