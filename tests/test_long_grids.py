"""Grids of hundreds of thousands of rows: a launch's blocks along y are at
most 65535, so kernels of few rows to a block must take more of them or leave
the work to a kernel that does.  One step of a grid of a few columns against
the oracle (FP64, 1e-9 of the field's scale as for whole steps elsewhere) and
the mixed mode against FP64 (1e-5 m: a step's float rounding of an elevation
of at most 0.2 m is below 1e-6 m)."""
import numpy as np
import pytest

from helpers import G, make_pair, maxrel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [262200, 400000])
def test_a_step_of_a_very_long_grid(fw, oracle_mod, rows):
    M = 4
    rng = np.random.default_rng(rows)
    depth = np.asfortranarray(1.5 + 0.3 * rng.uniform(size=(M, rows)))
    st = tuple(np.asfortranarray(a * rng.uniform(-1.0, 1.0, size=(M, rows))) for a in (0.1, 0.1, 0.1))
    p = {"Mglob": M, "Nglob": rows, "DX": 1.0, "DY": 1.0, "WAVEMAKER": "NONE", "MinDepth": 0.01, "MinDepthFrc": 0.1}
    s, o = make_pair(fw, oracle_mod, p, depth, st)
    assert s.step(1) == 0
    o.step()
    eta = s.get("Eta")
    for n in ("Eta", "U", "V"):
        assert maxrel(s.get(n), o[n]) <= 1e-9, n
    s.close()
    m = fw.Solver(fw.with_defaults(p), precision="MIXED")
    m.init(depth, *st)
    assert m.step(1) == 0
    assert np.abs(m.get("Eta")[G:-G, G:-G] - eta[G:-G, G:-G]).max() <= 1e-5
    m.close()
