"""EXCHANGE in one pass (k_exchange) where an interior cell is the source of
ghost cells on both sides of the domain at once (3 to 7 cells across), with
sponge, walls and periodic y: whole FP64 steps against the oracle, ghost cells
included (bc.F:426-529, 631-1272).  Tolerance: that of whole steps elsewhere,
1e-9 of the field's scale; masks exact."""
import numpy as np
import pytest

from helpers import make_pair, maxrel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("size", [(3, 3), (3, 8), (4, 5), (5, 3), (6, 6), (7, 4), (33, 5), (5, 33)])
def test_small_grids_match_oracle(fw, oracle_mod, size, periodic):
    M, N = size
    rng = np.random.default_rng(10 * M + N)
    depth = np.asfortranarray(1.5 + 0.4 * rng.uniform(size=(M, N)))
    depth[M // 2, N // 2] = -0.02
    st = tuple(np.asfortranarray(a * rng.normal(size=(M, N))) for a in (0.03, 0.05, 0.05))
    p = {"Mglob": M, "Nglob": N, "DX": 1.0, "DY": 1.0, "PERIODIC": periodic, "WAVEMAKER": "NONE", "MinDepth": 0.01,
         "MinDepthFrc": 0.1, "DIRECT_SPONGE": True, "Sponge_west_width": 2.0, "Sponge_north_width": 1.0}
    s, o = make_pair(fw, oracle_mod, p, depth, st)
    for _ in range(3):
        s.step(1)
        o.step()
    for n in ("Eta", "U", "V", "HU", "HV", "nu_break"):
        assert maxrel(s.get(n), o[n]) <= 1e-9, n
    assert np.array_equal(s.get("MASK"), o["MASK"])
    s.close()
