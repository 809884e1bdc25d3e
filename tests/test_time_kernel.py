"""fw_time_kernel: what it runs is the step's own kernel, and what it is not
said to change stays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("precision", ["MIXED", "FP64"])
@pytest.mark.parametrize("name,field", [("tri_x", "U"), ("tri_y", "V")])
def test_solving_again_gives_the_same(fw, name, field, precision, periodic):
    M, N = 61, 50
    rng = np.random.default_rng(9)
    p = fw.with_defaults({"Mglob": M, "Nglob": N, "DX": 1.0, "DY": 1.0, "PERIODIC": periodic, "WAVEMAKER": "NONE",
                          "MinDepth": 0.01, "MinDepthFrc": 0.1})
    s = fw.Solver(p, precision=precision)
    s.init(np.asfortranarray(rng.uniform(0.5, 2.0, size=(M, N))),
           *[np.asfortranarray(0.05 * rng.normal(size=(M, N))) for _ in range(3)])
    s.begin_step()
    s.cal_dispersion()
    s.fluxes()
    s.estimate_huv(1)
    s.time_kernel(name, 1)
    a = s.get(field)
    s.time_kernel(name, 12)
    assert np.array_equal(s.get(field), a)
    assert np.abs(a).max() > 0
    s.close()
