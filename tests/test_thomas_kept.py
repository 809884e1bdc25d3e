"""The FP64 solves with kept factors (viscosity breaking) against the ones
that eliminate at every call (without it), bit for bit: k_thomas_solve's
quotients are products with kept reciprocals where div_rcp's range allows, and
divisions elsewhere, and both round as the division.  The same fields give
both the same right-hand side (no breaking: nu is zero); still rows, tiny and
huge velocities take the solve through zero numerators and past both ends of
the range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("scale", [0.05, 1e-151, 1e-306, 3e150])
@pytest.mark.parametrize("size", [(8, 9), (33, 70), (101, 47)])
def test_kept_factors_give_the_elimination_s_bits(fw, size, scale, periodic):
    M, N = size
    rng = np.random.default_rng(M)
    depth = np.asfortranarray(rng.uniform(0.5, 2.0, size=(M, N)))
    got = []
    vel = [np.asfortranarray(scale * rng.normal(size=(M, N))) for _ in range(2)]
    for a in vel:
        a[M // 3:2 * M // 3, :] = 0.0
        a[:, N // 3:2 * N // 3] = 0.0
    for visc in (True, False):
        s = fw.Solver(fw.with_defaults({"Mglob": M, "Nglob": N, "DX": 1.0, "DY": 1.0, "PERIODIC": periodic,
                                        "WAVEMAKER": "NONE", "MinDepth": 0.01, "MinDepthFrc": 0.1, "Gamma2": 0.0,
                                        "VISCOSITY_BREAKING": visc, "FroudeCap": 1e300}), precision="FP64")
        s.init(depth, np.zeros((M, N)), np.zeros((M, N)), np.zeros((M, N)))
        m9 = s.get("MASK9")
        # the momentum the recovery starts from, with no flux or source
        for n, a in zip(("Ubar", "Vbar"), vel):
            f = s.get(n)
            f[3:-3, 3:-3] = a
            s.set(n, f)
        s.set_scalar("DT", 0.0)
        s.estimate_huv(1)
        got.append([s.get(n)[3:-3, 3:-3] for n in ("U", "V", "Ubar")] + [m9])
        s.close()
    assert np.array_equal(got[0][3], got[1][3])
    assert np.isfinite(got[0][0]).all() and np.abs(got[0][0]).max() > 0
    for a, b in zip(got[0][:3], got[1][:3]):
        assert np.array_equal(np.ascontiguousarray(a).view(np.uint64), np.ascontiguousarray(b).view(np.uint64))
