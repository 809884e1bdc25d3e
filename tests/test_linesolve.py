"""The mixed u/v recovery (k_linesolve, and the longer lines' kernels) at the
line lengths where its partition changes: one chunk, two chunks, chunks of
uneven length, one to eight blocks to a line, and lines beyond 4096 rows.

ESTIMATE_HUV on the same fields in the mixed and the FP64 mode (the
reference's Thomas recurrence, tridiagnal.F:59-398).  Tolerance: the inputs
are float values, so both modes solve the same system but for the rounding of
the right-hand side (three float terms, 2e-7 of their size) and of the
coefficients' refinement (float rounding of the result, 6e-8).  The inverse of
the matrix is bounded by 1 / min(tmp2^-1 (tmp2 - |tmp1| - |tmp3|)) <=
tmp2 = 1 + 0.78 (h/dx)^2 <= 4.2 for h <= 2 dx, so 2e-6 of the largest
velocity covers the mixed error; 1e-5 leaves a factor of five.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [2, 3, 15, 16, 17, 31, 32, 33, 47, 250, 255, 256, 257, 271, 496, 497, 511, 512, 513, 1023, 1100, 2048, 2049, 4095,
           4096, 4097, 4200]


def _case(M, N, periodic):
    rng = np.random.default_rng(M * 7919 + N)
    p = {"Mglob": M, "Nglob": N, "DX": 1.0, "DY": 1.0, "PERIODIC": periodic, "WAVEMAKER": "NONE",
         "VISCOSITY_BREAKING": True, "CFL": 0.5, "MinDepth": 0.01, "MinDepthFrc": 0.1, "DT_fixed": 0.01}
    depth = np.asfortranarray(rng.uniform(0.5, 2.0, size=(M, N)))
    f = [np.asfortranarray(a * rng.normal(size=(M, N)).astype(np.float32).astype(np.float64)) for a in (0.02, 0.1, 0.1)]
    return p, depth.astype(np.float32).astype(np.float64), f


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("L", LENGTHS)
@pytest.mark.parametrize("direction", ["x", "y"])
def test_mixed_line_solve_matches_fp64(fw, direction, L, periodic):
    if direction == "x" and periodic:
        pytest.skip("x lines are never periodic")
    M, N = (L, 13) if direction == "x" else (21, L)
    p, depth, (eta, u, v) = _case(M, N, periodic)
    got = []
    for prec in ("FP64", "MIXED"):
        s = fw.Solver(fw.with_defaults(p), precision=prec)
        s.init(depth, eta, u, v)
        s.begin_step()
        s.cal_dispersion()
        s.fluxes()
        s.estimate_huv(1)
        got.append([s.get(n)[3:-3, 3:-3] for n in ("U", "V")])
        s.close()
    scale = max(np.abs(a).max() for a in got[0])
    assert scale > 0
    for a, b in zip(*got):
        assert np.abs(a - b).max() <= 1e-5 * scale


@pytest.mark.parametrize("size", [(130, 70), (33, 300), (517, 40)])
def test_checkpoint_of_the_earlier_factor_layout_is_factored_again(fw, size, tmp_path):
    """A file whose header does not name this layout of the factors: the run
    continues as the one it was taken from."""
    p, depth, st = _case(*size, False)
    a = fw.Solver(fw.with_defaults(p), precision="MIXED")
    a.init(depth, *st)
    a.step(3)
    path = str(tmp_path / "ck")
    a.checkpoint(path)
    raw = bytearray(open(path, "rb").read())
    off = 8 + 4 + 4 + 4  # magic, sizeof_params, sizeof_grid, precision
    assert raw[off:off + 4] == (1).to_bytes(4, "little")
    raw[off:off + 4] = bytes(4)
    open(path, "wb").write(raw)
    b = fw.Solver(fw.with_defaults(p), precision="MIXED")
    b.restore(path)
    a.step(2)
    b.step(2)
    for n in ("Eta", "U", "V", "Ubar", "Vbar"):
        assert np.array_equal(a.get(n), b.get(n)), n
    a.close()
    b.close()


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("how", ["set", "set_f32", "set_fields", "mask9"])
def test_fp64_factors_follow_a_new_depth(fw, how, periodic):
    """The FP64 solves keep their factors while Depth, MASK9 and MASK stand:
    a run that solved before one of them was set gives the bits of one that
    did not."""
    M, N = 45, 70
    p, depth, st = _case(M, N, periodic)
    rng = np.random.default_rng(2)
    got = []
    for early in (True, False):
        s = fw.Solver(fw.with_defaults(p), precision="FP64")
        s.init(depth, *st)
        s.begin_step()
        names = ("U", "V", "Eta", "Ubar", "Vbar", "H", "HU", "HV", "P", "Q")
        keep = {n: s.get(n) for n in names}
        if early:
            s.cal_dispersion()
            s.fluxes()
            s.estimate_huv(1)
            for n in names:
                s.set(n, keep[n])
        new = np.asfortranarray((s.get("Depth") * 1.25).astype(np.float32).astype(np.float64))
        if how == "set":
            s.set("Depth", new)
        elif how == "set_f32":
            s.set_f32("Depth", new.astype(np.float32))
        elif how == "set_fields":
            s.set_fields({"Depth": new, "Eta": keep["Eta"]})
        else:
            m = s.get("MASK9")
            m[10:20, 15:30] = 0
            s.set("MASK9", m)
        s.cal_dispersion()
        s.fluxes()
        s.estimate_huv(1)
        got.append([s.get(n) for n in ("U", "V", "Eta")])
        s.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
