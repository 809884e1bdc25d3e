"""A caller may capture single parts of a step on the context's stream
(fw_stream): every part stays on that stream, so its capture ends with nothing
left on another, and needs nothing that another capture recorded."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("Eta", "U", "V", "Ubar", "Vbar", "HU", "HV", "MASK", "MASK9", "AGE")


@pytest.mark.parametrize("dispersion", [True, False])
@pytest.mark.parametrize("precision", ["MIXED", "FP64"])
def test_each_part_in_a_capture_of_its_own(fw, precision, dispersion):
    import torch
    M, N = 130, 70
    rng = np.random.default_rng(5)
    depth = np.asfortranarray(np.linspace(3.0, -0.5, M)[:, None] + 0.1 * rng.normal(size=(M, N)))
    st = tuple(np.asfortranarray(a * rng.normal(size=(M, N))) for a in (0.05, 0.05, 0.05))
    p = fw.with_defaults({"Mglob": M, "Nglob": N, "DX": 1.0, "DY": 1.0, "WAVEMAKER": "NONE", "MinDepth": 0.01,
                          "MinDepthFrc": 0.1, "DISPERSION": dispersion})
    got = []
    for captured in (True, False):
        s = fw.Solver(p, precision=precision)
        s.init(depth, *st)
        s.sync()
        stream = torch.cuda.ExternalStream(s.stream())
        parts = [s.begin_step, lambda: s.stage(1), lambda: s.stage(2), lambda: s.stage(3)]
        for part in parts:
            if not captured:
                part()
                continue
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=stream, capture_error_mode="thread_local"):
                part()
            with torch.cuda.stream(stream):
                g.replay()
            s.sync()
        s.end_step()
        got.append({n: s.get(n) for n in FIELDS})
        s.close()
    for n, a in got[0].items():
        assert np.array_equal(a, got[1][n]), n
    assert np.isfinite(got[0]["Eta"]).all()
