"""The line solver's kept factors follow every way of setting a field that
they depend on: a run that solved before Depth or MASK9 was set gives the
bits of one that did not (MIXED; FP64 in test_linesolve.py)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _set_fields_f32(s, arrays, pinned):
    L = s.L
    names = (ctypes.c_char_p * len(arrays))(*[n.encode() for n in arrays])
    keep, ptrs = [], []
    for a in arrays.values():
        a = np.asfortranarray(a, dtype=np.float32)
        if pinned:
            p = ctypes.c_void_p()
            assert L.fw_host_alloc(ctypes.c_size_t(a.nbytes), ctypes.byref(p)) == 0
            ctypes.memmove(p, a.ctypes.data, a.nbytes)
            ptrs.append(p.value)
        else:
            ptrs.append(a.ctypes.data)
        keep.append(a)
    host = (ctypes.c_void_p * len(ptrs))(*ptrs)
    assert L.fw_set_fields_f32(s.ctx, len(ptrs), names, host) == 0
    if pinned:
        for p in ptrs:
            assert L.fw_host_free(ctypes.c_void_p(p)) == 0


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("how", ["set", "set_f32", "set_fields", "set_fields_f32", "set_fields_f32_pinned", "mask9",
                                 "mask9_fields"])
def test_mixed_factors_follow_a_new_depth(fw, how, periodic):
    M, N = 45, 70
    rng = np.random.default_rng(3)
    p = fw.with_defaults({"Mglob": M, "Nglob": N, "DX": 1.0, "DY": 1.0, "PERIODIC": periodic, "WAVEMAKER": "NONE",
                          "MinDepth": 0.01, "MinDepthFrc": 0.1, "DT_fixed": 0.01})
    depth = np.asfortranarray(rng.uniform(0.5, 2.0, size=(M, N)))
    st = [np.asfortranarray(a * rng.normal(size=(M, N))) for a in (0.02, 0.1, 0.1)]
    names = ("U", "V", "Eta", "Ubar", "Vbar", "H", "HU", "HV", "P", "Q")
    got = []
    for early in (True, False):
        s = fw.Solver(p, precision="MIXED")
        s.init(depth, *st)
        s.begin_step()
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
            s.set_f32("Depth", new)
        elif how == "set_fields":
            s.set_fields({"Eta": keep["Eta"], "Depth": new})
        elif how.startswith("set_fields_f32"):
            _set_fields_f32(s, {"Depth": new, "Eta": keep["Eta"]}, how.endswith("pinned"))
        else:
            m = s.get("MASK9")
            m[10:20, 15:30] = 0
            if how == "mask9":
                s.set("MASK9", m)
            else:
                s.set_fields({"MASK9": m})
        s.cal_dispersion()
        s.fluxes()
        s.estimate_huv(1)
        got.append([s.get(n) for n in ("U", "V", "Eta")])
        s.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
