"""A checkpoint whose header does not name the present layout of the line
solver's factors (fw_restore) is factored again, whatever its factors are; one
that names it is continued with the factors it holds.  The file's factors are
overwritten here, so that a run that used them would leave the checkpointed
one's path."""
import struct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NG = 3
# the arena's planes up to the factors, in the order they are carved
N_REAL = 53                    # Eta .. Hmax
FIRST = {"A": 25, "Uxx": 29}   # A B C E; Uxx Vxy Uxy Vyy DUxx DVxy DUxy DVyy
HEADER = 80                    # bytes; the layout word is at 20


def _factor_ranges(precision, M, N):
    """(offset, bytes) of the factors in a checkpoint's arena."""
    def up(n):
        return (n + 255) // 256 * 256
    es = 8 if precision == "FP64" else 4
    pitch = (M + 2 * NG + 1 + 31) // 32 * 32
    cells = pitch * (N + 2 * NG + 1)
    real, dbl = up(cells * es), up(cells * 8)
    off = N_REAL * real + 4 * up(cells) + 2 * real  # reals, masks, right-hand sides: then ty tp tq tc
    if precision == "FP64":
        return [(k * real, cells * 8) for k in range(FIRST["A"], FIRST["A"] + 4)] + [(off + 2 * dbl, cells * 8)]
    out = [(FIRST["Uxx"] * real, 8 * real)]
    off += 4 * dbl + dbl + 256 + 3 * dbl  # .., DepthD, m9_dirty, the y factorisation's scratch
    for L, lines in ((M, N), (N, M)):
        m = max(16, (L + 255) // 256)
        P = 1 if L < 2 * m else L // m
        red = up(lines * (10 * P + 3) * 4)
        out.append((off, 10 * real + red))
        off += 10 * real + red
    return out


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("precision", ["MIXED", "FP64"])
@pytest.mark.parametrize("size", [(130, 70), (33, 300)])
def test_factors_of_another_layout_are_not_used(fw, size, precision, periodic, tmp_path):
    M, N = size
    rng = np.random.default_rng(M)
    p = fw.with_defaults({"Mglob": M, "Nglob": N, "DX": 1.0, "DY": 1.0, "PERIODIC": periodic, "WAVEMAKER": "NONE",
                          "MinDepth": 0.01, "MinDepthFrc": 0.1})
    depth = np.asfortranarray(rng.uniform(0.5, 2.0, size=(M, N)))
    a = fw.Solver(p, precision=precision)
    a.init(depth, *[np.asfortranarray(c * rng.normal(size=(M, N))) for c in (0.02, 0.05, 0.05)])
    a.step(3)
    path = str(tmp_path / "ck")
    a.checkpoint(path)
    a.step(2)
    fields = ("Eta", "U", "V", "Ubar", "Vbar")
    want = [a.get(n) for n in fields]
    a.close()
    raw = bytearray(open(path, "rb").read())
    sp, sg = struct.unpack_from("<II", raw, 8)
    layout, = struct.unpack_from("<i", raw, 20)
    arena = HEADER + sp + sg
    word = struct.pack("<d", 0.25) if precision == "FP64" else struct.pack("<f", 0.25)
    for off, n in _factor_ranges(precision, M, N):
        raw[arena + off:arena + off + n] = word * (n // len(word))
    got = {}
    for tag in (layout, 0):
        struct.pack_into("<i", raw, 20, tag)
        open(path, "wb").write(raw)
        b = fw.Solver(p, precision=precision)
        b.restore(path)
        b.step(2, check=False)
        got[tag] = [b.get(n) for n in fields]
        b.close()
    assert layout != 0
    for n, w, x in zip(fields, want, got[0]):
        assert np.array_equal(w, x), n
    assert not np.array_equal(want[1], got[layout][1])  # the planes overwritten are the factors
    assert not np.array_equal(want[2], got[layout][2])
