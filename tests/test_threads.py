"""Contexts of different sizes in host threads of their own.  A kernel's limit
of shared memory belongs to the process, not to a context, so no context may
set it to its own need: 1008- and 4096-cell x lines ask for 53 and 62 KB.  The
threads' results are those of the same calls made one context after the
other."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CALLS = 1500


def test_line_solves_of_two_sizes_at_once(fw):
    def context(M, N):
        rng = np.random.default_rng(M)
        p = fw.with_defaults({"Mglob": M, "Nglob": N, "DX": 1.0, "DY": 1.0, "WAVEMAKER": "NONE"})
        s = fw.Solver(p, precision="MIXED")
        s.init(np.asfortranarray(rng.uniform(0.5, 2.0, size=(M, N))),
               *[np.asfortranarray(0.05 * rng.normal(size=(M, N))) for _ in range(3)])
        s.set_scalar("DT", 0.0)
        return s

    def work(s, errors):
        try:
            for _ in range(CALLS):
                s.estimate_huv(1)
            s.sync()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    sizes, errors, alone = [(1008, 640), (4096, 8)], [], {}
    for size in sizes:
        s = context(*size)
        work(s, errors)
        alone[size] = s.get("U")
        s.close()
    runs = [(context(*size), size) for size in 2 * sizes]
    threads = [threading.Thread(target=work, args=(s, errors)) for s, _ in runs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
    for s, size in runs:
        assert np.isfinite(alone[size]).all()
        assert np.array_equal(s.get("U"), alone[size])
        s.close()
