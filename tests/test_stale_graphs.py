"""What an ensemble's or a network's captured graph was made with may change:
a context is initialised again (new wavemaker tables), a scalar is set, the
solver is another one, the network's workspace grows.  The next run then
gives what stepping gives, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("Eta", "U", "V", "Ubar", "Vbar", "MASK", "AGE", "nu_break")


def _case(fw, seed, M=200, N=40, **over):
    p, d, ph, _ = fw.cases.barred_beach(M, N, 1.0, seed=seed, wk_from_shore=120.0, nfreq=8, ntheta=2,
                                        shore_from_east=40.0, Hmo=0.5, Sponge_west_width=20.0)
    # low breaking thresholds: the sea of _init breaks
    p.update(dict({"Cbrk1": 0.02, "Cbrk2": 0.01, "DT_fixed": 0.02}, **over))
    return fw.with_defaults(p), d, ph


def _init(fw, s, d, ph, seed):
    s.init(d, *fw.cases.random_state(*d.shape, seed=seed, eta_amp=0.2, u_amp=0.3), ph)


def _same(a, b):
    for n in FIELDS:
        assert np.array_equal(a.get(n), b.get(n)), n


@pytest.mark.parametrize("what", ["T_brk", "init"])
def test_ensemble_after_a_change(fw, what):
    p, d, ph = _case(fw, 1)
    e = fw.Ensemble([(p, d, ph), _case(fw, 2, M=130)], precision="MIXED", single_launch=True)
    one = fw.Solver(p, precision="MIXED")
    for s in (e.solvers[0], one):
        _init(fw, s, d, ph, 3)
    e.step(4)
    one.step(4)
    _same(e.solvers[0], one)
    for s in (e.solvers[0], one):
        if what == "T_brk":
            s.set_scalar("T_brk", 0.05)
        else:
            _init(fw, s, d, _case(fw, 9)[2], 4)
    e.step(6)
    one.step(6)
    _same(e.solvers[0], one)
    assert (one.get("AGE") > 0).any()
    one.close()
    e.close()


@pytest.mark.parametrize("what", ["T_brk", "init", "other", "workspace"])
def test_correct_run_after_a_change(fw, what):
    import torch
    p, d, ph = _case(fw, 1)
    net, ref = fw.learned.Net(seed=7), fw.learned.Net(seed=7)
    a, b = fw.Solver(p, precision="MIXED"), fw.Solver(p, precision="MIXED")
    for s in (a, b):
        _init(fw, s, d, ph, 3)

    def loop(s, n):
        for _ in range(n):
            s.step(1)
            ref.correct(s, wait=False)
        s.sync()

    net.correct_run(a, 4)
    loop(b, 4)
    _same(a, b)
    if what == "T_brk":
        for s in (a, b):
            s.set_scalar("T_brk", 0.05)
    elif what == "init":
        for s in (a, b):
            _init(fw, s, d, _case(fw, 9)[2], 4)
    elif what == "other":  # the same sizes, at the same addresses or not
        for s in (a, b):
            s.close()
        p, d, ph = _case(fw, 1, DX=1.25, DY=1.5)
        a = fw.Solver(p, precision="MIXED")
        _init(fw, a, d, ph, 5)
    else:
        net.forward(torch.zeros(2, 300, 400, 5, device="cuda"))
        torch.cuda.synchronize()
    net.correct_run(a, 6)
    if what == "other":
        b = fw.Solver(p, precision="MIXED")
        _init(fw, b, d, ph, 5)
    loop(b, 6)
    _same(a, b)
    assert (a.get("AGE") > 0).any()
    for x in (a, b, net, ref):
        x.close()
