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


@pytest.mark.parametrize("precision", ["MIXED", "FP64"])
@pytest.mark.parametrize("name", ["post_mask_break", "break_a"])
def test_breaking_candidates_do_not_pile_up(fw, name, precision):
    """Every cell a candidate of the breaking sweep (0.35 sqrt(g H) <= ETAT <
    0.65 sqrt(g H), AGE 0), launched 60 times without the sweep: the list
    keeps to its place in memory, and the run goes on as after two launches."""
    p, depth, phases, _ = fw.cases.barred_beach(200, 24, 1.0, seed=3, wk_from_shore=120.0, shore_from_east=40.0)
    depth = np.asfortranarray(np.full_like(depth, 1.0))
    p = fw.with_defaults(p)
    sea = fw.cases.random_state(*depth.shape, seed=6)
    got = []
    for reps in (1, 59):
        s = fw.Solver(p, precision=precision)
        s.init(depth, *sea, phases)
        s.step(4)
        s.set("ETAT", np.full(s.shape("ETAT"), 1.5))
        s.set("AGE", np.zeros(s.shape("AGE")))
        s.time_kernel(name, reps)
        s.step(6)
        got.append([s.get(n) for n in ("Eta", "U", "V", "AGE", "nu_break", "MASK")])
        s.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    assert np.abs(got[0][0]).max() > 0


@pytest.mark.parametrize("precision", ["MIXED", "FP64"])
def test_update_is_timed_as_a_step_runs_it(fw, precision):
    """JON_2D: a step takes the wavemaker's mass from k_wm_band, so k_update's
    time does not grow with the frequencies (summed in every band cell, 4000 of
    them take tens of times the kernel's few microseconds)."""
    times = []
    for nf in (2, 4000):
        p, depth, phases, _ = fw.cases.barred_beach(200, 24, 1.0, seed=3, wk_from_shore=120.0, shore_from_east=40.0,
                                                    nfreq=nf, ntheta=1)
        s = fw.Solver(fw.with_defaults(p), precision=precision)
        s.init(depth, phases=phases)
        s.step(2)
        assert 0 < s.scalar("ihi") - s.scalar("ilo") < 200
        times.append(min(s.time_kernel("update", 20) for _ in range(3)))
        s.close()
    assert times[1] < 2.0 * times[0], times
