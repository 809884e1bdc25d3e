"""The work a user of this package has it do, as cases that can be timed.

Each case is one pass through the public entry points: a stretch of time
steps with the output that a time loop takes after it, an exchange with a
host model, an ensemble, or the correction network.  Sizes come from the
package's benchmark configurations (250 x 500, 2048 x 2048, 4096 x 4096, the
ensemble's 128 x 256 to 1024 x 1024, the coarse 1024 x 1024 run) and from
odd and ragged grids of the same range; every solver case starts from a
developed sea (a sum of wave trains over the case's own bathymetry), so that
waves, breaking and the wet/dry front are there from the first step.

A pass of a solver case ends with the output fields in page-locked host
arrays, as a time loop with output has them: float in MIXED, double (and
MASK) in FP64.
"""
import ctypes
import math

import numpy as np
import torch

import __graft_entry__

G = 3  # ghost cells on each side
GRAV = 9.81


def _fw():
    return __graft_entry__.load_package()


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest calls: a time loop that looks at its output after
        # every step, on the ensemble's smallest grid; latency and launches
        {"name": "loop_128x256", "kind": "run", "bathymetry": "planar", "nx": 128, "ny": 256, "dx": 2.5,
         "precision": "MIXED", "calls": 1, "steps": 1, "stats": False, "tuned": False},
        # a planar beach between two outputs, the everyday small run
        {"name": "beach_250x500", "kind": "run", "bathymetry": "planar", "nx": 250, "ny": 500, "dx": 1.0,
         "precision": "MIXED", "calls": 1, "steps": 20, "stats": False, "tuned": False},
        # the same beach in double, the reference's arithmetic
        {"name": "beach_250x500_fp64", "kind": "run", "bathymetry": "planar", "nx": 250, "ny": 500, "dx": 1.0,
         "precision": "FP64", "calls": 1, "steps": 4, "stats": False, "tuned": False},
        # the benchmark's grid: an irregular directional sea over a shoal
        {"name": "shoal_2048", "kind": "run", "bathymetry": "shoal", "nx": 2048, "ny": 2048, "dx": 2.0,
         "precision": "MIXED", "calls": 1, "steps": 8, "stats": False, "tuned": True},
        # the largest: a barred beach with rip channels, wetting and drying
        {"name": "barred_4096", "kind": "run", "bathymetry": "barred", "nx": 4096, "ny": 4096, "dx": 1.0,
         "precision": "MIXED", "calls": 1, "steps": 4, "stats": False, "tuned": True},
        # a ragged walled grid in double
        {"name": "shoal_701x937_fp64", "kind": "run", "bathymetry": "shoal", "nx": 701, "ny": 937, "dx": 4.0,
         "precision": "FP64", "calls": 1, "steps": 2, "stats": False, "tuned": False},
        # a production run with its maxima, means, radiation stress and
        # roller kept, on a ragged grid, stepped call by call
        {"name": "stats_997x1501", "kind": "run", "bathymetry": "barred", "nx": 997, "ny": 1501, "dx": 1.0,
         "precision": "MIXED", "calls": 4, "steps": 1, "stats": True, "tuned": False},
        # a host model that exchanges the state at every step
        {"name": "coupled_1024", "kind": "coupled", "bathymetry": "shoal", "nx": 1024, "ny": 1024, "dx": 4.0,
         "precision": "MIXED", "tuned": True},
        # sixteen independent runs of uneven size advanced together
        {"name": "ensemble_16", "kind": "ensemble", "members": 16, "layout": 3, "steps": 4},
        # the correction network on the coarse grid of the learned run
        {"name": "net_forward_1024", "kind": "net_forward", "batch": 1, "h": 1024, "w": 1024},
        # a training iteration on a minibatch of coarse patches
        {"name": "net_train_8x128", "kind": "net_train", "batch": 8, "h": 128, "w": 128},
        # the coarse run with the network's correction after every step
        {"name": "learned_1024", "kind": "learned", "bathymetry": "barred", "nx": 1024, "ny": 1024, "dx": 2.0,
         "steps": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "run64", "coupled", "ensemble", "net_forward", "net_train",
                       "learned"])
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(2, 24), "layout": rng.randint(10, 10 ** 6),
                "steps": rng.randint(1, 4)}
    if kind == "net_forward":
        return {"kind": kind, "batch": rng.randint(1, 4), "h": _log(rng, 64, 1024), "w": _log(rng, 64, 1024)}
    if kind == "net_train":
        return {"kind": kind, "batch": rng.randint(1, 8), "h": _log(rng, 32, 256), "w": _log(rng, 32, 256)}
    bath = rng.choice(["planar", "shoal", "barred"])
    if kind == "learned":
        bath = "barred"
    top = {"run": 3000, "run64": 900, "coupled": 1600, "learned": 1100}[kind]
    nx, ny = _log(rng, 120, top), _log(rng, 64, top)
    # enough metres for the case's beach, at the grid spacing of its kind
    need = {"planar": 300.0, "shoal": 2600.0, "barred": 900.0}[bath]
    dx = round(max({"planar": 1.0, "shoal": 2.0, "barred": 1.0}[bath], need / nx), 3)
    if kind == "learned":
        return {"kind": kind, "bathymetry": bath, "nx": nx, "ny": ny, "dx": dx, "steps": rng.randint(1, 4)}
    if kind == "coupled":
        return {"kind": kind, "bathymetry": bath, "nx": nx, "ny": ny, "dx": dx, "precision": "MIXED",
                "tuned": rng.random() < 0.5}
    fp64 = kind == "run64"
    return {"kind": "run", "bathymetry": bath, "nx": nx, "ny": ny, "dx": dx,
            "precision": "FP64" if fp64 else "MIXED", "calls": 1 if fp64 else rng.randint(1, 3),
            "steps": rng.randint(1, 2) if fp64 else rng.randint(1, 6), "stats": rng.random() < 0.25,
            "tuned": rng.random() < 0.5}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _beach(case, rng):
    """(params, interior depth, JON_2D phases) of the case's bathymetry."""
    fw = _fw()
    b, nx, ny, dx = case["bathymetry"], case["nx"], case["ny"], case["dx"]
    seed = int(rng.integers(1 << 30))
    if b == "planar":
        return fw.cases.planar_beach(nx, ny, dx=dx, seed=seed)
    if b == "shoal":
        return fw.cases.shoal_jonswap(nx, ny, dx=dx, seed=seed)
    p, depth, phases, _ = fw.cases.barred_beach(nx, ny, dx=dx, seed=seed)
    return p, depth, phases


def _sea(p, depth, rng, hs):
    """Interior eta, u, v of eight wave trains toward the shore over the
    alongshore-mean depth: local wave numbers, heights limited to a quarter
    of the depth, nothing on land.  Alongshore wave numbers fit the domain,
    so a periodic run starts periodic."""
    nx, ny = depth.shape
    h = np.maximum(depth.mean(axis=1), 0.0)
    hw = np.maximum(h, 0.05)
    ly = ny * p["DY"]
    y = np.arange(ny) * p["DY"]
    left, right, ul, vl = [], [], [], []
    for _ in range(8):
        om = 2.0 * math.pi / rng.uniform(6.0, 12.0)
        k = om * om / GRAV / np.sqrt(np.tanh(om * om * hw / GRAV))
        ky = 2.0 * math.pi * int(rng.integers(-3, 4)) / ly
        ky = float(np.clip(ky, -0.5 * k.min(), 0.5 * k.min()))
        if p.get("PERIODIC"):
            ky = 2.0 * math.pi * round(ky * ly / (2.0 * math.pi)) / ly
        kx = np.sqrt(k * k - ky * ky)
        ph = np.cumsum(kx) * p["DX"] + rng.uniform(0.0, 2.0 * math.pi)
        a = np.where(h > 0.1, np.minimum(hs, 0.25 * h) / 8.0, 0.0) * rng.uniform(0.5, 1.0)
        for f, g in ((np.cos, np.cos), (np.sin, np.sin)):
            left.append(a * f(ph))
            ul.append(a * f(ph) * om * kx / (k * k * hw))
            vl.append(a * f(ph) * om * ky / (k * k * hw))
            right.append(g(ky * y))
    r = np.asarray(right)
    wet = depth > 0.1
    eta, u, v = (np.asfortranarray((np.asarray(m).T @ r) * wet) for m in (left, ul, vl))
    return eta, u, v


def _solver(case, seed):
    fw = _fw()
    rng = np.random.default_rng(seed)
    p, depth, phases = _beach(case, rng)
    if case.get("stats"):
        p.update({"OUT_Hmax": True, "OUT_Hmin": True, "OUT_Umax": True, "OUT_MFmax": True, "OUT_Umean": True,
                  "OUT_Radiation": True, "ROLLER": True, "STEADY_TIME": 0.0, "T_INTV_mean": 60.0})
    p = fw.with_defaults(p)
    eta, u, v = _sea(p, depth, rng, 1.0)
    s = fw.Solver(p, precision=case.get("precision", "MIXED"))
    s.init(depth, eta, u, v, phases)
    if case.get("tuned"):
        s.autotune()
    return s


class _Fields:
    """Page-locked host arrays of a solver's fields (x fastest), and the
    calls that fill them or send them: float arrays through the _f32 entry
    points in MIXED, double arrays and MASK otherwise."""

    def __init__(self, s, names):
        self.s, self.f32 = s, s.precision == "MIXED"
        self.t = {}
        for n in names:
            w, h = s.shape(n)
            dt = torch.int32 if n == "MASK" else torch.float32 if self.f32 else torch.float64
            self.t[n] = torch.zeros((h, w), dtype=dt, pin_memory=True)
        k = len(names)
        self.n = k
        self.names = (ctypes.c_char_p * k)(*[n.encode() for n in names])
        self.ptrs = (ctypes.c_void_p * k)(*[self.t[n].data_ptr() for n in names])

    def get(self):
        f = self.s.L.fw_get_fields_f32 if self.f32 else self.s.L.fw_get_fields
        self._check(f(self.s.ctx, self.n, self.names, self.ptrs))
        return dict(self.t)

    def put(self):
        f = self.s.L.fw_set_fields_f32 if self.f32 else self.s.L.fw_set_fields
        self._check(f(self.s.ctx, self.n, self.names, self.ptrs))

    def _check(self, rc):
        if rc != 0:
            raise _fw().FwError(rc)


_NET = [(8, 32), (32, 32), (32, 32), (32, 3)]  # channels; the first layer's five inputs padded to eight


def _net_params(rng, last=1.0):
    """He-scaled weights w[9][cin][cout] then b[cout], layer by layer."""
    out = []
    for k, (ci, co) in enumerate(_NET):
        real = 5 if k == 0 else ci
        w = rng.normal(0.0, math.sqrt(2.0 / (9 * real)), size=(9, ci, co))
        w[:, real:, :] = 0.0
        s = last if k == len(_NET) - 1 else 1.0
        out += [(s * w).ravel(), s * rng.normal(0.0, 0.05, size=co)]
    return np.concatenate(out).astype(np.float32)


def _net_inputs(case, seed):
    """(params, x, target, wmask): features of a sea over a slope with a dry
    shore, and targets of the corrections' size."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    b, h, w = case["batch"], case["h"], case["w"]

    def rand(*s):
        return torch.randn(*s, device="cuda", generator=g)

    ix = torch.linspace(0.0, 1.0, w, device="cuda").expand(b, h, w)
    iy = torch.linspace(0.0, 1.0, h, device="cuda")[None, :, None].expand(b, h, w)
    ph = rand(b, 1, 1)
    eta = 0.5 * torch.sin(40.0 * ix + 9.0 * iy + 6.0 * ph) + 0.05 * rand(b, h, w)
    u = 0.7 * eta + 0.02 * rand(b, h, w)
    v = 0.1 * torch.cos(30.0 * ix + 20.0 * iy + 3.0 * ph) + 0.02 * rand(b, h, w)
    dep = 10.0 - 11.0 * ix
    wet = (dep > 0.0).float()
    x = torch.stack([eta * wet, u * wet, v * wet, dep / 10.0, wet], dim=-1).contiguous()
    t = (rand(b, h, w, 3) * wet[..., None]).contiguous()
    return _net_params(np.random.default_rng(seed)), x, t, wet.contiguous()


def prepare(case, seed):
    fw = _fw()
    kind = case["kind"]
    if kind == "run":
        s = _solver(case, seed)
        names = ["Eta", "U", "V", "Ubar", "Vbar"] + ([] if s.precision == "MIXED" else ["MASK"])
        if case["stats"]:
            names += ["HeightMax", "MomentumFluxMax", "ETAmean", "Umean"]
        return {"case": case, "s": s, "out": _Fields(s, names)}
    if kind == "coupled":
        s = _solver(case, seed)
        f = _Fields(s, ["Eta", "U", "V", "Ubar", "Vbar"])
        f.get()
        return {"case": case, "s": s, "out": f}
    if kind == "ensemble":
        rng = np.random.default_rng(seed)
        members = []
        for p, depth, phases in fw.cases.ensemble_members(case["members"], seed=case["layout"]):
            members.append((p, depth, np.asfortranarray(rng.uniform(0.0, 2.0 * np.pi, size=phases.shape))))
        e = fw.Ensemble(members, precision="MIXED", single_launch=True)
        for s, (p, depth, phases) in zip(e.solvers, members):
            s.init(depth, *_sea(s.params, depth, rng, p["Hmo"]), phases)
        return {"case": case, "e": e, "out": [_Fields(s, ["Eta", "U"]) for s in e.solvers]}
    if kind == "learned":
        s = _solver(case, seed)
        net = fw.learned.Net(seed=1)
        # small corrections, as a trained network's: a few millimetres
        net.set_params(_net_params(np.random.default_rng(seed), last=0.1))
        return {"case": case, "s": s, "net": net, "out": _Fields(s, ["Eta", "U", "V", "Ubar", "Vbar"])}
    params, x, t, wet = _net_inputs(case, seed)
    net = fw.learned.Net(seed=1)
    net.set_params(params)
    return {"case": case, "net": net, "x": x, "t": t, "w": wet}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "run":
        for _ in range(case["calls"]):
            state["s"].step(case["steps"])
        return state["out"].get()
    if kind == "coupled":
        state["out"].put()
        state["s"].step(1)
        return state["out"].get()
    if kind == "ensemble":
        state["e"].step(case["steps"])
        return [f.get() for f in state["out"]]
    if kind == "learned":
        status = state["net"].correct_run(state["s"], case["steps"])
        if status != 0:
            raise _fw().FwError(status, "correct_run")
        return state["out"].get()
    if kind == "net_forward":
        return state["net"].forward(state["x"])
    loss = state["net"].loss_grad(state["x"], state["t"], state["w"])
    grads = state["net"].grads()
    state["net"].adam(1e-3)
    return {"loss": loss, "grads": grads}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _step_work(cells, precision):
    """Bytes and operations of one step: the three stages' 61 reals (the
    state, its copy of the step's start and the depths read, the state
    written) and 6 mask bytes of every cell, and about 5000 operations of
    the scheme's arithmetic."""
    return cells * (494.0 if precision == "FP64" else 250.0), cells * 5000.0


def work(case):
    kind = case["kind"]
    if kind in ("net_forward", "net_train"):
        px = float(case["batch"]) * case["h"] * case["w"]
        conv = 2.0 * 9 * (5 * 32 + 2 * 32 * 32 + 32 * 3)  # one forward pass, per pixel
        if kind == "net_forward":
            return {"bytes": px * 4 * (5 + 3), "flops": px * conv}
        return {"bytes": px * 4 * (5 + 3 + 1), "flops": px * (3.0 * conv - 2.0 * 9 * 5 * 32)}
    if kind == "ensemble":
        bytes_, flops = 0.0, 0.0
        for p, _, _ in _fw().cases.ensemble_members(case["members"], seed=case["layout"]):
            b, f = _step_work(float(p["Mglob"]) * p["Nglob"], "MIXED")
            out = 2 * 2 * 4 * (p["Mglob"] + 2 * G) * (p["Nglob"] + 2 * G)
            bytes_, flops = bytes_ + b * case["steps"] + out, flops + f * case["steps"]
        return {"bytes": bytes_, "flops": flops}
    cells = float(case["nx"]) * case["ny"]
    plane = float(case["nx"] + 2 * G) * (case["ny"] + 2 * G)
    b, f = _step_work(cells, case.get("precision", "MIXED"))
    if kind == "coupled":
        return {"bytes": b + 5 * 2 * 2 * 4 * plane, "flops": f}
    if kind == "learned":
        # the network's forward pass on every step: the state read, the corrected state written
        conv = 2.0 * 9 * (5 * 32 + 2 * 32 * 32 + 32 * 3)
        n = case["steps"]
        return {"bytes": n * (b + cells * 4 * (5 + 8)) + 5 * 2 * 4 * plane, "flops": n * (f + cells * conv)}
    n = case["calls"] * case["steps"]
    word = 8 if case["precision"] == "FP64" else 4
    # the statistics' running fields, read and written: 4 maxima, 11 of the
    # means, 12 sums of the radiation stress
    extra = cells * n * 2 * word * (4 + 11 + 12) if case["stats"] else 0.0
    nout = 5 + (4 if case["stats"] else 0)
    return {"bytes": n * b + extra + nout * 2 * word * plane, "flops": n * f}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _net64(params, x):
    """The network's output in float64; params a float64 tensor."""
    a = torch.nn.functional.pad(x.double(), (0, 3))
    off = 0
    for k, (ci, co) in enumerate(_NET):
        w = params[off:off + 9 * ci * co].reshape(9, ci, co)
        off += 9 * ci * co
        b = params[off:off + co]
        off += co
        h, wd = a.shape[1], a.shape[2]
        p = torch.nn.functional.pad(a, (0, 0, 1, 1, 1, 1))
        y = b
        for t in range(9):
            ky, kx = t // 3, t % 3
            y = y + p[:, ky:ky + h, kx:kx + wd] @ w[t]
        a = torch.relu(y) if k < len(_NET) - 1 else y
    return a


def exact(case, seed):
    # A solver step has no plain 64-bit form short of the whole scheme: the
    # solver cases' own FP64 mode is that scheme in 64 bits.
    if case["kind"] not in ("net_forward", "net_train"):
        return None
    params, x, t, wet = _net_inputs(case, seed)
    w = torch.from_numpy(params).cuda().double()
    if case["kind"] == "net_forward":
        return _net64(w, x)
    w.requires_grad_(True)
    d = _net64(w, x) - t.double()
    loss = (wet.double()[..., None] * d * d).sum() / wet.numel()
    loss.backward()
    grads = w.grad.clone()
    pad = grads[:9 * 8 * 32].view(9, 8, 32)
    pad[:, 5:, :] = 0.0
    return {"loss": float(loss), "grads": grads.cpu().numpy()}
