"""The work that a user of the engine has it do, as cases that can be timed.

Every case goes through the public entry points of sevc.py / calibrate.py
(the ctypes mirror of include/sevc.h), from the inputs a program holds to
the host arrays it gets back.  Kinds:

  step       one sevc_step and a read-back of the mesh: a program that
             drives the engine step by step
  run        the steps between two snapshots (sevc_run), the last of them a
             snapshot step, then the mesh read back
  gate       the same past the 5/6 nucleation gate: removals, flips and
             nucleation attempts in every interval
  batch      the same for a batched handle (many small microstructures)
  whole      a whole small job: create, run, read back, destroy
  adjoint    forward steps on the tape, the area histogram and its gradients
  calibrate  one iteration of the calibration loop on a batch, from its
             checkpoint
  monitor    the statistics, histogram and invariant check of a running mesh

Meshes are periodic Voronoi diagrams of uniform seeds from the library's
generator; grains are about one unit across (domain sqrt(n), as in the
reference's example.ini) unless a case is on the unit square.
"""
import math
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "se-grain-growth-gpu_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import calibrate  # noqa: E402
import sevc  # noqa: E402

NBINS, AMAX = 64, 4.0


def listed():
    return [
        # the smallest call: a 300-grain mesh (the test fixtures' size) stepped
        # from a host loop that looks at the mesh after each step
        {"name": "step_300", "kind": "step", "n": 300, "gb_eps": 0.0, "dt": 1e-4},
        # the same at the size of one ensemble member, odd count, anisotropic
        # boundaries (GB_eps = 0.02: every boundary energy a cos^3)
        {"name": "step_20k_aniso", "kind": "step", "n": 20011, "gb_eps": 0.02, "dt": 1e-4},
        # the reference's own example: 2,000 grains, dt 1e-4, stored energy
        # 3..6, a snapshot every 100 steps
        {"name": "run_2k", "kind": "run", "n": 2000, "steps": 100, "dt": 1e-4, "se": "triangular"},
        # the benchmark's microstructure, 1M grains, one snapshot interval
        # at the start of the run (hardly any events)
        {"name": "run_1m", "kind": "run", "n": 1000000, "steps": 100, "dt": 2e-4, "se": "lognormal"},
        # past the 5/6 gate with stored energies for which nucleations are
        # accepted (one attempt every 5 steps), 100,000 grains
        {"name": "gate_100k", "kind": "gate", "n": 100003, "steps": 50, "dt": 1e-3, "se": "triangular", "gap": 5,
         "mc_k": 3.0},
        # past the gate in the benchmark's regime (lognormal stored energy,
        # one attempt every 10 steps), 400,000 grains, about as many events
        # per step as the benchmark's window
        {"name": "gate_400k", "kind": "gate", "n": 400000, "steps": 50, "dt": 2e-3, "se": "lognormal", "gap": 10,
         "mc_k": 1.0},
        # an ensemble of small microstructures in one handle (unit square,
        # dt 1e-6, stored energy U[0, 0.5])
        {"name": "batch_64", "kind": "batch", "ninst": 64, "lo": 500, "hi": 5000, "steps": 20, "dt": 1e-6},
        # a whole small job, with what every new handle pays for
        {"name": "whole_5k", "kind": "whole", "n": 5003, "steps": 50, "dt": 1e-4, "se": "uniform"},
        # gradients of the grain-size histogram: the benchmark's 10,000-grain
        # differentiable workload, a window of 100 steps
        {"name": "adjoint_10k", "kind": "adjoint", "n": 10000, "steps": 100, "every": 50, "dt": 4e-6},
        # one calibration iteration on a batch (the calibration test's sizes)
        {"name": "calibrate_16x2k", "kind": "calibrate", "ninst": 16, "lo": 1500, "hi": 2500, "steps": 40,
         "dt": 2e-4},
        # a running mesh looked at between steps: small and large
        {"name": "monitor_2k", "kind": "monitor", "n": 2000},
        {"name": "monitor_500k", "kind": "monitor", "n": 500009},
    ]


def _log_size(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi)))) | 1


def draw(rng):
    kind = rng.choice(["step", "run", "run", "gate", "batch", "whole", "adjoint", "calibrate", "monitor"])
    if kind == "step":
        return {"kind": kind, "n": _log_size(rng, 128, 60000), "gb_eps": rng.choice([0.0, 0.02]),
                "dt": rng.choice([1e-4, 2e-4])}
    if kind == "run":
        n = _log_size(rng, 300, 700000)
        return {"kind": kind, "n": n, "steps": rng.choice([20, 50, 100]), "dt": rng.choice([1e-4, 2e-4]),
                "se": rng.choice(["triangular", "lognormal", "uniform"])}
    if kind == "gate":
        return {"kind": kind, "n": _log_size(rng, 5000, 300000), "steps": rng.choice([20, 50]), "dt": 2e-3,
                "se": "lognormal", "gap": rng.choice([5, 10]), "mc_k": 1.0}
    if kind == "batch":
        lo = rng.choice([100, 500, 1000])
        return {"kind": kind, "ninst": _log_size(rng, 4, 128), "lo": lo, "hi": lo * rng.choice([2, 5]),
                "steps": rng.choice([10, 20]), "dt": 1e-6}
    if kind == "whole":
        return {"kind": kind, "n": _log_size(rng, 300, 30000), "steps": rng.choice([20, 50]), "dt": 1e-4,
                "se": "uniform"}
    if kind == "adjoint":
        return {"kind": kind, "n": _log_size(rng, 1000, 30000), "steps": rng.choice([40, 60, 100]),
                "every": rng.choice([20, 50]), "dt": 4e-6}
    if kind == "calibrate":
        lo = rng.choice([500, 1000])
        return {"kind": kind, "ninst": _log_size(rng, 4, 24), "lo": lo, "hi": 2 * lo, "steps": rng.choice([20, 40]),
                "dt": 2e-4}
    return {"kind": kind, "n": _log_size(rng, 1000, 400000)}


def _mesh(n, seed, se="uniform"):
    m = sevc.voronoi(n, seed + 1, "triangular" if se == "triangular" else "uniform")
    if se == "lognormal":
        m["se"] = np.random.default_rng(seed).lognormal(-1.0, 0.5, n)
    return m


def _options(n, dt, domain, snap_gap=10 ** 8, gb_eps=0.0, nucleation=None):
    """nucleation: None or (gap, MC_k); stored energies are used as given"""
    gap, mc_k = nucleation if nucleation else (0, 1.0)
    o = sevc.default_options(n_grains=n, dt=dt, dtau=gap * dt if nucleation else 1.0, nucleation_gap=gap,
                             domain_bound=domain, GB_eps=gb_eps, GB_scaling=1.0, SE_eps=1.0, SE_min=999.0,
                             SE_max=999.0, do_nucleation=1 if nucleation else 0, MC_k=mc_k, nmax=10 ** 8, tmax=-1,
                             snap_gap=snap_gap, n_blocks=32, n_threads=256)
    o.min_grains = -1
    return o


def _engine(opt, m):
    return sevc.Engine.from_arrays(opt, m["xy"], m["ridges"], m["oris"], m["se"])


def _batch_meshes(case, seed, scale):
    # the sizes belong to the case, the microstructures to the seed
    sizes = np.random.default_rng(case["ninst"]).integers(case["lo"], case["hi"] + 1, case["ninst"])
    meshes = [sevc.voronoi(int(n), seed * 1009 + i) for i, n in enumerate(sizes)]
    for m in meshes:
        m["se"] = m["se"] * scale
    return meshes


class _Calibration(calibrate.Calibration):
    def __del__(self):   # its checkpoint file goes with it
        if getattr(self, "ckpt", None) and os.path.exists(self.ckpt):
            self.close()


def prepare(case, seed):
    kind, s = case["kind"], {"case": case}
    if kind == "step":
        m = _mesh(case["n"], seed, "triangular")
        s["eng"] = _engine(_options(case["n"], case["dt"], math.sqrt(case["n"]), gb_eps=case["gb_eps"]), m)
    elif kind in ("run", "gate"):
        n, k = case["n"], case["steps"]
        m = _mesh(n, seed, case["se"])
        nucl = (case["gap"], case["mc_k"]) if kind == "gate" else None
        s["eng"] = _engine(_options(n, case["dt"], math.sqrt(n), snap_gap=k, nucleation=nucl), m)
        info = s["eng"].step()          # step 0 is a snapshot step: intervals of k steps follow, each ending in one
        if kind == "gate":
            while info.curr_n_grains > 5 * n // 6:
                info = s["eng"].run(k)[-1]
            s["eng"].run(k)             # an interval past the gate: attempts have begun
    elif kind == "batch":
        meshes = _batch_meshes(case, seed, 0.5)
        o = _options(len(meshes[0]["oris"]), case["dt"], 1.0, snap_gap=case["steps"])
        s["eng"] = sevc.Engine.from_batch(o, meshes)
        s["eng"].step()
    elif kind == "whole":
        s["mesh"] = _mesh(case["n"], seed, case["se"])
        s["opt"] = _options(case["n"], case["dt"], math.sqrt(case["n"]), snap_gap=case["steps"] - 1)
    elif kind == "adjoint":
        m = _mesh(case["n"], seed)
        m["se"] = m["se"] * 0.5
        s["eng"] = _engine(_options(case["n"], case["dt"], 1.0), m)
        s["w"] = np.linspace(1.0, -1.0, NBINS) / NBINS
    elif kind == "calibrate":
        meshes = _batch_meshes(case, seed, 1.0)
        domain = math.sqrt(sum(len(m["oris"]) for m in meshes) / len(meshes))
        s["cal"] = _Calibration(meshes, case["dt"], case["steps"], checkpoint_every=20, domain=domain)
        s["target"] = s["cal"].histogram(1.0, 1.0, 1.0)
    else:
        m = _mesh(case["n"], seed, "lognormal")
        s["eng"] = _engine(_options(case["n"], 2e-4, math.sqrt(case["n"])), m)
        s["eng"].run(3)
    return s


# what a step reports, beside its own times and launch count
_INFO = ("n", "curr_n_grains", "n_flips", "n_removals", "n_two_three", "n_nucleations", "n_conflicts",
         "polling_iters", "nucleation_attempted", "outputs_complete")


def _infos(infos):
    return {f: np.array([getattr(i, f) for i in infos], np.int64) for f in _INFO} | {
        "nucleated_area": np.array([i.nucleated_area for i in infos])}


def _state(eng, complete):
    """The mesh on the host.  Extinction times and dA/dt of entities that no
    event can reach are computed on snapshot steps only (outputs_complete):
    after another step they are not outputs."""
    st = eng.get_state()
    if not complete:
        del st["btext"], st["gdadt"]
    return st


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        info = s["eng"].step()
        return {"info": _infos([info]), "state": _state(s["eng"], False)}
    if kind in ("run", "gate", "batch"):
        infos = s["eng"].run(case["steps"])
        return {"info": _infos(infos), "state": _state(s["eng"], True)}
    if kind == "whole":
        eng = _engine(s["opt"], s["mesh"])
        infos = eng.run(case["steps"])
        st = _state(eng, True)
        eng.close()
        return {"info": _infos(infos), "state": st}
    if kind == "adjoint":
        eng = s["eng"]
        eng.tape_start(case["every"])
        infos = eng.run(case["steps"])
        hist = eng.area_histogram(NBINS, AMAX)
        gse, ggb, gmu = eng.adjoint_histogram(NBINS, AMAX, s["w"])
        eng.tape_stop()
        return {"info": _infos(infos), "hist": hist, "grad_se": gse, "grad_gb": ggb, "grad_mu": gmu}
    if kind == "calibrate":
        loss, grad = s["cal"].loss_and_grad(1.3, 0.8, 0.6, s["target"])
        return {"loss": loss, "grad": grad}
    eng = s["eng"]
    return {"stats": eng.grain_stats(), "hist": eng.area_histogram(NBINS, AMAX), "violations": eng.check_data()}


# Per grain of a mesh of V = 2G vertices and B = 3G boundaries: a step reads
# and writes each field once (72 V + 25 B + 20 G + 4 per list entry), the
# host copy is every field of the mesh, and a step cannot do without about
# 400 binary64 operations (the two finite-difference passes).
_STEP_BYTES, _STATE_BYTES, _STEP_FLOPS = 263, 734, 400


def work(case):
    kind = case["kind"]
    if kind in ("batch", "calibrate"):
        n = case["ninst"] * (case["lo"] + case["hi"]) / 2
    else:
        n = case["n"]
    k = case.get("steps", 1)
    if kind in ("step", "run", "gate", "batch", "whole"):
        return {"bytes": n * (k * _STEP_BYTES + _STATE_BYTES), "flops": n * k * _STEP_FLOPS}
    if kind in ("adjoint", "calibrate"):   # forward, replay, backward
        return {"bytes": 3 * n * k * _STEP_BYTES, "flops": 3 * n * k * _STEP_FLOPS}
    # each pass reads the lists, the positions, and for the check the slots
    return {"bytes": n * (3 * (24 + 2 * 16) + 2 * 32 + 3 * 8), "flops": n * 100}


# ---- the same values in 64 bits, by plain numpy ----

def _wrap(d, D):
    return d - D * np.round(d / D)


def _polygons(st, D):
    """Every enabled grain's unwrapped polygon as padded arrays (its list
    closed on the first vertex, repeated to the end): x, y of (grains, most
    sides + 1), and the signed areas."""
    n = st["gvlen"]
    w = int(n.max()) + 1
    L = st["glist"].reshape(-1, sevc.MAXV)[:, :min(w, sevc.MAXV)]
    if L.shape[1] < w:
        L = np.concatenate([L, L[:, :1]], axis=1)
    col = np.arange(w)[None, :]
    L = np.where(col < n[:, None], L, L[:, :1])
    L = np.where(L < 0, 0, L)
    x, y = st["px"][L], st["py"][L]
    z = np.zeros((len(n), 1))
    ax = np.concatenate([z, np.cumsum(_wrap(np.diff(x, axis=1), D), axis=1)], axis=1)
    ay = np.concatenate([z, np.cumsum(_wrap(np.diff(y, axis=1), D), axis=1)], axis=1)
    area = 0.5 * np.sum(ax[:, :-1] * ay[:, 1:] - ay[:, :-1] * ax[:, 1:], axis=1)
    return L, area


def _exact_step(s, case):
    """Arclengths, boundary energies, areas and the moved positions of one
    step from the mesh it starts on: the gradient of the energy instead of
    the difference quotient.  Vertices that an event moves are not followed
    (a few, by less than a short edge)."""
    D, eps = s["eng"].opt.domain_bound, case["gb_eps"]
    st = s["eng"].get_state()
    a, b = st["bini"], st["bend"]
    dx, dy = _wrap(st["px"][b] - st["px"][a], D), _wrap(st["py"][b] - st["py"][a], D)
    length = np.hypot(dx, dy)
    vg = st["vg"].reshape(-1, 3)
    ga, gb = vg[a], vg[b]
    shared = (ga[:, :, None] == gb[:, None, :]).any(axis=2)
    two = np.sort(np.where(shared, ga, -1), axis=1)[:, 1:]
    gamma = 1 + 0.5 * eps * (1 - np.cos(4 * (st["gori"][two[:, 0]] - st["gori"][two[:, 1]])) ** 3)
    L, area = _polygons(st, D)
    # dE/dx: line tension of the three boundaries, then the stored energy
    gx, gy = np.zeros_like(st["px"]), np.zeros_like(st["px"])
    for end, sign in ((a, -1.0), (b, 1.0)):
        np.add.at(gx, end, sign * gamma * dx / length)
        np.add.at(gy, end, sign * gamma * dy / length)
    n = st["gvlen"]
    c = st["gse"] * np.sign(area)
    for p in range(int(n.max())):
        g = np.nonzero(p < n)[0]
        v, nx, pv = L[g, p], L[g, (p + 1) % n[g]], L[g, (p - 1) % n[g]]
        hx = _wrap(st["px"][nx] - st["px"][v], D) + _wrap(st["px"][v] - st["px"][pv], D)
        hy = _wrap(st["py"][nx] - st["py"][v], D) + _wrap(st["py"][v] - st["py"][pv], D)
        np.add.at(gx, v, 0.5 * c[g] * hy)
        np.add.at(gy, v, -0.5 * c[g] * hx)
    px, py = (st["px"] - case["dt"] * gx) % D, (st["py"] - case["dt"] * gy) % D
    known = {"px": px, "py": py, "blen": length, "benergy": gamma, "garea": area}
    out = {f: known.get(f) for f in st if f not in ("btext", "gdadt")}
    return {"info": {f: None for f in _INFO + ("nucleated_area",)}, "state": out}


def _exact_monitor(s):
    D = s["eng"].opt.domain_bound
    st = s["eng"].get_state()
    on = st["gen"] > 0
    area, sides = np.abs(_polygons(st, D)[1])[on], st["gvlen"][on]
    t = area * on.sum() / (D * D) / (AMAX / NBINS)
    hist = np.zeros(NBINS)
    for k in range(NBINS):
        d = np.abs(t - k - 0.5)
        hist[k] = np.sum(np.where(d <= 0.5, 0.75 - d * d, np.where(d <= 1.5, 0.5 * (1.5 - d) ** 2, 0.0)))
    stats = {"n_grains": int(on.sum()), "n_three_sided": int((sides == 3).sum()), "mean_area": float(area.mean()),
             "std_area": float(area.std()), "min_area": float(area.min()), "max_area": float(area.max()),
             "mean_sides": float(sides.mean())}
    return {"stats": stats, "hist": hist / on.sum(), "violations": None}


def exact(case, seed):
    """The steps of the longer cases follow hundreds of discrete events: no
    plain restatement of them runs in a few seconds."""
    if case["kind"] == "step":
        return _exact_step(prepare(case, seed), case)
    if case["kind"] == "monitor":
        return _exact_monitor(prepare(case, seed))
    return None
