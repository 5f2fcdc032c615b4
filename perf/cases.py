"""What a user of this framework has it do, as cases that can be timed.

A tracking program keeps one MPBeam handle, advances the train turn by turn
(the drop-in calls cg_run_turns for one turn at a time) and reads the moments
of every bunch after each call; the macroparticles and the ion clouds stay on
the device and are fetched when somebody wants to see them.  The other two
kinds are the call for programs that own their particles (moments of a bunch
in the caller's device buffers) and one gradient of the field surrogate, the
work its training repeats.

The trains with ions run at bunch currents at which the ions oscillate
regularly (0.02 mA in the 80-bunch train, less in the long ones): near the
trapping threshold their motion over hundreds of passages is chaotic, and two
correct codes then agree in statistics only.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from cetasim_b200 import _abi, configs, surrogate
from cetasim_b200.beam import MPBeam

RINGS = {"plain_single": (1, 1, 1e5), "fast_ion": (20, 80, 2e4), "batched_uneven": (50, 900, None),
         "large_trapping": (50, 1000, 5e4)}  # sections, bunches, macroparticles per bunch


def listed():
    return [
        # a program that owns its particles asks for one bunch's moments each
        # turn: a bunch of the fast-ion train, and the largest accepted call
        {"name": "moments_bunch", "kind": "moments", "n": 20000},
        {"name": "moments_largest", "kind": "moments", "n": 1048576},
        # single-bunch short-range wake study: the smallest turn there is
        track("single_bunch", "plain_single", scale=1.0, ma=1.0),
        # fast-ion instability in a short train, 20 interaction points
        track("fast_ion_train", "fast_ion", scale=1.0, ma=0.02),
        # the benchmark's ragged 900-bunch train: ions at 50 points, HOM, FIR
        track("uneven_train", "batched_uneven", scale=1.0, ma=0.002),
        # trapped clouds round a uniform fill, SR and LR wakes, FIR
        track("trapped_clouds", "large_trapping", scale=0.2, ma=0.0002, clouds=200000),
        # space charge in each of 20 sections: the 2.5-D PIC and the
        # Bassetti-Erskine slices
        track("space_charge_pic", "fast_ion", scale=1.0, ma=0.125, ions=False, space_charge=2,
              mesh_x=32, mesh_y=32, slices=33),
        track("space_charge_slices", "fast_ion", scale=1.0, ma=0.125, ions=False, space_charge=1,
              mesh_x=32, mesh_y=32, slices=33),
        # broadband impedance with a one-turn map, from the impedance table
        # and from the wake table
        track("impedance_spectrum", "fast_ion", scale=1.0, ma=0.125, ions=False, sections=1,
              impedance="spectrum", rows=640, turns=4),
        track("impedance_wake", "fast_ion", scale=1.0, ma=0.125, ions=False, sections=1,
              impedance="wake", rows=400, turns=4),
        # beam loading, bin by bin: the main cavity and a passive harmonic one
        track("beam_loading", "batched_uneven", scale=0.1, ma=0.125, ions=False, sections=1,
              wakes=False, loading=True, rf_bins=40, turns=4),
        # one gradient of the surrogate's training batch
        {"name": "surrogate_gradient", "kind": "gradient", "n": 2048},
    ]


def track(name, ring, scale, ma, *, bunches=None, sections=None, ions=None, wakes=True, clouds=0,
          space_charge=0, mesh_x=0, mesh_y=0, slices=0, impedance="", rows=0, loading=False,
          rf_bins=0, turns=1):
    """One call of MPBeam.Run for `turns` turns: `ring` of configs.make with
    its macroparticle counts times `scale`, `ma` mA per bunch, its first
    `bunches` bunches and `sections` equal sections."""
    k, m, _ = RINGS[ring]
    d = {"kind": "track", "ring": ring, "scale": scale, "ma": ma, "bunches": bunches or m,
         "sections": sections or k, "ions": ring != "plain_single" if ions is None else ions,
         "wakes": wakes, "clouds": clouds, "space_charge": space_charge, "mesh_x": mesh_x,
         "mesh_y": mesh_y, "slices": slices, "impedance": impedance, "rows": rows,
         "loading": loading, "rf_bins": rf_bins, "turns": turns}
    return {"name": name, **d} if name else d


def draw(rng):
    def between(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["moments", "single", "fast_ion", "uneven", "trapped", "space_charge",
                       "impedance", "loading", "gradient"])
    if kind == "moments":
        return {"kind": "moments", "n": int(between(1000, 1048576))}
    if kind == "gradient":
        return {"kind": "gradient", "n": 128 * int(between(1, 128))}
    if kind == "single":
        return track("", "plain_single", between(0.02, 1.0), 1.0, turns=rng.randint(1, 16))
    if kind == "fast_ion":
        return track("", "fast_ion", between(0.02, 1.0), between(0.005, 0.02),
                     bunches=rng.randint(16, 80), turns=rng.randint(1, 3))
    if kind == "uneven":
        return track("", "batched_uneven", between(0.01, 0.5), between(0.0005, 0.002),
                     bunches=rng.randint(150, 900), sections=rng.choice([10, 20, 50]))
    if kind == "trapped":
        return track("", "large_trapping", between(0.01, 0.15), between(0.0001, 0.0002),
                     bunches=rng.randint(150, 1000), sections=rng.choice([10, 20, 50]),
                     clouds=int(between(5000, 150000)))
    if kind == "space_charge":
        return track("", "fast_ion", between(0.02, 1.0), 0.125, ions=False,
                     bunches=rng.randint(4, 80), space_charge=rng.choice([1, 2, 2, 3]),
                     mesh_x=rng.randint(12, 40), mesh_y=rng.randint(12, 40),
                     slices=rng.randint(7, 40))
    if kind == "impedance":
        spectrum = rng.random() < 0.5
        return track("", "fast_ion", between(0.02, 1.0), 0.125, ions=False, sections=1,
                     bunches=rng.randint(1, 80), impedance="spectrum" if spectrum else "wake",
                     rows=rng.randint(640, 1200) if spectrum else rng.randint(300, 600),
                     turns=rng.randint(1, 8))
    return track("", "batched_uneven", between(0.01, 0.2), 0.125, ions=False, sections=1,
                 bunches=rng.randint(80, 900), wakes=False, loading=True,
                 rf_bins=rng.randint(20, 100), turns=rng.randint(1, 8))


# ---- the train and its settings ---------------------------------------------

def workload(case, seed):
    ring, nb, k = case["ring"], case["bunches"], case["sections"]
    wl = configs.make(ring, n_scale=case["scale"], bunch_current=case["ma"] * 1e-3)
    wl.n_macro, wl.harm, wl.ne = wl.n_macro[:nb].copy(), wl.harm[:nb].copy(), wl.ne[:nb].copy()
    cfg = wl.cfg
    cfg.seed = seed
    lib = _abi.load()
    if k != cfg.n_sections:
        secs = configs.ring_sections(cfg.ring, k)
        if lib.cg_lattice_init(C.byref(cfg.ring), secs, k):
            raise RuntimeError("cg_lattice_init failed")
        wl.sections, cfg.sections, cfg.n_sections = secs, configs.C_cast(secs), k
    if not case["ions"]:
        cfg.flag_beam_ion = 0
    if not case["wakes"]:
        cfg.flag_sr_wake = cfg.flag_lr_wake = cfg.flag_fir = 0
    if case["space_charge"]:
        cfg.flag_sc = case["space_charge"]
        cfg.sc_mesh[:] = [case["mesh_x"], case["mesh_y"], case["slices"]]
    if case["impedance"] == "spectrum":
        wl.set_bbi(impedance_table(case["rows"]), 0)
    elif case["impedance"] == "wake":
        wl.set_bbi(wake_table(case["rows"]), 1)
    if case["loading"]:
        r = cfg.ring
        r.n_cav = 2
        r.cav_phase[0] = math.pi - math.asin(r.u0 / r.cav_vol[0]) - math.pi / 2
        r.cav_harm[1], r.cav_vol[1], r.cav_phase[1] = 3, 0.0, 0.0
        main = {"rf_mode": 1, "res_type": 1, "res_rs": 5e6, "res_q0": 2e4, "res_coupling": 2.0,
                "res_detune": -20e3, "res_excite": 1}
        passive = {"rf_mode": 1, "res_type": 0, "res_rs": 2e6, "res_q0": 1e4, "res_coupling": 0.0,
                   "res_detune": 150e3, "res_excite": 1, "res_cold": 1}
        for i, fields in enumerate((main, passive)):
            for name, v in fields.items():
                getattr(r, name)[i] = v
        r.rf_bunch_bins = case["rf_bins"]
        if lib.cg_config_derive(C.byref(cfg)):
            raise RuntimeError("cg_config_derive failed")
    return wl


def impedance_table(n, fmax=300e9):
    """A broadband resonator per plane, n frequencies up to fmax."""
    f = np.arange(n) * (fmax / (n - 1))
    t = np.zeros((n, 11))
    t[:, 0] = f
    with np.errstate(divide="ignore", invalid="ignore"):
        for p, (rs, fr) in enumerate(((2e4, 40e9), (4e5, 30e9), (4e5, 30e9), (1e5, 30e9), (1e5, 30e9))):
            z = rs / (1 + 1j * (fr / f - f / fr)) * (fr / f if p else 1.0)
            z[0] = 0
            t[:, 1 + p], t[:, 6 + p] = z.real, z.imag
    return t


def wake_table(nw, dz=0.5e-3, cen=40):
    """A smoothed damped oscillation on a grid through z = 0."""
    z = (np.arange(nw) - cen) * dz
    env = np.exp(-0.5 * (z / 1.5e-3) ** 2) + np.where(z > 0, np.exp(-z / 20e-3), 0.0)
    t = np.zeros((nw, 6))
    t[:, 0] = z
    for p, a in enumerate((3e13, 2e15, 2e15, 5e14, 5e14)):
        t[:, 1 + p] = a * env * np.cos(2 * np.pi * z / 6e-3 + 0.3 * p)
    t[cen, 0] = 0.0
    return t


MOMENTS = np.dtype([("n_alive", "i4"), ("n_macro", "i4"), ("mean", "f8", 6), ("emit", "f8", 3),
                    ("eff_emit", "f8", 3), ("rms_x", "f8"), ("rms_y", "f8"), ("eff_rms_x", "f8"),
                    ("eff_rms_y", "f8"), ("bunch_length", "f8"), ("energy_spread", "f8"),
                    ("z_min", "f8"), ("z_max", "f8"), ("transmission", "f8")])
PLANES = ("x", "px", "y", "py", "z", "dp")
CLOUD = ("coeff", "rms_x", "rms_y", "aver_x", "aver_y", "count")


class Tracked(dict):
    """A tracked train: the moments that the call brought back, and what it
    left on the device, which comes to the host when it is read: the
    particles, the number of ions at each section and the Gaussian of the
    cloud that each bunch met there (the ions themselves differ in number from
    input to input)."""

    def __init__(self, beam, moments):
        super().__init__((name, None) for name in PLANES + ("lost",))
        self.beam, self.host = beam, {}
        m = np.frombuffer(moments, dtype=MOMENTS)
        for name in MOMENTS.names:
            v = m[name]
            for i in range(v.shape[1] if v.ndim == 2 else 0):
                super().__setitem__("%s_%d" % (name, i), v[:, i])
            if v.ndim == 1:
                super().__setitem__(name, v)
        if beam.wl.cfg.flag_beam_ion:
            for name in ("ions",) + tuple("cloud_" + c for c in CLOUD):
                super().__setitem__(name, None)

    def fetch(self):
        b, h = self.beam, self.host
        h.update({name: [] for name, v in self.items() if v is None})
        for j in range(b.wl.n_bunches):
            c, lost = b.download(j)
            for q, name in enumerate(PLANES):
                h[name].append(c[q])
            h["lost"].append(lost)
        for k in range(b.wl.cfg.n_sections if "ions" in h else 0):
            h["ions"].append(np.array([len(b.ions(k)[0])]))
            rec = b.cloud_record(k)
            for q, name in enumerate(CLOUD):
                h["cloud_" + name].append(rec[:, 0, q])
        for name in h:
            h[name] = np.concatenate(h[name])

    def __getitem__(self, name):
        v = super().__getitem__(name)
        if v is None:
            if not self.host:
                self.fetch()
            v = self.host[name]
        return v


# ---- preparation and one pass -----------------------------------------------

def bunch(n, seed):
    """A Gaussian bunch off axis, a fiftieth of its particles lost."""
    rng = np.random.default_rng(seed)
    scale = np.array([1.4e-5, 1.4e-6, 6.3e-6, 6.3e-7, 2.5e-3, 9e-4])[:, None]
    off = scale * rng.normal(0.0, 0.2, (6, 1))
    return rng.normal(0.0, 1.0, (6, n)) * scale + off, (rng.random(n) < 0.02).astype(np.uint8)


def batch(n, seed):
    """The surrogate's initial weights and a training batch: positions and
    aspect ratios with the field of the Gaussian at them, from
    G_x = x/2 Int_0^1 exp(-u x^2/2 - u y^2/(2 q)) q^(-1/2) du,
    G_y = y/2 Int_0^1 exp(...) q^(-3/2) du, q = 1 - u (1 - r^2)."""
    rng = np.random.default_rng(seed)
    w = []
    for count, fan_in in ((192, 3), (64, 3), (4096, 64), (64, 64), (4096, 64), (64, 64), (128, 64), (2, 64)):
        w.append(rng.uniform(-1, 1, count) / math.sqrt(fan_in))
    x = rng.random((n, 3))
    x[:, 2] = np.where(rng.random(n) < 0.5, 0.05 ** (1 - x[:, 2]), 0.05 + 0.95 * x[:, 2])
    x = x.astype(np.float32)
    a, b, r = x.astype(np.float64).T
    px, py = 8 * a, 8 * b * r
    nodes, weights = np.polynomial.legendre.leggauss(96)
    gx, gy = np.zeros(n), np.zeros(n)
    for s, ws in zip(nodes, weights):
        u = 0.5 * (s + 1)
        q = 1 - u * (1 - r * r)
        e = 0.5 * ws * np.exp(-u * px * px / 2 - u * py * py / (2 * q)) / np.sqrt(q)
        gx += 0.5 * px * e
        gy += 0.5 * py * e / q
    return np.concatenate(w).astype(np.float32), x, np.stack([gx, gy], 1).astype(np.float32)


def prepare(case, seed):
    if case["kind"] == "gradient":
        return {"kind": "gradient", "batch": batch(case["n"], seed)}
    if case["kind"] == "moments":
        coords, lost = bunch(case["n"], seed)
        out = torch.zeros(MOMENTS.itemsize, dtype=torch.uint8, device="cuda")
        return {"kind": "moments", "n": case["n"], "lib": _abi.load(),
                "coords": torch.from_numpy(coords).cuda(), "lost": torch.from_numpy(lost).cuda(),
                "out": out, "read": {"alive": out[:8].view(torch.int32),
                                     **dict(zip(FIELDS, out[8:].view(torch.float64)))}}
    beam = MPBeam(workload(case, seed))
    beam.generate(seed)
    if case["clouds"]:
        for k, cloud in enumerate(configs.preload_clouds(beam.wl, case["clouds"], seed)):
            beam.upload_ions(k, 0, *cloud)
    return {"kind": "track", "beam": beam, "turn": 0, "turns": case["turns"]}


def run(state):
    if state["kind"] == "gradient":
        loss, grad = surrogate.gradient(*state["batch"])
        return {"loss": np.float64(loss), **layers(grad)}
    if state["kind"] == "moments":
        rc = state["lib"].cg_bunch_moments_noalloc(
            state["coords"].data_ptr(), state["n"], state["lost"].data_ptr(), state["n"], 10.0, 10.0,
            state["out"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        if rc:
            raise _abi.CgError(rc, "cg_bunch_moments_noalloc")
        return state["read"]
    state["beam"].Run(state["turn"], state["turns"])
    state["turn"] += state["turns"]
    return Tracked(state["beam"], state["beam"].moments())


FIELDS = tuple("mean_" + p for p in PLANES) + tuple("emit_" + p for p in "xyz") + tuple(
    "eff_emit_" + p for p in "xyz") + ("rms_x", "rms_y", "eff_rms_x", "eff_rms_y", "bunch_length",
                                       "energy_spread", "z_min", "z_max", "transmission")


def layers(g):
    cuts = {"w1": 192, "b1": 256, "w2": 4352, "b2": 4416, "w3": 8512, "b3": 8576, "w4": 8704, "b4": 8706}
    out, at = {}, 0
    for name, to in cuts.items():
        out[name], at = g[at:to], to
    return out


# ---- what a pass cannot do without -------------------------------------------

def work(case):
    n = case["n"] if case["kind"] != "track" else 0
    if case["kind"] == "moments":
        return {"bytes": 49.0 * n + MOMENTS.itemsize, "flops": 30.0 * n}
    if case["kind"] == "gradient":  # forward and two backward products of 8512 weights
        return {"bytes": 20.0 * n + 8 * 8706, "flops": 6 * 8512.0 * n}
    k, m = case["sections"], case["bunches"]
    per = RINGS[case["ring"]][2]
    n = m * max(1, int(per * case["scale"])) if per else int(
        configs.make(case["ring"], n_scale=case["scale"]).n_macro[:m].sum())
    # per particle and section: the map, the moments, the ion kick (two w(z)),
    # the space charge; per turn the longitudinal tail and the wakes
    flops = n * (k * (110.0 + 30.0 + (438.0 if case["ions"] else 0.0) + (90.0 if case["space_charge"] else 0.0)) + 250.0)
    if case["ions"]:
        flops += k * 438.0 * (m * m / 2 + m * case["clouds"])
    # the beam read and written in each section (97 B a particle with its
    # flag) and once more in the turn's tail, by bunches that share no cache
    return {"bytes": case["turns"] * 97.0 * n * (k + 1), "flops": case["turns"] * flops}


# ---- the same in 64 bits by plain numpy ----------------------------------------

def exact(case, seed):
    if case["kind"] == "moments":
        return exact_moments(*bunch(case["n"], seed))
    if case["kind"] == "gradient":
        return exact_gradient(*batch(case["n"], seed))
    return None  # many coupled stages per turn: no plain restatement of this size


def exact_moments(c, lost):
    alive = lost == 0
    v = c[:, alive].astype(np.longdouble)
    mean = v.mean(axis=1)
    d = v - mean[:, None]
    m2 = [[(d[i] * d[j]).mean() for j in range(6)] for i in range(6)]
    out = {"alive": None}
    out.update({"mean_" + p: np.float64(mean[i]) for i, p in enumerate(PLANES)})
    emit, eff = [], []
    for i in (0, 2, 4):
        a, b, ab = m2[i][i], m2[i + 1][i + 1], m2[i][i + 1]
        emit.append(np.sqrt(a * b - ab * ab))
        ra, rb, rab = a + mean[i] ** 2, b + mean[i + 1] ** 2, ab + mean[i] * mean[i + 1]
        eff.append(np.sqrt(ra * rb - rab * rab))
    for i, p in enumerate("xyz"):
        out["emit_" + p], out["eff_emit_" + p] = np.float64(emit[i]), np.float64(eff[i])
    for i, p in enumerate("xy"):
        out["rms_" + p], out["eff_rms_" + p] = np.float64(np.sqrt(emit[i] * 10)), np.float64(np.sqrt(eff[i] * 10))
    out["bunch_length"], out["energy_spread"] = np.float64(np.sqrt(m2[4][4])), np.float64(np.sqrt(m2[5][5]))
    z = np.append(c[4, alive], c[4, 0])
    out["z_min"], out["z_max"] = z.min() - 1e-6, z.max() + 1e-6
    out["transmission"] = alive.sum() / len(lost)
    return out


def bf16(a):
    return torch.from_numpy(a).to(torch.bfloat16).double().numpy()


def exact_gradient(w, x, t):
    p = layers(w)
    n = len(x)
    w1, w2, w3, w4 = (bf16(p[k]).reshape(s) for k, s in (("w1", (64, 3)), ("w2", (64, 64)), ("w3", (64, 64)), ("w4", (2, 64))))
    b1, b2, b3, b4 = (p[k].astype(np.float64) for k in ("b1", "b2", "b3", "b4"))
    a, b, r = x.astype(np.float64).T
    x0 = np.stack([2 * a - 1, 2 * b - 1, 2 * np.log(r / 0.05) / math.log(20.0) - 1], 1)

    def silu(z):
        s = 1 / (1 + np.exp(-z))
        return z * s, s * (1 + z * (1 - s))

    h1, g1 = silu(x0 @ w1.T + b1)
    h2, g2 = silu(h1 @ w2.T + b2)
    h3, g3 = silu(h2 @ w3.T + b3)
    odd = np.stack([a, b], 1)
    e = (h3 @ w4.T + b4) * odd - t
    d4 = e * odd / n
    d3 = (d4 @ w4) * g3
    d2 = (d3 @ w3) * g2
    d1 = (d2 @ w2) * g1
    return {"loss": np.float64((e * e).sum() / (2 * n)), "w1": (d1.T @ x0).ravel(), "b1": d1.sum(0),
            "w2": (d2.T @ h1).ravel(), "b2": d2.sum(0), "w3": (d3.T @ h2).ravel(), "b3": d3.sum(0),
            "w4": (d4.T @ h3).ravel(), "b4": d4.sum(0)}
