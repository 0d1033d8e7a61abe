"""Performance cases: the calls a user of this framework makes, at the sizes
they are made in earnest, through its public entry points.

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  the objects a program holds before the call
    run(state)           one pass through the entry point, and its outputs
    work(case)           bytes and operations one pass cannot do without
    exact(case, seed)    the outputs in plain float64 torch

Every case is a machine study on one lattice, the 12-sector scaling FFA of
the benchmark (300 MeV protons, k = 7.6, r 8.0-9.3 m at 1 mm, 0.005 degrees
of azimuth per map node).  The kinds:

    push   Pusher.push: a bunch through `steps` fused steps on the device
    step   FFAG_RungeKutta.Boris_solve: one step of a host matrix
    host   MatrixTracker.run: a host matrix through `steps` steps and back
    sc     SpaceCharge.update: one 2.5D space-charge update
    map    LearnedSectorMap.apply: learned sector maps on a bunch
    train  Trainer.graph_step: one optimiser step of the learned map
    orbit  SectorTracker.run: azimuth-domain tracks (closed orbits, tunes)
"""
from __future__ import annotations

import math

import numpy as np
import torch

# ------------------------------------------------------------------ machine
Q, C = 1.60217662e-19, 2.99792458e8
E0_MEV = 938.2723
E0 = E0_MEV * 1e6 * Q
M0 = E0 / C ** 2
EPS0 = 8.854187817e-12
B0, K, NSEC = 1.4369567177144435e-07, 7.6, 12
PERIOD = 2 * math.pi / NSEC
RMIN, RMAX, DR, DTH = 8.0, 9.3, 0.001, math.radians(0.005)
NR, NTH = 1301, 6000
ORDERS = 4
# flutter magnets: start, end, fringe [rad], signed amplitude
MAGNETS = [(0.1308996938995747, 0.2945243112740431, 0.19144080232812802, 1.0),
           (0.3436116964863836, 0.39269908169872414, 0.05743224069843841, -1.3)]
# closed orbit at 300 MeV, azimuth 0, and its revolution time
R_CO, PR_CO, T_REV = 8.12743880049872, 0.11755478732238835, 2.677375361028528e-07
DT = T_REV / 720
GAPS, GAP_WIDTH, VOLTAGE = (3.75, 183.75), 0.2, 100e3
APERTURE = (7.5, 9.5, -0.1, 0.1)
COLS = {"r": 0, "vr": 1, "z": 2, "vz": 3, "fi": 4, "f5": 5, "rf": 9, "esc_r": 10, "esc_z": 11, "esc_fi": 12}
FLAGS = {"inj": 7, "surv": 8}
SC_STEPS = 60            # steps between space-charge updates (12 updates a turn)
DEV = "cuda"
_kept = {}


def momentum(ek):
    return math.sqrt((ek * 1e6 * Q + E0) ** 2 - E0 ** 2) / C


def flutter(th, nder):
    """The flutter and its first nder azimuth derivatives (float64 tensors)."""
    polys, base = [np.polynomial.Polynomial([0.0, 1.0])], np.polynomial.Polynomial([0.0, 1.0, -1.0])
    for _ in range(nder):
        polys.append(polys[-1].deriv() * base)

    def at(p, s):
        v = torch.zeros_like(s)
        for c in p.coef[::-1]:
            v = v * s + float(c)
        return v
    out = [torch.zeros_like(th) for _ in range(nder + 1)]
    for x0, x1, w, y in MAGNETS:
        k = 16.0 / w
        a = [k ** m * at(polys[m], torch.sigmoid(k * (th - x0))) for m in range(nder + 1)]
        b = [(-k) ** m * at(polys[m], torch.sigmoid(-k * (th - x1))) for m in range(nder + 1)]
        for m in range(nder + 1):
            for j in range(m + 1):
                out[m] += y * math.comb(m, j) * a[j] * b[m - j]
    return out


def tables():
    """z-Taylor tables (Bz, Bfi, Br), each (ORDERS + 1, NR, NTH), of the field
    expanded about the mid-plane (div B = curl B = 0 order by order)."""
    if "tables" not in _kept:
        r = torch.linspace(RMIN, RMAX, NR, dtype=torch.float64, device=DEV)[:, None]
        th = torch.linspace(0.0, PERIOD, NTH, dtype=torch.float64, device=DEV)
        P = flutter(th, 2 * ORDERS + 2)
        out = [torch.zeros((ORDERS + 1, NR, NTH), dtype=torch.float64, device=DEV) for _ in range(3)]
        for n in range(ORDERS + 1):
            e = K - 2 * n
            out[0][n] = B0 * r ** e * P[0]
            out[1][n] = B0 * r ** (e - 1) * P[1] / (2 * n + 1)
            out[2][n] = B0 * e * r ** (e - 1) * P[0] / (2 * n + 1)
            P = [-(e ** 2 * P[m] + P[m + 2]) / ((2 * n + 2) * (2 * n + 1)) for m in range(len(P) - 2)]
        _kept["tables"] = out
    return _kept["tables"]


def freq_curve():
    """RF program: time, frequency, voltage, energy (300 to 310 MeV in 1000 turns)."""
    t = np.linspace(-200e-9, -200e-9 + 1050 * T_REV, 2001)
    ek = 300.0 + 10.0 * np.clip(t / (1000 * T_REV), 0.0, 1.0)
    p = np.sqrt((ek * 1e6 * Q + E0) ** 2 - E0 ** 2) / C
    v = p * C ** 2 / (ek * 1e6 * Q + E0)
    r = 8.33 * (p / momentum(300.0)) ** (1.0 / (K + 1))
    return np.column_stack([t, v / (2 * np.pi * r), np.full_like(t, VOLTAGE), ek])


def machine(order, rf):
    """The framework's description of the machine (lattice, RF, aperture)."""
    key = ("machine", order, rf)
    if key not in _kept:
        import warnings
        from pyffa_b200.constants import FFAG_GlobalParameters
        from pyffa_b200.fields import FFAG_Bfield_analytical, FFAG_EField_new
        cfg = {"Bmap": {"NSector": NSEC, "rmin_max_step_m": [RMIN, RMAX, DR], "SpiralAngle_deg": 0.0,
                        "theta_step_rad": DTH, "interval_1": [0.25, 0.3125, 0.09375, 0.09375, 0.25],
                        "positive_or_negative_1": [0, 1, 0, -1.3, 0], "fringe_width_1": [0, 1.17, 0, 1.17, 0],
                        "Bmean": None, "r_axis": None, "coefficients_tupel": [B0, K]}, "config": {"folder": "."}}
        stacks = None
        if order:
            if "stacks" not in _kept:
                _kept["stacks"] = [t.cpu().numpy() for t in tables()]
            stacks = _kept["stacks"]
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")
            bm = FFAG_Bfield_analytical(config=cfg, max_order=order, stacks=stacks, AddNumricalMap=False)
        head = {"acc_phi_paint": 30.0, "gap_azimuth": list(GAPS), "gap_width": GAP_WIDTH, "E_rmin": 8.0,
                "E_rmax": 9.3, "harmonic": 1, "rf_shift": [0.0, 0.0]}
        gp = FFAG_GlobalParameters()
        gp.AddBMap(bm)
        gp.AddEMap(FFAG_EField_new(header=head, data=freq_curve(), EnableFlag=bool(rf)))
        gp.AddAperture(*APERTURE)
        bm.device_map(torch.device(DEV, torch.cuda.current_device()))
        _kept[key] = gp
    return _kept[key]


# ------------------------------------------------------------------ inputs
def normals(seed, *shape):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return torch.randn(shape, dtype=torch.float64, device=DEV, generator=g)


def orbit_table():
    """Azimuth, radius and vr / v of the 300 MeV closed orbit over one sector."""
    if "orbit" not in _kept:
        v = momentum(300.0) * C ** 2 / (300e6 * Q + E0)
        s = torch.zeros((1, 16), dtype=torch.float64, device=DEV)
        c = PR_CO / math.sqrt(1 + PR_CO ** 2)
        s[0, 0], s[0, 1], s[0, 5], s[0, 7], s[0, 8] = R_CO, v * c, v * math.sqrt(1 - c * c) / R_CO, 1, 1
        rows, dt = [], DT / 8
        for k in range(520):
            rows.append([float(s[0, 4]), float(s[0, 0]), float(s[0, 1]) / v])
            boris(s, dt, 0.0, 0.0, False, 0)
        _kept["orbit"] = np.array(rows).T
    return _kept["orbit"]


def bunch(case, seed):
    """v-format rows (n, 16) on the device: 6D Gaussian at azimuth 0 (2 mm,
    1 mrad, 1e-3) or, with space charge, a KV bunch of 4 mm radii spread 20 ns
    in time, on the closed orbit of each particle's azimuth."""
    n = case["n"]
    w = normals(seed, 6, n)
    a = torch.zeros((n, 16), dtype=torch.float64, device=DEV)
    if case.get("sc"):
        u = w[:4] / w[:4].norm(dim=0)
        fi = math.pi - 2 * math.pi * 20e-9 / T_REV * w[4]
        th, r, s = orbit_table()
        f = torch.remainder(fi, PERIOD).cpu().numpy()
        a[:, 0] = torch.from_numpy(np.interp(f, th, r)).to(DEV) + 4e-3 * u[0]
        tr = torch.from_numpy(np.interp(f, th, s / np.sqrt(1 - s * s))).to(DEV) + 2e-3 * u[1]
        a[:, 2], tz, dp = 4e-3 * u[2], 2e-3 * u[3], 1e-4 * w[5]
    else:
        fi = torch.zeros(n, dtype=torch.float64, device=DEV)
        a[:, 0] = R_CO + 2e-3 * w[0]
        tr = PR_CO + 1e-3 * w[1]
        a[:, 2], tz, dp = 2e-3 * w[2], 1e-3 * w[3], 1e-3 * w[4]
    p = momentum(300.0) * (1 + dp)
    e = torch.sqrt((p * C) ** 2 + E0 ** 2)
    v = p * C ** 2 / e / torch.sqrt(1 + tr ** 2 + tz ** 2)
    a[:, 1], a[:, 3], a[:, 4] = v * tr, v * tz, fi
    a[:, 5] = e if case.get("solver") == "RK4" else v / a[:, 0]
    a[:, 7] = a[:, 8] = 1.0
    a[:, 14] = a[:, 15] = torch.arange(n, device=DEV)
    return a


def endpoints(case, seed):
    """Two successive space-charge fields per particle [V/m]."""
    return 2e4 * normals(seed + 1000, 6, case["n"])


# ------------------------------------------------------- learned-map inputs
SHAPES = [("W1", 16, 256), ("b1", 1, 256), ("W2", 256, 256), ("b2", 1, 256), ("W3", 256, 256), ("b3", 1, 256),
          ("W4", 256, 8), ("b4", 1, 8), ("Ws", 8, 8), ("bs", 1, 8), ("Wq", 16, 8)]
PAIRS = [(i, j) for i in range(5) for j in range(i, 5)]


def blocks(p):
    out, o = {}, 0
    for name, r, c in SHAPES:
        out[name] = p[o:o + r * c].view(r, c)
        o += r * c
    return out


def network(seed, trained):
    """Parameters: the initial ones of a training run, or a map's: a rotation
    by the sector's phase advances, small second and higher orders."""
    p = torch.zeros(sum(r * c for _, r, c in SHAPES), dtype=torch.float32, device=DEV)
    b, w = blocks(p), normals(seed + 7, 256 * 600).float()
    b["W1"][:6] = w[:1536].view(6, 256) * (1.5 / math.sqrt(6))
    b["W2"][:] = w[1536:67072].view(256, 256) * math.sqrt(2 / 256)
    b["W3"][:] = w[67072:132608].view(256, 256) * math.sqrt(2 / 256)
    for j, q in ((0, 3.595 / NSEC), (2, 0.781 / NSEC)):
        c, s = math.cos(2 * math.pi * q), math.sin(2 * math.pi * q)
        b["Ws"][j:j + 2, j:j + 2] = torch.tensor([[c - 1, -s], [s, c - 1]])
    b["Wq"][:15, :4] = 1e-4 * w[140000:140060].view(15, 4)
    b["b1"][0] = 0.1 * w[133000:133256]
    if trained:
        b["W4"][:, :4] = 1e-5 * w[134000:135024].view(256, 4)
    else:
        b["W4"][:, :4] = 1e-2 * w[134000:135024].view(256, 4)
    return p


def states(n, seed, radius):
    """(n, 8) float32 states uniform in the discs of `radius`, e in [-0.9, 0.9]."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    u = torch.rand((5, n), dtype=torch.float64, device=DEV, generator=g)
    s = torch.zeros((n, 8), dtype=torch.float32, device=DEV)
    for j in (0, 2):
        rho = radius * u[j].sqrt()
        s[:, j], s[:, j + 1] = rho * torch.cos(2 * math.pi * u[j + 1]), rho * torch.sin(2 * math.pi * u[j + 1])
    s[:, 4] = 1.8 * u[4] - 0.9
    return s


def targets(x):
    """What the network is to learn of the next sector entrance (scaled residual included)."""
    t = torch.zeros_like(x)
    t[:, 0], t[:, 1] = 0.2 * x[:, 0] - 0.9 * x[:, 1], 0.9 * x[:, 0] + 0.2 * x[:, 1]
    t[:, 2], t[:, 3] = 0.8 * x[:, 2] - 0.4 * x[:, 3], 0.4 * x[:, 2] + 0.8 * x[:, 3]
    t[:, :4] += 0.5 * torch.sin(3 * x[:, :4] * x[:, 4:5])
    return t


def tracks(case, seed):
    """(m, 5) r, pr, z, pz, P around the scaled closed orbits of 300-600 MeV."""
    w = normals(seed, 4, case["m"])
    ek = torch.linspace(300.0, 600.0, case["m"], dtype=torch.float64, device=DEV)
    p = torch.sqrt((ek * 1e6 * Q + E0) ** 2 - E0 ** 2) / C
    x = torch.empty((case["m"], 5), dtype=torch.float64, device=DEV)
    x[:, 0] = R_CO * (p / momentum(300.0)) ** (1 / (K + 1)) + 1e-3 * w[0]
    x[:, 1] = PR_CO / math.sqrt(1 + PR_CO ** 2) + 1e-3 * w[1]
    x[:, 2], x[:, 3], x[:, 4] = 1e-3 * w[2], 1e-3 * w[3], p
    return x


# -------------------------------------------------------------------- cases
def listed():
    push = {"kind": "push", "solver": "Boris", "precision": "fp64", "steps": 720, "order": 2, "rf": True, "sc": False}
    return [
        # an A/B check against the reference's single step, or a program that
        # still keeps its own step loop: the smallest call, all latency
        {"name": "host_single_step", "kind": "step", "n": 2000, "order": 2, "rf": True},
        # one turn of a small bunch through the full-order map without RF:
        # dynamic aperture and tune studies
        dict(push, name="boris_small_order4", n=10_000, order=4, rf=False),
        # one turn of an accelerated bunch: the tracking loop's main path
        dict(push, name="boris_turn_rf", n=100_000),
        # the same with the float32 field
        dict(push, name="boris_fp32c_turn_rf", n=100_000, precision="fp32c"),
        # the steps between two space-charge updates of a large bunch
        dict(push, name="boris_sc_interval", n=1_000_000, steps=SC_STEPS, rf=False, sc=True),
        # one turn with the other solver
        dict(push, name="rk4_turn_rf", n=100_000, solver="RK4"),
        # a ragged host bunch through a turn, host memory to host memory
        {"name": "host_turn", "kind": "host", "n": 50_021, "solver": "Boris", "precision": "fp64", "steps": 720,
         "order": 2, "rf": True},
        # the space-charge update of a large bunch, open boundary
        {"name": "sc_open_large", "kind": "sc", "n": 1_000_000, "ns": 64, "grid": 128, "open": True, "sc": True},
        # and of a ragged small one, the reference's periodic boundary
        {"name": "sc_periodic_small", "kind": "sc", "n": 100_003, "ns": 32, "grid": 64, "open": False, "sc": True},
        # one turn of a bunch with the learned sector map
        {"name": "learned_turn", "kind": "map", "n": 262_221, "maps": 12},
        # one optimiser step of the learned map's training
        {"name": "learned_train_step", "kind": "train", "batch": 8192},
        # the tracks of one tune search over 256 energies (five each), one sector
        {"name": "orbit_tracks", "kind": "orbit", "m": 1280, "steps": 523},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["push", "push", "push", "push", "step", "host", "sc", "sc", "map", "train", "orbit"])
    if kind == "step":
        return {"kind": kind, "n": size(100, 20_000), "order": rng.choice([0, 2, 4]), "rf": rng.random() < 0.5}
    if kind == "sc":
        return {"kind": kind, "n": size(20_000, 1_000_000), "ns": rng.randint(8, 64), "grid": rng.choice([32, 64, 128]),
                "open": rng.random() < 0.5, "sc": True}
    if kind == "map":
        return {"kind": kind, "n": size(1000, 262_000), "maps": rng.randint(1, 12)}
    if kind == "train":
        return {"kind": kind, "batch": size(1024, 8000)}
    if kind == "orbit":
        return {"kind": kind, "m": size(3, 20_000), "steps": size(64, 523)}
    c = {"kind": kind, "n": size(1000, 100_000), "solver": rng.choice(["Boris", "Boris", "RK4"]), "precision": "fp64",
         "steps": size(30, 720), "order": rng.choice([0, 1, 2, 3, 4]), "rf": rng.random() < 0.5}
    if kind == "push":
        c["sc"] = rng.random() < 0.3
        if c["sc"]:
            c["n"], c["steps"] = size(10_000, 1_000_000), rng.randint(10, SC_STEPS)
        if c["solver"] == "Boris" and rng.random() < 0.25:
            c["precision"] = "fp32c"
    return c


def work(case):
    """A push reads and writes each particle's state once (10 float64 columns
    and 2 flags in, 82 bytes out; 36 more in with the two field endpoints) and
    does about 300 (Boris) or 980 (RK4) operations a step; the tables it
    touches are shared by the bunch and not counted."""
    k = case["kind"]
    if k in ("push", "step", "host"):
        n, steps = case["n"], case.get("steps", 1)
        per = 2 * 128 if k != "push" else 164 + (50 if case["sc"] else 0)
        return {"bytes": n * per, "flops": n * steps * (980 if case.get("solver") == "RK4" else 300)}
    if k == "sc":
        cells = case["ns"] * case["grid"] ** 2
        side = case["grid"] * (2 if case["open"] else 1)
        # r, vr, z, vz, fi, f5, flag, old endpoint and mask in; fields, both
        # endpoints and masks out; charge, potential and two field cubes out
        return {"bytes": case["n"] * (49 + 25 + 74) + 16 * cells,
                "flops": case["n"] * 150 + case["ns"] * 2 * 5 * side * side * 2 * math.log2(side) / 2}
    if k == "map":
        return {"bytes": case["n"] * 68 + 280_000, "flops": case["n"] * case["maps"] * 266_752}
    if k == "train":
        return {"bytes": case["batch"] * 64 + 138_192 * 4 * 7, "flops": 3 * case["batch"] * 266_752}
    return {"bytes": case["m"] * 72, "flops": case["m"] * case["steps"] * 4 * 150}


# ------------------------------------------------------------------ product
def prepare(case, seed):
    k = case["kind"]
    s = {"kind": k}
    if k == "map":
        from pyffa_b200 import learned
        s["map"] = learned.LearnedSectorMap(None, None, network(seed, True))
        s["start"] = states(case["n"], seed, 0.6)
        s["state"] = torch.empty_like(s["start"])
        s["applied"] = torch.zeros(case["n"], dtype=torch.int32, device=DEV)
        s["maps"] = case["maps"]
        return s
    if k == "train":
        from pyffa_b200 import learned
        lr = torch.full((1 << 20,), 1e-3, dtype=torch.float32, device=DEV)
        s["trainer"] = learned.Trainer(network(seed, False), batch=case["batch"], lr_table=lr)
        s["x"] = states(case["batch"], seed, 1.0)
        s["t"] = targets(s["x"])
        return s
    if k == "orbit":
        from pyffa_b200 import learned
        s["tracker"] = learned.SectorTracker(machine(0, False).Bmap, Q, steps_per_sector=case["steps"])
        s["x"] = tracks(case, seed)
        return s
    rows = bunch(case, seed)
    if k == "sc":
        from pyffa_b200.bunch import FFAG_Bunch
        from pyffa_b200.space_charge import SpaceCharge
        b = FFAG_Bunch(rows.cpu().numpy(), marcosize=1e13 / case["n"],
                       sc_grid_size=(case["ns"], case["grid"], case["grid"], 12.0))
        s["sc"] = SpaceCharge(b, hockney=case["open"], seo={n: v.cpu().numpy() for n, v in orbits().items()})
        s["bunch"] = b
        return s
    gp = machine(case["order"], case["rf"])
    if k == "step":
        from pyffa_b200.track import FFAG_RungeKutta
        s["rk"], s["gp"] = FFAG_RungeKutta(), gp
        s["start"] = rows.cpu().numpy()
        s["rows"] = s["start"].copy()
        return s
    if k == "host":
        from pyffa_b200.track import MatrixTracker
        s["in"] = rows.cpu().pin_memory()
        s["out"] = torch.empty_like(s["in"]).pin_memory()
        s["out"].copy_(s["in"])
        s["tracker"] = MatrixTracker(case["n"], gp, case["solver"], case["precision"])
        s["tracker"].bind_clock(0.0, DT, case["steps"])
        s["steps"] = case["steps"]
        return s
    from pyffa_b200.bunch import FFAG_Bunch
    from pyffa_b200.track import Pusher, StepClock
    b = FFAG_Bunch(rows.cpu().numpy(), BunchType=case["solver"])
    if case["sc"]:
        for name, v in zip(("e_pp_r", "e_pp_z", "e_pp_fi", "e_pre_r", "e_pre_z", "e_pre_fi"), endpoints(case, seed)):
            b.cols[name].copy_(v)
        b.cols["sc_pre"].fill_(1)
        b.cols["sc_pp"].fill_(1)
    s["bunch"], s["pusher"] = b, Pusher(b, gp, case["solver"], case["precision"])
    s["clock"] = StepClock(0.0, DT, gp.Emap, case["solver"], b.device)
    s["clock"].ensure(2 * SC_STEPS + case["steps"])
    s["first"], s["steps"] = (2 * SC_STEPS, case["steps"]) if case["sc"] else (0, case["steps"])
    s["sc_step"] = SC_STEPS if case["sc"] else 0
    s["cols"] = [[b.cols[c] for c in names] for names in (COLS, FLAGS)]
    s["start"] = [[c.clone() for c in group] for group in s["cols"]]
    return s


def run(s):
    k = s["kind"]
    if k == "push":
        # the bunch as it enters the machine, then the steps
        for to, start in zip(s["cols"], s["start"]):
            torch._foreach_copy_(to, start)
        s["pusher"].push(s["clock"], s["first"], s["steps"], s["sc_step"])
        return {c: s["bunch"].cols[c] for c in (*COLS, *FLAGS)}
    if k == "step":
        np.copyto(s["rows"], s["start"])
        return s["rk"].Boris_solve(0.0, s["rows"], DT, s["gp"])
    if k == "host":
        s["tracker"].run(s["in"], s["out"], 0, s["steps"])
        return s["out"]
    if k == "sc":
        s["sc"].update()
        return {c: s["bunch"].cols[c] for c in ("esc_r", "esc_z", "esc_fi", "e_pre_r", "e_pre_z", "e_pre_fi", "sc_pre")}
    if k == "map":
        s["state"].copy_(s["start"])
        s["map"].apply(s["state"], s["maps"], s["applied"])
        return {"state": s["state"], "applied": s["applied"]}
    if k == "train":
        tr = s["trainer"]
        tr.graph_step(s["x"], s["t"])
        return {"params": tr.p, "grads": tr.g, "m": tr.m, "v": tr.v}
    return s["tracker"].run(s["x"], 1)


# -------------------------------------------------------------------- exact
def field(r, fi, z, order):
    """Bz, Br, Bfi: mid-plane field with its z-linear terms, then the tables."""
    fm = fi - PERIOD * torch.floor(fi / PERIOD)
    F, Fp = flutter(fm, 1)
    b = B0 * r ** K
    Bz, Bfi, Br = b * F, b * Fp / r * z, K * b / r * F * z
    if order:
        qr, qt = (r - RMIN) / DR, fm / (PERIOD / (NTH - 1))
        i, j = qr.long().clamp(0, NR - 2), qt.long().clamp(0, NTH - 2)
        tr, tt = qr - i, qt - j
        at, w = i * NTH + j, ((1 - tr) * (1 - tt), (1 - tr) * tt, tr * (1 - tt), tr * tt)
        T = [t.view(ORDERS + 1, -1) for t in tables()]
        for n in range(1, order + 1):
            v = [sum(wk * t[n][at + o] for wk, o in zip(w, (0, 1, NTH, NTH + 1))) for t in T]
            Bz = Bz + v[0] * z ** (2 * n)
            Bfi = Bfi + v[1] * z ** (2 * n + 1)
            Br = Br + v[2] * z ** (2 * n + 1)
    return Bz, Br, Bfi


def gap(r, fi, phase, acc):
    """Er, Efi of the last RF gap's rectangle."""
    th = math.radians(GAPS[-1])
    x, y = r * torch.cos(fi), r * torch.sin(fi)
    u, w = x * math.cos(th) + y * math.sin(th), y * math.cos(th) - x * math.sin(th)
    e = acc * torch.sin(phase) * ((u >= 8.0) & (u <= 9.3) & (w.abs() <= GAP_WIDTH / 2))
    d = th + math.pi / 2 - fi
    return e * torch.cos(d), e * torch.sin(d)


def curve(t):
    d = freq_curve()
    x0, dx = d[0, 0], d[1, 0] - d[0, 0]
    i = min(max(int(math.floor((t - x0) / dx)), 0), len(d) - 2)
    u = (t - x0 - i * dx) / dx
    return d[i, 1] + u * (d[i + 1, 1] - d[i, 1]), (d[i, 2] + u * (d[i + 1, 2] - d[i, 2])) / GAP_WIDTH


def boris(a, dt, f, acc, rf, order):
    """One relativistic Boris step of the rows `a`, in place, in Cartesian axes."""
    r, z, fi = a[:, 0], a[:, 2], a[:, 4]
    Bz, Br, Bfi = field(r, fi, z, order)
    Er, Ez, Ef = a[:, 10].clone(), a[:, 11], a[:, 12].clone()
    if rf:
        er, ef = gap(r, fi, a[:, 9], acc)
        Er, Ef = Er + er, Ef + ef
    lost = (r > APERTURE[1]) | (r < APERTURE[0]) | (z > APERTURE[3]) | (z < APERTURE[2])
    live = (a[:, 7] == 1) & (a[:, 8] == 1)
    s, c = torch.sin(fi), torch.cos(fi)
    vf = r * a[:, 5]
    v = torch.stack([a[:, 1] * c - vf * s, a[:, 1] * s + vf * c, a[:, 3]])
    E = torch.stack([Er * c - Ef * s, Er * s + Ef * c, Ez])
    B = -torch.stack([Br * c - Bfi * s, Br * s + Bfi * c, Bz])
    p = M0 * v / torch.sqrt(1 - (v * v).sum(0) / C ** 2) + 0.5 * dt * Q * E
    t = 0.5 * dt * Q / (M0 * torch.sqrt(1 + (p * p).sum(0) / (M0 * C) ** 2)) * B
    p = p + torch.linalg.cross(p + torch.linalg.cross(p, t, dim=0), 2 / (1 + (t * t).sum(0)) * t, dim=0)
    p = p + 0.5 * dt * Q * E
    v = p / (M0 * torch.sqrt(1 + (p * p).sum(0) / (M0 * C) ** 2))
    x, y = r * c + v[0] * dt, r * s + v[1] * dt
    rn, d = torch.sqrt(x * x + y * y), torch.atan2(y * c - x * s, x * c + y * s)
    cn, sn = x / rn, y / rn
    new = [rn, v[0] * cn + v[1] * sn, z + v[2] * dt, v[2], fi + d, (v[1] * cn - v[0] * sn) / rn]
    for col, val in enumerate(new):
        a[:, col] = torch.where(live, val, a[:, col])
    a[:, 8] = torch.where(live & lost, 0.0, a[:, 8])
    a[:, 9] += f * 2 * math.pi * dt


def rk4(a, dt, t, rf, order):
    live = ((a[:, 7] == 1) & (a[:, 8] == 1)).double()

    def rhs(y, f, acc):
        r, vr, z, vz, fi, E, ph = y
        Bz, Br, Bfi = field(r, fi, z, order)
        Er, Ez, Ef = a[:, 10], a[:, 11], a[:, 12]
        if rf:
            er, ef = gap(r, fi, ph, acc)
            Er, Ef = Er + er, Ef + ef
        w = torch.sqrt((1 - (E0 / E) ** 2) * C ** 2 - vr ** 2 - vz ** 2)
        Ev = vr * Er + w * Ef + vz * Ez
        q = Q * C ** 2 / E
        return torch.stack([vr, w * w / r + q * (Er - w * Bz + vz * Bfi) - Q * vr / E * Ev, vz,
                            q * (Ez + w * Br - vr * Bfi) - Q * vz / E * Ev, w / r, Q * Ev,
                            torch.full_like(r, f * 2 * math.pi)])
    y = torch.stack([a[:, c] for c in (0, 1, 2, 3, 4, 5, 9)])
    k1 = dt * rhs(y, *curve(t))
    k2 = dt * rhs(y + 0.5 * k1, *curve(t + 0.5 * dt))
    k3 = dt * rhs(y + 0.5 * k2, *curve(t + 0.5 * dt))
    k4 = dt * rhs(y + k3, *curve(t + dt))
    y = y + live * (k1 + 2 * k2 + 2 * k3 + k4) / 6
    for c, v in zip((0, 1, 2, 3, 4, 5, 9), y):
        a[:, c] = v


def pushed(case, seed):
    a = bunch(case, seed)
    sc, steps = case.get("sc"), case.get("steps", 1)
    first = 2 * SC_STEPS if sc else 0
    e = endpoints(case, seed) if sc else None
    t = np.add.accumulate(np.concatenate([[0.0], np.full(first + steps, DT)]))
    for s in range(first, first + steps):
        if sc:
            w = (s % SC_STEPS) / SC_STEPS
            a[:, 10:13] = (e[3:] + w * (e[3:] - e[:3])).T
        if case.get("solver") == "RK4":
            rk4(a, DT, float(t[s]), case["rf"], case["order"])
        else:
            boris(a, DT, *curve(float(t[s])), case["rf"], case["order"])
    return a


def orbits():
    """Closed-orbit tables (energy, azimuth) by the scaling law."""
    th, r, s = orbit_table()
    fi = np.linspace(0, 2 * np.pi, 721)
    ek = np.linspace(280.0, 320.0, 9)
    f = np.array([(momentum(e) / momentum(300.0)) ** (1 / (K + 1)) for e in ek])[:, None]
    x = np.mod(fi, PERIOD)
    out = {"Ek_axis": ek, "fi_axis": fi, "r": f * np.interp(x, th, r),
           "pr": np.ones_like(f) * np.interp(x, th, s / np.sqrt(1 - s * s)), "perimeter": 52.37912270488599 * f[:, 0]}
    return {k: torch.from_numpy(v).to(DEV) for k, v in out.items()}


def space_charge(case, seed):
    a, T, ns, g, two = bunch(case, seed), orbits(), case["ns"], case["grid"], 2 * math.pi
    vf = a[:, 0] * a[:, 5]
    gam = 1 / torch.sqrt(1 - (a[:, 1] ** 2 + a[:, 3] ** 2 + vf ** 2) / C ** 2)
    fm = a[:, 4] - two * torch.floor(a[:, 4] / two)

    def look(tab):
        x, y = ((gam - 1) * E0_MEV - T["Ek_axis"][0]) / (T["Ek_axis"][1] - T["Ek_axis"][0]), fm / (two / 720)
        i, j = x.floor().long().clamp(0, 7), y.floor().long().clamp(0, 719)
        u, v = x - i, y - j
        return (1 - u) * (1 - v) * tab[i, j] + (1 - u) * v * tab[i, j + 1] + u * (1 - v) * tab[i + 1, j] + u * v * tab[i + 1, j + 1]
    x, z, pr = a[:, 0] - look(T["r"]), a[:, 2], look(T["pr"])
    spans = []
    for sh in (0.0, math.pi, math.pi / 2, 1.5 * math.pi):
        m = (fm + sh) - two * torch.floor((fm + sh) / two)
        spans.append((float(m.max() - m.min()), float(m.min()) - sh, float(m.max()) - sh))
    _, lo, hi = min(spans, key=lambda v: v[0])
    lo, hi = lo % two, hi % two
    hi += two if hi <= lo else 0.0
    mg = float(gam.mean())
    per = np.interp((mg - 1) * E0_MEV, T["Ek_axis"].cpu().numpy(), T["perimeter"].cpu().numpy())
    length = per * (hi - lo) / two
    s = ((fm + two * (fm < lo) - lo) / ((hi - lo) / (ns - 1))).long().clamp(0, ns - 1)
    box = []
    for u in (x, z):
        m, sg = float(u.mean()), float(((u * u).mean() - u.mean() ** 2).sqrt())
        box.append((m - 12 * sg, 24 * sg / g))
    (x0, dx), (z0, dz) = box

    def cell(u, u0, du):
        q = (u - u0) / du
        i = q.floor().long()
        f = torch.where(i < 0, 0.0, torch.where(i >= g - 1, 1.0, q - i))
        return i.clamp(0, g - 2), f, q
    ix, fx, qx = cell(x, x0, dx)
    iz, fz, qz = cell(z, z0, dz)
    at = (s * g + iz) * g + ix
    rho = torch.zeros(ns * g * g, dtype=torch.float64, device=DEV)
    for o, w in ((0, (1 - fx) * (1 - fz)), (1, fx * (1 - fz)), (g, (1 - fx) * fz), (g + 1, fx * fz)):
        rho.index_add_(0, at + o, w)
    rho = rho.view(ns, g, g) * (1e13 / case["n"] * Q / length * ns / (dx * dz))
    if case["open"]:
        N = 2 * g
        i = torch.arange(N, device=DEV, dtype=torch.float64)
        i = torch.minimum(i, N - i)
        X, Z = (dx * i)[None, :], (dz * i)[:, None]
        G = -torch.log(torch.clamp(X * X + Z * Z, min=1e-300)) / (4 * math.pi * EPS0)
        h, k = dx / 2, dz / 2
        G[0, 0] = -(h * k * (math.log(h * h + k * k) - 3) + h * h * math.atan(k / h) + k * k * math.atan(h / k)) / (h * k) / (4 * math.pi * EPS0)
        phi = torch.fft.irfft2(torch.fft.rfft2(rho, s=(N, N)) * torch.fft.rfft2(G * dx * dz), s=(N, N))[:, :g, :g]
    else:
        kx, kz = (two / (g * d) * torch.fft.fftfreq(g, 1 / g, dtype=torch.float64, device=DEV) for d in (dx, dz))
        k2 = kx[None, :] ** 2 + kz[:, None] ** 2
        phi = torch.fft.ifft2(torch.fft.fft2(rho) * torch.where(k2 == 0, 0.0, 1 / (EPS0 * k2.clamp(min=1e-300)))).real
    Ex, Ez = torch.empty_like(phi), torch.empty_like(phi)
    Ex[:, :, 1:-1] = -(phi[:, :, 2:] - phi[:, :, :-2]) / (2 * dx)
    Ex[:, :, 0], Ex[:, :, -1] = -(phi[:, :, 1] - phi[:, :, 0]) / dx, -(phi[:, :, -1] - phi[:, :, -2]) / dx
    Ez[:, 1:-1] = -(phi[:, 2:] - phi[:, :-2]) / (2 * dz)
    Ez[:, 0], Ez[:, -1] = -(phi[:, 1] - phi[:, 0]) / dz, -(phi[:, -1] - phi[:, -2]) / dz
    at, u, v = (s * g + iz) * g + ix, qx - ix, qz - iz
    er, ez = (sum(w * f.reshape(-1)[at + o] for o, w in ((0, (1 - u) * (1 - v)), (1, u * (1 - v)), (g, (1 - u) * v),
                                                         (g + 1, u * v))) / mg ** 2 for f in (Ex, Ez))
    rt = torch.sqrt(1 + pr * pr)
    return {"esc_r": er / rt, "esc_z": ez, "esc_fi": -er * pr / rt}


def forward(b, x):
    h = x[:, :6]
    for i in (1, 2, 3):
        h = torch.nn.functional.silu(h @ b["W%d" % i][:h.shape[1]] + b["b%d" % i])
    quad = torch.stack([x[:, i] * x[:, j] for i, j in PAIRS], 1)
    return x[:, :6] + (h @ b["W4"] + b["b4"] + x[:, :6] @ b["Ws"][:6] + b["bs"] + quad @ b["Wq"][:15])[:, :6]


def exact(case, seed):
    k = case["kind"]
    if k in ("push", "step", "host"):
        a = pushed(case, seed)
        if k != "push":
            return a
        return {**{c: a[:, i] for c, i in COLS.items()}, "inj": None, "surv": None}
    if k == "sc":
        e = space_charge(case, seed)
        return {**e, "e_pre_r": e["esc_r"], "e_pre_z": e["esc_z"], "e_pre_fi": e["esc_fi"], "sc_pre": None}
    if k == "map":
        b, x = blocks(network(seed, True).double()), states(case["n"], seed, 0.6).double()
        for _ in range(case["maps"]):
            x[:, :4] = torch.cat([forward(b, part)[:, :4] for part in x.split(65536)])
        return {"state": x, "applied": None}
    if k == "train":
        p = network(seed, False).double().requires_grad_(True)
        x = states(case["batch"], seed, 1.0)
        t = targets(x).double()
        loss = ((forward(blocks(p), x.double())[:, :4] - t[:, :4]) ** 2).mean()
        g, = torch.autograd.grad(loss, p)
        p = p.detach()
        m, v = 0.1 * g, 0.001 * g * g
        step = 1e-3 * (m / 0.1) / (torch.sqrt(v / 0.001) + 1e-8)
        for n, blk in blocks(step).items():
            if n in ("Ws", "bs", "Wq"):
                blk.zero_()
                blocks(m)[n].zero_()
                blocks(v)[n].zero_()
        return {"params": p - step, "grads": g, "m": m, "v": v}
    x, h = tracks(case, seed), PERIOD / case["steps"]
    qP = Q / x[:, 4]

    def rhs(th, y):
        r, pr, z, pz = y
        Bz, Br, Bfi = field(r, torch.full_like(r, th), z, 0)
        pf = torch.sqrt(1 - pr ** 2 - pz ** 2)
        return torch.stack([r * pr / pf, pf - qP * (r * Bz - r * pz / pf * Bfi), r * pz / pf,
                            qP * (r * Br - r * pr / pf * Bfi)])
    y = x[:, :4].T.contiguous()
    for s in range(case["steps"]):
        k1 = h * rhs(s * h, y)
        k2 = h * rhs(s * h + 0.5 * h, y + 0.5 * k1)
        k3 = h * rhs(s * h + 0.5 * h, y + 0.5 * k2)
        k4 = h * rhs(s * h + h, y + k3)
        y = y + (k1 + 2 * k2 + 2 * k3 + k4) / 6
    return y.T
