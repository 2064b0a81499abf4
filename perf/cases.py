"""The work that programs have this engine do, as cases that can be timed and compared: NVT dynamics of one system and
of a serving batch, the per-step call of a plugin, batched and fresh single points, the analysis step, and the charge
solve by itself. Every case goes through the public front end (metal-reax_b200/rxcuda.py, or the C ABI of
include/rxcuda.h for the entry point that takes device pointers).

`exact` restates the ReaxFF energy, the charge equilibration and the integrator in plain FP64 torch (the gradient by
automatic differentiation), on the force-field file itself.
"""
import ctypes
import math
import sys
from pathlib import Path

import numpy as np
import torch

PKG = Path(__file__).resolve().parents[1] / "metal-reax_b200"
if str(PKG) not in sys.path:
    sys.path.insert(0, str(PKG))

import rxcuda  # noqa: E402
import systems  # noqa: E402

MASS = [12.0, 1.008, 15.999]
DT, TDAMP, CHAIN = 0.25, 25.0, 3
FRAMES = 16     # frames of the periodic orbit that a plugin's or a screening loop's positions follow
MAX_BONDS = 64  # columns of a bond table (the engine's random carbon reaches about 20)
LEAVE = 2       # requests that leave and join in a serving round


# ------------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # The smallest system of the engine's acceptance runs (216 H2O) under NVT: launches and latency count.
        {"name": "md_water_648", "kind": "md", "matter": "water", "atoms": 648, "steps": 20, "charges": True},
        # The headline workload: 8000 H2O, NVT at 300 K, charges re-equilibrated every step.
        {"name": "md_water_24000", "kind": "md", "matter": "water", "atoms": 24000, "steps": 10, "charges": True},
        # The largest box of the published size series (21,952 H2O).
        {"name": "md_water_65856", "kind": "md", "matter": "water", "atoms": 65856, "steps": 5, "charges": True},
        # The graphitization example: random carbon at 4000 K, one element, no charge solve; dense in bonds and torsions.
        {"name": "md_carbon_30000", "kind": "md", "matter": "carbon", "atoms": 30000, "steps": 10, "charges": False},
        # The per-step call of a plugin that integrates on the host: page-locked positions in, charges solved, energies,
        # gradient, virial and charges out.
        {"name": "step_water_24000", "kind": "step", "matter": "water", "atoms": 24000, "pinned": True, "tilted": False},
        # The two calls of the LAMMPS pair style and charge fix, on LAMMPS's own (pageable) arrays.
        {"name": "split_water_5184", "kind": "split", "matter": "water", "atoms": 5184, "pinned": False, "tilted": False},
        # Screening: 512 mixed CHO systems of 64-1024 atoms as one batch, fresh single points.
        {"name": "batch_cho_512", "kind": "batch", "systems": 512, "nmin": 64, "nmax": 1024},
        # One round of the serving loop: two of 16 CHO requests of 100-5000 atoms leave, two join, ten NVT steps.
        {"name": "serve_cho_16", "kind": "serve", "systems": 16, "nmin": 100, "nmax": 5000, "steps": 10},
        # One fresh small system handed over, evaluated once and answered (an odd size).
        {"name": "point_cho_333", "kind": "point", "matter": "cho", "atoms": 333},
        # The analysis step of a run: per-atom energies and virials, the decision census and the bond table.
        {"name": "analysis_water_5184", "kind": "analysis", "matter": "water", "atoms": 5184},
        # The charge solve alone from a cold start at the tight tolerance of the reference's NVE comparison.
        {"name": "charges_water_24000", "kind": "charges", "matter": "water", "atoms": 24000, "tol": 1e-10},
        # The allocation-free charge solve on a CSR matrix that the caller holds on the device.
        {"name": "static_water_2592", "kind": "static", "matter": "water", "atoms": 2592, "tol": 1e-6},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["md", "md", "step", "split", "batch", "serve", "point", "analysis", "charges", "static"])
    matter = rng.choice(["water", "water", "cho", "carbon"])
    if kind == "md":
        return {"kind": kind, "matter": matter, "atoms": _log_int(rng, 300, 50000 if matter != "cho" else 8000),
                "steps": rng.randint(3, 10), "charges": matter != "carbon"}
    if kind in ("step", "split"):
        matter = rng.choice(["water", "water", "cho"])
        return {"kind": kind, "matter": matter, "atoms": _log_int(rng, 300, 40000 if matter == "water" else 8000),
                "pinned": rng.random() < 0.5, "tilted": rng.random() < 0.3}
    if kind == "batch":
        return {"kind": kind, "systems": _log_int(rng, 8, 400), "nmin": 64, "nmax": rng.choice([300, 700, 1024])}
    if kind == "serve":
        return {"kind": kind, "systems": rng.randint(4, 24), "nmin": 100, "nmax": rng.choice([1000, 2500, 5000]),
                "steps": rng.randint(3, 10)}
    if kind == "point":
        return {"kind": kind, "matter": "water" if matter == "water" else "cho", "atoms": _log_int(rng, 64, 4000)}
    if kind == "analysis":
        return {"kind": kind, "matter": matter, "atoms": _log_int(rng, 300, 20000 if matter != "cho" else 6000)}
    if kind == "charges":
        return {"kind": kind, "matter": "water", "atoms": _log_int(rng, 300, 40000), "tol": rng.choice([1e-6, 1e-8, 1e-10])}
    return {"kind": kind, "matter": "water", "atoms": _log_int(rng, 200, 6000), "tol": rng.choice([1e-6, 1e-8])}


# ------------------------------------------------------------------------------------------------------- inputs
def _water(atoms, rng):
    """About `atoms` / 3 water molecules on a jittered lattice at 1 g/cm3 with random orientations (whole lattices fill
    their box as systems.water_box does; other counts leave some sites empty)."""
    nmol = max(1, int(atoms) // 3)
    side = 1
    while side ** 3 < nmol:
        side += 1
    h = ((2 * 1.008 + 15.999) * systems.AMU_G) ** (1.0 / 3.0) * 1e8
    site = np.sort(rng.permutation(side ** 3)[:nmol])
    cell = np.stack([site // (side * side), (site // side) % side, site % side], axis=1)
    centre = (cell + 0.5) * h + rng.uniform(-0.3, 0.3, size=(nmol, 3))
    quat = rng.normal(size=(nmol, 4))
    a, b, c, d = (quat / np.linalg.norm(quat, axis=1, keepdims=True)).T
    rot = np.array([[a * a + b * b - c * c - d * d, 2 * (b * c - a * d), 2 * (b * d + a * c)],
                    [2 * (b * c + a * d), a * a - b * b + c * c - d * d, 2 * (c * d - a * b)],
                    [2 * (b * d - a * c), 2 * (c * d + a * b), a * a - b * b - c * c + d * d]]).transpose(2, 0, 1)
    half = math.radians(104.5) / 2
    local = np.array([[0.0, 0.0, 0.0], [0.96 * math.sin(half), 0.0, 0.96 * math.cos(half)],
                      [-0.96 * math.sin(half), 0.0, 0.96 * math.cos(half)]])
    x = (centre[:, None, :] + np.einsum("ka,mca->mkc", local, rot)).reshape(-1, 3)
    t = np.tile(np.array([2, 1, 1], dtype=np.int32), nmol)
    return _periodic(h * side, x, t)


def _periodic(length, x, t):
    return {"name": "water%d" % len(t), "origin": np.zeros(3), "box": np.eye(3) * length, "periodic": np.ones(3, dtype=np.int32),
            "x": np.ascontiguousarray(x - length * np.floor(x / length)), "type": np.ascontiguousarray(t, dtype=np.int32),
            "tag": np.arange(1, len(t) + 1, dtype=np.int64), "mass": np.array(MASS)[t]}


def _one(case, seed):
    atoms = int(case["atoms"])
    if case["matter"] == "water":
        s = _water(atoms, np.random.default_rng([seed, 1]))
    elif case["matter"] == "carbon":
        s = systems.random_carbon(atoms, seed=seed)
    else:
        s = systems.serving_request(0, seed=seed, nmin=atoms, nmax=atoms)[0]
    return systems.triclinic(s) if case.get("tilted") else s


def _many(case, seed, count):
    """CHO systems of the serving workload's kind; their sizes (log-uniform) go with the case, all else with the seed."""
    sizes = np.exp(np.random.default_rng(case["nmin"] + case["nmax"]).uniform(math.log(case["nmin"]), math.log(case["nmax"]), size=count))
    return [systems.serving_request(k, seed=seed, nmin=int(n), nmax=int(n))[0] for k, n in enumerate(np.round(sizes))]


def _orbit(x, rng):
    """FRAMES snapshots of a smooth periodic motion about x, about as far from one to the next as an MD step moves."""
    amp = rng.normal(scale=0.03, size=x.shape)
    phase = rng.uniform(0.0, 2.0 * math.pi, size=(len(x), 1))
    return np.stack([x + amp * np.sin(2.0 * math.pi * k / FRAMES + phase) for k in range(FRAMES)])


def _field():
    return (PKG / "data" / "ffield.synthetic.cho").read_text()


def _engine(ss, tol=1e-6):
    e = rxcuda.Engine(0)
    e.set_forcefield(_field())
    e.set_control()
    e.set_qeq(0.0, 10.0, tol, 200)
    if ss:
        e.set_systems(ss)
    return e


def _temperature(case):
    return 4000.0 if case.get("matter") == "carbon" else 300.0


def _serve_pool(case, seed):
    """The requests of a serving state: the batch it starts with and those that join later (used round robin)."""
    ss = _many(case, seed, case["systems"] + 4 * LEAVE)
    temps = np.random.default_rng([seed, 3]).uniform(300.0, 3000.0, size=len(ss))
    vels = [systems.maxwell_velocities(s, t, seed=seed + 7 * k) for k, (s, t) in enumerate(zip(ss, temps))]
    return ss, temps, vels


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng([seed, 2])
    if kind == "md":
        s = _one(case, seed)
        e = _engine([s])
        temp = _temperature(case)
        e.md_setup(MASS, dt=DT, t_start=temp, t_damp=TDAMP, chain=CHAIN)
        if not case["charges"]:
            e.set_charges(np.zeros(len(s["type"])))
            e.md_charges(False)
        e.set_velocities(systems.maxwell_velocities(s, temp, seed=seed))
        return {"kind": kind, "e": e, "s": s, "steps": case["steps"], "x0": s["x"].copy(), "box": np.diag(s["box"]).copy()}
    if kind in ("step", "split", "batch"):
        ss = _many(case, seed, case["systems"]) if kind == "batch" else [_one(case, seed)]
        frames = _orbit(np.concatenate([s["x"] for s in ss]), rng)
        n = frames.shape[1]
        grad = None
        if case.get("pinned"):
            locked = rxcuda.pinned_array(frames.shape)
            locked[:] = frames
            frames, grad = locked, rxcuda.pinned_array((n, 3))
        return {"kind": kind, "e": _engine(ss), "frames": frames, "grad": grad, "at": 0}
    if kind == "serve":
        ss, temps, vels = _serve_pool(case, seed)
        k = case["systems"]
        e = _engine(ss[:k])
        e.md_setup(MASS, dt=DT, t_start=300.0, t_damp=TDAMP, chain=CHAIN)
        e.set_velocities(np.concatenate(vels[:k]))
        return {"kind": kind, "e": e, "ss": ss, "temps": temps, "vels": vels, "now": list(range(k)), "next": k,
                "steps": case["steps"]}
    if kind == "point":
        return {"kind": kind, "e": _engine([]), "s": _one(case, seed)}
    if kind == "analysis":
        s = _one(case, seed)
        e = _engine([s])
        if case["matter"] != "carbon":
            e.qeq_solve()
        return {"kind": kind, "e": e}
    if kind == "charges":
        return {"kind": kind, "e": _engine([_one(case, seed)], case["tol"])}
    s = _one(case, seed)
    rs, col, val, eta, chi = _charge_csr(s)
    out = {k: torch.zeros(len(s["type"]), dtype=torch.float64, device="cuda") for k in ("s", "t", "q")}
    counts = torch.zeros(2, dtype=torch.int32, device="cuda")
    rel = torch.zeros(2, dtype=torch.float64, device="cuda")
    lib = rxcuda.load()
    if lib.rx_qeq_solve_static(0, *([None] * 8), 1e-6, 1, None, None, None, None, 0) != 0:
        raise RuntimeError("rx_qeq_solve_static: set-up failed")
    return {"kind": kind, "lib": lib, "rs": rs, "col": col, "val": val, "eta": eta, "chi": chi, "counts": counts, "rel": rel,
            "tol": case["tol"], **out}


# ------------------------------------------------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "static":
        state["s"].zero_()
        state["t"].zero_()
        stream = torch.cuda.current_stream().cuda_stream
        p = {k: v.data_ptr() for k, v in state.items() if isinstance(v, torch.Tensor)}
        err = ctypes.create_string_buffer(128)
        rc = state["lib"].rx_qeq_solve_static(len(state["eta"]), p["rs"], p["col"], p["val"], p["eta"], p["chi"], p["s"], p["t"],
                                              p["q"], state["tol"], 200, p["counts"], p["rel"], stream, err, len(err))
        if rc != 0:
            raise RuntimeError(err.value.decode())
        return {"q": state["q"], "s": state["s"], "t": state["t"]}
    e = state["e"]
    if kind == "md":
        out = e.md_run(state["steps"])
        d = e.get_positions() - state["x0"]     # how far the atoms have gone, in the image nearest their start
        d -= state["box"] * np.round(d / state["box"])
        return {"e": out["e"], "T": out["T"], "moved": d, "v": e.get_velocities(), "q": e.get_charges(), "grad": e.gradient()}
    if kind == "serve":
        joining = [(state["next"] + k) % len(state["ss"]) for k in range(LEAVE)]
        state["next"] += LEAVE
        state["now"] = state["now"][LEAVE:] + joining
        e.update_systems(list(range(LEAVE, len(state["now"]))), [state["ss"][k] for k in joining],
                         [state["vels"][k] for k in joining])
        e.md_targets([float(state["temps"][k]) for k in state["now"]], [1] * len(state["now"]))
        out = e.md_run(state["steps"])
        return {"e": out["e"], "T": out["T"], "v": e.get_velocities(), "q": e.get_charges(), "grad": e.gradient()}
    if kind == "point":
        e.set_systems([state["s"]])
        out = e.compute(qeq=True, cold=True)
        return {"e": out["e"], "grad": out["grad"], "q": e.get_charges(), "virial": e.virial()}
    if kind == "analysis":
        out = e.compute(census=True, peratom=True)
        pe, pv = e.peratom()
        b = e.bonds()
        partner, bo = _bond_table(b["start"], b["partner"], b["bo"])
        return {"e": out["e"], "grad": out["grad"], "virial": e.virial(), "eatom": pe, "vatom": pv, "census": out["census"],
                "partner": partner, "bo": bo, "total_bo": b["total_bo"], "nlp": b["nlp"]}
    if kind == "charges":
        e.qeq_reset()
        return {"q": e.qeq_solve()["q"]}
    x = state["frames"][state["at"] % FRAMES]
    state["at"] += 1
    e.set_positions(x)
    if kind == "batch":
        out = e.compute(qeq=True, cold=True)
        return {"e": out["e"], "grad": out["grad"], "q": e.get_charges(), "virial": e.virial()}
    if kind == "step":
        out = e.compute(qeq=True, grad_out=state["grad"])
        return {"e": out["e"], "grad": out["grad"], "q": e.get_charges(), "virial": e.virial()}
    q = e.qeq_solve()["q"]
    e.set_positions(x)
    e.set_charges(q)
    out = e.compute(grad_out=state["grad"])
    return {"e": out["e"], "grad": out["grad"], "q": q, "virial": e.virial()}


def _bond_table(start, partner, bo):
    """One row per atom (the layout of LAMMPS's fix reaxff/bonds), its bonds in the order of their partners."""
    owner = np.repeat(np.arange(len(start) - 1), np.diff(start))
    order = np.argsort(owner * len(start) + partner, kind="stable")
    col = np.arange(len(owner)) - np.asarray(start)[owner]
    rows = np.full((len(start) - 1, MAX_BONDS), -1, dtype=np.int32), np.zeros((len(start) - 1, MAX_BONDS))
    for table, v in zip(rows, (partner, bo)):
        table[owner, col] = v[order]
    return rows


# ------------------------------------------------------------------------------------------------------- its size
def _density(case):
    """Atoms per A^3 of what a case is made of (water, carbon at 1 g/cm3; a typical CHO request)."""
    return {"water": 0.1003, "carbon": 0.0502}.get(case.get("matter"), 0.12)


def _mean_size(case):
    lo, hi = case["nmin"], case["nmax"]
    return (hi - lo) / math.log(hi / lo)


def work(case):
    """bytes: the state that comes in and goes out once (positions, velocities, charges, gradient, energies; the CSR matrix
    where the caller hands it over). flops: per step and unordered pair within 10 A, 120 for the pair terms, 40 for its
    charge-matrix entry and 8 per fused iteration of the charge solve; per atom, 4000 for the bonded terms (carbon at
    4000 K, with six bonds an atom: 40000)."""
    kind = case["kind"]
    atoms = case["atoms"] if "atoms" in case else case["systems"] * _mean_size(case)
    pairs = atoms * _density(case) * 4.0 / 3.0 * math.pi * 1000.0 / 2.0
    bonded = atoms * (40000.0 if case.get("matter") == "carbon" else 4000.0)
    if kind == "static":
        return {"bytes": 2 * pairs * 12.0 + atoms * 56.0, "flops": 8.0 * pairs * 32}
    if kind == "charges":
        return {"bytes": atoms * 32.0, "flops": pairs * (40.0 + 8.0 * 60)}
    if kind == "analysis":
        return {"bytes": atoms * (24 + 8 + 24 + 56 + 28 + 16 + 48.0), "flops": pairs * 120.0 + bonded}
    if kind in ("md", "serve"):
        solve = 40.0 + 8.0 * 9 if case.get("charges", True) else 0.0
        return {"bytes": atoms * (48 + 48 + 32.0), "flops": case["steps"] * (pairs * (120.0 + solve) + bonded)}
    passes = {"step": 9, "split": 9}.get(kind, 40)
    return {"bytes": atoms * (24 + 24 + 8.0), "flops": pairs * (160.0 + 8.0 * passes) + bonded}


def tolerance(case):
    """About four times the largest relative difference seen when the charge solve's sums are taken in another order, its
    tolerance moved by a fifth or the Verlet rows built with another skin (first and third pass on a state), and of the
    error against `exact`. Charges set it where they are solved (to 1e-6 of the residual): water 4e-6 of the charges, CHO
    systems (worse conditioned) 1.2e-5; without a solve the single-precision pair terms do (1e-6 of the gradient). A
    solve by itself is good to its own tolerance."""
    kind, matter = case["kind"], case.get("matter", "cho")
    if kind in ("charges", "static"):
        return {"rel": max(2e-9, (15.0 if kind == "charges" else 5.0) * case["tol"])}
    if matter == "carbon":
        return {"rel": 5e-6}
    if kind in ("batch", "serve", "point"):
        return {"rel": 5e-5}
    if kind == "md":
        return {"rel": 2e-5}
    return {"rel": 5e-6 if matter == "water" else 3e-5}


# ------------------------------------------------------------------------------------------------------- exact
def exact(case, seed):
    with torch.enable_grad():
        return _exact(case, seed)


_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.asarray(a), device=_DEV)


class _Tables:
    """The force-field file in FP64: one tensor per parameter, indexed by type (`a`), pair (`p`) and so on."""

    def __init__(self):
        rows = [line.split("!")[0].split() for line in _field().splitlines()[1:]]
        at = 0

        def take(n):
            nonlocal at
            at += n
            return rows[at - n:at]

        gp = [float(r[0]) for r in take(int(take(1)[0][0]))]
        nt = int(take(1)[0][0])
        take(3)
        names = ["r_s valency mass r_vdw epsilon gamma r_pi valency_e", "alpha gamma_w valency_boc p_ovun5 - chi eta p_hbond",
                 "r_pi2 p_lp2 - b131 b132 b133 - -", "p_ovun2 p_val3 - valency_val p_val5 rcore ecore acore"]
        a = {}
        self.names = []
        for i in range(nt):
            block = take(4)
            self.names.append(block[0].pop(0))
            for line, row in zip(names, block):
                for nm, v in zip(line.split(), row):
                    a.setdefault(nm, []).append(float(v))
        a = {k: np.array(v) for k, v in a.items() if k != "-"}
        a["eta"] = 2.0 * a["eta"]
        a["nlp_opt"] = 0.5 * (a["valency_e"] - a["valency"])
        a["valency_val"] = np.where(a["mass"] < 21, a["valency_boc"], a["valency_val"])
        p = {}
        count = int(take(1)[0][0])
        take(1)

        def both(nm, i, j, v):
            p.setdefault(nm, np.zeros((nt, nt)))
            p[nm][i, j] = p[nm][j, i] = v

        for _ in range(count):
            u, w = take(2)
            i, j = int(u[0]) - 1, int(u[1]) - 1
            for nm, v in zip("de_s de_p de_pp p_be1 p_bo5 v13 p_bo6 p_ovun1".split(), u[2:]):
                both(nm, i, j, float(v))
            for nm, v in zip("p_be2 p_bo3 p_bo4 - p_bo1 p_bo2 ovc".split(), w):
                both(nm, i, j, float(v))
        mean = lambda v: 0.5 * (v[:, None] + v[None, :])  # noqa: E731
        geo = lambda v: np.sqrt(v[:, None] * v[None, :])  # noqa: E731
        p["r_s"], p["r_p"], p["r_pp"] = mean(a["r_s"]), mean(a["r_pi"]), mean(a["r_pi2"])
        p["p_boc3"], p["p_boc4"], p["p_boc5"] = geo(a["b132"]), geo(a["b131"]), geo(a["b133"])
        p["D"], p["alpha"], p["r_vdw"], p["gamma_w"] = geo(a["epsilon"]), geo(a["alpha"]), 2.0 * geo(a["r_vdw"]), geo(a["gamma_w"])
        p["shield"] = (a["gamma"][:, None] * a["gamma"][None, :]) ** -1.5
        p["rcore"], p["ecore"], p["acore"] = geo(a["rcore"]), geo(a["ecore"]), geo(a["acore"])
        for r in take(int(take(1)[0][0])):
            i, j = int(r[0]) - 1, int(r[1]) - 1
            for nm, scale, v in zip("D r_vdw alpha r_s r_p r_pp".split(), (1, 2, 1, 1, 1, 1), map(float, r[2:])):
                if v > 0:
                    both(nm, i, j, scale * v)
        co = np.isclose(a["mass"], 12.0)[:, None] & np.isclose(a["mass"], 15.999)[None, :]
        p["triple"] = (co | co.T).astype(float)
        # valence sets (up to two a triple in this file), torsions with their wildcards, hydrogen bonds
        th = np.zeros((nt, nt, nt, 2, 7))
        used = np.zeros((nt, nt, nt), dtype=int)
        for r in take(int(take(1)[0][0])):
            i, j, k = (int(v) - 1 for v in r[:3])
            for key in {(i, j, k), (k, j, i)}:
                th[key][used[key]] = [float(v) for v in r[3:10]]
                used[key] += 1
        fb, on, own = np.zeros((nt,) * 4 + (5,)), np.zeros((nt,) * 4, dtype=bool), set()
        for r in take(int(take(1)[0][0])):
            i, j, k, m = (int(v) - 1 for v in r[:4])
            for ii in range(nt) if i < 0 else [i]:
                for mm in range(nt) if m < 0 else [m]:
                    for key in ((ii, j, k, mm), (mm, k, j, ii)):
                        if i >= 0:
                            own.add(key)
                        elif key in own:
                            continue
                        fb[key], on[key] = [float(v) for v in r[4:9]], True
        hb, hon = np.zeros((nt,) * 3 + (4,)), np.zeros((nt,) * 3, dtype=bool)
        for r in take(int(take(1)[0][0])):
            key = tuple(int(v) - 1 for v in r[:3])
            hb[key], hon[key] = [float(v) for v in r[3:7]], True
        self.gp = gp
        self.a = {k: _t(v) for k, v in a.items()}
        self.p = {k: _t(v) for k, v in p.items()}
        self.th, self.fb, self.fb_on, self.hb, self.hb_on = _t(th), _t(fb), _t(on), _t(hb), _t(hon)
        self.carbon = _t(np.array([nm == "C" for nm in self.names]))


def _pairs(x, box, rc, shift=0):
    """Unordered pairs within rc over periodic images: (i, j, L.s) with x_j + L.s - x_i the separation; indices + shift."""
    L = _t(np.asarray(box, dtype=np.float64))
    inv = torch.linalg.inv(L)
    h = (1.0 / inv.norm(dim=0)).tolist()
    n = len(x)
    out = []
    nearest = min(h) > 2.0 * rc
    reach = [0, 0, 0] if nearest else [math.ceil(rc / v) + 1 for v in h]   # + 1: positions may sit outside the cell
    images = [(a, b, c) for a in range(-reach[0], reach[0] + 1) for b in range(-reach[1], reach[1] + 1)
              for c in range(-reach[2], reach[2] + 1)]
    rows = max(1, int(6e7) // n)
    for i0 in range(0, n, rows):
        d0 = x[None, :, :] - x[i0:i0 + rows, None, :]
        if nearest:
            d0 = d0 - torch.round(d0 @ inv) @ L
        i = torch.arange(i0, min(n, i0 + rows), device=x.device)[:, None]
        j = torch.arange(n, device=x.device)[None, :]
        for s in images:
            sv = torch.tensor(s, dtype=torch.float64, device=x.device) @ L
            keep = (j > i) | ((j == i) & (s > (0, 0, 0)))
            hit = torch.nonzero(keep & (((d0 + sv) ** 2).sum(-1) <= rc * rc))
            a, b = hit[:, 0] + i0, hit[:, 1]
            out.append((a + shift, b + shift, d0[hit[:, 0], b] + sv - (x[b] - x[a])))
    return tuple(torch.cat(v) for v in zip(*out))


def _taper(r, rc):
    t = r / rc
    return 1.0 - t ** 4 * (35.0 - 84.0 * t + 70.0 * t ** 2 - 20.0 * t ** 3)


def _lists(ss, xs, rc=10.0):
    got, off = [], 0
    for s, x in zip(ss, xs):
        got.append(_pairs(x, s["box"], rc, off))
        off += len(x)
    return tuple(torch.cat(v) for v in zip(*got))


def _solve_charges(ff, types, sys_of, nsys, x, lists, tol, x0=None, imax=200):
    """The stock charge solve: Jacobi-preconditioned CG on (diag(eta) + H) s = -chi and H t = -1, each system and right-hand
    side stopping at sqrt(r.M^-1 r) / |b| <= tol; q = s - (sum s / sum t) t. Returns q and (s, t)."""
    i, j, sv = lists
    r = (x[j] + sv - x[i]).norm(dim=1)
    h = 14.4 * _taper(r, 10.0) / (r ** 3 + ff.p["shield"][types[i], types[j]]) ** (1.0 / 3.0)
    eta = ff.a["eta"][types][:, None]
    b = torch.stack([-ff.a["chi"][types], -torch.ones_like(x[:, 0])], dim=1)
    n = len(types)
    # the sum over images of a self pair counts twice: both directions are entries of the row
    A = torch.sparse_coo_tensor(torch.stack([torch.cat([i, j]), torch.cat([j, i])]), torch.cat([h, h]), (n, n)).coalesce().to_sparse_csr()
    total = lambda v: torch.zeros(nsys, 2, dtype=torch.float64, device=v.device).index_add_(0, sys_of, v)  # noqa: E731
    z = torch.zeros_like(b) if x0 is None else x0.clone()
    res = b - (eta * z + A @ z)
    d = res / eta
    bn = total(b * b).sqrt()
    sig = total(res * d)
    for _ in range(1, imax):
        live = sig.sqrt() / bn > tol
        if not live.any():
            break
        q = eta * d + A @ d
        alpha = torch.where(live, sig / total(d * q), torch.zeros_like(sig))[sys_of]
        z = z + alpha * d
        res = res - alpha * q
        p = res / eta
        new = torch.where(live, total(res * p), sig)
        d = torch.where(live[sys_of], p + (new / sig)[sys_of] * d, d)
        sig = new
    sums = total(z)
    return z[:, 0] - (sums[:, 0] / sums[:, 1])[sys_of] * z[:, 1], z


def _grouped(owner, n):
    """Every ordered pair of different entries with the same owner, from `owner` sorted ascending."""
    cnt = torch.bincount(owner, minlength=n)
    start = torch.cumsum(cnt, 0) - cnt
    first = torch.repeat_interleave(torch.arange(len(owner), device=owner.device), cnt[owner])
    base = torch.cumsum(cnt[owner], 0) - cnt[owner]
    second = start[owner[first]] + torch.arange(len(first), device=owner.device) - base[first]
    return first, second


def _sorted_by(owner, *more):
    order = torch.argsort(owner, stable=True)
    return tuple(v[order] for v in (owner,) + more)


def _energies(ff, types, sys_of, nsys, x, lists, q):
    """The 13 energies of every system (nsys, 13): bond, over, under, lone pair, valence, penalty, coalition, H-bond,
    torsion, conjugation, van der Waals, Coulomb, polarization."""
    gp, a, p = ff.gp, ff.a, ff.p
    n, dev = len(types), x.device
    terms = [None] * 13

    def per_system(v, atom):
        return torch.zeros(nsys, dtype=torch.float64, device=dev).index_add(0, sys_of[atom], v)

    def per_atom(v, atom):
        return torch.zeros(n, dtype=torch.float64, device=dev).index_add(0, atom, v)

    # ---- pairs
    i, j, sv = lists
    r = (x[j] + sv - x[i]).norm(dim=1)
    P = {k: v[types[i], types[j]] for k, v in p.items() if k in ("D", "alpha", "r_vdw", "gamma_w", "rcore", "ecore", "acore", "shield")}
    tap = _taper(r, gp[12])
    fn = (r ** gp[28] + P["gamma_w"] ** -gp[28]) ** (1.0 / gp[28])
    e2 = torch.exp(0.5 * P["alpha"] * (1.0 - fn / P["r_vdw"]))
    terms[10] = per_system(tap * (P["D"] * (e2 * e2 - 2.0 * e2) + P["ecore"] * torch.exp(P["acore"] * (1.0 - r / P["rcore"]))), i)
    terms[11] = per_system(332.06371 * q[i] * q[j] * tap / (r ** 3 + P["shield"]) ** (1.0 / 3.0), i)
    every = torch.arange(n, device=dev)
    terms[12] = per_system(23.02 * (a["chi"][types] * q + 0.5 * a["eta"][types] * q * q), every)
    # ---- bond orders of the directed bonds
    bo_cut = 0.01 * gp[29]
    near = torch.nonzero(r.detach() <= 5.0)[:, 0]
    bi, bj = torch.cat([i[near], j[near]]), torch.cat([j[near], i[near]])
    bs = torch.cat([sv[near], -sv[near]])

    def uncorrected(bi, bj, bs):
        dv = x[bj] + bs - x[bi]
        d = dv.norm(dim=1)
        ti, tj = types[bi], types[bj]

        def part(reach, r0, p1, p2, scale):
            has = (a[reach][ti] > 0) & (a[reach][tj] > 0)
            ratio = d / torch.where(has, p[r0][ti, tj], torch.ones_like(d))
            return torch.where(has, scale * torch.exp(p[p1][ti, tj] * ratio ** p[p2][ti, tj]), torch.zeros_like(d))
        return dv, d, part("r_s", "r_s", "p_bo1", "p_bo2", 1.0 + bo_cut), part("r_pi", "r_p", "p_bo3", "p_bo4", 1.0), \
            part("r_pi2", "r_pp", "p_bo5", "p_bo6", 1.0)
    with torch.no_grad():
        _, _, s0, s1, s2 = uncorrected(bi, bj, bs)
        keep = torch.nonzero(s0 + s1 + s2 >= bo_cut)[:, 0]
    bi, bj, bs = _sorted_by(bi[keep], bj[keep], bs[keep])
    dv, d, sg, pi, pp = uncorrected(bi, bj, bs)
    ti, tj = types[bi], types[bj]
    B = {k: v[ti, tj] for k, v in p.items()}
    bo = sg + pi + pp - bo_cut
    tbo = per_atom(bo, bi)
    Dp, Dpb = tbo - a["valency"][types], tbo - a["valency_val"][types]
    e1, eb2 = torch.exp(-gp[0] * Dp), torch.exp(-gp[1] * Dp)
    f2 = e1[bi] + e1[bj]
    f3 = -torch.log(0.5 * (eb2[bi] + eb2[bj])) / gp[1]
    vi, vj = a["valency"][ti], a["valency"][tj]
    one = torch.ones_like(bo)
    f1 = torch.where(B["ovc"] >= 0.001, 0.5 * ((vi + f2) / (vi + f2 + f3) + (vj + f2) / (vj + f2 + f3)), one)
    f45 = one
    for end in (bi, bj):
        f45 = f45 * torch.where(B["v13"] >= 0.001, 1.0 / (1.0 + torch.exp(-(B["p_boc4"] * bo * bo - Dpb[end]) * B["p_boc3"] + B["p_boc5"])), one)
    full = bo * f1 * f45
    pi, pp = pi * f1 * f1 * f45, pp * f1 * f1 * f45
    sg = full - pi - pp
    bo, sg, pi, pp = (torch.where(v < 1e-10, torch.zeros_like(v), v) for v in (full, sg, pi, pp))
    tbo = per_atom(bo, bi)
    A = {k: v[types] for k, v in a.items()}
    Delta, De, Dboc, Dval = (tbo - A[k] for k in ("valency", "valency_e", "valency_boc", "valency_val"))
    trunc = torch.trunc(De.detach() / 2.0)
    vlpex = De - 2.0 * trunc
    nlp = torch.exp(-gp[15] * (2.0 + vlpex) ** 2) - trunc
    Dlp = A["nlp_opt"] - nlp
    # ---- bond energy (both directions of a bond share it), with the triple-bond term of C-O
    positive = sg > 0
    power = torch.where(positive, torch.where(positive, sg, one) ** B["p_be2"], torch.zeros_like(sg))
    eb = -B["de_s"] * sg * torch.exp(B["p_be1"] * (1.0 - power)) - B["de_p"] * pi - B["de_pp"] * pp
    hu = gp[10] * torch.exp(-gp[7] * (bo - 2.5) ** 2) / (1.0 + 25.0 * torch.exp(gp[4] * (Delta[bi] + Delta[bj]))) * \
        (torch.exp(-gp[3] * (tbo[bi] - bo)) + torch.exp(-gp[3] * (tbo[bj] - bo)))
    eb = eb + torch.where((bo >= 1.0) & (B["triple"] > 0), hu, torch.zeros_like(hu))
    terms[0] = 0.5 * per_system(eb, bi)
    # ---- lone pair, C2
    terms[3] = per_system(A["p_lp2"] * Dlp / (1.0 + torch.exp(torch.clamp(-75.0 * Dlp, max=700.0))), every)
    vov = bo - Delta[bi] - 0.04 * Delta[bi] ** 4
    c2 = ff.carbon[ti] & ff.carbon[tj] & (vov > 3.0)
    terms[3] = terms[3] + per_system(torch.where(c2, gp[5] * (vov - 3.0) ** 2, torch.zeros_like(vov)), bi)
    # ---- over and under coordination (no type of this file is heavier than 21)
    sum1 = per_atom(B["p_ovun1"] * B["de_s"] * bo, bi)
    sum2 = per_atom((Delta - Dlp)[bj] * (pi + pp), bi)
    sexp = lambda v: torch.exp(torch.clamp(v, max=700.0))  # noqa: E731
    corr = Delta - Dlp / (1.0 + gp[32] * sexp(gp[31] * sum2))
    terms[1] = per_system(sum1 * corr / (corr + A["valency"] + 1e-8) / (1.0 + sexp(A["p_ovun2"] * corr)), every)
    terms[2] = per_system(-A["p_ovun5"] * (1.0 - sexp(gp[6] * corr)) / (1.0 + sexp(-A["p_ovun2"] * corr)) /
                          (1.0 + gp[8] * sexp(gp[9] * sum2)), every)
    # ---- valence angles, penalty, coalition: unordered pairs of bonds of one centre
    thb = 0.001
    u, w = _grouped(bi, n)
    b0 = bo.detach()
    sel = (u < w) & (b0[u] > thb) & (b0[w] > thb) & (b0[u] * b0[w] > 1e-5)
    u, w = u[sel], w[sel]
    c = bi[u]
    sbop = per_atom(pi + pp, bi)
    prod = torch.exp(-per_atom(bo ** 8, bi))
    sbo = sbop + (1.0 - prod) * (-Dboc - gp[33] * torch.where(vlpex >= 0, torch.zeros_like(nlp), nlp))
    lowp, highp = (sbo > 0) & (sbo <= 1), (sbo > 1) & (sbo < 2)
    half = torch.full_like(sbo, 0.5)
    sbo2 = torch.where(lowp, torch.where(lowp, sbo, half) ** gp[16], torch.where(
        highp, 2.0 - (2.0 - torch.where(highp, sbo, half)) ** gp[16], torch.where(sbo >= 2, 2.0 * torch.ones_like(sbo), torch.zeros_like(sbo))))
    cosine = ((dv[u] * dv[w]).sum(1) / (d[u] * d[w])).clamp(-1.0 + 1e-14, 1.0 - 1e-14)
    theta = torch.acos(cosine)
    Bu, Bw = bo[u] - thb, bo[w] - thb
    ex6 = torch.exp(gp[14] * Dboc[c])
    pen3, pen4 = torch.exp(-gp[20] * Delta[c]), torch.exp(gp[21] * Delta[c])
    va, pe, co = 0.0, 0.0, 0.0
    for k in range(ff.th.shape[3]):
        t00, v1, v2, coa1, v7, pen1, v4 = ff.th[types[bj[u]], types[c], types[bj[w]], k].unbind(1)
        has = v1.abs() > 0.001
        f7 = [1.0 - torch.exp(-A["p_val3"][c] * v ** v4) for v in (Bu, Bw)]
        v5 = A["p_val5"][c]
        f8 = v5 - (v5 - 1.0) * (2.0 + ex6) / (1.0 + ex6 + torch.exp(-v7 * Dboc[c]))
        t0 = (180.0 - t00 * (1.0 - torch.exp(-gp[17] * (2.0 - sbo2[c])))) * 3.14159265 / 180.0
        bell = torch.exp(-v2 * (t0 - theta) ** 2)
        zero = torch.zeros_like(bell)
        va = va + torch.where(has, f7[0] * f7[1] * f8 * torch.where(v1 >= 0, v1 * (1.0 - bell), -v1 * bell), zero)
        pe = pe + torch.where(has, pen1 * (2.0 + pen3) / (1.0 + pen3 + pen4) * torch.exp(-gp[19] * ((Bu - 2.0) ** 2 + (Bw - 2.0) ** 2)), zero)
        co = co + torch.where(has, coa1 / (1.0 + torch.exp(gp[2] * Dval[c])) * torch.exp(
            -gp[38] * ((tbo[bj[u]] - Bu) ** 2 + (tbo[bj[w]] - Bw) ** 2) - gp[30] * ((Bu - 1.5) ** 2 + (Bw - 1.5) ** 2)), zero)
    terms[4], terms[5], terms[6] = per_system(va, c), per_system(pe, c), per_system(co, c)
    # ---- hydrogen bonds: donor bond of a hydrogen x acceptor within 7.5 A of it
    hb_kind = a["p_hbond"].long()
    hi, hj, hs = torch.cat([i, j]), torch.cat([j, i]), torch.cat([sv, -sv])
    ok = (hb_kind[types[hi]] == 1) & (hb_kind[types[hj]] == 2) & (torch.cat([r, r]).detach() <= 7.5)
    hi, hj, hs = _sorted_by(hi[ok], hj[ok], hs[ok])
    donor = torch.nonzero((hb_kind[ti] == 1) & (hb_kind[tj] == 2) & (b0 >= 1e-2))[:, 0]
    cnt = torch.bincount(hi, minlength=n)
    first = torch.cumsum(cnt, 0) - cnt
    m = cnt[bi[donor]]
    db = torch.repeat_interleave(donor, m)
    ac = first[bi[db]] + torch.arange(len(db), device=dev) - torch.repeat_interleave(torch.cumsum(m, 0) - m, m)
    ok = (bj[db] != hj[ac]) & ff.hb_on[types[bj[db]], types[bi[db]], types[hj[ac]]]
    db, ac = db[ok], ac[ok]
    r0, h1, h2, h3 = ff.hb[types[bj[db]], types[bi[db]], types[hj[ac]]].unbind(1)
    dk = x[hj[ac]] + hs[ac] - x[hi[ac]]
    rk = dk.norm(dim=1)
    cs = (dv[db] * dk).sum(1) / (d[db] * rk)
    terms[7] = per_system(h1 * (1.0 - torch.exp(-h2 * bo[db])) * torch.exp(-h3 * (r0 / rk + rk / r0 - 2.0)) * (0.5 * (1.0 - cs)) ** 2, bi[db])
    # ---- torsions and conjugation: central bond c (one of its two directions), bond u of its atom, bond w of the other
    code = lambda s: (s * 1e3).round().long()  # noqa: E731
    sc = code(bs)
    later = (sc[:, 0] > 0) | ((sc[:, 0] == 0) & ((sc[:, 1] > 0) | ((sc[:, 1] == 0) & (sc[:, 2] > 0))))
    central = torch.nonzero((b0 > thb) & ((bi < bj) | ((bi == bj) & later)))[:, 0]
    nb = torch.bincount(bi, minlength=n)
    bstart = torch.cumsum(nb, 0) - nb
    combos = nb[bi[central]] * nb[bj[central]]
    ce = torch.repeat_interleave(central, combos)
    rank = torch.arange(len(ce), device=dev) - torch.repeat_interleave(torch.cumsum(combos, 0) - combos, combos)
    u = bstart[bi[ce]] + torch.div(rank, nb[bj[ce]], rounding_mode="floor")
    w = bstart[bj[ce]] + rank % nb[bj[ce]]
    back = (bj[w] == bi[ce]) & ((bs[w] + bs[ce]).abs().sum(1) < 1e-6)
    same = (bj[u] == bj[w]) & ((bs[ce] + bs[w] - bs[u]).abs().sum(1) < 1e-6)
    ok = (u != ce) & ~back & ~same & (b0[u] > thb) & (b0[w] > thb) & (b0[u] * b0[ce] * b0[w] > thb) & \
        ff.fb_on[types[bj[u]], types[bi[ce]], types[bj[ce]], types[bj[w]]]
    ce, u, w = ce[ok], u[ok], w[ok]
    V1, V2, V3, t1, c1 = ff.fb[types[bj[u]], types[bi[ce]], types[bj[ce]], types[bj[w]]].unbind(1)
    dij, djk, dkl = dv[u], dv[ce], dv[w]
    dot = lambda m1, m2: (m1 * m2).sum(1)  # noqa: E731
    cos1 = dot(djk, dij) / (d[ce] * d[u])
    cos2 = -dot(djk, dkl) / (d[ce] * d[w])
    sin1 = torch.sqrt((1.0 - cos1 * cos1).clamp(min=1e-20))
    sin2 = torch.sqrt((1.0 - cos2 * cos2).clamp(min=1e-20))
    uc = -dot(dij, djk) * dot(djk, dkl) + d[ce] ** 2 * dot(dij, dkl)
    us = -d[ce] * dot(dij, torch.linalg.cross(djk, dkl))
    co = uc / torch.sqrt(uc * uc + us * us)
    cos2w, cos3w = 2.0 * co * co - 1.0, co * (4.0 * co * co - 3.0)
    Dsum = Dboc[bi[ce]] + Dboc[bj[ce]]
    x3, x4 = torch.exp(-gp[24] * Dsum), torch.exp(gp[25] * Dsum)
    f11 = (2.0 + x3) / (1.0 + x3 + x4)
    boa = [bo[k] - thb for k in (u, ce, w)]
    f10 = 1.0
    f12 = 1.0
    for v in boa:
        f10 = f10 * (1.0 - torch.exp(-gp[23] * v))
        f12 = f12 * torch.exp(-gp[27] * (v - 1.5) ** 2)
    CV = 0.5 * (V1 * (1.0 + co) + V2 * torch.exp(t1 * (2.0 - pi[ce] - f11) ** 2) * (1.0 - cos2w) + V3 * (1.0 + cos3w))
    terms[8] = per_system(f10 * sin1 * sin2 * CV, bi[ce])
    terms[9] = per_system(c1 * f12 * (1.0 + (co * co - 1.0) * sin1 * sin2), bi[ce])
    return torch.stack(terms, dim=1), (bi, bj, bs, bo, tbo, nlp)


def _evaluate(ff, ss, xs, types, sys_of, q=None, tol=1e-6, guess=None):
    """Energies, gradient, charges, the solve's (s, t) and the bond table of positions xs, with charges solved unless given."""
    x = torch.cat(xs).detach().requires_grad_(True)
    lists = _lists(ss, [v.detach() for v in xs])
    z = None
    if q is None:
        with torch.no_grad():
            q, z = _solve_charges(ff, types, sys_of, len(ss), x.detach(), lists, tol, guess)
    # the energy of all systems on positions x + strain x gives the virial as well: -dE/dstrain
    strain = torch.zeros(len(ss), 3, 3, dtype=torch.float64, device=x.device, requires_grad=True)
    full = x + (x[:, None, :] @ strain[sys_of])[:, 0]
    i, j, sv = lists
    svs = sv + (sv[:, None, :] @ strain[sys_of[i]])[:, 0]
    e, bonds = _energies(ff, types, sys_of, len(ss), full, (i, j, svs), q)
    g, w = torch.autograd.grad(e.sum(), (x, strain))
    w = -w
    vir = torch.stack([w[:, 0, 0], w[:, 1, 1], w[:, 2, 2], w[:, 0, 1], w[:, 0, 2], w[:, 1, 2]], dim=1)
    return {"e": e.detach(), "grad": g, "q": q, "z": z, "virial": vir, "bonds": [v.detach() for v in bonds]}


def _host(v):
    return v.detach().cpu().numpy()


def _exact(case, seed):
    kind = case["kind"]
    ff = _Tables()
    if kind == "serve" or (kind == "md" and (case["atoms"] > 3000 or not case["charges"])):
        return None   # tens of evaluations of tens of thousands of atoms: a whole call, compared with another run only
    if kind == "batch":
        if case["systems"] > 200:
            return None
        ss = _many(case, seed, case["systems"])
    else:
        ss = [_one(case, seed)]
    types = torch.cat([_t(s["type"]).long() for s in ss])
    sys_of = torch.repeat_interleave(torch.arange(len(ss), device=_DEV), torch.tensor([len(s["type"]) for s in ss], device=_DEV))
    xs = [_t(s["x"]) for s in ss]
    if kind in ("step", "split", "batch"):
        frame = _orbit(np.concatenate([s["x"] for s in ss]), np.random.default_rng([seed, 2]))[0]
        xs = list(torch.split(_t(frame), [len(s["type"]) for s in ss]))
    if kind in ("charges", "static"):
        with torch.no_grad():
            q, z = _solve_charges(ff, types, sys_of, 1, xs[0], _lists(ss, xs), case["tol"])
        return {"q": _host(q)} if kind == "charges" else {"q": _host(q), "s": _host(z[:, 0]), "t": _host(z[:, 1])}
    if kind == "md":
        return _exact_md(ff, case, seed, ss, xs, types, sys_of)
    q = None if kind != "analysis" or case["matter"] != "carbon" else torch.zeros(len(types), dtype=torch.float64, device=_DEV)
    r = _evaluate(ff, ss, xs, types, sys_of, q)
    out = {k: _host(r[k]) for k in ("e", "grad", "virial")}
    if kind == "analysis":
        bi, bj, bs, bo, tbo, nlp = (_host(v) for v in r["bonds"])
        start = np.searchsorted(bi, np.arange(len(tbo) + 1))
        partner, bo = _bond_table(start, bj, bo)
        out.update(eatom=None, vatom=None, census=None, partner=partner, bo=bo, total_bo=tbo, nlp=nlp)
        return out
    return dict(out, q=_host(r["q"]))


def _exact_md(ff, case, seed, ss, xs, types, sys_of):
    """Velocity Verlet with a Nose-Hoover chain (Martyna, Tuckerman and Klein, Mol. Phys. 87, 1117 (1996)) applied for dt/2 on
    each side of a step, the charge guesses extrapolated from the last four solutions."""
    temp = _temperature(case)
    v = _t(systems.maxwell_velocities(ss[0], temp, seed=seed))
    m = _t(ss[0]["mass"])[:, None]
    ftm = 1.0 / 48.88821291 ** 2
    n = len(types)
    kT, nf = 0.0019872067 * temp, 3.0 * n - 3.0
    Q = [nf * kT * TDAMP ** 2] + [kT * TDAMP ** 2] * (CHAIN - 1)
    vx = [0.0] * CHAIN
    hist = [torch.zeros(n, 2, dtype=torch.float64, device=_DEV) for _ in range(4)]
    box = _t(np.diag(ss[0]["box"]))
    x = xs[0].clone()

    def forces():
        h = hist
        guess = torch.stack([4 * (h[0][:, 0] + h[2][:, 0]) - (6 * h[1][:, 0] + h[3][:, 0]), h[2][:, 1] + 3 * (h[0][:, 1] - h[1][:, 1])], dim=1)
        r = _evaluate(ff, ss, [x], types, sys_of, guess=guess)
        hist.insert(0, r["z"])
        hist.pop()
        return r

    def chain(v):
        ke2 = float((m * v * v).sum()) / ftm

        def push(k):
            return ((ke2 - nf * kT) if k == 0 else (Q[k - 1] * vx[k - 1] ** 2 - kT)) / Q[k]
        vx[-1] += push(CHAIN - 1) * 0.25 * DT
        for k in range(CHAIN - 2, -1, -1):
            f = math.exp(-vx[k + 1] * 0.125 * DT)
            vx[k] = (vx[k] * f + push(k) * 0.25 * DT) * f
        scale = math.exp(-vx[0] * 0.5 * DT)
        ke2 *= scale * scale
        for k in range(CHAIN - 1):
            f = math.exp(-vx[k + 1] * 0.125 * DT)
            vx[k] = (vx[k] * f + push(k) * 0.25 * DT) * f
        vx[-1] += push(CHAIN - 1) * 0.25 * DT
        return v * scale, ke2 / (nf * 0.0019872067)

    r = forces()
    for _ in range(case["steps"]):
        v, _t0 = chain(v)
        v = v - 0.5 * DT * ftm * r["grad"] / m
        x = x + DT * v
        r = forces()
        v = v - 0.5 * DT * ftm * r["grad"] / m
        v, heat = chain(v)
    d = x - xs[0]
    d = d - box * torch.round(d / box)
    return {"e": _host(r["e"]), "T": np.array([heat]), "moved": _host(d), "v": _host(v), "q": _host(r["q"]), "grad": _host(r["grad"])}


def _charge_csr(s):
    """The charge matrix of a system as CSR on the device (every image of a pair summed into its entry), eta and chi."""
    ff = _Tables()
    types = _t(s["type"]).long()
    x = _t(s["x"])
    i, j, sv = _pairs(x, s["box"], 10.0)
    r = (x[j] + sv - x[i]).norm(dim=1)
    h = 14.4 * _taper(r, 10.0) / (r ** 3 + ff.p["shield"][types[i], types[j]]) ** (1.0 / 3.0)
    n = len(types)
    A = torch.sparse_coo_tensor(torch.stack([torch.cat([i, j]), torch.cat([j, i])]), torch.cat([h, h]), (n, n)).coalesce().to_sparse_csr()
    return (A.crow_indices().int().contiguous(), A.col_indices().int().contiguous(), A.values().contiguous(),
            ff.a["eta"][types].contiguous(), ff.a["chi"][types].contiguous())
