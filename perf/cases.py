"""The work users have the engine do, as cases to be timed and compared.

Every case goes through the public entry points of `tis_gb300`.  The systems are the
repository's own synthetic TIS chains (76, 346 and 1500 nucleotides, and lengths in
between) with explicit Mg2+, Cl- and K+ ions, equilibrated before they are measured: the
set-up chain is strained and its lists are all equally old, which no running simulation
meets.  A case is a dict of plain values:

  kind        md | dropin | upload | terms | param_grad | traj_grad | pair_lists | analysis
  n_nt, box   chain length and cubic box side (A)
  replicas    independent replicas advanced together (Mg2+ swept over mg_lo .. mg_hi mM)
  kcl         K+ concentration, mM (Cl- neutralises)
  rc, debye   Coulomb cutoff (A) and screening length (A; 0: unscreened)
  fp64        True: the all-FP64 path; False: the mixed-precision path
  steps       steps of one pass
  interval    traj_grad: checkpoint interval; analysis: steps between frames
"""
import math
import os
import shutil
import sys
import tempfile
from concurrent.futures import ThreadPoolExecutor
from functools import lru_cache

os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")  # as bench.py: a hardware queue per replica group

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "16s-central-folding_gb300"))

from tis_gb300 import (ENERGY_NAMES, PREC_FP64, PREC_MIXED, STATE_NAMES, TERM_BONDED, TERM_LR, TERM_SR,  # noqa: E402
                       TERM_STACK, Engine, System, synth)
from tis_gb300.api import pair_lists_noalloc  # noqa: E402

T_298 = 0.59219
STEP = 0.05  # integration step of the force field's time unit
SIG0 = 1.5852
SR_LIST, LR_SKIN = 15.0, 3.0  # SR list radius; skin added to rc for the LR list
MG, CL, K_ION = 3, 4, 5
FORCE_TERMS = TERM_SR | TERM_LR | TERM_BONDED | TERM_STACK


def _case(kind, n_nt, box, replicas=1, mg=(5.0, 5.0), kcl=76.0, rc=30.0, debye=0.0, fp64=False, steps=1, interval=0):
    return dict(kind=kind, n_nt=n_nt, box=box, replicas=replicas, mg_lo=mg[0], mg_hi=mg[1], kcl=kcl, rc=rc, debye=debye,
                fp64=fp64, steps=steps, interval=interval)


def listed():
    small = dict(n_nt=76, box=200.0, mg=(2.0, 2.0), kcl=50.0)
    central = dict(n_nt=346, box=350.0)
    large = dict(n_nt=1500, box=600.0, mg=(10.0, 10.0), kcl=150.0)
    cases = [
        # one replica of the shortest chain in double precision, read back often: latency and launches
        ("md_small_fp64", _case("md", **small, fp64=True, steps=20)),
        # one replica of the central-domain-size chain, the single-trajectory user
        ("md_central", _case("md", **central, steps=100)),
        # a few replicas of an odd size at the engine's default 50 A cutoff with screened Coulomb, a step
        # count that is no multiple of the graph length
        ("md_ragged", _case("md", n_nt=203, box=277.5, replicas=7, mg=(0.0, 7.5), kcl=90.0, rc=50.0, debye=10.0, steps=33)),
        # the benchmark's batch: 64 replicas, Mg2+ swept over 0-20 mM
        ("md_batch64", _case("md", **central, replicas=64, mg=(0.0, 20.0), steps=100)),
        # the largest system: 16 replicas of the 1500-nt chain, 48.9k particles each
        ("md_large16", _case("md", **large, replicas=16, steps=40)),
        # the reference's run loop with its four routines called one by one
        ("dropin_central", _case("dropin", **central, steps=10)),
        # a sampler that moves states between host and engine: upload, list build, 20 steps, a frame back
        ("upload_batch64", _case("upload", **central, replicas=64, mg=(0.0, 20.0), steps=20)),
        # a frame's force terms and energies (parity checks, minimisers, analysis)
        ("terms_central", _case("terms", **central)),
        # dU/dtheta of 64 stored frames (force-field fitting)
        ("param_grad64", _case("param_grad", **central, replicas=64)),
        # gradient through a fixed-noise trajectory of 16 replicas, checkpoints every 10 steps
        ("traj_grad16", _case("traj_grad", **central, replicas=16, steps=40, interval=10)),
        # the allocation-free pair list of the largest system on caller-owned device buffers
        ("pair_lists_large", _case("pair_lists", **large)),
        # ion observables along a run: fitted density grid and bound ions every 20 steps
        ("analysis_central", _case("analysis", **central, steps=100, interval=20)),
    ]
    return [dict(c, name=n) for n, c in cases]


def draw(rng):
    kind = rng.choice(["md", "md", "md", "md", "dropin", "upload", "terms", "param_grad", "traj_grad", "pair_lists", "analysis"])

    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    n_nt = log_int(76, 1500 if kind in ("md", "pair_lists", "upload") else 700)
    box = round(200.0 * (n_nt / 76.0) ** 0.368 * rng.uniform(0.95, 1.1), 1)
    # replicas: up to the batch of 64, within the particle count of the largest listed case
    most = {"md": 64, "upload": 64, "param_grad": 64, "traj_grad": 16, "dropin": 8}.get(kind, 1)
    kcl = round(rng.uniform(50.0, 150.0), 1)
    mg = sorted((round(rng.uniform(0.0, 10.0), 2), round(rng.uniform(0.0, 20.0), 2)))
    per = 3 * n_nt + sum(_ion_numbers(mg[1], kcl, box, n_nt))
    budget = {"md": 700000, "upload": 340000, "param_grad": 340000, "traj_grad": 80000}.get(kind, 60000)
    replicas = log_int(1, max(1, min(most, budget // per)))
    c = _case(kind, n_nt, box, replicas, mg, kcl, rc=rng.choice([30.0, 30.0, 40.0, 50.0]) if box > 212.0 else 30.0,
              debye=rng.choice([0.0, 0.0, 10.0]), fp64=rng.random() < 0.25 and per * replicas < 60000)
    if kind == "md":
        c["steps"] = log_int(7, 40 if per * replicas > 350000 or c["fp64"] else 100)
    elif kind in ("dropin", "upload"):
        c["steps"] = log_int(3, 20)
    elif kind == "traj_grad":
        c.update(steps=log_int(5, 30), interval=rng.randint(3, 10))
    elif kind == "analysis":
        c["interval"] = log_int(5, 30)
        c["steps"] = c["interval"] * rng.randint(2, 5)
    return c


# ---- systems ---------------------------------------------------------------------------
def _ion_numbers(mg_mm, kcl_mm, box, n_nt):
    return synth.ion_counts_for(mg_mm * 1e-3, kcl_mm * 1e-3, box, 2 * n_nt - 1)


@lru_cache(maxsize=None)
def _chain(n_nt, box, rc):
    """Arrays of the ion-free chain; every replica of a case is the same molecule: the first of the
    generator's that came out without overlapping beads, each try in a wider coil."""
    d = tempfile.mkdtemp(prefix="tis_chain_")
    try:
        for k in range(8):
            f = synth.generate(d, "chain", n_nt, seed=4000 + k, n_hb_pairs=max(4, n_nt // 3),
                               density=(400.0 if n_nt < 400 else 900.0) * (1 + 0.25 * k))
            s = System.load(f["pdb"], f["bonds"], f["stacks"], f["maxikey"], T=T_298, box=box, rc=rc, n_mg=0, n_cl=0, n_k=0,
                            seed=1, center=(3 * n_nt) // 2, rng=1)
            a = s.to_dict()
            x = torch.from_numpy(np.stack([a["x"], a["y"], a["z"]], 1))
            if float(torch.nn.functional.pdist(x).min()) > 3.3:
                return a
        raise RuntimeError("no chain of %d nucleotides without overlaps" % n_nt)
    finally:
        shutil.rmtree(d)


def _arrays(case, seed, r):
    """One replica: the chain, ions at random non-overlapping places, thermal velocities."""
    rng = np.random.default_rng([int(seed), r])
    a = dict(_chain(case["n_nt"], case["box"], case["rc"]))
    L = case["box"]
    mg = case["mg_lo"] + (case["mg_hi"] - case["mg_lo"]) * (r / max(1, case["replicas"] - 1))
    counts = _ion_numbers(mg, case["kcl"], L, case["n_nt"])
    n_ion = sum(counts)
    beads = np.stack([a["x"], a["y"], a["z"]], 1)
    # sites of a 7 A lattice, jittered by up to 1.5 A (so at least 4 A apart), away from the beads
    m = int(L / 7.0)
    taken = np.zeros((m, m, m), dtype=bool)
    at = np.floor(np.mod(beads, L) / (L / m)).astype(int) % m
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                taken[(at[:, 0] + dx) % m, (at[:, 1] + dy) % m, (at[:, 2] + dz) % m] = True
    free = np.flatnonzero(~taken.reshape(-1))
    site = np.stack(np.unravel_index(rng.choice(free, n_ion, replace=False), (m, m, m)), 1)
    pos = (site + 0.5) * (L / m) + rng.uniform(-1.5, 1.5, (n_ion, 3))
    kind = np.repeat([MG, CL, K_ION], counts).astype(np.int32)
    a["kind"] = np.concatenate([a["kind"], kind])
    a["type"] = np.concatenate([a["type"], kind + 4]).astype(np.int32)
    x = np.concatenate([beads, pos])
    v = rng.normal(size=x.shape) * np.sqrt(T_298 / a["mass"][a["type"] - 1])[:, None]
    for c, k in enumerate("xyz"):
        a[k], a["o" + k], a["v" + k] = x[:, c].copy(), x[:, c] - STEP * v[:, c], v[:, c].copy()
    a["n_particles"] = np.array([len(x)], dtype=np.int64)
    a["n_ions"] = np.array(counts, dtype=np.int32)
    a["seed"] = np.array([1000 * (int(seed) % 1000003) + r + 1], dtype=np.int64)
    a["debye"] = np.array([case["debye"]])
    return a


def _systems(case, seed):
    _chain(case["n_nt"], case["box"], case["rc"])
    with ThreadPoolExecutor(8) as ex:
        arrays = list(ex.map(lambda r: _arrays(case, seed, r), range(case["replicas"])))
    return arrays, [System.from_arrays(a) for a in arrays]


def _equilibrated(case, systems):
    """The replicas' states after mixed-precision steps from their set-up: enough for the strained
    angles of the generated chain to open (measured: folded P-S-B triples are gone after 3000)."""
    steps = 4000 if len(systems) * case["n_nt"] < 10000 else 3000 if case["n_nt"] < 700 else 1500
    e = Engine(systems, precision=PREC_MIXED)
    e.populate_lists()
    e.step(steps)
    e.sync()
    st = e.get_states()
    e.close()
    return st


def _pinned(n):
    return torch.zeros(n, dtype=torch.float64).pin_memory().numpy()


def _pinned_states(st):
    out = {k: _pinned(v.size) for k, v in st.items()}
    for k, v in st.items():
        out[k][:] = v
    return out


# ---- the measured calls -----------------------------------------------------------------
def prepare(case, seed):
    arrays, systems = _systems(case, seed)
    n = sum(a["x"].size for a in arrays)
    precision = PREC_FP64 if case["fp64"] else PREC_MIXED
    s = dict(case=case)
    if case["kind"] == "pair_lists":
        st = _equilibrated(case, systems)
        xyz = np.mod(np.stack([st[k] for k in "xyz"]), case["box"])
        s["xyz"] = torch.from_numpy(xyz).cuda()
        s["part"] = torch.from_numpy(arrays[0]["kind"]).cuda()
        rho = n / case["box"] ** 3
        caps = [int(0.5 * n * rho * 4.19 * (1.3 * r) ** 3) + 40 * 3 * case["n_nt"] for r in (SR_LIST, case["rc"] + LR_SKIN)]
        s["sr"], s["lr"] = (torch.zeros((c, 2), dtype=torch.int32, device="cuda") for c in caps)
        s["counts"] = torch.zeros(3, dtype=torch.int64, device="cuda")
        return s
    one_group = dict(groups=1) if case["kind"] in ("param_grad", "traj_grad") else {}
    st = _pinned_states(_equilibrated(case, systems))
    e = Engine(systems, precision=precision, **one_group)
    e.set_states(st)
    s["engine"] = e
    if case["kind"] in ("md", "upload", "dropin", "analysis"):
        e.populate_lists()
        if case["kind"] != "dropin":  # a running program has captured its graphs; the lists age as in a run
            e.step(case["interval"] or case["steps"])
            e.sync()
    s["out"] = {k: _pinned(n) for k in (("x", "y", "z") if case["kind"] == "upload" else STATE_NAMES)}
    s["energies"] = torch.zeros((case["replicas"], 5), dtype=torch.float64).pin_memory().numpy()
    if case["kind"] in ("upload", "param_grad", "traj_grad"):
        s["states"] = st
    if case["kind"] == "terms":
        s["state"] = {k: v.copy() for k, v in st.items()}
    if case["kind"] == "traj_grad":
        rng = np.random.default_rng([int(seed), 77])
        s["seed"] = {k: rng.normal(size=n) for k in ("x", "y", "z", "vx", "vy", "vz")}
    if case["kind"] == "analysis":
        beads = np.flatnonzero(arrays[0]["kind"] == 0).astype(np.int32)  # the phosphates of the chain
        ref = np.stack([st[k][beads] for k in "xyz"], 1)
        s["grid"] = e.density(0, K_ION, (0.0, 0.0, 0.0), 5.0, (int(case["box"] / 5.0),) * 3, beads, ref)
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "pair_lists":
        x, y, z = s["xyz"]
        n, L, sr, lr = x.numel(), case["box"], s["sr"], s["lr"]
        pair_lists_noalloc(x.data_ptr(), y.data_ptr(), z.data_ptr(), s["part"].data_ptr(), n, [L, L, L], SR_LIST,
                           case["rc"] + LR_SKIN, sr.data_ptr(), len(sr), lr.data_ptr(), len(lr), s["counts"].data_ptr(),
                           torch.cuda.current_stream().cuda_stream)
        # the call leaves the pairs in no order: a caller that wants reproducible sums sorts them
        return [s["counts"]] + [torch.sort(p[:, 0].long() * n + p[:, 1]).values for p in (sr, lr)]
    e = s["engine"]
    if kind == "md":
        e.step(case["steps"])
        e.sync()
        return dict(e.get_states(out=s["out"]), energies=e.all_energies(out=s["energies"]))
    if kind == "dropin":
        for _ in range(case["steps"]):
            e.deterministic_forces()
            e.full_forces()
            e.move_rigid_units()
            e.check_shifts()
        e.sync()
        return dict(e.get_states(out=s["out"]), energies=e.all_energies(out=s["energies"]))
    if kind == "upload":
        e.set_states(s["states"])
        e.populate_lists()
        e.step(case["steps"])
        e.sync()
        return dict(e.get_states(("x", "y", "z"), out=s["out"]), energies=e.all_energies(out=s["energies"]))
    if kind == "terms":
        e.set_state(0, s["state"])
        f, en = e.forces(0, FORCE_TERMS)
        return {"forces": f, "energies": np.array([en[k] for k in ENERGY_NAMES])}
    if kind == "param_grad":
        e.set_states(s["states"])
        g = e.param_grad()
        return {"stacks": g[:, :5], "hbonds": g[:, 5], "pairs": g[:, 6:]}
    if kind == "traj_grad":
        e.set_states(s["states"])
        g, d0 = e.traj_grad(case["steps"], case["interval"], s["seed"], want_state=True)
        return {"theta": g, "state": d0}
    counts = []
    for _ in range(case["steps"] // case["interval"]):
        e.step(case["interval"])
        s["grid"].add()
        counts += [e.ion_counts(0, k, 7.2684)[0] for k in (MG, K_ION)]
    grid, frames, rmsd = s["grid"].get()
    return {"grid": grid, "frames": frames, "rmsd": rmsd, "bound": counts}


def work(case):
    """Inputs read once, outputs written once; the arithmetic of the interactions inside the cutoffs."""
    L, reps, steps = case["box"], case["replicas"], case["steps"]
    mg = 0.5 * (case["mg_lo"] + case["mg_hi"])
    n = (3 * case["n_nt"] - 1 + sum(_ion_numbers(mg, case["kcl"], L, case["n_nt"]))) * reps
    rho = n / reps / L ** 3
    sr = 0.5 * n * rho * 4.19 * 12.0 ** 3 + 10.0 * case["n_nt"] * reps  # pairs: the solution's, and the chain's own
    lr = 0.5 * n * rho * 4.19 * case["rc"] ** 3
    topo = 12.0 * case["n_nt"] * reps  # bonds, angles, stacks, H-bond candidates
    step = 30.0 * sr + 3.0 * lr + 200.0 * topo + 60.0 * n
    state = 72.0 * n
    kind = case["kind"]
    if kind in ("md", "dropin", "analysis"):
        return {"bytes": 2 * state, "flops": steps * step}
    if kind == "upload":
        return {"bytes": state + 24.0 * n, "flops": steps * step + 10.0 * (sr + lr)}
    if kind == "terms":
        return {"bytes": state + 24.0 * n, "flops": 40.0 * (sr + lr) + 300.0 * topo}
    if kind == "param_grad":
        return {"bytes": state + 128.0 * reps, "flops": 60.0 * (sr + lr) + 300.0 * topo}
    if kind == "traj_grad":
        return {"bytes": 3 * state, "flops": 4.0 * steps * step}
    return {"bytes": 28.0 * n + 8.0 * (sr + lr), "flops": 10.0 * (sr + lr)}


# ---- 64-bit values ----------------------------------------------------------------------
def exact(case, seed):
    """FP64 values of the force terms and of dU/dtheta, from the energies by automatic
    differentiation.  Trajectories have none: their Monte Carlo decisions and rounding are part
    of the path; neither has the H-bond column, which follows the same Monte Carlo."""
    if case["kind"] not in ("terms", "param_grad"):
        return None
    arrays, systems = _systems(case, seed)
    st = _equilibrated(case, systems)
    values, at = [], 0
    for a in arrays:
        n = a["x"].size
        x = np.stack([st[k][at:at + n] for k in "xyz"], 1)
        values.append(_terms64(case, a, x) if case["kind"] == "terms" else _grad64(case, a, x))
        at += n
    if case["kind"] == "terms":
        return {"forces": values[0][0], "energies": values[0][1]}
    g = np.stack(values)
    return {"stacks": g[:, :5], "hbonds": None, "pairs": g[:, 6:]}


def _f64(v):
    return torch.as_tensor(np.asarray(v), dtype=torch.float64, device="cuda" if torch.cuda.is_available() else "cpu")


def _index(v):
    return torch.as_tensor(np.asarray(v).astype(np.int64), device="cuda" if torch.cuda.is_available() else "cpu")


def _image(d, L):
    return d - L * torch.round(d / L)


def _pairs64(x, L, cut):
    """Index pairs i < j within `cut`."""
    found = []
    for b in range(0, len(x), 1024):
        d = _image(x[b:b + 1024, None, :] - x[None, :, :], L)
        i, j = torch.nonzero((d * d).sum(-1) <= cut * cut, as_tuple=True)
        i = i + b
        found.append(torch.stack([i, j])[:, i < j])
    return torch.cat(found, 1)


def _bonded_pairs(a):
    ends = np.where(a["bt_kind"] == 1, a["bt_c"], a["bt_b"])
    return np.stack([np.minimum(a["bt_a"], ends), np.maximum(a["bt_a"], ends)])


def _lj(a, i, j, r, elj, rlj):
    """E (s^12 - 2 s^6 + 1) inside the contact distance D, s = sig0 / (r + sig0 - D)."""
    t = _index(a["type"]) - 1
    ion = (t[i] > 5) | (t[j] > 5)
    D = torch.where(ion, rlj[t[i]] + rlj[t[j]], torch.full_like(r, 3.2))
    inside = r <= D
    s6 = (SIG0 / torch.where(inside, r + SIG0 - D, torch.full_like(r, SIG0))) ** 6
    E = torch.sqrt(elj[t[i]] * elj[t[j]])
    return torch.where(inside, E * (s6 * s6 - 2 * s6 + 1), torch.zeros_like(r)), E, D


def _coulomb(a, case, i, j, r, lB, debye):
    q = _f64(a["qc"])[_index(a["type"]) - 1]
    u = q[i] * q[j] * lB / r
    if case["debye"] > 0:
        u = u * torch.exp(-r / debye)
    return torch.where(r <= case["rc"], u, torch.zeros_like(u))


def _angle(x, i, j, k):
    a, b = x[i] - x[j], x[k] - x[j]
    return torch.atan2(torch.linalg.norm(torch.linalg.cross(a, b), dim=-1), (a * b).sum(-1))


def _dihedral(x, i, j, k, m):
    v1, v2, v3 = x[j] - x[i], x[k] - x[j], x[m] - x[k]
    p, n = torch.linalg.cross(v1, v2), torch.linalg.cross(v2, v3)
    return torch.atan2((v1 * n).sum(-1) * torch.linalg.norm(v2, dim=-1), (p * n).sum(-1))


def _wrapped(psi, native):
    d = psi - native
    return d - 2 * math.pi * torch.round(d.detach() / (2 * math.pi))


def _stacks64(a, x):
    """(1 / D of every secondary stack that is on, 1 / D of every tertiary stack)."""
    k = _index(a["st2_idx"]).reshape(-1, 7).T
    dr = torch.linalg.norm(x[k[5]] - x[k[2]], dim=-1) - _f64(a["st2_r0"])
    d1 = _wrapped(_dihedral(x, k[0], k[1], k[3], k[4]), -2.58684)
    d2 = _wrapped(_dihedral(x, k[6], k[4], k[3], k[1]), 3.07135)
    u2 = 1 / (1 + 1.4 * dr * dr + 4 * d1 * d1 + 4 * d2 * d2)
    m = _index(a["st3_idx"]).reshape(-1, 6).T
    nat = _f64(a["st3_native"]).reshape(-1, 6).T
    dr = torch.linalg.norm(x[m[4]] - x[m[1]], dim=-1) - nat[0]
    q = 1 + 5 * dr * dr + 1.5 * (_angle(x, m[0], m[1], m[4]) - nat[1]) ** 2 + 1.5 * (_angle(x, m[3], m[4], m[1]) - nat[2]) ** 2
    for at, ids in ((3, (0, 1, 4, 3)), (4, (4, 1, 0, 2)), (5, (1, 4, 3, 5))):
        q = q + 0.15 * _wrapped(_dihedral(x, *(m[t] for t in ids)), nat[at]) ** 2
    off = np.zeros(a["st2_E"].size)  # secondary stacks that a formed tertiary stack on their site switches off
    near = (dr < 10.0).cpu().numpy()
    for t, at in enumerate(a["st3_off"].reshape(-1, 2)):
        off[at[at >= 0]] += near[t]
    return u2 * _f64(off == 0), 1 / q


def _terms64(case, a, pos):
    L = case["box"]
    x = _f64(pos).requires_grad_(True)
    i, j = _pairs64(x.detach(), L, max(case["rc"], SR_LIST))
    r = torch.linalg.norm(_image(x[i] - x[j], L), dim=-1)
    elj, rlj, lB = _f64(a["elj"]), _f64(a["rlj"]), float(a["lB"][0])
    bi, bj = _index(_bonded_pairs(a))
    rb = torch.linalg.norm(_image(x[bi] - x[bj], L), dim=-1)
    u_lj, E, D = _lj(a, i, j, r, elj, rlj)
    u_ex, Eb, Db = _lj(a, bi, bj, rb, elj, rlj)
    u_c = _coulomb(a, case, i, j, r, lB, case["debye"])
    kind, ta, tb, tc = (_index(a["bt_" + k]) for k in ("kind", "a", "b", "c"))
    k0, x0 = _f64(a["bt_k0"]), _f64(a["bt_x0"])
    bond, ang = kind == 0, kind == 1
    u_bond = k0[bond] * (torch.linalg.norm(x[tb[bond]] - x[ta[bond]], dim=-1) - x0[bond]) ** 2
    u_ang = k0[ang] * (_angle(x, ta[ang], tb[ang], tc[ang]) - x0[ang]) ** 2
    u2, u3 = _stacks64(a, x)
    e2, e3 = (u2 * _f64(a["st2_E"])).sum(), (u3 * _f64(a["st3_E"])).sum()
    u = u_lj.sum() - u_ex.sum() + u_c.sum() + u_bond.sum() + u_ang.sum() + e2 + e3
    f = -torch.autograd.grad(u, x)[0]
    # reported LJ energies are clamped at very short distances; the forces are not
    low, lowb = r < D - 0.4406141861 * SIG0, rb < Db - 0.4406141861 * SIG0
    near = r <= SR_LIST
    rna = x[:int(a["n_rna"][0])].detach()
    e = {"E_lj": torch.where(low, 1001.0 * E, u_lj).sum(), "E_coul_sr": u_c[near].sum(), "E_coul_lr": u_c[~near].sum(),
         "E_bond": u_bond.sum(), "E_angle": u_ang.sum(), "E_excl": -torch.where(lowb, 1001.0 * Eb, u_ex).sum(),
         "E2_STACK": e2, "E3_STACK": e3, "E2_HB": 0.0, "E3_HB": 0.0,
         "Rg": torch.sqrt(((rna - rna.mean(0)) ** 2).sum(-1).mean())}
    return f.reshape(-1).cpu().numpy(), np.array([float(torch.as_tensor(e[k]).detach()) for k in ENERGY_NAMES])


def _grad64(case, a, pos):
    L = case["box"]
    x = _f64(pos)
    i, j = _pairs64(x, L, max(case["rc"], 12.0))
    r = torch.linalg.norm(_image(x[i] - x[j], L), dim=-1)
    n = len(x)
    bonded = np.sort(np.asarray(_bonded_pairs(a), dtype=np.int64)[0] * n + _bonded_pairs(a)[1])
    key = (i * n + j).cpu().numpy()
    times = np.searchsorted(bonded, key, "right") - np.searchsorted(bonded, key, "left")
    elj, rlj = _f64(a["elj"]).requires_grad_(True), _f64(a["rlj"]).requires_grad_(True)
    lB, debye = _f64(a["lB"][0]).requires_grad_(True), _f64(case["debye"]).requires_grad_(True)
    u = (_lj(a, i, j, r, elj, rlj)[0] * _f64(1.0 - times)).sum() + _coulomb(a, case, i, j, r, lB, debye).sum()
    ge, gr, gl, gd = (g if g is not None else torch.zeros_like(v)
                      for v, g in zip((elj, rlj, lB, debye), torch.autograd.grad(u, (elj, rlj, lB, debye), allow_unused=True)))
    u2, u3 = _stacks64(a, x)
    cls = a["st2_cls"]
    u2 = u2.cpu().numpy() * a["st2_dss"]
    ss = [u2[cls == c].sum() for c in range(4)]
    ge, gr = ge.cpu().numpy(), gr.cpu().numpy()
    return np.array(ss + [-float(u3.sum()), 0.0, ge[0], ge[1], ge[2:6].sum(), ge[6], ge[7], ge[8], gr[6], gr[8],
                          float(gl), float(gd)])
