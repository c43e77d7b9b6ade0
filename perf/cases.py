"""The framework's work, as cases that can be timed and compared.

Each case goes through the public entry points as a user's program does: the
per-call functions that mirror the reference's (forces, a step of
update_sc_nospline on the caller's arrays), the device-resident stepper (one
system, many replicas, a centroid run with a learned correction) and the
training step of that correction. Starts are waters at liquid density on a
jittered lattice of like orientations (as the reference starts), in a cell of the
lattice's shape (cubic, or orthorhombic as ice), some molecules a cell vector away
(coordinates are never wrapped), beads spread as a free ring polymer.

Outputs of the FP64 form come back as float64. The mixed form computes its forces
in FP32, and the Suzuki-Chin force is a finite difference that keeps about eight
digits: what follows from those is returned as float32.
"""
import math

import numpy as np
import torch

import qtip4pf_water_gb300 as q

# qTIP4P/F and unit constants in atomic units (the reference's truncated pi)
PI = 3.14159265359
BOHR = 1.0 / 0.529177210903
KCAL = 1.5936e-3
ME, NA = 9.10938356e-31, 6.0221409e23
M_O, M_H = 0.001 * 15.9994 / (NA * ME), 0.001 * 1.0080 / (NA * ME)
K_AU = 1.38064852e-23 / 4.3597447222071e-18
MOL_VOLUME = (15.9994 + 2.0 * 1.0080) / NA / 0.997 * 1e24 * BOHR ** 3
EPS_EWALD, EPS_SC, TEMP = 1e-6, 1e-5, 298.0
R_CUT = 9.0 * BOHR
N_PARAMS, N_WEIGHTS = q.MLP_NPARAMS, q.MLP_NW


def listed():
    return [
        # a classical water droplet-sized box, one force call: the smallest call there is, all latency
        {"name": "forces_64_fp64", "kind": "forces", "mols": 64, "beads": 1, "precision": "fp64", "lists": False},
        # lists and forces of a ring polymer in an orthorhombic (ice-like) cell, in the default precision:
        # what a run does at its start and an analysis for every stored configuration
        {"name": "forces_336_p8_fp64", "kind": "forces", "mols": 336, "beads": 8, "precision": "fp64", "lists": True},
        # the benchmark's system (512 waters, 32 beads), its forces by one call in the mixed form
        {"name": "forces_512_p32_mixed", "kind": "forces", "mols": 512, "beads": 32, "precision": "mixed", "lists": False},
        # the reference's own force: Suzuki-Chin in FP64, as the drop-in evaluates it by default
        {"name": "sc_216_p8_fp64", "kind": "sc", "mols": 216, "beads": 8, "precision": "fp64"},
        # the benchmark's system stepped call by call on the caller's page-locked arrays (update_sc_nospline)
        {"name": "step_512_p32_mixed", "kind": "step", "mols": 512, "beads": 32, "precision": "mixed", "propagator": "trotter"},
        # classical Langevin dynamics of 216 waters on the device: launches and latency
        {"name": "md_216_p1_mixed", "kind": "md", "mols": 216, "beads": 1, "precision": "mixed", "propagator": "trotter", "steps": 200},
        # the benchmark: 512 waters, 32 beads, Trotter and PILE-G on the device
        {"name": "md_512_p32_mixed", "kind": "md", "mols": 512, "beads": 32, "precision": "mixed", "propagator": "trotter", "steps": 50},
        # Suzuki-Chin on the device, 512 waters and 16 beads
        {"name": "md_512_p16_sc_mixed", "kind": "md", "mols": 512, "beads": 16, "precision": "mixed", "propagator": "sc", "steps": 20},
        # the FP64 form of the 216-water, 32-bead Trotter run (the parity form)
        {"name": "md_216_p32_fp64", "kind": "md", "mols": 216, "beads": 32, "precision": "fp64", "propagator": "trotter", "steps": 4},
        # 48 uneven replicas (64 to 512 waters, 8 to 32 beads) in one context
        {"name": "replicas_48_mixed", "kind": "replicas", "count": 48, "steps": 20},
        # centroid dynamics of 4096 waters with the learned correction attached
        {"name": "cmd_4096_mixed", "kind": "cmd", "mols": 4096, "steps": 50},
        # one training step of the learned correction over a large batch of molecules
        {"name": "train_442368", "kind": "train", "rows": 442368},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(mols):
    """Lattice cells a side of a near-cubic lattice of that many waters and waters a cell (1, or 2: body-centred); None if there is none."""
    for per in (1, 2):
        n = mols // per
        for a in range(round(n ** (1.0 / 3.0)) + 1, 0, -1):
            for b in range(a, a + 3):
                for c in range(b, a + 3):
                    if per * a * b * c == mols:
                        return (a, b, c), per
    return None


def _mols(rng, lo, hi):
    n = _spread(rng, lo, hi)
    while _sides(n) is None:
        n -= 1
    return n


def draw(rng):
    kind = rng.choice(["forces", "forces", "sc", "step", "md", "md", "md", "replicas", "cmd", "train"])
    if kind == "train":
        return {"kind": kind, "rows": _spread(rng, 2000, 442368)}
    if kind == "replicas":
        return {"kind": kind, "count": rng.randint(3, 40), "steps": rng.randint(5, 15)}
    if kind == "cmd":
        return {"kind": kind, "mols": _mols(rng, 256, 4096), "steps": rng.randint(10, 50)}
    precision = rng.choice(["fp64", "mixed", "mixed"])
    sc = kind == "sc" or (kind in ("step", "md") and rng.random() < 0.4)
    # waters times beads: the FP64 form's cost is held below the largest listed case's
    most = 3000 if precision == "fp64" else 16384
    mols = _mols(rng, 27, min(900, most // 8) if sc else 900)
    if sc:  # the reference's assembly takes even rings; with fewer than eight beads its steps are not stable
        beads = 2 * rng.randint(4, max(4, min(16, most // mols // 2)))
    else:  # single configurations, odd and even rings
        beads = rng.choice([1, _spread(rng, 1, max(1, min(32, most // mols))), _spread(rng, 1, max(1, min(32, most // mols)))])
    case = {"kind": kind, "mols": mols, "beads": beads, "precision": precision}
    if kind == "forces":
        case["lists"] = rng.random() < 0.5
    if kind in ("step", "md"):
        case["propagator"] = "sc" if sc else "trotter"
    if kind == "md":
        case["steps"] = rng.randint(2, 4) if precision == "fp64" else rng.randint(10, 40)
    return case


# ---- starts ---------------------------------------------------------------------------

def _box(mols):
    sides, per = _sides(mols)
    return np.array(sides, dtype=np.float64) * (per * MOL_VOLUME) ** (1.0 / 3.0)


def _modes(beads):
    """The orthonormal bead -> normal mode matrix of a ring."""
    b = np.arange(beads)
    rows = [np.full(beads, math.sqrt(1.0 / beads))]
    for k in range(1, beads):
        w = 2.0 * math.pi * b * k / beads
        if 2 * k == beads:
            rows.append(math.sqrt(1.0 / beads) * np.cos(w))
        else:
            rows.append(math.sqrt(2.0 / beads) * (np.cos(w) if 2 * k < beads else np.sin(w)))
    return np.array(rows)


def _masses(mols):
    return np.tile(np.repeat(np.array([M_O, M_H, M_H]), 3), mols)


def _water(mols, beads, box, seed, temp=TEMP):
    """Positions and momenta, each double[beads][9 mols]."""
    rng = np.random.default_rng(seed)
    sides, per = _sides(mols)
    k = np.arange(mols) // per
    grid = np.stack([k % sides[0], k // sides[0] % sides[1], k // (sides[0] * sides[1])], 1) + 0.5 * (np.arange(mols) % per)[:, None]
    at = (grid + 0.25) * (box / sides) + rng.normal(scale=0.15, size=(mols, 3))
    at += box * rng.choice([-1.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 1.0], size=(mols, 3))
    r, half = 0.9419 * BOHR, 0.5 * 107.4 * math.pi / 180.0
    body = np.array([[0.0, 0.0, 0.0], [r * math.sin(half), 0.0, r * math.cos(half)], [-r * math.sin(half), 0.0, r * math.cos(half)]])
    turn, _ = np.linalg.qr(np.eye(3) + rng.normal(scale=0.25, size=(mols, 3, 3)))  # tilts of some fifteen degrees
    turn *= np.sign(np.einsum("nii->ni", turn))[:, None]
    x = (at[:, None] + np.einsum("nij,aj->nai", turn, body) + rng.normal(scale=0.02, size=(mols, 3, 3))).reshape(-1)
    beta_n, mass = 1.0 / (K_AU * temp) / beads, _masses(mols)
    modes = np.zeros((beads, 9 * mols))
    modes[0] = math.sqrt(beads) * x
    for k in range(1, beads):
        w = (2.0 / beta_n) * math.sin(k * math.pi / beads)
        modes[k] = rng.normal(size=9 * mols) / np.sqrt(beta_n * mass * w * w)
    pos = _modes(beads).T @ modes
    mom = rng.normal(size=(beads, 9 * mols)) * np.sqrt(mass / beta_n)
    mom -= np.tile(mom.reshape(-1, 3).mean(0), 3 * mols)
    return np.ascontiguousarray(pos), np.ascontiguousarray(mom)


def _replicas(count, seed):
    """(mols, beads, temperature) of every replica."""
    rng = np.random.default_rng(1000 + count)  # the same batch for every seed: the seed makes its configurations
    return [(int(rng.choice([64, 128, 216, 343, 512])), int(rng.choice([8, 16, 32])), float(rng.uniform(250.0, 350.0))) for _ in range(count)]


def _precision(case):
    return q.MIXED if case.get("precision") == "mixed" else q.FP64


def _float32(*arrays):
    return [np.asarray(a, dtype=np.float32) for a in arrays]


def _joined(forces, *energies):
    """FP32 forces with the energies behind them: the mixed form's energy is what is left of terms many times its
    size, so its error goes by their scale, as the forces' does, and not by its own."""
    out = np.empty(forces.size + len(energies), dtype=np.float32)
    out[:forces.size] = forces.reshape(-1)
    out[forces.size:] = energies
    return out


# ---- prepare --------------------------------------------------------------------------

def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, int(seed))


def _prepare_forces(case, seed):
    box = _box(case["mols"])
    pos, _ = _water(case["mols"], case["beads"], box, seed)
    s = q.System.create(case["mols"], case["beads"], box, precision=_precision(case), temp_K=TEMP,
                        propagator=q.SUZUKI_CHIN if case["kind"] == "sc" else q.TROTTER)
    point, lst, _ = s.build_lists(pos)
    return {"case": case, "s": s, "pos": pos, "f": np.zeros_like(pos), "fphys": np.zeros_like(pos), "charge": s.charges(), "mass": s.masses(),
            "point": point, "list": lst}


_prepare_sc = _prepare_forces


def _propagator(case):
    return q.SUZUKI_CHIN if case["propagator"] == "sc" else q.TROTTER


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def _prepare_step(case, seed):
    box = _box(case["mols"])
    pos, mom = (a.reshape(-1) for a in _water(case["mols"], case["beads"], box, seed))
    s = q.System.create(case["mols"], case["beads"], box, precision=_precision(case), temp_K=TEMP, dt_fs=0.25, propagator=_propagator(case),
                        thermostat=q.PILE_G, seed=seed)
    point, lst, disp = s.build_lists(pos)
    f, fphys = np.zeros_like(pos), np.zeros_like(pos)
    if case["propagator"] == "sc":
        s.force_eval_sc_nospline(pos, f, s.charges(), s.masses(), point, lst, fphys)
    else:
        s.force_eval_trotter(pos, f, s.charges(), point, lst)
    st = {"case": case, "s": s, "charge": s.charges(), "mass": s.masses(), "point": point, "list": lst, "heat": 0.0}
    st |= {k: _pinned(a) for k, a in (("q", pos), ("p", mom), ("f", f), ("fphys", f), ("disp", disp))}
    return st


def _start(ctx, starts):
    for s, (pos, mom) in zip(ctx.systems, starts):
        s.set_state(pos, mom)
    ctx.init_forces()


def _prepare_md(case, seed):
    box = _box(case["mols"])
    one = case["beads"] == 1
    d = q.system_desc(case["mols"], case["beads"], box, temp_K=TEMP, dt_fs=0.5 if one else 0.25, propagator=_propagator(case),
                      thermostat=q.PILE_L if one else q.PILE_G, seed=seed)
    ctx = q.Context([d], _precision(case))
    _start(ctx, [_water(case["mols"], case["beads"], box, seed)])
    return {"case": case, "ctx": ctx}


def _prepare_replicas(case, seed):
    descs, starts = [], []
    for k, (mols, beads, temp) in enumerate(_replicas(case["count"], seed)):
        box = _box(mols)
        descs.append(q.system_desc(mols, beads, box, temp_K=temp, dt_fs=0.25, propagator=q.TROTTER, thermostat=q.PILE_G, seed=seed + k))
        starts.append(_water(mols, beads, box, seed + 7919 * k, temp))
    ctx = q.Context(descs, q.MIXED)
    _start(ctx, starts)
    return {"case": case, "ctx": ctx}


def _network(seed):
    """FP32 parameters (weights, then biases) and the BF16 weights, on the device."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.zeros(N_PARAMS, device="cuda")
    w[:64 * 96].normal_(0.0, math.sqrt(1.0 / 96), generator=g)
    w[64 * 96:64 * 160].normal_(0.0, math.sqrt(1.0 / 64), generator=g)
    w[64 * 160:64 * 169].normal_(0.0, math.sqrt(1.0 / 64), generator=g)
    w[N_WEIGHTS:N_WEIGHTS + 128].normal_(0.0, 0.1, generator=g)
    return w, w[:N_WEIGHTS].to(torch.bfloat16)


def _weights(w, wbf):
    a, b = wbf.data_ptr(), w.data_ptr()
    return q.MlpWeights(a, a + 2 * 64 * 96, a + 2 * 64 * 160, b + 4 * N_WEIGHTS, b + 4 * (N_WEIGHTS + 64), b + 4 * (N_WEIGHTS + 128))


def _prepare_cmd(case, seed):
    box = _box(case["mols"])
    d = q.system_desc(case["mols"], 1, box, temp_K=TEMP, dt_fs=0.25, propagator=q.TROTTER, thermostat=q.PILE_L, seed=seed)
    ctx = q.Context([d], q.MIXED)
    pos, mom = _water(case["mols"], 1, box, seed)
    ctx.systems[0].set_state(pos, mom)
    w, wbf = _network(seed)
    norm = np.concatenate([np.full(96, 0.5), np.full(96, 0.2)]).astype(np.float32)
    ctx.systems[0].attach_surrogate(_weights(w, wbf), norm, 1e-4)  # small beside the forces, as an untrained network must not steer the run
    ctx.init_forces()
    return {"case": case, "ctx": ctx, "keep": (w, wbf)}


def _prepare_train(case, seed):
    m = case["rows"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    w, wbf = _network(seed)
    t = torch.zeros((m, 16), device="cuda")
    t[:, :9].normal_(generator=g)
    ctas = 512
    return {"case": case, "x": torch.randn((m, 96), device="cuda", generator=g).to(torch.bfloat16), "t": t, "w": w, "wbf": wbf,
            "m1": torch.zeros_like(w), "m2": torch.zeros_like(w), "part": torch.zeros((ctas, N_PARAMS + 1), device="cuda"), "ctas": ctas,
            "grad": torch.zeros(N_PARAMS + 1, device="cuda"), "step": 0}


# ---- run ------------------------------------------------------------------------------

def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


def _run_forces(st):
    s, case = st["s"], st["case"]
    out = {}
    if case["lists"]:
        st["point"], st["list"], _ = s.build_lists(st["pos"])
        out["point"] = st["point"]
    if case["beads"] == 1:
        energy = s.get_forces_nospline(st["pos"], st["f"], st["charge"], st["point"], st["list"])
    else:
        energy, _ = s.force_eval_trotter(st["pos"], st["f"], st["charge"], st["point"], st["list"])
    if case["precision"] == "mixed":
        out["f"] = _joined(st["f"], energy)
    else:
        out["f"], out["energy"] = st["f"], energy
    return out


def _run_sc(st):
    energy, pot = st["s"].force_eval_sc_nospline(st["pos"], st["f"], st["charge"], st["mass"], st["point"], st["list"], st["fphys"])
    if st["case"]["precision"] == "mixed":
        return {"f": _float32(st["f"])[0], "fphys": _joined(st["fphys"], energy, pot)}
    return {"f": _float32(st["f"])[0], "fphys": st["fphys"], "energy": energy, "pot": pot}


def _run_step(st):
    energy, st["heat"], pot = st["s"].update_sc_nospline(st["q"], st["p"], st["mass"], st["f"], st["fphys"], st["charge"], st["point"], st["list"],
                                                         st["disp"], True, st["heat"])
    if st["case"]["precision"] == "mixed":
        p, heat = _float32(st["p"], st["heat"])
        return {"q": st["q"], "p": p, "f": _joined(st["f"], energy, pot), "heat": heat}
    out = {"q": st["q"], "p": st["p"], "f": st["f"], "fphys": st["fphys"], "energy": energy, "heat": st["heat"], "pot": pot}
    if st["case"]["propagator"] == "sc":
        out["p"], out["f"] = _float32(out["p"], out["f"])
    return out


def _block(ctx, steps):
    """A block of steps, its estimator records and the state it ends in."""
    ctx.run_steps(steps, is_nvt=True)
    records = ctx.systems[0].estimators()
    ctx.reset_estimators()
    return records, ctx.systems[0].get_state()


def _run_md(st):
    case = st["case"]
    records, state = _block(st["ctx"], case["steps"])
    if case["precision"] == "mixed" or case["propagator"] == "sc":
        records, state = ({k: _float32(a)[0] for k, a in d.items()} for d in (records, state))
    return {"records": records, "state": state}


def _run_replicas(st):
    st["ctx"].run_steps(st["case"]["steps"], is_nvt=True)
    states = [s.get_state() for s in st["ctx"].systems]
    return {k: np.concatenate([d[k] for d in states], dtype=np.float32, casting="same_kind") for k in ("q", "p", "fphys")}


def _run_cmd(st):
    records, state = _block(st["ctx"], st["case"]["steps"])
    return {"pot": _float32(records["pot"])[0], "kin": _float32(records["kin"])[0], "state": {k: _float32(state[k])[0] for k in ("q", "p", "fphys")}}


def _run_train(st):
    m = st["case"]["rows"]
    q.mlp_train_batch(_weights(st["w"], st["wbf"]), st["x"].data_ptr(), st["t"].data_ptr(), m, 2.0 / (9 * m), st["part"].data_ptr(), st["ctas"],
                      st["grad"].data_ptr())
    st["step"] += 1
    q.adam_step(st["w"].data_ptr(), st["m1"].data_ptr(), st["m2"].data_ptr(), st["grad"].data_ptr(), N_PARAMS, st["step"], 1e-4, st["wbf"].data_ptr(),
                N_WEIGHTS)
    return {"grad": st["grad"], "w": st["w"]}


# ---- work -----------------------------------------------------------------------------

def _ewald(mols, box):
    """kappa, real-space cutoff, reciprocal cutoff."""
    vol, acc = float(np.prod(box)), math.sqrt(-math.log(EPS_EWALD))
    kappa = 2.6 * (3.0 * mols / vol / vol) ** (1.0 / 6.0)
    rc = acc / kappa
    if rc > 0.5 * box.min():
        rc = 0.5 * float(box.min())
        kappa = acc / rc
    return kappa, rc, 2.0 * acc * kappa


def _evaluation_flops(mols):
    """One configuration: 60 a site pair within the cutoff, 30 an O-O pair, 20 a (site, k), 150 a molecule."""
    box = _box(mols)
    vol = float(np.prod(box))
    _, rc, kc = _ewald(mols, box)
    sphere = 4.0 / 3.0 * math.pi
    sites = 3.0 * mols
    nk = 0.5 * sphere * kc ** 3 * vol / (2.0 * math.pi) ** 3
    return (30.0 * sites * sites * min(1.0, sphere * rc ** 3 / vol) + 15.0 * mols * mols * min(1.0, sphere * R_CUT ** 3 / vol) + 20.0 * sites * nk
            + 150.0 * mols)


def _evaluations(beads, sc):
    return beads + (beads // 2) * 2 if sc else beads  # the force gradient of an odd bead: two evaluations' worth


def work(case):
    kind = case["kind"]
    if kind == "train":
        m = case["rows"]
        return {"bytes": m * (96 * 2 + 16 * 4) + 5 * 4 * N_PARAMS, "flops": 6.0 * m * (96 * 64 + 64 * 64 + 64 * 16)}
    if kind == "replicas":
        sizes = _replicas(case["count"], 0)
        steps = case["steps"]
        return {"bytes": sum(40 * 9 * n * p for n, p, _ in sizes) * steps, "flops": sum(_evaluation_flops(n) * p for n, p, _ in sizes) * steps}
    n = case["mols"]
    if kind == "cmd":
        per = _evaluation_flops(n) + 2 * n * 2.0 * (96 * 64 + 64 * 64 + 64 * 16) + 3 * n * 90 * 60.0
        return {"bytes": 40 * 9 * n * case["steps"], "flops": per * case["steps"]}
    p = case["beads"]
    sc = kind == "sc" or case.get("propagator") == "sc"
    flops = _evaluation_flops(n) * _evaluations(p, sc)
    per_dof = {"forces": 16, "sc": 24, "step": 64, "md": 40}[kind]
    steps = case.get("steps", 1)
    return {"bytes": per_dof * 9 * n * p * steps, "flops": flops * steps}


# ---- exact ----------------------------------------------------------------------------

def exact(case, seed):
    kind = case["kind"]
    if kind in ("forces", "sc"):
        return _exact_forces(case, int(seed))
    if kind == "train":
        return _exact_train(case, int(seed))
    return None  # a trajectory: its forces are those of the cases above


def _exact_forces(case, seed):
    mols, beads = case["mols"], case["beads"]
    box = _box(mols)
    pos, _ = _water(mols, beads, box, seed)
    pos, L = torch.from_numpy(pos).cuda(), torch.from_numpy(box).cuda()
    sets = [_force(pos[b], mols, box, L) for b in range(beads)]
    f = torch.stack([s[0] for s in sets])
    e = [s[1] for s in sets]
    mixed = case["precision"] == "mixed"

    def joined(forces, *energies):
        return torch.cat([forces.reshape(-1), torch.tensor(energies, dtype=f.dtype, device="cuda")])

    if case["kind"] == "forces":
        out = {"f": joined(f, sum(e))} if mixed else {"f": f, "energy": sum(e)}
        return out | {"point": None} if case["lists"] else out
    mass = torch.from_numpy(_masses(mols)).cuda()
    omega_sq = (K_AU * TEMP * beads) ** 2
    total, pot, fsc = 0.0, 0.0, torch.empty_like(f)
    for b in range(beads):
        if b % 2 == 0:
            total, pot = total + 2.0 * e[b], pot + e[b]
            fsc[b] = 2.0 * f[b] / 3.0
            continue
        u = f[b] / mass
        total += 4.0 * e[b] + float((f[b] * u).sum()) / (3.0 * omega_sq)
        # the force's derivative along f / m, by a central difference whose step leaves the most digits in 64 bits
        h = 1e-4 / float(u.square().mean().sqrt())
        d = [_force(pos[b] + k * h * u, mols, box, L)[0] for k in (-2, -1, 1, 2)]
        fsc[b] = 4.0 * f[b] / 3.0 - (8.0 * (d[2] - d[1]) - (d[3] - d[0])) / (6.0 * h) / (9.0 * omega_sq)
    total, pot = total / 3.0, 2.0 * pot / beads
    return {"f": fsc, "fphys": joined(f, total, pot)} if mixed else {"f": fsc, "fphys": f, "energy": total, "pot": pot}


def _image(d, L):
    return d - L * torch.round(d / L)


def _force(x, mols, box, L):
    """Forces (9 mols) and energy of one configuration, in 64 bits."""
    r = x.reshape(mols, 3, 3)
    f = torch.zeros_like(r)
    # Lennard-Jones between oxygens
    eps, sig = 0.1852 * KCAL, 3.1589 * BOHR
    d = _image(r[:, None, 0] - r[None, :, 0], L)
    r2 = d.square().sum(-1)
    near = (r2 < R_CUT * R_CUT) & ~torch.eye(mols, dtype=torch.bool, device=x.device)
    i2 = torch.where(near, 1.0 / torch.where(near, r2, torch.ones_like(r2)), torch.zeros_like(r2))
    s6 = i2 ** 3 * sig ** 6
    cut = 4.0 * eps * ((sig / R_CUT) ** 12 - (sig / R_CUT) ** 6)
    energy = 0.5 * float((4.0 * eps * (s6 * s6 - s6) - cut * near).sum())
    f[:, 0] += ((24.0 * eps * (2.0 * s6 * s6 - s6) * i2)[..., None] * d).sum(1)
    # quartic Morse bonds and the harmonic angle
    ar, depth = 2.287 / BOHR, 116.09 * KCAL
    v = [_image(r[:, 0] - r[:, k], L) for k in (1, 2)]
    ln = [a.square().sum(-1).sqrt() for a in v]
    for k in (0, 1):
        y = ln[k] - 0.9419 * BOHR
        energy += float((depth * (ar ** 2 * y ** 2 - ar ** 3 * y ** 3 + 7.0 / 12.0 * ar ** 4 * y ** 4)).sum())
        g = (depth * (2.0 * ar ** 2 * y - 3.0 * ar ** 3 * y ** 2 + 7.0 / 3.0 * ar ** 4 * y ** 3) / ln[k])[:, None] * v[k]
        f[:, 0] -= g
        f[:, 1 + k] += g
    kt, th0 = 87.85 * KCAL, 107.4 * PI / 180.0
    c = (v[0] * v[1]).sum(-1) / (ln[0] * ln[1])
    th = torch.acos(c) - th0
    energy += 0.5 * kt * float(th.square().sum())
    g = kt * th / (1.0 - c * c).sqrt()  # -dE/dc
    for k in (0, 1):
        dc = v[1 - k] / (ln[0] * ln[1])[:, None] - (c / ln[k] ** 2)[:, None] * v[k]
        f[:, 0] += g[:, None] * dc
        f[:, 1 + k] -= g[:, None] * dc
    # Ewald over the charge sites (M in the oxygen's place)
    gm = 0.73612
    site = r.clone()
    site[:, 0] = gm * r[:, 0] + 0.5 * (1.0 - gm) * (r[:, 1] + r[:, 2])
    site = site.reshape(-1, 3)
    n = site.shape[0]
    qo = -1.1128
    chg = torch.tensor([qo, -0.5 * qo, -0.5 * qo], dtype=x.dtype, device=x.device).repeat(mols)
    kappa, rc, kc = _ewald(mols, box)
    pref = 2.0 * kappa / math.sqrt(PI)
    fs = torch.zeros_like(site)
    for lo in range(0, n, 1024):
        i = torch.arange(lo, min(n, lo + 1024), device=x.device)
        d = _image(site[i][:, None] - site[None], L)
        r2 = d.square().sum(-1)
        j = torch.arange(n, device=x.device)
        on = (r2 < rc * rc) & (i[:, None] != j[None])
        r2 = torch.where(on, r2, torch.ones_like(r2))
        rl = r2.sqrt()
        qq = torch.where(on, chg[i][:, None] * chg[None], torch.zeros_like(r2))
        same = i[:, None] // 3 == j[None] // 3
        e = qq / rl * torch.where(same, -torch.erf(kappa * rl), torch.erfc(kappa * rl))
        energy += 0.5 * float(e.sum())
        fs[i] = (((e + qq * pref * torch.exp(-(kappa * kappa) * r2)) / r2)[..., None] * d).sum(1)
    b = [2.0 * PI / float(s) for s in box]
    km = int(kc * float(box.max()) / (2.0 * PI))
    ks = []
    for kx in range(km + 1):
        ky, kz = np.meshgrid(np.arange(-km, km + 1), np.arange(-km, km + 1), indexing="ij")
        k2 = (b[0] * kx) ** 2 + (b[1] * ky) ** 2 + (b[2] * kz) ** 2
        on = np.where((ky == 0) & (kz == 0), (k2 > 0) & (k2 < kc * kc), k2 <= kc * kc)
        ks.append(np.stack([np.full(on.sum(), b[0] * kx), b[1] * ky[on], b[2] * kz[on]], 1))
    k = torch.from_numpy(np.concatenate(ks)).cuda()
    vol = float(np.prod(box))
    k2 = k.square().sum(-1)
    coef = 2.0 * PI / vol * torch.exp(-k2 / (4.0 * kappa * kappa)) / k2 * torch.where(k[:, 0] > 0, 2.0, 1.0)
    for lo in range(0, len(k), 2048):
        kk, cc = k[lo:lo + 2048], coef[lo:lo + 2048]
        ph = site @ kk.T
        co, si = ph.cos() * chg[:, None], ph.sin() * chg[:, None]
        sr, si_ = co.sum(0), si.sum(0)
        energy += float((cc * (sr * sr + si_ * si_)).sum())
        fs += ((sr * si - si_ * co) * (2.0 * cc)) @ kk
    energy -= 0.5 * pref * float(chg.square().sum())
    fs = fs.reshape(mols, 3, 3)
    f[:, 0] += gm * fs[:, 0]
    f[:, 1] += fs[:, 1] + 0.5 * (1.0 - gm) * fs[:, 0]
    f[:, 2] += fs[:, 2] + 0.5 * (1.0 - gm) * fs[:, 0]
    return f.reshape(-1), energy


def _exact_train(case, seed):
    st = _prepare_train(case, seed)
    m = case["rows"]
    a = st["wbf"].double()
    w = [t.clone().requires_grad_() for t in (a[:64 * 96].reshape(64, 96), a[64 * 96:64 * 160].reshape(64, 64), a[64 * 160:].reshape(16, 64))]
    bias = [t.double().clone().requires_grad_() for t in (st["w"][N_WEIGHTS:N_WEIGHTS + 64], st["w"][N_WEIGHTS + 64:N_WEIGHTS + 128],
                                                          st["w"][N_WEIGHTS + 128:])]
    total = 0.0
    for lo in range(0, m, 65536):
        h = st["x"][lo:lo + 65536].double()
        for k in range(3):
            h = h @ w[k].T + bias[k]
            h = torch.nn.functional.silu(h) if k < 2 else h
        err = (h - st["t"][lo:lo + 65536].double())[:, :9].square().sum()
        (err / (9 * m)).backward()
        total += float(err.detach())
    grad = torch.cat([t.grad.reshape(-1) for t in w + bias] + [torch.tensor([total], dtype=torch.float64, device="cuda")])
    new = st["w"].double() - 1e-4 * grad[:-1] / (grad[:-1].abs() + 1e-8)  # Adam's first step
    return {"grad": grad, "w": new}
