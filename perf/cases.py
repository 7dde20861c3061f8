"""The work this library is measured on: its public entry points over the range of systems
that the benchmark configurations (cgppd_gb300/workloads.py) span.

kinds of case
  energy     one call of the drop-in energy module on a packed replica: the reference's
             callers issue one per Monte Carlo step (synchronous, non-crowder or
             asynchronous form)
  recompute  every replica's energy from scratch (Engine.recompute), as after an upload
             or to drop accumulated rounding
  mc         one exchange block: Engine.run, then every replica's state and potential
             downloaded into page-locked buffers
  grad       loss and gradient of the pair-energy network on one mini-batch
  predict    its inference on host features
  train      one epoch of Adam training over collected samples

Energies are returned in FP32: they are sums of FP32 pair terms, and the asynchronous
energy call and torch's own scalars are FP32 too.
"""
import ctypes
import functools
import math

import numpy as np
import torch

import cgppd_gb300
from cgppd_gb300 import engine as eng
from cgppd_gb300 import surrogate as sg
from cgppd_gb300 import workloads as wlm

LADDER = (288.0, 450.0)          # temperatures of every configuration
TABLE_SEED = 20261203            # the contact table is a parameter file, not an input


# ------------------------------------------------------------------ cases

def listed():
    return [
        # the reference's own test system (two 76-residue chains): launch latency
        {"name": "energy_two_chains", "kind": "energy", "form": "sync", "lengths": "76x2", "crowders": 0,
         "flexible": 0.0, "box": 150.0},
        # a mid-size replica with flexible segments (exclusions inside molecules), odd size
        {"name": "energy_flexible", "kind": "energy", "form": "sync", "lengths": "162x5 203x1", "crowders": 0,
         "flexible": 0.1, "box": 180.0},
        # one replica of the crowded configuration on a caller's stream, as replicas issue it
        {"name": "energy_crowded", "kind": "energy", "form": "async", "lengths": "60-160x24", "crowders": 40,
         "flexible": 0.0, "box": 250.0},
        # the largest replicas: the non-crowder sum that the sampling takes
        {"name": "energy_large", "kind": "energy", "form": "nc", "lengths": "40-400x80", "crowders": 40,
         "flexible": 0.0, "box": 450.0},
        # fresh energies of the crowded configuration's ladder
        {"name": "recompute_crowded", "kind": "recompute", "system": "rigid", "sims": 1, "lengths": "60-160x24",
         "crowders": 40, "replicas": 32, "box": 250.0},
        # the flexible-linker configuration: one chain of 76 + 10 + 76, step latency
        {"name": "mc_linker", "kind": "mc", "system": "linker", "sims": 1, "lengths": "76x2", "linker": 10,
         "crowders": 0, "replicas": 32, "box": 150.0, "steps": 100, "cluster": 8, "threads": 256},
        # eight copies of one protein
        {"name": "mc_copies", "kind": "mc", "system": "copies", "sims": 1, "lengths": "76x8", "crowders": 0,
         "replicas": 32, "box": 120.0, "steps": 100, "cluster": 4, "threads": 512},
        # the crowded configuration: 24 proteins and 40 crowders
        {"name": "mc_crowded", "kind": "mc", "system": "rigid", "sims": 1, "lengths": "60-160x24", "crowders": 40,
         "replicas": 32, "box": 250.0, "steps": 100, "cluster": 4, "threads": 512},
        # many uneven simulations in one launch
        {"name": "mc_batched", "kind": "mc", "system": "rigid", "sims": 32, "lengths": "40-400x2-12", "crowders": 0,
         "replicas": 24, "box": 0.0, "steps": 40, "cluster": 1, "threads": 512},
        # one training step of the pair-energy network: forward and backward
        {"name": "net_gradient", "kind": "grad", "rows": 8192},
        # its inference over a pose table of odd size
        {"name": "net_predict", "kind": "predict", "rows": 50001},
        # one epoch over collected samples: the whole training call
        {"name": "net_train", "kind": "train", "rows": 131072},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["energy", "energy", "recompute", "mc", "mc", "mc", "grad", "predict", "train"])
    if kind == "energy":
        n, longest = _logint(rng, 2, 80), _logint(rng, 60, 400)
        c = rng.choice([0, 0, rng.randint(1, 40)])
        residues = n * 0.5 * (longest + 30) + 20 * c
        return {"kind": "energy", "form": rng.choice(["sync", "nc", "async"]), "lengths": "30-%dx%d" % (longest, n),
                "crowders": c, "flexible": rng.choice([0.0, 0.0, 0.1]),
                "box": round(max(150.0, 2.0 * (residues * 500.0) ** (1 / 3)), 1)}
    if kind == "recompute":
        n, c, r = _logint(rng, 2, 24), rng.choice([0, rng.randint(1, 40)]), _logint(rng, 4, 32)
        return {"kind": "recompute", "system": "rigid", "sims": 1, "lengths": "40-%dx%d" % (_logint(rng, 60, 160), n),
                "crowders": c, "replicas": r, "box": 250.0}
    if kind == "mc":
        system = rng.choice(["linker", "copies", "rigid", "batched"])
        steps = _logint(rng, 20, 100)
        r = _logint(rng, 8, 32)
        c = {"kind": "mc", "system": system, "sims": 1, "crowders": 0, "replicas": r, "steps": steps, "cluster": 4,
             "threads": 512}
        if system == "linker":
            c.update(lengths="%dx2" % rng.randint(30, 76), linker=rng.randint(5, 12), box=150.0, cluster=8,
                     threads=256)
        elif system == "copies":
            c.update(lengths="%dx%d" % (_logint(rng, 30, 120), rng.randint(2, 8)), box=150.0)
        elif system == "rigid":
            c.update(lengths="60-%dx%d" % (rng.randint(80, 160), rng.randint(4, 24)), crowders=rng.randint(0, 40),
                     box=250.0)
        else:
            c.update(system="rigid", sims=rng.randint(8, 31), lengths="40-%dx2-%d" % (_logint(rng, 80, 400),
                                                                                      rng.randint(3, 12)),
                     box=0.0, steps=min(steps, 40), replicas=rng.randint(8, 24), cluster=1)
        return c
    if kind == "grad":
        # batches up to 1024 rows in steps of 128, larger ones in steps of 1024
        return {"kind": "grad", "rows": rng.choice([128 * rng.randint(1, 8), 1024 * rng.randint(1, 7)])}
    if kind == "predict":
        return {"kind": "predict", "rows": _logint(rng, 100, 50000)}
    return {"kind": "train", "rows": _logint(rng, 16000, 131000)}


# ------------------------------------------------------------------ systems

def _sizes(case):
    """Residue counts of the proteins of each simulation: 'LENxCOUNT' terms, either a
    range 'a-b' (log-uniform lengths, uniform counts), drawn from the text alone."""
    rng = np.random.default_rng(sum(map(ord, case["lengths"])) + 7 * case.get("sims", 1))
    out = []
    for _ in range(case.get("sims", 1)):
        lens = []
        for term in case["lengths"].split():
            length, count = term.split("x")
            if "-" in count:
                a, b = map(int, count.split("-"))
                count = int(rng.integers(a, b + 1))
            for _ in range(int(count)):
                if "-" in length:
                    a, b = map(int, length.split("-"))
                    lens.append(int(round(math.exp(rng.uniform(math.log(a), math.log(b))))))
                else:
                    lens.append(int(length))
        out.append(lens)
    return out


@functools.lru_cache(maxsize=None)
def _globule(n):
    """A compact fold of n residues: the n lattice points nearest the centre (95 A^3 per
    residue, the density of the repository's synthetic chains) along a serpentine."""
    side = int(math.ceil((2.0 * n) ** (1 / 3))) + 2
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3).astype(np.float64)
    keep = np.argsort(((g - (side - 1) / 2.0 + 0.01) ** 2).sum(1), kind="stable")[:n]
    g = g[np.sort(keep)]
    x = 4.57 * g + np.random.default_rng(n).normal(scale=0.35, size=g.shape)
    return x - x.mean(0)


@functools.lru_cache(maxsize=None)
def _linker_chain(na, nl, nb):
    for seed in range(4):   # a walk may run into its own domain: the next one
        try:
            return wlm.two_domain_linker(np.random.default_rng([seed, na, nl, nb]), na, nl, nb).astype(np.float64)
        except RuntimeError:
            continue
    raise RuntimeError("no linker structure of %d + %d + %d residues" % (na, nl, nb))


@functools.lru_cache(maxsize=None)
def _parameters():
    """The parameter files of a run: contact table (20 types and the crowder type), vdW
    radius per type, torsion tables."""
    rng = np.random.default_rng(TABLE_SEED)
    radius = rng.uniform(4.5, 7.0, size=21).astype(np.float32)
    table = wlm.contact_table(rng, with_crowder=True, crowder_eps=0.1)
    V = rng.uniform(0.0, 1.5, size=(20, 20, 4))
    S = rng.uniform(0.0, 2 * math.pi, size=(20, 20, 4))
    return table, radius, V, S


def _rotations(rng, n):
    q = rng.normal(size=(n, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    return np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], -1).reshape(n, 3, 3)


def _molecules(rng, lens, crowders, box, copies=False, linker=0):
    """Placed molecules of one simulation: the fold by length, orientation, centre,
    residue types and charges from rng."""
    _, radius, _, _ = _parameters()
    if linker:
        x = _linker_chain(lens[0], linker, lens[1])
        x = (x - x.mean(0)) @ _rotations(rng, 1)[0].T + box / 2.0
        n = len(x)
        types, charges, _ = wlm.residue_params(rng, n, radius)
        seg = list(range(lens[0] - 1, lens[0] + linker + 1))
        return [wlm.Molecule(x, types, charges, radius[types], segments=[seg])]
    folds = [_globule(n) for n in lens] + [_globule(20)] * crowders
    rad = [float(np.sqrt((f ** 2).sum(1).max())) for f in folds]
    centres = wlm.place_centres(rng, [0.8 * r for r in rad], box)
    rot = _rotations(rng, len(folds))
    mols, first = [], None
    for k, f in enumerate(folds):
        x = f @ rot[k].T + centres[k]
        if k >= len(lens):
            mols.append(wlm.Molecule(x, np.full(20, wlm.CROWDER_TYPE, np.int32), np.zeros(20, np.float32),
                                     np.full(20, 5.0, np.float32), crowder=True))
            continue
        if not copies or first is None:
            types, charges, _ = wlm.residue_params(rng, len(f), radius)
            first = types, charges
        mols.append(wlm.Molecule(x, first[0], first[1], radius[first[0]]))
    return mols


def _box(case, lens):
    return case["box"] or max(150.0, 2.2 * (sum(lens) * 2000.0) ** (1 / 3))


def _workload(case, seed):
    rng = np.random.default_rng(seed)
    table, _, V, S = _parameters()
    linker = case.get("linker", 0)
    R = case["replicas"]
    sims = []
    for lens in _sizes(case):
        box = _box(case, lens)
        mols = _molecules(rng, lens, case["crowders"], box, case["system"] == "copies", linker)
        weights = (0.35, 0.35, 0.30, 0.35) if linker else (1, 1, 1, 1)
        sims.append(wlm.Simulation(mols, box, wlm.ladder(*LADDER, R), wlm.ladder(0.5, 2.0, R),
                                   wlm.ladder(0.2, 0.2, R), move_weights=weights))
    return wlm.Workload("case", sims, table, V if linker else None, S if linker else None, seed=seed)


def _packed(case, seed):
    """A replica packed as the reference uploads it: float4 (x, y, z, rigid-domain uid +
    bond fraction) and (type, charge, radius, molecule id + chain fraction or -1 for a
    crowder), padded to 32 residues."""
    rng = np.random.default_rng(seed)
    lens = _sizes(case)[0]
    mols = _molecules(rng, lens, case["crowders"], case["box"])
    n = sum(m.n for m in mols)
    P = -(-n // 32) * 32
    pos, meta = np.zeros((P, 4), np.float32), np.zeros((P, 4), np.float32)
    pos[:, 3], meta[:, 0] = -2.0, 20.0
    i = 0
    for k, m in enumerate(mols):
        sl = slice(i, i + m.n)
        pos[sl, :3] = m.xyz
        domain = np.full(m.n, k + 1.0, np.float32)
        if case["flexible"] and not m.crowder:
            # a flexible segment: no rigid domain, bonded to the domains at both ends
            width = max(4, int(case["flexible"] * m.n))
            a = int(rng.integers(4, max(5, m.n - width - 4)))
            domain[a:a + width] = 0.0
            domain[a - 1:a + 1] += 0.25
        pos[sl, 3] = domain
        meta[sl, 0] = np.minimum(m.types, 19)
        meta[sl, 1] = m.charges
        meta[sl, 2] = m.radii
        meta[sl, 3] = -1.0 if m.crowder else (k + 1) + (k + 1) / 1024.0
        i += m.n
    return pos, meta


# ------------------------------------------------------------------ network inputs

def _poses(seed, rows):
    """Pose features of molecule pairs as the collector writes them, and energies: a
    smooth well in the distance and the orientation, and noise."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))
    d = torch.randn(rows, 3, generator=g, device="cuda") * 1.3
    r = 20.0 * d.norm(dim=1).clamp_min(0.2)
    q = torch.randn(rows, 4, generator=g, device="cuda")
    q = q / q.norm(dim=1, keepdim=True)
    q = torch.where(q[:, :1] < 0, -q, q)
    X = torch.cat([d, (10.0 / r)[:, None], q], 1)
    y = 8.0 * torch.exp(-((r - 22.0) / 9.0) ** 2) * (q[:, 1] - 1.0) + 0.3 * torch.randn(rows, generator=g, device="cuda")
    return X.cpu().numpy(), y.cpu().numpy()


def _network(flat):
    """float64 parameters on the GPU by name."""
    return {k: torch.from_numpy(np.asarray(v, np.float64)).cuda() for k, v in sg.unpack(flat).items()}


def _forward64(p, X):
    h = X
    for layer in "1234":
        h = torch.nn.functional.silu(h @ p["W" + layer].T + p["b" + layer])
    return h @ p["w5"] + p["b5"]


# ------------------------------------------------------------------ prepare and run

def _bind_table():
    L = cgppd_gb300.lib()
    t20 = np.ascontiguousarray(_parameters()[0][:20, :20])
    a = L.cgppd_aminoacids_create()
    L.cgppd_aminoacids_set_table(a, t20.ctypes.data_as(ctypes.POINTER(ctypes.c_float)))
    dev = L.LJPotentialDataToDevice(a)
    L.cgppd_aminoacids_destroy(a)
    L.bindLJTexture(dev)


_bound = []


def prepare(case, seed):
    kind = case["kind"]
    if kind == "energy":
        if not _bound:
            _bind_table()
            _bound.append(True)
        pos, meta = _packed(case, seed)
        L = cgppd_gb300.lib()
        L.CUDA_setBoxDimension(case["box"])
        st = {"kind": kind, "form": case["form"], "L": L, "P": len(pos), "pos": torch.from_numpy(pos).cuda(),
              "meta": torch.from_numpy(meta).cuda(), "result": ctypes.c_double(0.0)}
        if case["form"] == "async":
            st["stream"] = torch.cuda.Stream()
            side = len(pos) // 32
            st["out"] = torch.zeros(side * side, dtype=torch.float32, device="cuda")
        return st
    if kind in ("grad", "predict", "train"):
        rows = case["rows"]
        X, y = _poses(seed, rows)
        s = sg.Surrogate(batch=8192, seed=seed)
        if kind == "train":
            s.add_samples(X, y)
        return {"kind": kind, "net": s, "X": X, "y": y}
    wl = _workload(case, seed)
    e = eng.from_workload(wl, cluster=case.get("cluster", 4), threads=case.get("threads", 512))
    st = {"kind": kind, "engine": e, "steps": case.get("steps", 0), "bufs": []}
    if kind == "mc":
        # one page-locked buffer per array, every simulation's replicas in a row
        info = [e.sim_info(si) for si in range(len(wl.sims))]
        count = lambda f: sum(f(*x) for x in info)  # noqa: E731
        st["all"] = {"positions": torch.zeros(count(lambda N, M, R: 4 * R * N)).pin_memory(),
                     "relative": torch.zeros(count(lambda N, M, R: 4 * R * N)).pin_memory(),
                     "centres": torch.zeros(count(lambda N, M, R: 4 * R * M)).pin_memory(),
                     "potentials": torch.zeros(count(lambda N, M, R: R), dtype=torch.float64).pin_memory()}
        at = [x.data_ptr() for x in st["all"].values()]
        for N, M, R in info:
            st["bufs"].append(tuple(at))
            at = [a + 8 * n for a, n in zip(at, (2 * R * N, 2 * R * N, 2 * R * M, R))]
    else:
        pos = torch.from_numpy(_replica_positions(wl, seed)).pin_memory()
        e.upload(0, pos.data_ptr(), None, None, recompute=False)
        e.synchronize()
    return st


def _replica_positions(wl, seed):
    """Every replica of the one simulation with its molecules shifted by about 1 A."""
    rng = np.random.default_rng(seed + 1)
    sim = wl.sims[0]
    R = len(sim.temperatures)
    out = np.zeros((R, sim.n_residues, 4), np.float32)
    i = 0
    for m in sim.molecules:
        out[:, i:i + m.n, :3] = m.xyz[None] + rng.normal(size=(R, 1, 3)).astype(np.float32)
        i += m.n
    return out


def run(state):
    kind = state["kind"]
    if kind == "energy":
        L, P = state["L"], state["P"]
        pos, meta = ctypes.c_void_p(state["pos"].data_ptr()), ctypes.c_void_p(state["meta"].data_ptr())
        if state["form"] == "async":
            L.CUDA_EonDevice_async(pos, meta, None, None, None, None, ctypes.c_void_p(state["out"].data_ptr()),
                                   P // 32, 32, P, 0, ctypes.c_void_p(state["stream"].cuda_stream))
            return state["out"]
        call = L.CUDA_EonDeviceNC if state["form"] == "nc" else L.CUDA_EonDevice
        call(pos, meta, None, None, None, None, ctypes.byref(state["result"]), 32, P, 0)
        return state["result"].value
    if kind == "recompute":
        return state["engine"].recompute().astype(np.float32)
    if kind == "mc":
        e = state["engine"]
        e.run(1, state["steps"])
        for si, b in enumerate(state["bufs"]):
            e.download(si, *b)
        e.synchronize()
        return {**state["all"], "potentials": state["all"]["potentials"].float()}
    net = state["net"]
    if kind == "grad":
        loss, g = net.loss_grad(state["X"], state["y"])
        return {"loss": loss, "gradient": g}
    if kind == "predict":
        return net.predict(state["X"])
    history = net.train(1)
    return {"parameters": net.params, "history": history}


# ------------------------------------------------------------------ work

def _pairs_per_step(lens):
    n = np.asarray(lens, np.float64)
    return float((n * (n.sum() - n)).sum() / len(n))


PAIR_FLOPS = 30   # the Lennard-Jones term of a pair; charged pairs' further term left out


def work(case):
    kind = case["kind"]
    if kind == "energy":
        lens = _sizes(case)[0] + [20] * (0 if case["form"] == "nc" else case["crowders"])
        n = np.asarray(lens, np.float64)
        P = 32 * -(-(sum(_sizes(case)[0]) + 20 * case["crowders"]) // 32)
        return {"bytes": 32.0 * P, "flops": PAIR_FLOPS * float(n.sum() ** 2 - (n * n).sum()) / 2}
    if kind == "recompute":
        n = np.asarray(_sizes(case)[0] + [20] * case["crowders"], np.float64)
        R = case["replicas"]
        return {"bytes": 16.0 * float(n.sum()) * R, "flops": PAIR_FLOPS * R * float(n.sum() ** 2 - (n * n).sum()) / 2}
    if kind == "mc":
        R, byt, fl = case["replicas"], 0.0, 0.0
        for lens in _sizes(case):
            if case["system"] == "linker":
                na, nb = lens
                n = na + nb + case["linker"]
                fl += 0.3 * PAIR_FLOPS * R * case["steps"] * na * nb   # the moves that change internal distances
                byt += 96.0 * n * R
                continue
            lens = lens + [20] * case["crowders"]
            fl += PAIR_FLOPS * R * case["steps"] * _pairs_per_step(lens)
            byt += 96.0 * (sum(lens) + len(lens)) * R   # state in, state out, downloaded
        return {"bytes": byt, "flops": fl}
    rows = case["rows"]
    layers = 2.0 * rows * (8 * 256 + 3 * 256 * 256 + 256)
    if kind == "predict":
        return {"bytes": rows * 36.0 + sg.N_PARAMS * 4.0, "flops": layers}
    if kind == "grad":
        return {"bytes": rows * 36.0 + 2 * sg.N_PARAMS * 4.0, "flops": 3 * layers}
    n = rows - int(0.05 * rows)
    steps = n // 8192
    return {"bytes": rows * 36.0 + steps * 7 * 4.0 * sg.N_PARAMS, "flops": (3 * steps * 8192 + rows - n) / rows * layers}


# ------------------------------------------------------------------ 64-bit values

RT_KCAL, DH_FACTOR = float(np.float32(0.59218674898147583)), float(np.float32(4.1507959365844727))


def _pair_sum(xyz, types, charges, radii, eps, box, keep):
    """Sum over pairs i < j with keep(i, j) of the Kim-Hummer term in kcal/mol."""
    n = len(xyz)
    total = torch.zeros((), dtype=torch.float64, device="cuda")
    idx = torch.arange(n, device="cuda")
    for a in range(0, n, 1024):
        i = idx[a:a + 1024, None]
        j = idx[None, a:]
        mask = (j > i) & keep(i, j)
        d = xyz[a:a + 1024, None, :] - xyz[None, a:, :]
        d = d - box * torch.round(d / box)
        r2 = (d * d).sum(-1).clamp_min(1e-30)
        r = r2.sqrt()
        e = eps[types[a:a + 1024]][:, types[a:]]
        s6 = (0.25 * (radii[a:a + 1024, None] + radii[None, a:]) ** 2 / r2) ** 3
        u = -4.0 * e * s6 * (s6 - 1.0)
        u = torch.where((e > 0) & (s6 > 0.5), 2.0 * e - u, u) * RT_KCAL
        u = u + DH_FACTOR * charges[a:a + 1024, None] * charges[None, a:] * torch.exp(-r / 10.0) / r
        total += torch.where(mask, u, torch.zeros_like(u)).sum()
    return total


def _eps64(table):
    return torch.from_numpy(float(wlm.LAMBDA) * (table.astype(np.float64) - float(wlm.E0))).cuda()


def exact(case, seed):
    kind = case["kind"]
    if kind == "energy":
        pos, meta = (torch.from_numpy(x).cuda().double() for x in _packed(case, seed))
        real = pos[:, 3] != -2.0
        P = len(pos)
        pos, meta = pos[real], meta[real]
        domain, chain, mol = pos[:, 3].trunc(), meta[:, 3].frac(), meta[:, 3].trunc()
        bond = pos[:, 3].frac()
        crowder = meta[:, 3] == -1.0

        def keep(i, j):
            if case["form"] == "nc":
                return ~crowder[i] & ~crowder[j] & (mol[i] != mol[j])
            return ~(((domain[i] != 0) & (domain[i] == domain[j])) | ((bond[i] != 0) & (bond[i] == bond[j])) |
                     ((chain[i] == chain[j]) & ((j - i) < 4)))

        e = _pair_sum(pos[:, :3], meta[:, 0].long(), meta[:, 1], meta[:, 2], _eps64(_parameters()[0][:20, :20]),
                      float(np.float32(case["box"])), keep)
        if case["form"] == "async":
            out = torch.zeros((P // 32) ** 2, dtype=torch.float64, device="cuda")
            out[0] = e
            return out
        return e
    if kind == "recompute":
        wl = _workload(case, seed)
        sim = wl.sims[0]
        pos = torch.from_numpy(_replica_positions(wl, seed)).cuda().double()
        types, charges, radii = (torch.from_numpy(np.concatenate([getattr(m, k) for m in sim.molecules])).cuda()
                                 for k in ("types", "charges", "radii"))
        mol = torch.from_numpy(np.repeat(np.arange(len(sim.molecules)), [m.n for m in sim.molecules])).cuda()
        eps = _eps64(wl.lj_raw)
        return torch.stack([_pair_sum(p[:, :3], types.long(), charges.double(), radii.double(), eps, sim.box,
                                      lambda i, j: mol[i] != mol[j]) for p in pos])
    if kind in ("grad", "predict"):
        X, y = _poses(seed, case["rows"])
        s = sg.Surrogate(batch=128, seed=seed)   # for its seeded parameters only
        p = _network(s.params)
        s.close()
        X = torch.from_numpy(X).cuda().double()
        if kind == "predict":
            return _forward64(p, X)
        for v in p.values():
            v.requires_grad_(True)
        loss = ((_forward64(p, X) - torch.from_numpy(y).cuda().double()) ** 2).mean()
        loss.backward()
        return {"loss": loss.detach(), "gradient": torch.cat([p[k].grad.reshape(-1) for k in sg.OFF])}
    return None   # a trajectory, or an optimiser's path, has no value apart from its steps' rounding
