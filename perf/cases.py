"""Performance cases of the simulation step: what a user of this package has it do, through its public
entry points, over the range of sizes, models, semantics and precisions it is used with.

A case is a dict of plain values; `kind` names the call it stands for:

  sim      one Simulation: set a state, advance it, read the counts and statistics back.  This is one
           checkpoint interval of a run (the state comes from host memory, as a snapshot or a fresh
           initial condition does, and the counts go back to be logged).  Models: the small A/B network,
           the Schlogl model, random sparse networks of 3-16 species (all on reflective lattices), and an
           enzyme network in a cell of irregular shape, given as a neighbour table with a membrane and a
           cytosol compartment.
  learned  the same with a learned tau proposer attached (corrected semantics).
  batch    a Batch: an ensemble of independent replicas (uneven Brusselator lattices with their own rate
           constants, or equal Schlogl lattices), every state set, all advanced together, every state read.
  train    Learner.train on a buffer of trace records: a whole (short) training, weights returned.
  argmin   plis_tau_argmin_noalloc over a device array of taus.

Counts, times and statistics of a simulation are draws from its random stream: they have no value that
64-bit arithmetic without the stream could give, so exact() returns None for them.
"""
import ctypes
import math

import numpy as np
import torch

from pliscuda_b200 import Model, Simulation, _lib, workloads
from pliscuda_b200.batch import Batch
from pliscuda_b200.learned import N_WEIGHTS, TRACE_DTYPE, Learner


def listed():
    return [
        # one step of a small system and a look at it: the smallest call, all latency
        {"name": "ab10_one_step", "kind": "sim", "model": "ab", "x": 10, "y": 10, "z": 10, "mode": "reference",
         "precision": "fp64", "steps": 1},
        # the small plain run: 1,000 subvolumes, a few hundred steps, bound by the step's latency
        {"name": "ab10_run", "kind": "sim", "model": "ab", "x": 10, "y": 10, "z": 10, "mode": "reference",
         "precision": "fp64", "steps": 300},
        # the headline workload: Schlogl on 64^3, reference semantics, binary64
        {"name": "schlogl64_fp64", "kind": "sim", "model": "schlogl", "x": 64, "y": 64, "z": 64, "mode": "reference",
         "precision": "fp64", "steps": 256},
        # the binary32 form with corrected semantics on a lattice of odd sides
        {"name": "schlogl_odd_fp32", "kind": "sim", "model": "schlogl", "x": 67, "y": 45, "z": 53, "mode": "corrected",
         "precision": "fp32", "steps": 256},
        # learned tau proposals on a large lattice
        {"name": "learned128_fp64", "kind": "learned", "x": 128, "y": 128, "z": 128, "precision": "fp64", "steps": 24},
        # a network of many species and reactions, binary32, medium lattice
        {"name": "net64_fp32", "kind": "sim", "model": "net", "species": 10, "reactions": 20, "network": 7, "x": 64,
         "y": 64, "z": 64, "mode": "reference", "precision": "fp32", "steps": 64},
        # the same network in binary64 on the largest lattice: the largest call
        {"name": "net128_fp64", "kind": "sim", "model": "net", "species": 10, "reactions": 20, "network": 7, "x": 128,
         "y": 128, "z": 128, "mode": "reference", "precision": "fp64", "steps": 64},
        # an irregular cell with two compartments (neighbour table), about 9,000 subvolumes
        {"name": "cell_table_fp64", "kind": "sim", "model": "cell", "x": 26, "y": 26, "z": 26, "mode": "reference",
         "precision": "fp64", "steps": 256},
        # an uneven ensemble with its own parameters per replica: 256 Brusselator lattices of side 8..48
        {"name": "batch_brusselator256", "kind": "batch", "model": "brusselator", "replicas": 256, "low": 8, "high": 48,
         "mode": "reference", "precision": "fp64", "steps": 64},
        # an ensemble of equal small systems for statistics, corrected semantics, binary32
        {"name": "batch_schlogl16x128", "kind": "batch", "model": "schlogl", "replicas": 128, "low": 16, "high": 16,
         "mode": "corrected", "precision": "fp32", "steps": 250},
        # training of a proposer
        {"name": "train_proposer", "kind": "train", "records": 400_000, "batch": 16384, "iterations": 200,
         "quantile": 0.25},
        # the arg-min of the taus of a 256^3 lattice, on the caller's stream
        {"name": "argmin_16m", "kind": "argmin", "n": 1 << 24},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi, cells):
    """Three sides, log-uniform and odd as often as even, with at most `cells` subvolumes."""
    while True:
        d = [_log_int(rng, lo, hi) for _ in range(3)]
        if d[0] * d[1] * d[2] <= cells:
            return {"x": d[0], "y": d[1], "z": d[2]}


def draw(rng):
    kind = rng.choice(["ab", "schlogl", "schlogl", "net", "cell", "learned", "brusselator", "ensemble", "train", "argmin"])
    forms = {"mode": rng.choice(["reference", "corrected"]), "precision": rng.choice(["fp64", "fp32"])}
    if kind == "ab":
        return {"kind": "sim", "model": "ab", **_sides(rng, 2, 20, 4096), **forms, "steps": _log_int(rng, 1, 400)}
    if kind == "schlogl":
        d = _sides(rng, 8, 128, 1 << 21)
        most = max(2, min(256, (1 << 26) // (d["x"] * d["y"] * d["z"])))
        return {"kind": "sim", "model": "schlogl", **d, **forms, "steps": _log_int(rng, 2, most)}
    if kind == "net":
        d = _sides(rng, 8, 96, 1 << 19)
        most = max(2, min(64, (1 << 24) // (d["x"] * d["y"] * d["z"])))
        species, reactions, network = rng.choice([(10, 20, 7), (6, 12, 7), (5, 9, 11), (16, 30, 7), (3, 7, 11)])
        return {"kind": "sim", "model": "net", "species": species, "reactions": reactions, "network": network, **d,
                **forms, "steps": _log_int(rng, 2, most)}
    if kind == "cell":
        return {"kind": "sim", "model": "cell", **_sides(rng, 6, 48, 40_000), **forms, "steps": _log_int(rng, 8, 256)}
    if kind == "learned":
        d = _sides(rng, 8, 128, 1 << 21)
        most = max(2, min(128, (1 << 25) // (d["x"] * d["y"] * d["z"])))
        return {"kind": "learned", **d, "precision": forms["precision"], "steps": _log_int(rng, 2, most)}
    if kind == "brusselator":
        low = rng.randint(4, 16)
        return {"kind": "batch", "model": "brusselator", "replicas": _log_int(rng, 4, 256), "low": low,
                "high": rng.randint(low, 40), **forms, "steps": _log_int(rng, 2, 48)}
    if kind == "ensemble":
        side = rng.randint(5, 20)
        return {"kind": "batch", "model": "schlogl", "replicas": _log_int(rng, 2, 128), "low": side, "high": side,
                **forms, "steps": _log_int(rng, 4, 200)}
    if kind == "train":
        return {"kind": "train", "records": _log_int(rng, 1000, 1_000_000), "batch": 128 * _log_int(rng, 1, 160),
                "iterations": _log_int(rng, 10, 250), "quantile": round(rng.uniform(0.1, 0.5), 3)}
    return {"kind": "argmin", "n": _log_int(rng, 1, 1 << 26)}


# -- models ------------------------------------------------------------------------------------------
def _on_lattice(m, dims):
    """The network of the lattice model m on a lattice of other sides."""
    return Model(n_subvolumes=dims[0] * dims[1] * dims[2], n_species=m.n_species, n_reactions=m.n_reactions,
                 reactants=m.reactants, products=m.products, reaction_rates=m.reaction_rates,
                 diffusion_rates=m.diffusion_rates, lattice=dims)


def _cell(dims, rng):
    """An ellipsoid cut out of a lattice: subvolumes inside it, numbered as the lattice is, as a 6-wide
    neighbour table padded with the own index; its outer layer is the membrane compartment.  Enzyme
    kinetics E + S <-> ES -> E + P, P -> S, with faster catalysis at the membrane."""
    X, Y, Z = dims
    z, y, x = np.meshgrid(np.arange(Z), np.arange(Y), np.arange(X), indexing="ij")
    r2 = (((x + 0.5) / X - 0.5) ** 2 + ((y + 0.5) / Y - 0.5) ** 2 + ((z + 0.5) / Z - 0.5) ** 2).reshape(-1)
    inside = r2 <= 0.25
    n = int(inside.sum())
    number = np.full(X * Y * Z + 1, -1, np.int64)
    number[:-1][inside] = np.arange(n)
    cells = np.nonzero(inside)[0]
    cx, cy, cz = cells % X, (cells // X) % Y, cells // (X * Y)
    nb = np.empty((n, 6), np.int64)
    for j, (there, step) in enumerate(((cx > 0, -1), (cx + 1 < X, 1), (cy > 0, -X), (cy + 1 < Y, X), (cz > 0, -X * Y),
                                       (cz + 1 < Z, X * Y))):
        nb[:, j] = number[np.where(there, cells + step, X * Y * Z)]
    membrane = (nb < 0).any(axis=1)
    own = np.arange(n)[:, None]
    key = np.where(nb < 0, 6, np.arange(6))
    nb = np.take_along_axis(np.where(nb < 0, own, nb), np.argsort(key, axis=1, kind="stable"), axis=1)
    E, S, ES, P = range(4)
    re = np.zeros((4, 4), np.int32)
    pr = np.zeros((4, 4), np.int32)
    for r, (reac, prod) in enumerate((((E, S), (ES,)), ((ES,), (E, S)), ((ES,), (E, P)), ((P,), (S,)))):
        re[list(reac), r] = 1
        pr[list(prod), r] = 1
    m = Model(n_subvolumes=n, n_species=4, n_reactions=4, reactants=re.reshape(-1), products=pr.reshape(-1),
              reaction_rates=[0.02, 0.5, 0.5, 0.1, 0.02, 0.5, 2.0, 0.1],
              diffusion_rates=[0.5, 1.0, 0.4, 1.0, 0.2, 1.0, 0.2, 1.0], neighbours=nb.reshape(-1).astype(np.uint32),
              n_compartments=2, compartment=membrane.astype(np.int32))
    state = np.concatenate([rng.poisson(30, n), rng.poisson(120, n), rng.poisson(15, n), rng.poisson(5, n)])
    return m, state.astype(np.uint32)


def _model(case, seed):
    """(model, initial counts) of a sim or learned case; the counts come from the seed."""
    rng = np.random.default_rng(seed)
    dims = (case["x"], case["y"], case["z"])
    n = dims[0] * dims[1] * dims[2]
    kind = case.get("model", "schlogl")
    if kind == "cell":
        return _cell(dims, rng)
    if kind == "ab":  # Poisson(50) counts of both species
        return _on_lattice(workloads.small_ab(2)[0], dims), rng.poisson(50.0, 2 * n).astype(np.uint32)
    if kind == "schlogl":  # low state on one half in x, high state on the other, with their fluctuations
        mean = np.where(np.arange(n) % dims[0] < dims[0] // 2, 100.0, 600.0)
        return _on_lattice(workloads.schlogl(2)[0], dims), rng.poisson(mean).astype(np.uint32)
    m = workloads.random_network(2, case["species"], case["reactions"], case["network"])[0]
    counts = np.exp(rng.random(case["species"] * n, dtype=np.float32) * np.float32(math.log(1e5)))
    return _on_lattice(m, dims), counts.astype(np.uint32)


def _weights(rng):
    """Proposer weights with hidden activations of order one that propose about 8 times the plain tau,
    and feature statistics of the Schlogl model."""
    w = np.zeros(N_WEIGHTS, np.float32)
    for off, fan, count, scale in ((0, 8, 512, 1.0), (576, 64, 4096, 1.0), (4736, 64, 4096, 1.0), (8896, 64, 64, 0.05)):
        w[off:off + count] = rng.uniform(-1, 1, count) * math.sqrt(6 / fan) * scale
    w[8960] = math.log(8.0)
    w[8961:8969] = (5.5, 5.5, 5.5, 6.0, 5.3, 6.5, -5.5, 7.5)
    w[8969:8977] = (1.1, 1.1, 0.7, 0.4, 1.0, 1.0, 1.0, 1.0)
    return w


# -- cases -------------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("sim", "learned"):
        model, counts = _model(case, seed)
        sim = Simulation(model, mode=case.get("mode", "corrected"), precision=case["precision"], seed=seed)
        if kind == "learned":
            sim.set_state(counts)
            sim.set_proposer(_weights(np.random.default_rng(3)), 16.0)
        return {"kind": "sim", "sim": sim, "counts": counts, "steps": case["steps"]}
    if kind == "batch":
        rng = np.random.default_rng(seed)
        models, counts = [], []
        # the lattice sides belong to the ensemble; rate constants and counts come from the seed
        for side in np.random.default_rng(3).integers(case["low"], case["high"] + 1, case["replicas"]).tolist():
            n = side ** 3
            if case["model"] == "schlogl":
                models.append(_on_lattice(workloads.schlogl(2)[0], (side, side, side)))
                mean = np.where(np.arange(n) % side < side // 2, 100.0, 600.0)
                counts.append(rng.poisson(mean).astype(np.uint32))
            else:
                a, b = rng.uniform(50, 200), rng.uniform(100, 600)
                models.append(_on_lattice(workloads.brusselator(2, a, b)[0], (side, side, side)))
                counts.append(np.concatenate([rng.poisson(a, n), rng.poisson(b / a * 1e4, n)]).astype(np.uint32))
        batch = Batch.from_models(models, mode=case["mode"], precision=case["precision"], seed=seed)
        return {"kind": kind, "batch": batch, "counts": counts, "steps": case["steps"]}
    if kind == "train":
        learner = Learner(case["records"])
        learner.set_records(_records(case, seed))
        return {"kind": kind, "learner": learner, "seed": seed, **{k: case[k] for k in ("batch", "iterations", "quantile")}}
    g = torch.Generator(device="cuda").manual_seed(seed)
    tau = torch.empty(case["n"], dtype=torch.float64, device="cuda").exponential_(1.0, generator=g)
    return {"kind": kind, "tau": tau, "min": torch.empty(1, dtype=torch.float64, device="cuda"),
            "arg": torch.empty(1, dtype=torch.int64, device="cuda")}


def _statistics(st):
    return [int(st.steps), int(st.rollbacks), int(st.events), int(st.exact_events), int(st.stop_reason)]


def run(state):
    kind = state["kind"]
    if kind == "sim":
        sim = state["sim"]
        sim.set_state(state["counts"])
        st = sim.step(state["steps"])
        return {"counts": sim.get_state(), "time": float(st.time), "stats": np.array(_statistics(st))}
    if kind == "batch":
        batch = state["batch"]
        for r, c in enumerate(state["counts"]):
            batch.set_state(r, c)
        batch.step(state["steps"])
        counts = np.concatenate([batch.get_state(r) for r in range(len(state["counts"]))])
        stats = [batch.stats(r) for r in range(len(state["counts"]))]
        return {"counts": counts, "time": np.array([s.time for s in stats]),
                "stats": np.array([_statistics(s) for s in stats])}
    if kind == "train":
        learner = state["learner"]
        learner.train(iterations=state["iterations"], batch=state["batch"], quantile=state["quantile"],
                      seed=state["seed"])
        return {"weights": learner.weights()}
    tau = state["tau"]
    rc = _lib.lib.plis_tau_argmin_noalloc(ctypes.c_void_p(tau.data_ptr()), tau.numel(),
                                          ctypes.c_void_p(state["min"].data_ptr()),
                                          ctypes.c_void_p(state["arg"].data_ptr()),
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    return {"min": state["min"], "arg": state["arg"]}


def _sizes(case):
    """(subvolumes, species, reactions, bytes of the neighbour table read per step) of a case."""
    if case["kind"] == "batch":
        sides = np.arange(case["low"], case["high"] + 1, dtype=np.float64)
        n = case["replicas"] * float(np.mean(sides ** 3))
        return n, (1 if case["model"] == "schlogl" else 2), 4, 0.0
    n = case["x"] * case["y"] * case["z"]
    kind = case.get("model", "schlogl")
    if kind == "cell":
        n = n * math.pi / 6
        return n, 4, 4, 24.0 * n
    return (n, *{"ab": (2, 3), "schlogl": (1, 4), "net": (case.get("species"), case.get("reactions"))}[kind], 0.0)


def work(case):
    """Bytes: every step reads and writes the counts (and reads the neighbour table, where there is
    one); the state crosses from and to host memory once.  Flops: per subvolume and step, a
    propensity (4), a Poisson mean and its exponential (24) per reaction and species, and the leap
    bound (10 per reaction, 30 per species); per record and parameter of a training step, 6."""
    if case["kind"] == "train":
        per = case["iterations"] * case["batch"]
        return {"bytes": 36.0 * per + case["iterations"] * 6 * 4.0 * 8961 + 64.0 * case["records"], "flops": 6.0 * 8768 * per}
    if case["kind"] == "argmin":
        return {"bytes": 8.0 * case["n"] + 16, "flops": float(case["n"])}
    n, s, r, table = _sizes(case)
    flops = n * (r * 38 + s * 58 + (17_000 if case["kind"] == "learned" else 0))
    return {"bytes": case["steps"] * (8.0 * s * n + table) + 8.0 * s * n, "flops": case["steps"] * flops}


# -- 64-bit values -----------------------------------------------------------------------------------
def _records(case, seed):
    """Trace records with features of the size of the Schlogl model's and labels that depend on them."""
    rng = np.random.default_rng(seed)
    recs = np.zeros(case["records"], TRACE_DTYPE)
    f = rng.standard_normal((case["records"], 8), dtype=np.float32)
    f[:, 2:] += 0.5 * f[:, :1]
    noise = rng.standard_normal(case["records"], dtype=np.float32)
    recs["label"] = 1.0 + np.tanh(f[:, 0]) + 0.3 * f[:, 6] * f[:, 1] + 0.3 * noise
    recs["features"] = f * np.float32(0.8) + np.array([5.5, 5.5, 5.5, 6, 5, 6.5, -5.5, 7.5], np.float32)
    recs["tau_cao"] = 1.0
    return recs


def _philox(c, k0, k1):
    """Philox4x32-10 blocks of the counters c (four uint64 arrays holding 32-bit words)."""
    m32 = np.uint64(0xFFFFFFFF)
    c = [np.asarray(v, np.uint64) for v in c]
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & m32, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _exact_training(case, seed):
    """Learner.train in binary64: He-uniform start, pinball loss of minibatches drawn by Philox, Adam."""
    recs = _records(case, seed)
    lo, hi = seed & 0xFFFFFFFF, seed >> 32
    count = 8 * 64 + 2 * 64 * 64 + 64
    u = (_philox((np.arange(count), np.full(count, 0x1417), np.zeros(count), np.zeros(count)), lo, hi)[0]
         >> np.uint64(8)).astype(np.float64)
    u = 2.0 * ((u + 0.5) / 16777216.0) - 1.0
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    w = torch.zeros(8961, dtype=torch.float64, device=dev)
    at = 0
    for off, fan, n in ((0, 8, 512), (576, 64, 4096), (4736, 64, 4096), (8896, 64, 64)):
        w[off:off + n] = torch.from_numpy((u[at:at + n] * math.sqrt(6.0 / fan)).astype(np.float32).astype(np.float64))
        at += n
    feats = torch.from_numpy(recs["features"].astype(np.float64)).to(dev)
    label = torch.from_numpy(recs["label"].astype(np.float64)).to(dev)
    mean = feats.mean(0)
    inv = 1.0 / torch.sqrt(torch.clamp((feats * feats).mean(0) - mean * mean, min=1e-6))
    w[8960] = label.mean()
    m, v = torch.zeros_like(w), torch.zeros_like(w)
    t = np.arange(case["batch"])
    for it in range(case["iterations"]):
        c = _philox((t, np.full(t.size, it), np.zeros(t.size), np.full(t.size, 0x7A11)), lo, hi)
        pick = torch.from_numpy((((c[0] << np.uint64(32)) | c[1]) % np.uint64(case["records"])).astype(np.int64)).to(dev)
        f, lab = (feats[pick] - mean) * inv, label[pick]
        W1, W2, W3 = w[0:512].view(8, 64), w[576:4672].view(64, 64), w[4736:8832].view(64, 64)
        h1 = torch.clamp(f @ W1 + w[512:576], min=0)
        h2 = torch.clamp(h1 @ W2 + w[4672:4736], min=0)
        h3 = torch.clamp(h2 @ W3 + w[8832:8896], min=0)
        res = lab - (h3 @ w[8896:8960] + w[8960])
        q = case["quantile"]
        dy = ((1.0 - q) * (res < 0).double() - q * (res > 0).double()) / case["batch"]
        g3 = dy[:, None] * w[8896:8960] * (h3 > 0)
        g2 = (g3 @ W3.T) * (h2 > 0)
        g1 = (g2 @ W2.T) * (h1 > 0)
        g = torch.cat([(f.T @ g1).reshape(-1), g1.sum(0), (h1.T @ g2).reshape(-1), g2.sum(0), (h2.T @ g3).reshape(-1),
                       g3.sum(0), h3.T @ dy, dy.sum().reshape(1)])
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        w = w - 1e-3 * (m / (1 - 0.9 ** (it + 1))) / (torch.sqrt(v / (1 - 0.999 ** (it + 1))) + 1e-8)
    return torch.cat([w, mean, inv]).cpu()


def exact(case, seed):
    if case["kind"] == "train":
        return {"weights": _exact_training(case, seed)}
    if case["kind"] == "argmin":
        tau = prepare(case, seed)["tau"]
        return {"min": tau.min().reshape(1), "arg": None}
    return None
