"""Timed cases of the framework's public entry points.

Each case is one thing a user's program does with this package: advance a
lattice between two records of a trajectory, take a whole solve through host
buffers, advance an ensemble of replicates together, serve a handful of solve
requests, run a well-mixed ensemble, or bring row-major frames in and out.
The models are the shapes of ``lattice_microbes_b200.configs`` (bimolecular,
rod cell, crowded cell, serving requests, two-state gene); the particle
lattices of the larger ones are placed on the GPU so that inputs are quick to
make.  Every output is a whole number, so every result has to be the same.
"""
import numpy as np
import torch

from lattice_microbes_b200 import configs
from lattice_microbes_b200.solver import Batch, CMEEnsemble, Context, Lattice, Model, Server

# kind "run": `records` records of a trajectory, `steps` timesteps each: the
#   inner loop of a solver (timesteps, then species counts).  `tune` says
#   whether the program lets the autotuner choose the schedule once.
# kind "solve": one whole solve through pinned host buffers (upload,
#   timesteps, download).
# kind "batch": an ensemble of bimolecular replicates of mixed edges.
# kind "serve": requests submitted, served to the end and collected.
# kind "cme": a well-mixed ensemble run and its records collected.
# kind "frames": a row-major lattice set, counted and read back.


def listed():
    return [
        # The smallest call: one record of a 16^3 replicate, 32 timesteps.
        dict(name="small replicate", kind="run", model="bimolecular", X=16, Y=16, Z=16, slots=8, bytes=1,
             density=0.06, species=3, records=1, steps=32, tune=True),
        # The plain drop-in run: A + B <-> C on 32^3, a record every 128 timesteps.
        dict(name="plain 32^3", kind="run", model="bimolecular", X=32, Y=32, Z=32, slots=8, bytes=1, density=0.061,
             species=3, records=2, steps=128, tune=True),
        # The rod cell as the solver classes run it: default schedule, a record every 64 timesteps.
        dict(name="rod cell records", kind="run", model="rod", X=64, Y=64, Z=128, slots=8, bytes=1, density=0.0103,
             species=5, records=3, steps=64, tune=False),
        # The rod cell as one solve through host buffers, autotuned.
        dict(name="rod cell solve", kind="solve", model="rod", X=64, Y=64, Z=128, slots=8, bytes=1, density=0.0103,
             species=5, records=1, steps=256, tune=True),
        # The crowded cell at full size: IntLattice of 16 slots, 1M particles, 200 species, 500 reactions.
        dict(name="crowded cell", kind="run", model="crowded", X=128, Y=128, Z=256, slots=16, bytes=4, density=0.238,
             species=200, records=1, steps=16, tune=True),
        # A large serving-sized solve: about 1.25 particles on every site.
        dict(name="dense 96^3", kind="run", model="dense", X=96, Y=96, Z=96, slots=8, bytes=1, density=1.25, species=26,
             records=1, steps=32, tune=True),
        # Ragged edges, ByteLattice of 16 slots, two particles per site.
        dict(name="ragged byte-16", kind="run", model="dense", X=100, Y=60, Z=72, slots=16, bytes=1, density=2.0,
             species=40, records=1, steps=32, tune=True),
        # An IntLattice of 8 slots with obstacles, rows no multiple of 16, default schedule.
        dict(name="obstacles int-8", kind="run", model="crowded", X=72, Y=40, Z=88, slots=8, bytes=4, density=0.4,
             species=60, records=2, steps=24, tune=False),
        # An ensemble of replicates of uneven size advanced together.
        dict(name="mixed ensemble", kind="batch", model="bimolecular", replicates=40, steps=32),
        # Continuous batching: requests of mixed size, density and length served to the end.
        dict(name="served requests", kind="serve", model="dense", requests=6, edge_min=16, edge_max=64, steps=96),
        # Gene-expression ensemble, every replicate's records collected on the host.
        dict(name="gene ensemble", kind="cme", model="gene", replicates=16384, t_end=600.0, interval=60.0),
        # Frames in and out in the .lm file's row-major order, with a species count.
        dict(name="row-major frames", kind="frames", model="dense", X=64, Y=64, Z=128, slots=8, bytes=1, density=0.5,
             species=30),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    pick = rng.random()
    if pick < 0.12:
        return dict(kind="batch", model="bimolecular", replicates=log_int(4, 40), steps=rng.randint(8, 32))
    if pick < 0.22:
        return dict(kind="serve", model="dense", requests=rng.randint(2, 6), edge_min=16,
                    edge_max=rng.choice([24, 32, 48, 64]), steps=log_int(24, 96))
    if pick < 0.32:
        return dict(kind="cme", model="gene", replicates=log_int(100, 16384), t_end=float(log_int(60, 600)),
                    interval=float(rng.choice([10, 30, 60])))
    slots, width = rng.choice([(4, 1), (8, 1), (8, 1), (8, 1), (16, 1), (16, 1), (32, 1), (4, 4), (8, 4), (16, 4),
                               (16, 4)])
    X, Y, Z = (log_int(9, 128) for _ in range(3))
    if rng.random() < 0.5:
        X = max(32, (X + 31) // 32 * 32)
    if pick < 0.42:
        return dict(kind="frames", model="dense", X=X, Y=Y, Z=Z, slots=slots, bytes=width,
                    density=0.01 * (slots * 10) ** rng.random(), species=rng.randint(2, 60))
    model = rng.choice(["bimolecular", "rod", "crowded", "dense", "dense"])
    # Mean particles per site, up to an eighth of the slots (fuller lattices overflow their queue).
    density = {"bimolecular": 0.06, "rod": 0.01}.get(model) or 0.05 * (slots * 2.4) ** rng.random()
    case = dict(kind="run" if rng.random() < 0.75 else "solve", model=model, X=X, Y=Y, Z=Z,
                slots=8 if model == "rod" else slots, bytes=1 if model == "rod" else width, density=density,
                species={"bimolecular": 3, "rod": 5}.get(model) or rng.randint(2, 200), records=rng.randint(1, 3),
                tune=rng.random() < 0.6)
    if model == "rod":  # the capsule needs room for its cytoplasm
        case.update(X=max(X, 24), Y=max(Y, 24), Z=max(Z, max(X, Y, 24) + 8))
    # No more site-timesteps than the crowded cell's pass.
    sites = case["X"] * case["Y"] * case["Z"]
    if case["kind"] == "solve":
        case["records"] = 1
    case["steps"] = max(2, min(log_int(4, 96), 16 * 128 * 128 * 256 // (sites * case["records"] * 4)))
    return case


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def place(X, Y, Z, slots, width, site_types, onto, count, species, seed):
    """A native lattice (numpy uint32) of `count` particles at random sites of
    type `onto` (any site when None), species drawn evenly, each in the first
    free slot; particles that find their site full are left out."""
    dev = "cuda"
    gen = torch.Generator(device=dev).manual_seed(seed)
    N = X * Y * Z
    where = torch.randint(0, N, (count,), generator=gen, device=dev)
    if onto is not None:
        allowed = torch.nonzero(torch.from_numpy(site_types).to(dev) == onto).reshape(-1)
        where = allowed[where % allowed.numel()]
    where = torch.sort(where)[0]
    at = torch.arange(count, device=dev)
    new = torch.ones(count, dtype=torch.bool, device=dev)
    new[1:] = where[1:] != where[:-1]
    rank = at - torch.cummax(torch.where(new, at, torch.zeros_like(at)), 0)[0]
    kind = torch.randint(1, species + 1, (count,), generator=gen, device=dev)
    ok = rank < slots
    where, rank, kind = where[ok], rank[ok], kind[ok]
    if width == 1:
        lat = torch.zeros(slots * N, dtype=torch.uint8, device=dev)
        lat[((rank // 4) * N + where) * 4 + rank % 4] = kind.to(torch.uint8)
        return lat.cpu().numpy().view(np.uint32)
    lat = torch.zeros(slots * N, dtype=torch.int32, device=dev)
    lat[rank * N + where] = kind.to(torch.int32)
    return lat.cpu().numpy().view(np.uint32)


def conversions(ns, nr, nst, spacing, N, rng, first, second):
    """Reactions that keep the particle number: A -> B at rates `first` and
    A + B -> C + D at rates `second` (log-uniform), each reactant pair once."""
    rtype = np.zeros(nr, dtype=np.uint32)
    K = np.zeros(nr)
    S = np.zeros((ns, nr), dtype=np.int32)
    D = np.zeros((ns, nr), dtype=np.uint32)
    RL = np.zeros((nr, nst), dtype=np.uint32)
    RL[:, 0] = 1
    RL[:, 1:] = rng.random((nr, nst - 1)) < 0.2
    pairs = set()
    for j in range(nr):
        a, b = (int(v) for v in rng.choice(ns, size=2, replace=False))
        if rng.random() < 0.5 and (min(a, b), max(a, b)) not in pairs:
            pairs.add((min(a, b), max(a, b)))
            rtype[j] = configs.SECOND
            K[j] = configs.lm_rate(np.exp(rng.uniform(*np.log(second))), 2, spacing, N)
            S[a, j] -= 1
            S[b, j] -= 1
            D[a, j] = D[b, j] = 1
            for p in rng.choice(ns, size=2):
                S[p, j] += 1
        else:
            rtype[j] = configs.FIRST
            K[j] = np.exp(rng.uniform(*np.log(first)))
            S[a, j] -= 1
            S[b, j] += 1
            D[a, j] = 1
    return rtype, K, S, D, RL


def problem(model, X, Y, Z, slots, width, density, species, seed):
    """A configs.ModelSpec of the named shape."""
    rng = np.random.default_rng(seed)
    N = X * Y * Z
    if model == "rod":
        # The rod cell's chemistry, with its D_ATP and E spread over the cytoplasm at the given density.
        spec = configs.config1(seed=seed, X=X, Y=Y, Z=Z)
        if spec.lattice.size != 2 * N or (X, Y, Z) != (64, 64, 128):
            lat = place(X, Y, Z, slots, width, spec.sites, 1, max(1, int(density * N)), 1, seed)
            spec.lattice = lat
        return spec
    if model == "bimolecular":
        # A + B <-> C, 32 nm, 50 us, D = 1e-12 m^2/s.
        spec = configs.config0(seed=seed, edge=4)
        spec.X, spec.Y, spec.Z, spec.slots, spec.bytes_per_slot = X, Y, Z, slots, width
        spec.K = np.array([configs.lm_rate(1.07e6, 2, spec.spacing, N), configs.lm_rate(0.351, 1, spec.spacing, N)])
        spec.sites = np.zeros(N, dtype=np.uint8)
        spec.lattice = place(X, Y, Z, slots, width, spec.sites, None, max(1, int(density * N)), 2, seed)
        return spec
    if model == "crowded":
        # Free cytoplasm and 7 obstacle classes over 20 % of the volume, 10 nm, 10 us, 2.5 reactions per species.
        spacing, tau, nst = 10e-9, 10e-6, 8
        sites = configs.obstacle_sites(X, Y, Z, 0.20, nst, rng, 2.0, min(6.0, min(X, Y, Z) / 2.0))
        Dsp = np.exp(rng.uniform(np.log(1e-14), np.log(5e-12), size=species))
        DF = np.zeros((nst, nst, species))
        DF[0, 0, :] = Dsp
        for s in range(species):
            t = 1 + s % (nst - 1)
            DF[0, t, s] = DF[t, 0, s] = DF[t, t, s] = Dsp[s] * 0.1
        rx = conversions(species, max(2, (5 * species) // 2), nst, spacing, N, rng, (1e-3, 1e2), (1e5, 1e7))
        lat = place(X, Y, Z, slots, width, sites, 0, max(1, int(density * N)), species, seed)
    else:
        # A serving request: one site type, 32 nm, 50 us, about one reaction per species.
        spacing, tau, nst = 32e-9, 50e-6, 1
        sites = np.zeros(N, dtype=np.uint8)
        DF = np.exp(rng.uniform(np.log(1e-14), np.log(5e-12), size=species)).reshape(1, 1, species)
        rx = conversions(species, species, nst, spacing, N, rng, (0.1, 10.0), (1e5, 1e7))
        lat = place(X, Y, Z, slots, width, sites, None, max(1, int(density * N)), species, seed)
    return configs.ModelSpec("%s-%dx%dx%d" % (model, X, Y, Z), X, Y, Z, slots, width, species, nst, tau, spacing,
                             rx[0], rx[1], rx[2], rx[3], DF, rx[4], lat, sites)


def of_case(case, seed):
    return problem(case["model"], case["X"], case["Y"], case["Z"], case["slots"], case["bytes"], case["density"],
                   case["species"], seed)


class DeviceWords:
    """A lattice's current particle buffer, for torch to look at in place; it
    keeps the lattice for as long as a tensor looks at it."""

    def __init__(self, lattice):
        self.lattice = lattice
        ptr, _ = lattice.device_buffers()
        self.__cuda_array_interface__ = dict(shape=(lattice.words * lattice.nsites,), typestr="<i4",
                                             data=(ptr, False), version=2)


def words_of(lattice):
    return torch.as_tensor(DeviceWords(lattice), device="cuda")


def batch_members(case, seed):
    edges = configs.batch_edges(count=case["replicates"])
    return [problem("bimolecular", e, e, e, 8, 1, 0.061, 3, seed * 1009 + j) for j, e in enumerate(edges)]


def serve_members(case, seed):
    # The mix of sizes belongs to the case, the models and particles to the seed.
    rng = np.random.default_rng(case["requests"] * 1000 + case["edge_max"])
    out = []
    for k in range(case["requests"]):
        # The first request is the largest, the others are spread over the range.
        e = case["edge_max"] if k == 0 else int(rng.integers(case["edge_min"], case["edge_max"] + 1))
        out.append((problem("dense", e, e, e, 8, 1, float(rng.uniform(0.5, 2.0)), int(rng.integers(2, 51)),
                            seed * 1009 + k), max(1, case["steps"] - 7 * k)))
    return out


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case, ctx=Context(0), seed=seed & 0x7FFFFFFF)
    ctx = state["ctx"]
    if kind in ("run", "solve", "frames"):
        spec = of_case(case, seed)
        lat = Lattice(ctx, spec.X, spec.Y, spec.Z, spec.slots, spec.bytes_per_slot)
        state.update(lattice=lat, t=0, ns=spec.ns, nst=spec.nst)
        if kind == "frames":
            lat.set_native(spec.lattice, spec.sites)
            state["particles"], state["sites"] = lat.get_row_major()
            return state
        state["model"] = Model.from_spec(ctx, spec)
        lat.set_native(spec.lattice, spec.sites)
        if case["tune"]:
            lat.autotune(state["model"], state["seed"], 0, 16)
        if kind == "solve":
            pin = [torch.from_numpy(a.copy()).pin_memory() for a in (spec.lattice.view(np.int32), spec.sites)]
            state.update(words_in=pin[0], sites_in=pin[1], words_out=torch.empty_like(pin[0]).pin_memory())
        return state
    if kind == "batch":
        specs = batch_members(case, seed)
        state["lattices"] = []
        state["models"] = [Model.from_spec(ctx, s) for s in specs]
        for s in specs:
            lat = Lattice(ctx, s.X, s.Y, s.Z, s.slots, s.bytes_per_slot)
            lat.set_native(s.lattice, s.sites)
            state["lattices"].append(lat)
        state["batch"] = Batch(ctx, state["lattices"], state["models"])
        state["seeds"] = [(state["seed"] + 77 * j) & 0x7FFFFFFF for j in range(len(specs))]
        state["t"] = 0
        return state
    if kind == "serve":
        state["requests"] = serve_members(case, seed)
        state["server"] = Server(ctx, hbm_budget_bytes=16 << 30, max_active=16, chunk_timesteps=32)
        return state
    state["ensemble"] = CMEEnsemble(ctx, configs.two_state_gene(), case["replicates"])
    return state


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------

def run(state):
    case, seed = state["case"], state["seed"]
    kind = case["kind"]
    if kind == "run":
        # The next stretch of the trajectory: timesteps and a record of the species counts, `records` times.
        lat, out = state["lattice"], []
        for _ in range(case["records"]):
            _, st, counts = lat.run_counts(state["model"], seed, state["t"], case["steps"], state["ns"])
            state["t"] += case["steps"]
            out += [counts, np.array([st.reactions, st.overflows], dtype=np.uint64)]
        return out + [words_of(lat)]
    if kind == "solve":
        lat = state["lattice"]
        lat.run_native_async(state["model"], seed, 0, case["steps"], state["words_in"].data_ptr(),
                             state["sites_in"].data_ptr(), state["words_out"].data_ptr())
        _, st = lat.wait()
        return [state["words_out"], np.array([st.reactions, st.overflows], dtype=np.uint64)]
    if kind == "batch":
        _, stats = state["batch"].run(state["seeds"], state["t"], case["steps"])
        state["t"] += case["steps"]
        return [np.array([[s.reactions, s.overflows] for s in stats], dtype=np.uint64),
                torch.cat([words_of(lat) for lat in state["lattices"]])]
    if kind == "serve":
        server, done = state["server"], {}
        for k, (spec, steps) in enumerate(state["requests"]):
            server.submit(k, spec, (seed + 31 * k) & 0x7FFFFFFF, steps)
        while len(done) < len(state["requests"]):
            server.step()
            while True:
                got = server.pop_result()
                if got is None:
                    break
                info, words, counts = got
                done[int(info.id)] = [np.array([info.stats.status, info.stats.steps_done], dtype=np.int64), counts,
                                      words]
        return [done[k] for k in sorted(done)]
    if kind == "cme":
        ens = state["ensemble"]
        ens.run(seed, case["t_end"], case["interval"])
        events, finished = ens.stats()
        return [ens.counts(), np.array([events, finished], dtype=np.uint64)]
    lat = state["lattice"]
    lat.set_row_major(state["particles"], state["sites"], state["ns"], state["nst"])
    counts = lat.species_counts(state["ns"])
    particles, sites = lat.get_row_major()
    return [counts, particles, sites]


# ---------------------------------------------------------------------------
# What a pass needs, and what it has to give
# ---------------------------------------------------------------------------

def work(case):
    """Per timestep: the particles and site types read once and the particles
    written once (the lattice is larger than a kernel keeps on chip), and for
    each particle three hop draws and one reaction draw of about 24
    operations each.  A pass that goes through host or row-major buffers also
    reads and writes each of those once."""
    kind = case["kind"]
    if kind == "cme":
        records = case["replicates"] * 4 * 4 * (1 + int(case["t_end"] / case["interval"]))
        # About 17 events per second of model time and replicate, about 60 operations an event.
        return {"bytes": 2 * records, "flops": case["replicates"] * case["t_end"] * 17 * 60}
    if kind == "batch":
        sites = case["replicates"] * (16 ** 3 + 24 ** 3 + 32 ** 3 + 48 ** 3 + 64 ** 3) / 5
        particles, width, steps, extra = 0.061 * sites, 1, case["steps"], 0
    elif kind == "serve":
        sites = case["edge_max"] ** 3 + (case["requests"] - 1) * ((case["edge_min"] + case["edge_max"]) / 2) ** 3
        particles, width, steps, extra = 1.25 * sites, 1, case["steps"] - 3 * case["requests"], 2 * 9 * sites
    else:
        sites = case["X"] * case["Y"] * case["Z"]
        particles, width = case["density"] * sites, case["bytes"]
        steps = case.get("steps", 0) * case.get("records", 1)
        extra = 0 if kind == "run" else (2 * case["slots"] * width + 1) * sites
        if kind == "frames":
            return {"bytes": 2 * extra, "flops": 0}
    return {"bytes": max(1, steps) * (2 * particles * width + sites) + extra, "flops": steps * particles * 4 * 24}


def tolerance(case):
    return "exact"


def exact(case, seed):
    """Frames come back as they were set, packed; every other output is the
    end of a chain of seeded whole-number steps with no 64-bit form."""
    if case["kind"] != "frames":
        return None
    spec = of_case(case, seed)
    X, Y, Z, S = spec.X, spec.Y, spec.Z, spec.slots
    if spec.bytes_per_slot == 1:
        flat = spec.lattice.view(np.uint8).reshape(S // 4, Z, Y, X, 4)
        particles = np.ascontiguousarray(flat.transpose(3, 2, 1, 0, 4)).reshape(X, Y, Z, S)
    else:
        particles = np.ascontiguousarray(spec.lattice.reshape(S, Z, Y, X).transpose(3, 2, 1, 0))
    counts = np.bincount(particles.reshape(-1), minlength=spec.ns + 1)[: spec.ns + 1].astype(np.uint64)
    counts[0] = 0
    return [counts, particles, np.ascontiguousarray(spec.sites.reshape(Z, Y, X).transpose(2, 1, 0))]
