"""The work a user of this framework has it do, as timed cases.

Each case is one call sequence of a user's program through the public
binding (spatial_cell_gb300.native), at a size such programs run:

* ``steps``     a resident simulation advanced by some steps, then its frame
                (the frames.dat payload) taken to the host: the main loop of
                every program, from the smallest cell the request loop admits
                to the large periodic box;
* ``batch``     many replica cells of different sizes stepped as one sim;
* ``vesicle``   the crowded lipid vesicle with reflecting walls;
* ``request``   a new request served from nothing: sim, scene, preparation,
                horizon, last frame;
* ``roundtrip`` a reference-layout state taken from host records through
                preparation and steps back to host records, with every rule
                kind of the engine;
* ``analysis``  FP64 observables and a pair histogram of a loaded frame;
* ``sort``      the allocation-free cell sort on a caller's device buffers.

A case is a dict of plain values.  Densities are the measured workloads'
(particles 0.0082 per nm^3; metabolic items 2 to 5 per particle).
"""
import ctypes
import math

import numpy as np
import torch

from spatial_cell_gb300 import abi, native, scenes

KINDS = (scenes.LIPID, scenes.DUMMY, scenes.TYPE_A, scenes.TYPE_B)
DENSITY = 65536 / 200.0 ** 3  # particles per nm^3 of the measured workloads
CELL, REACH, SPREAD = 6.0, 5.5, 6.0  # nm: grid cell, interaction distance, diffusion distance
COORD, RELAX, DIFFUSE = 16, 32, 8  # sub-iterations of a step (the reference's config.json)


def listed():
    return [
        # The smallest cell the request loop admits, watched live: ten steps, its frame, and the caller waits for it.
        dict(name="steps_smallest", kind="steps", n=4096, nm=8192, species=8, lipids=0.4, pairs=1, steps=10, wait=True),
        # The small workload (200 nm box), frames streamed while it runs on.
        dict(name="steps_small", kind="steps", n=65536, nm=131072, species=8, lipids=0.4, pairs=1, steps=10, wait=False),
        # A mid-size request, lipid-rich, sizes that fill no tile or warp evenly, few species, watched live.
        dict(name="steps_ragged", kind="steps", n=250007, nm=500009, species=4, lipids=0.7, pairs=1, steps=5, wait=True),
        # The large workload: 2 M particles and 8 M metabolic items in a 635 nm periodic box.
        dict(name="steps_large", kind="steps", n=2097152, nm=8388608, species=8, lipids=0.4, pairs=1, steps=4, wait=False),
        # A dense metabolic gas in the memory-lean form of its pair pool, every species simulated.
        dict(name="steps_lean", kind="steps", n=196613, nm=983041, species=10, lipids=0.4, pairs=0, steps=5, wait=False),
        # Replica cells from a few thousand to 262 k particles stepped as one sim.
        dict(name="batch", kind="batch", replicas=24, lo=2048, hi=262144, steps=2),
        # The crowded vesicle at 1/16 of its full size: membrane, chain-bonded complexes, gas crowding the walls.
        dict(name="vesicle", kind="vesicle", scale=0.0625, steps=2),
        # A request's whole life: admission, device-generated scene, twenty steps, last frame, retirement.
        dict(name="request", kind="request", n=30011, steps=20),
        # A saved state with chains, transitions and polymerisation resumed for two steps and saved again.
        dict(name="roundtrip", kind="roundtrip", n=20003, nm=40009, steps=2),
        # Mean squared displacement, totals and g(r) of a frame of a trajectory.
        dict(name="analysis", kind="analysis", n=131072, nm=262144, bins=128),
        # A framework that owns the GPU's memory sorting its items into cells, at the entry's largest size.
        dict(name="sort_cells", kind="sort", n=262144, box=320.0, periodic=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "batch", "vesicle", "request", "roundtrip", "analysis", "sort"])
    if kind == "steps":
        n = _log(rng, 4096, 1500000)
        nm = int(n * rng.uniform(2.0, 4.0))
        pairs = rng.choice([1, 1, 0])
        return dict(kind=kind, n=n, nm=nm, species=rng.choice([1, 3, 4, 5, 8, 9, 10]), lipids=round(rng.uniform(0.1, 0.8), 3),
                    pairs=pairs, steps=max(1, min(10, 2000000 // (n + nm))), wait=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, replicas=rng.randint(2, 24), lo=2048, hi=_log(rng, 16384, 262144), steps=rng.randint(1, 2))
    if kind == "vesicle":
        return dict(kind=kind, scale=round(math.exp(rng.uniform(math.log(0.004), math.log(0.0625))), 5), steps=rng.randint(1, 2))
    if kind == "request":
        return dict(kind=kind, n=_log(rng, 4096, 262144), steps=rng.randint(10, 20))
    if kind == "roundtrip":
        n = _log(rng, 1000, 60000)
        return dict(kind=kind, n=n, nm=int(n * rng.uniform(1.0, 3.0)), steps=rng.randint(1, 2))
    if kind == "analysis":
        n = _log(rng, 8192, 200000)
        return dict(kind=kind, n=n, nm=2 * n + rng.randint(0, 999), bins=rng.choice([50, 64, 100, 128]))
    n = _log(rng, 1024, 262144)
    return dict(kind="sort", n=n, box=round((n / DENSITY) ** (1.0 / 3.0) + 20.0, 3), periodic=rng.choice([0, 1]))


def _mix(lipids):
    rest = 1.0 - lipids
    return (lipids, rest * 2 / 3, rest / 6, rest / 6)


class _Frames:
    """A pinned host frame the sim's frames land in, and its fields."""

    def __init__(self, n, nm):
        self.p = torch.empty(n * abi.REDUCED_DTYPE.itemsize, dtype=torch.uint8, pin_memory=True)
        self.m = torch.empty(nm * abi.REDUCED_METABOLIC_DTYPE.itemsize, dtype=torch.uint8, pin_memory=True)

    def take(self, sim, wait):
        t = sim.reduce_frame_async_ptr(ctypes.c_void_p(self.p.data_ptr()), ctypes.c_void_p(self.m.data_ptr()))
        if wait:
            sim.frame_wait(t)

    def fields(self):
        out = {}
        for name, buf, size in (("particles", self.p, abi.REDUCED_DTYPE.itemsize),
                                ("metabolic", self.m, abi.REDUCED_METABOLIC_DTYPE.itemsize)):
            out[name + "_words"] = buf.view(torch.int32).view(-1, size // 4)[:, :3]  # id, type, flags and state
            out[name + "_values"] = buf.view(torch.float16).view(-1, size // 2)[:, 6:]
        return out


def _analysis_inputs(case, seed):
    """Two frames of a small trajectory as arrays: the first's positions, and the second's records' values."""
    rng = np.random.default_rng(seed)
    box = float((case["n"] / DENSITY) ** (1.0 / 3.0))
    out = {"box": np.float32(box)}
    for name, n in (("p", case["n"]), ("m", case["nm"])):
        a = (rng.random((n, 3)) * box).astype(np.float32)
        b = a + rng.normal(0.0, 2.0, (n, 3)).astype(np.float32)
        b = np.where(b < 0, b + np.float32(box), np.where(b >= np.float32(box), b - np.float32(box), b)).astype(np.float32)
        b = np.minimum(b, np.nextafter(np.float32(box), np.float32(0)))
        out[name] = dict(first=a, pos=b, vel=rng.normal(0.0, 0.5, (n, 3)).astype(np.float32),
                         active=rng.random(n) < 0.9)
    out["type"] = rng.choice(np.array(KINDS, np.int32), case["n"], p=_mix(0.4))
    out["met"] = (rng.random((case["nm"], 8)) * 10.0).astype(np.float32)
    return out


def _sort_inputs(case, seed):
    rng = np.random.default_rng(seed)
    n = case["n"]
    pos = np.empty((n, 4), np.float32)
    pos[:, :3] = np.minimum((rng.random((n, 3)) * case["box"]).astype(np.float32),
                            np.nextafter(np.float32(case["box"]), np.float32(0)))
    pos[:, 3] = 2.5
    info = np.zeros((n, 4), np.int32)
    info[:, 0] = np.arange(n)
    info[:, 2] = rng.random(n) < 0.95
    return pos, info


def prepare(case, seed):
    kind = case["kind"]
    types = scenes.baseline_types()
    if kind == "steps":
        n, nm = case["n"], case["nm"]
        box = (n / DENSITY) ** (1.0 / 3.0)
        cfg = abi.make_config(num_particles=n, num_metabolic_particles=nm, sim_size=box, grid_cell_size=CELL,
                              max_interaction_distance=REACH, max_diffusion_distance=SPREAD,
                              num_metabolites=case["species"], seed=seed, periodic=1, metabolic_pairs=case["pairs"],
                              **scenes.WORKLOAD_EXTENSIONS)
        sim = native.Simulation(cfg, types, scenes.workload_rules())
        sim.generate_uniform(n, nm, KINDS, _mix(case["lipids"]), seed)
        sim.prepare()
        return dict(kind=kind, sim=sim, steps=case["steps"], wait=case["wait"], frames=_Frames(n, nm))
    if kind == "batch":
        specs = scenes.batch_specs(case["replicas"], seed=seed, n_lo=case["lo"], n_hi=case["hi"])
        # the sizes are the case's, the seeds and mixes the seed's
        sizes = [s[:3] for s in scenes.batch_specs(case["replicas"], seed=3, n_lo=case["lo"], n_hi=case["hi"])]
        specs = [(*a, *b[3:]) for a, b in zip(sizes, specs)]
        cfg, reps = scenes.batch_sim_args(specs)
        sim = native.Simulation(cfg, types, scenes.workload_rules(), replicas=reps)
        sim.generate_batch([s[0] for s in specs], [s[1] for s in specs], KINDS, [s[3] for s in specs],
                           [s[4] for s in specs])
        sim.prepare()
        return dict(kind="steps", sim=sim, steps=case["steps"], wait=False,
                    frames=_Frames(sim.cfg.num_particles, sim.cfg.num_metabolic_particles))
    if kind == "vesicle":
        cfg, groups, nm = scenes.vesicle_workload(case["scale"], seed=seed)
        sim = native.Simulation(cfg, types, scenes.workload_rules())
        sim.generate_scene(groups, nm, seed)
        sim.prepare()
        return dict(kind="steps", sim=sim, steps=case["steps"], wait=False,
                    frames=_Frames(cfg.num_particles, cfg.num_metabolic_particles))
    if kind == "request":
        n, nm = case["n"], 2 * case["n"]
        cfg = scenes.measured_config("plain_small", num_particles=n, num_metabolic_particles=nm,
                                     sim_size=float((n / DENSITY) ** (1.0 / 3.0)), seed=seed)
        return dict(kind=kind, cfg=cfg, types=types, rules=scenes.workload_rules(), n=n, nm=nm, seed=seed,
                    steps=case["steps"], frames=_Frames(n, nm))
    if kind == "roundtrip":
        box = float(48.0 * (case["n"] / 1500.0) ** (1.0 / 3.0))
        cfg, types, rules, p, m, nid = scenes.test_scene(seed, n=case["n"], nm=case["nm"], box=box, walls=1)
        cfg.noise_coordination_steps, cfg.relaxation_steps, cfg.metabolite_diffusion_steps = COORD, RELAX, DIFFUSE
        return dict(kind=kind, sim=native.Simulation(cfg, types, rules), p=p, m=m, nid=nid, steps=case["steps"])
    if kind == "analysis":
        x = _analysis_inputs(case, seed)
        cfg = scenes.measured_config("plain_small", num_particles=case["n"], num_metabolic_particles=case["nm"],
                                     sim_size=float(x["box"]), seed=seed)
        sim = native.Simulation(cfg, types, scenes.workload_rules())
        recs = []
        for name, n, dtype in (("p", case["n"], abi.PARTICLE_DTYPE), ("m", case["nm"], abi.METABOLIC_DTYPE)):
            r = scenes.blank_particles(n, dtype)
            r["id"] = np.arange(n)
            r["type"] = x["type"] if name == "p" else scenes.METABOLIC
            r["radius"] = types["radius"][r["type"]]
            r["hydrophobic"] = types["hydrophobic"][r["type"]]
            r["flags"] = x[name]["active"]
            r["velocity"] = x[name]["vel"]
            r["pos"] = x[name]["first"]
            recs.append(r)
        recs[1]["metabolites"][:, :8] = x["met"]
        sim.load_state(recs[0], recs[1])
        sim.mark_positions()
        for r, name in zip(recs, ("p", "m")):
            r["pos"] = x[name]["pos"]
        sim.load_state(recs[0], recs[1])
        return dict(kind=kind, sim=sim, bins=case["bins"])
    pos, info = _sort_inputs(case, seed)
    cfg = abi.make_config(sim_size=case["box"], grid_cell_size=CELL, max_interaction_distance=REACH,
                          max_diffusion_distance=SPREAD, periodic=case["periodic"])
    cells = abi.grid_dims(cfg)[2]
    return dict(kind=kind, cfg=cfg, n=case["n"], pos=torch.from_numpy(pos).cuda(), info=torch.from_numpy(info).cuda(),
                perm=torch.zeros(case["n"], dtype=torch.int32, device="cuda"),
                starts=torch.zeros(cells + 1, dtype=torch.int32, device="cuda"))


def run(state):
    kind = state["kind"]
    if kind == "steps":
        sim = state["sim"]
        sim.step(state["steps"])
        state["frames"].take(sim, state["wait"])
        return state["frames"].fields()
    if kind == "request":
        with native.Simulation(state["cfg"], state["types"], state["rules"]) as sim:
            sim.generate_uniform(state["n"], state["nm"], KINDS, (0.4, 0.4, 0.1, 0.1), state["seed"])
            sim.prepare()
            sim.step(state["steps"])
            state["frames"].take(sim, True)
        return state["frames"].fields()
    if kind == "roundtrip":
        sim = state["sim"]
        sim.load_state(state["p"], state["m"], step=0, next_particle_id=state["nid"])
        sim.prepare()
        sim.step(state["steps"])
        p, m = sim.export_state()
        return {"p": {k: p[k] for k in p.dtype.names}, "m": {k: m[k] for k in m.dtype.names}}
    if kind == "analysis":
        sim = state["sim"]
        out = {k: np.asarray(v) for k, v in sim.observe().items()}
        out["all_pairs"] = sim.pair_histogram(-1, -1, REACH, state["bins"]).view(np.int64)
        out["a_b_pairs"] = sim.pair_histogram(scenes.TYPE_A, scenes.TYPE_B, REACH, state["bins"]).view(np.int64)
        return out
    stream = torch.cuda.current_stream().cuda_stream
    rc = native.lib().sc_sort_cells_static(
        ctypes.byref(state["cfg"]), ctypes.c_void_p(state["pos"].data_ptr()), ctypes.c_void_p(state["info"].data_ptr()),
        state["n"], ctypes.c_void_p(state["perm"].data_ptr()), ctypes.c_void_p(state["starts"].data_ptr()),
        ctypes.c_void_p(stream))
    if rc:
        raise native.ScError(f"sc_sort_cells_static failed ({rc})")
    return {"perm": state["perm"], "starts": state["starts"]}


# Per-item state of the step's layout: position, velocity, orientation, angular velocity, both noises, debug vector and
# record (16 bytes each), state words, bonds.
_STATE_P = 8 * 16 + 16 + 24 * 4
_FRAME_P, _FRAME_M = 36, 44


def _step_work(n, nm, species, volume, steps, lipids):
    """State in and out once per step, the frame out once; flops: the pair terms of every sub-iteration that acts on
    pairs (20 a pair), at the densities' mean pair counts (metabolic items not displaced by lipids)."""
    state_m = 8 * 16 + 8 + 4 * species
    nbytes = steps * 2 * (n * _STATE_P + nm * state_m) + n * _FRAME_P + nm * _FRAME_M
    sphere = lambda r: 4.0 / 3.0 * math.pi * r ** 3  # noqa: E731
    free = nm * math.exp(-lipids * n / volume * sphere(3.5))
    rho_p, rho_m = n / volume, free / volume
    pairs = RELAX * n * rho_p * sphere(4.0) + RELAX / 2 * free * (rho_m + lipids * rho_p) * sphere(REACH) \
        + RELAX / 2 * lipids * n * rho_m * sphere(REACH)
    exchanges = DIFFUSE * free * rho_m * sphere(SPREAD) * 3 * species
    return {"bytes": nbytes, "flops": steps * (20.0 * pairs + exchanges)}


def work(case):
    kind = case["kind"]
    if kind == "steps":
        return _step_work(case["n"], case["nm"], case["species"], case["n"] / DENSITY, case["steps"], case["lipids"])
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for s in scenes.batch_specs(case["replicas"], seed=3, n_lo=case["lo"], n_hi=case["hi"]):
            w = _step_work(s[0], s[1], 8, s[2] ** 3, case["steps"], 1.0 / 3.0)
            total = {k: total[k] + w[k] for k in total}
        return total
    if kind == "vesicle":
        cfg, groups, nm = scenes.vesicle_workload(case["scale"])
        return _step_work(cfg.num_particles, nm, 8, cfg.sim_size ** 3, case["steps"], 0.2)
    if kind == "request":
        return _step_work(case["n"], 2 * case["n"], 8, case["n"] / DENSITY, case["steps"], 0.4)
    if kind == "roundtrip":
        w = _step_work(case["n"], case["nm"], 10, 48.0 ** 3 * case["n"] / 1500.0, case["steps"], 0.35)
        return {"bytes": w["bytes"] + 2 * (case["n"] * 256 + case["nm"] * 304), "flops": w["flops"]}
    if kind == "analysis":
        n, nm = case["n"], case["nm"]
        pairs = 2 * n * DENSITY * 4.0 / 3.0 * math.pi * REACH ** 3
        return {"bytes": n * (4 * 16 + 4) + nm * (4 * 16 + 32) + 2 * n * 32, "flops": 20.0 * pairs + 30.0 * (n + nm)}
    cells = abi.grid_dims(abi.make_config(sim_size=case["box"], grid_cell_size=CELL))[2]
    return {"bytes": case["n"] * (16 + 16 + 4) + 4 * (cells + 1), "flops": 0}


def _pair_counts(pos, keep_a, keep_b, box, r_max, bins):
    """Histogram of the distances below r_max of ordered pairs (a, b), a in keep_a, b in keep_b, in a periodic box."""
    pos = pos.astype(np.float64)
    n = max(1, int(box // r_max))
    cell = np.minimum((pos / (box / n)).astype(np.int64), n - 1)
    key = (cell[:, 0] * n + cell[:, 1]) * n + cell[:, 2]
    order = np.argsort(key, kind="stable")
    start = np.searchsorted(key[order], np.arange(n ** 3 + 1))
    counts = np.zeros(bins, np.int64)
    a = np.nonzero(keep_a)[0]
    around = {tuple((np.array(o) % n).tolist()): o for o in np.ndindex(3, 3, 3)} if n < 3 else None
    for o in np.ndindex(3, 3, 3) if around is None else around.values():
        c = (cell[a] + np.array(o) - 1) % n
        k = (c[:, 0] * n + c[:, 1]) * n + c[:, 2]
        lo, num = start[k], start[k + 1] - start[k]
        i = np.repeat(a, num)
        j = order[np.repeat(lo - np.concatenate([[0], np.cumsum(num)[:-1]]), num) + np.arange(num.sum())]
        use = (i != j) & keep_b[j]
        d = pos[j[use]] - pos[i[use]]
        d -= box * np.round(d / box)
        r = np.sqrt((d * d).sum(1))
        b = (r[r < r_max] * bins / r_max).astype(np.int64)
        counts += np.bincount(b[b < bins], minlength=bins)
    return counts


def exact(case, seed):
    """What run() returns where plain arithmetic gives it: the analysis of a frame, and the sorted order.  A step's
    result has no such value (its noise, rules and neighbour order are the framework's own)."""
    if case["kind"] == "analysis":
        x = _analysis_inputs(case, seed)
        box = float(x["box"])
        sets = [x["p"], x["m"]]
        act = [s["active"] for s in sets]
        msd, v2 = [], []
        for s, k in zip(sets, act):
            d = s["pos"][k].astype(np.float64) - s["first"][k].astype(np.float64)
            d -= box * np.round(d / box)
            msd.append((d * d).sum(1).mean())
            v2.append((s["vel"][k].astype(np.float64) ** 2).sum(1).mean())
        n_act = np.array([int(k.sum()) for k in act], np.int64)
        met = np.zeros(10)
        met[:8] = x["met"][act[1]].astype(np.float64).sum(0)
        kinds = x["type"]
        pairs = lambda a, b: _pair_counts(x["p"]["pos"], act[0] & a, act[0] & b, box, REACH, case["bins"])  # noqa: E731
        every = np.ones(case["n"], bool)
        return {"msd": np.array(msd), "msd_items": n_act, "mean_v2": np.array(v2), "active": n_act,
                "bond_slots": np.asarray(0), "metabolites": met, "all_pairs": pairs(every, every),
                "a_b_pairs": pairs(kinds == scenes.TYPE_A, kinds == scenes.TYPE_B)}
    if case["kind"] == "sort":
        pos, info = _sort_inputs(case, seed)
        box, size = np.float32(case["box"]), np.float32(CELL)
        axis = max(2, 1 << max(0, math.ceil(math.log2(math.ceil(case["box"] / CELL)))))
        used = int(box // size) if case["periodic"] else axis
        width = box / np.float32(used) if case["periodic"] else size
        g = np.minimum((pos[:, :3] / width).astype(np.int64), used - 1)
        key = np.where(info[:, 2] & 1, (g[:, 0] * axis + g[:, 1]) * axis + g[:, 2], 1 << 40)
        perm = np.argsort(key, kind="stable")
        return {"perm": perm.astype(np.int32), "starts": np.searchsorted(key[perm], np.arange(axis ** 3 + 1)).astype(np.int32)}
    return None
