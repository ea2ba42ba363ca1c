"""The calls whose speed this framework is judged by: the work a program has it do, through its
public entry points (`Simulation`, `Ensemble` and the device-buffer form of `cs_render_view`).

Every output is a whole number or a view value k / 255 that is written exactly, so two versions of
the framework agree bit for bit or not at all; no output has a 64-bit counterpart to compare with.

A case is a dict:

  family     "plane"      the 64 x 64 x 1 three-species model (A + B <-> C, K = 8), or its like
             "cell"       a spherical cell: membrane shell, cytoplasm, outside (8 species, K = 16)
             "multi"      nested nucleus, cytoplasm, membrane and outside (16 species, K = 16)
             "stiff"      one region, 12 species, rates over seven decades (K = 16)
             "tissue"     one region, three species, crowded (K = 8)
             "ensemble"   replicates of the three-species model with edges lo..hi (K = 8)
             "sweep"      replicates of the stiff model with edges lo..hi (K = 16)
  x, y, z    lattice resolution (lattices); replicates, lo, hi (ensembles)
  particles  particles placed (per replicate for ensembles)
  rng        "philox" (production) or "reference" (the reference's own random numbers)
  frames     frames per pass (one step call)
  log        write_freq of the step call (0: no samples)
  tuned      whether the program calls autotune once after preparing, as the integration notes advise
  precision  0 mixed, 1 FP32, 2 FP64 (production only)
  reads      what the program reads after the call: "counts", "view" (counts and the majority-species
             view in device memory), "lattice" (counts and the whole state), "slots" (ensembles)
  uploads    whether the pass starts from a lattice uploaded by the caller
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cell_simulation_gb300 import RNG_PHILOX, RNG_REFERENCE, Ensemble, LatticeParams, Simulation, configs
from cell_simulation_gb300 import native

K_OF = {"plane": 8, "cell": 16, "multi": 16, "stiff": 16, "tissue": 8, "ensemble": 8, "sweep": 16}
SPECIES = {"plane": 3, "cell": 8, "multi": 16, "stiff": 12, "tissue": 3, "ensemble": 3, "sweep": 12}
REACTIONS = {"plane": 2, "cell": 10, "multi": 30, "stiff": 24, "tissue": 2, "ensemble": 2, "sweep": 24}
ENSEMBLES = ("ensemble", "sweep")


def _lattice(name, family, xyz, particles, frames, rng="philox", log=0, tuned=False, reads="counts", uploads=False):
    c = {"family": family, "x": xyz[0], "y": xyz[1], "z": xyz[2], "particles": particles, "rng": rng, "frames": frames,
         "log": log, "tuned": tuned, "precision": 0, "reads": reads, "uploads": uploads}
    return dict(c, name=name) if name else c


def _replicates(name, family, n, lo, hi, particles, frames, tuned=False, precision=0, reads="counts"):
    c = {"family": family, "replicates": n, "lo": lo, "hi": hi, "particles": particles, "rng": "philox",
         "frames": frames, "log": 0, "tuned": tuned, "precision": precision, "reads": reads, "uploads": False}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: one frame of the reference's small example, then the counts and the view
        # that an interactive front end shows after every frame (latency and launches)
        _lattice("plane_frame", "plane", (64, 64, 1), 400, 1, reads="view"),
        # the same model run in earnest: a batch of frames with logged counts, tuned, state read back
        _lattice("plane_run", "plane", (64, 64, 1), 400, 500, log=50, tuned=True, reads="lattice"),
        # the same under the reference's own random numbers (bit-parity runs)
        _lattice("plane_reference", "plane", (64, 64, 1), 400, 100, rng="reference", reads="lattice"),
        # an ordinary single cell in a frame-by-frame loop with counts and view
        _lattice("cell_frame", "cell", (128, 128, 128), 22000, 1, reads="view"),
        # the same cell under the reference's random numbers
        _lattice("cell_reference", "cell", (128, 128, 128), 22000, 20, rng="reference", reads="view"),
        # a lattice of odd edges with several regions, default step, logged counts
        _lattice("multi_ragged", "multi", (61, 97, 45), 16000, 50, log=10, reads="view"),
        # the large multi-region cell, tuned: the framework's headline workload
        _lattice("multi_large", "multi", (256, 256, 256), 1000000, 20, tuned=True, reads="view"),
        # the same cell under the reference's random numbers
        _lattice("multi_large_reference", "multi", (256, 256, 256), 1000000, 10, rng="reference", reads="view"),
        # a stiff network on a large lattice, default step: particles move in most frames
        _lattice("stiff_large", "stiff", (192, 192, 192), 1000000, 20, reads="view"),
        # a crowded lattice handed over by the caller and read back whole (a host that owns the state)
        _lattice("tissue_exchange", "tissue", (48, 40, 37), 120000, 50, reads="lattice", uploads=True),
        # a production ensemble: many uneven replicates, tuned, counts read per batch of frames
        _replicates("ensemble_large", "ensemble", 512, 32, 96, 400, 20, tuned=True),
        # a parameter sweep of small replicates in FP64 selection, whole lattices read back
        _replicates("sweep_small", "sweep", 96, 12, 24, 600, 100, precision=2, reads="slots"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["plane", "cell", "multi", "multi", "stiff", "tissue", "ensemble", "sweep"])
    if family in ENSEMBLES:
        small = family == "sweep"
        lo = rng.randint(10, 16) if small else rng.randint(17, 48)
        hi = lo + (rng.randint(1, 12) if small else rng.randint(8, 48))
        n = _log_int(rng, 8, 128) if small else _log_int(rng, 16, 400)
        return _replicates(None, family, n, lo, hi, rng.randint(100, 800), _log_int(rng, 5, 100 if small else 20),
                           tuned=not small and rng.random() < 0.5, precision=rng.choice([0, 1, 2]),
                           reads="slots" if small else "counts")
    if family == "plane":
        xyz = (_log_int(rng, 20, 110), _log_int(rng, 20, 110), rng.choice([1, 1, 1, 2, 3]))
    elif family == "tissue":
        xyz = tuple(_log_int(rng, 17, 60) for _ in range(3))
    else:
        edge = _log_int(rng, 44, 200)
        xyz = tuple(int(edge * rng.uniform(1.0, 1.25)) for _ in range(3))
    V = xyz[0] * xyz[1] * xyz[2]
    if family == "cell":
        particles = 22000
    else:
        lo, hi = {"plane": (0.03, 0.2), "multi": (0.02, 0.08), "stiff": (0.04, 0.2), "tissue": (0.5, 2.0)}[family]
        particles = int(V * math.exp(rng.uniform(math.log(lo), math.log(hi))))
    most = max(1, min(500 if family == "plane" else 60, int(2.5e8 // V), int(1.5e7 // max(particles, 1))))
    frames = _log_int(rng, 1, most)
    reference = family != "stiff" and rng.random() < 0.3
    if family == "tissue":
        return _lattice(None, family, xyz, particles, frames, reads="lattice", uploads=True)
    return _lattice(None, family, xyz, particles, frames, rng="reference" if reference else "philox",
                    log=rng.choice([0, 0, 10]), tuned=not reference and rng.random() < 0.3,
                    reads="lattice" if family == "plane" and rng.random() < 0.5 else "view")


def _one_region(case, seed, names, counts, reactions):
    """A model on one region (every species diffuses at 1e-12) on a lattice of the case's size."""
    res = (case["x"], case["y"], case["z"])
    D = 1e-12
    sim = Simulation(LatticeParams([r * configs.LAMBDA for r in res], list(res), configs.stable_tau(D), configs.LAMBDA,
                                   K_OF[case["family"]]))
    sim.seed_placement(seed)
    sim.prepare_regions()
    sim.set_diffusion_rate("background", D)
    for name, n in zip(names, counts):
        sim.add_particle_count(name, "background", n, True, False)
    sim.set_diffusion_rate("background", D)
    for reactants, products, k in reactions:
        sim.add_reaction([names[i] for i in reactants], [names[i] for i in products], k)
    return sim


def _simulation(case, seed):
    res = (case["x"], case["y"], case["z"])
    if case["family"] == "cell":
        return configs.c2_single_cell(seed, res=res, r_ext=0.4375 * min(res)).sim
    if case["family"] == "multi":
        return configs.c3_multi_region(seed, res=res, r_nuc=0.15625 * min(res), r_cyt=0.4296875 * min(res),
                                       total_particles=case["particles"]).sim
    if case["family"] == "stiff":
        # the configured network itself: its particle number is steady, so passes stay alike
        names = [f"Q{i}" for i in range(SPECIES["stiff"])]
        return _one_region(case, seed, names, [case["particles"] // len(names)] * len(names), configs.c5_network())
    half = case["particles"] // 2
    return _one_region(case, seed, ["A", "B", "C"], [half, case["particles"] - half, 0],
                       [([0, 1], [2], configs.per_voxel_rate(1e6)), ([2], [0, 1], 0.1)])


def prepare(case, seed):
    state = {"case": case, "seed": int(seed) % (1 << 31) + 1, "frame": 0}
    if case["family"] in ENSEMBLES:
        rng = np.random.default_rng(seed)
        n = case["replicates"]
        # edges spread over lo..hi in a fixed mixed order: the seed changes the replicates' contents and rates
        edges = case["lo"] + np.arange(n) * 7919 % n * (case["hi"] - case["lo"] + 1) // n
        res = np.stack([edges, edges, edges], axis=1).astype(np.uint32)
        seeds = rng.integers(1, 2 ** 63, size=n, dtype=np.uint64)
        mult = np.exp(rng.uniform(math.log(0.5), math.log(2.0), size=n)).astype(np.float32)
        S = SPECIES[case["family"]]
        init = np.zeros(S + 1, np.uint32)
        if case["family"] == "ensemble":
            model = configs.c4_ensemble_template(8)
            init[1:3] = case["particles"] // 2
        else:
            model = configs.c5_ensemble_template()
            init[1:] = case["particles"] // S
        ens = Ensemble(model, res, seeds, mult, init)
        model.close()
        ens.set_precision(case["precision"])
        if case["tuned"]:
            ens.autotune(3)
        state["ens"] = ens
        return state
    sim = _simulation(case, seed)
    if case["uploads"]:
        state["lattice"] = sim.get_lattice()[0]
    sim.prepare_for_gpu(RNG_PHILOX if case["rng"] == "philox" else RNG_REFERENCE, 0)
    if case["tuned"]:
        sim.autotune(10)
    if case["reads"] == "view":
        state["view"] = torch.empty((case["x"], case["y"], case["z"]), dtype=torch.float32, device="cuda")
    state["sim"] = sim
    return state


def run(state):
    case, n = state["case"], state["case"]["frames"]
    if "ens" in state:
        ens = state["ens"]
        ens.step(n)
        out = {"counts": ens.counts()}
        if case["reads"] == "slots":
            out["slots"] = ens.slots()
        return out
    sim = state["sim"]
    if case["uploads"]:
        sim.set_lattice(state["lattice"])
    sim.stats.clear()
    if case["rng"] == "philox":
        sim.step_philox(n, state["seed"], case["log"])
    else:
        # the clock words of these frames (the reference reads the wall clock per frame)
        itimes = (np.arange(state["frame"], state["frame"] + n, dtype=np.uint64) * 7919 + state["seed"]).astype(np.uint32)
        state["frame"] += n
        sim.step(itimes, case["log"])
    out = {"counts": sim.counts(), "log": np.array([s.value for s in sim.stats], np.int32)}
    if case["reads"] == "lattice":
        out["slots"], out["occupancy"], out["concentrations"] = sim.get_lattice()
    elif case["reads"] == "view":
        # the view into the caller's device memory: the C entry point takes the buffer
        native.check(native.load().cs_render_view(sim._h, 0, 0, 0, None, state["view"].data_ptr()))
        out["view"] = state["view"]
    return out


def work(case):
    """What a pass cannot do without.  Bytes: the slots of the occupied voxels read and written once,
    one bit per voxel to know which those are, and the inputs and outputs of the call.  Operations
    (integer and floating point alike), per particle and frame: production, one Philox4x32-10 block (80),
    three move tests (12 each) and the reaction test (14); reference, one PCG and xorshift draw with the
    cumulative move test (60) and, per occupied voxel, every reaction's propensity (6 each)."""
    f = case["family"]
    K, S1 = K_OF[f], SPECIES[f] + 1
    if f in ENSEMBLES:
        n = case["replicates"]
        lo, hi = case["lo"], case["hi"]
        V = n * sum(e ** 3 for e in range(lo, hi + 1)) / (hi - lo + 1)
        particles = n * case["particles"]
        out = 8 * n * S1 + (V * K if case["reads"] == "slots" else 0)
    else:
        V = case["x"] * case["y"] * case["z"]
        particles = case["particles"]
        out = 8 * S1
        if case["reads"] == "view":
            out += 4 * V
        elif case["reads"] == "lattice":
            out += 4 * V * (K + 1 + S1)
        if case["uploads"]:
            out += 4 * V * K
    occupied = min(V, particles)
    ops = particles * 130.0 if case["rng"] == "philox" else particles * 60.0 + occupied * 6.0 * REACTIONS[f]
    return {"bytes": 2.0 * K * occupied + V / 8.0 + out, "flops": case["frames"] * ops}
