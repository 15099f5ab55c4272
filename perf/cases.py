"""What a user's program has the sweep engine do, as cases that can be timed and compared.

A pass is the call a simulation program repeats: advance a system (or a set of systems) by some
Monte Carlo steps and take the positions back, with the move counters or the observables where such
a program reads them. Every output is a whole number, so passes compare bit for bit.

Calls (`call`):
  run     one system: runSimulationOnGPU(mcs), positions into a pinned array, counters (the shape of
          the reference adapter's execute())
  sample  one system: `samples` times runSimulationOnGPU(mcs) and the observables, then the positions
  batch   `members` systems in one Batch: run(mcs), then every member's positions
  serve   `members` jobs of about `mcs` steps each through the job server, observables every `every`
          steps: submit all, wait, take every job's positions and samples

Layouts (`layout`): chains (serpentine_chains of `length` monomers at volume fraction `phi`),
network (the 128^3 six-functional network: 64-bit bond codes), square (four-functional network of
side `lx`), rings (odd rings and free monomers, three colours). `walls` is a bit mask of the axes
that are not periodic.
"""
from __future__ import annotations

import random

import numpy as np
import torch

import pscbfm_b200 as P
from pscbfm_b200 import systems as S

RELAX_MCS = 200        # steps before the first pass: a running simulation is not on its start lattice
LARGEST_MOVES = 1.3e8  # attempted moves of one pass of the largest case


def _case(name, call, layout, l, mcs, length=0, phi=0.0, walls=0, members=1, samples=0, every=0):
    lx, ly, lz = (l, l, l) if isinstance(l, int) else l
    return {"name": name, "call": call, "layout": layout, "lx": lx, "ly": ly, "lz": lz, "length": length,
            "phi": phi, "walls": walls, "mcs": mcs, "members": members, "samples": samples, "every": every}


def listed():
    return [
        # a program that steps a small system and looks at it after every MCS (a viewer, a coupling to
        # another code): launch and read-back latency
        _case("chains64_1mcs", "run", "chains", 64, 1, length=32, phi=0.25),
        # a single small chain system between two frames of a trajectory
        _case("chains32_1000mcs", "run", "chains", 32, 1000, length=16, phi=0.3),
        # the 64^3 chain system of the benchmark, a frame every 1000 MCS
        _case("chains64_1000mcs", "run", "chains", 64, 1000, length=32, phi=0.25),
        # the six-functional network of the benchmark (64-bit bond codes), a frame every 500 MCS
        _case("network128_500mcs", "run", "network", 128, 500),
        # a film between two walls, sides that are no powers of two along the walls, ragged chains
        _case("slit64x64x50_500mcs", "run", "chains", (64, 64, 50), 500, length=37, phi=0.35, walls=4),
        # a mid-size melt sampled as in an equilibration run: observables every 100 MCS
        _case("melt128_sampled", "sample", "chains", 128, 100, length=256, phi=0.5, samples=3),
        # a semi-dilute solution in a large box
        _case("dilute256_100mcs", "run", "chains", 256, 100, length=128, phi=0.1),
        # the 1M-monomer melt of the benchmark, a frame every 100 MCS
        _case("melt256_100mcs", "run", "chains", 256, 100, length=64, phi=0.5),
        # the same melt watched closely: a frame every 10 MCS
        _case("melt256_10mcs", "run", "chains", 256, 10, length=64, phi=0.5),
        # many replicas of a small system, one batch
        _case("replicas32_x128", "batch", "chains", 32, 200, length=32, phi=0.4, members=128),
        # a batch of mixed systems (the benchmark's ensemble draws)
        _case("ensemble_x32", "batch", "mixed", 128, 100, members=32),
        # a burst of jobs through the server
        _case("served_x16", "serve", "mixed", 64, 400, members=16, every=100),
    ]


def _monomers(case):
    return sum(s.n for s in _systems(case))


def draw(rng):
    call = rng.choice(["run"] * 5 + ["sample", "batch", "batch", "serve"])
    while True:
        log = lambda lo, hi: int(round(lo * (hi / lo) ** rng.random()))  # noqa: E731
        length, phi = log(5, 256), round(rng.uniform(0.1, 0.5), 3)
        if call in ("run", "sample"):
            layout = rng.choice(["chains"] * 6 + ["network", "square", "rings"])
            if layout == "network":
                case = _case("", call, layout, 128, log(1, 1000))
            elif layout == "square":
                case = _case("", call, layout, rng.choice([32, 64, 128]), log(1, 1000))
            elif layout == "rings":
                case = _case("", call, layout, rng.choice([32, 64, 128]), log(1, 1000))
            else:
                l = [rng.choice([32, 64, 128, 256]) for _ in range(3)]
                walls = rng.choice([0, 0, 0, 4, 6, 7])
                for a in range(3):
                    if (walls >> a) & 1:
                        l[a] = rng.randint(24, 160)
                case = _case("", call, layout, tuple(l), log(1, 1000), length=length, phi=phi, walls=walls)
            if call == "sample":
                case.update(samples=rng.randint(1, 4), mcs=log(10, 300))
        elif call == "batch":
            members = log(2, 64)
            if rng.random() < 0.5:
                case = _case("", call, "mixed", rng.choice([64, 128]), log(10, 300), members=members)
            else:
                case = _case("", call, "chains", rng.choice([32, 64]), log(10, 300), length=length, phi=phi,
                             members=members)
        else:
            case = _case("", call, "mixed", 64, log(50, 500), members=rng.randint(2, 20),
                         every=rng.choice([50, 100, 200]))
        case.pop("name")
        n, vol = _monomers(case), case["lx"] * case["ly"] * case["lz"]
        if n <= 1_100_000 and vol <= 256 ** 3 and n * case["mcs"] * max(case["samples"], 1) <= LARGEST_MOVES:
            return case


def _one(layout, l, length, phi, walls):
    if layout == "network":
        return S.crosslinked_network()
    if layout == "square":
        return S.square_network(l[0])
    if layout == "rings":
        return S.rings_and_free(l[0])
    s = S.serpentine_chains(l if len(set(l)) > 1 else l[0], length, phi)
    return S.walled(s, walls) if walls else s


def _systems(case):
    """The systems of a case in their start layout (the seeds and the relaxation make the inputs)."""
    l = (case["lx"], case["ly"], case["lz"])
    if case["layout"] == "mixed":
        # the ensemble's own draws (box, chain length, volume fraction), boxes up to lx
        out = []
        for side, length, phi in S.ensemble_params(4 * case["members"]):
            if side <= case["lx"] and len(out) < case["members"]:
                out.append(S.serpentine_chains(side, length, phi))
        return out
    s = _one(case["layout"], l, case["length"], case["phi"], case["walls"])
    return [s] * case["members"]


def _steps_of_job(case, k):
    """Jobs of a burst differ in length: from half of mcs to one and a half times it."""
    return max(1, case["mcs"] // 2 + (case["mcs"] * ((k * 7) % 16)) // 16)


def prepare(case, seed):
    systems = _systems(case)
    draws = random.Random(seed)
    seeds = [draws.getrandbits(48) for _ in systems]
    call = case["call"]
    if call == "serve":
        setups = [P.UpdaterGPUScBFM_AB_Type(0).load_system(s, seed=q, initialize=False)
                  for s, q in zip(systems, seeds)]
        return {"case": case, "setups": setups, "n": [s.n for s in systems], "server": P.Server(0)}
    members = [P.UpdaterGPUScBFM_AB_Type(0).load_system(s, seed=q) for s, q in zip(systems, seeds)]
    n = [s.n for s in systems]
    at = np.concatenate([[0], np.cumsum(n)])
    xyz = torch.empty((int(at[-1]), 3), dtype=torch.int32, pin_memory=True).numpy()
    state = {"case": case, "members": members, "at": at, "xyz": xyz}
    if call == "batch":
        state["batch"] = P.Batch(members)
        state["batch"].run(RELAX_MCS)
    else:
        members[0].runSimulationOnGPU(RELAX_MCS)
        if call == "sample":
            members[0].reset_msd_reference()
    return state


def run(state):
    case = state["case"]
    if case["call"] == "serve":
        srv = state["server"]
        jobs = [srv.submit_setup(u, _steps_of_job(case, k), case["every"], n=n)
                for k, (u, n) in enumerate(zip(state["setups"], state["n"]))]
        for j in jobs:
            srv.wait(j)
        got = [srv.result(j)[:2] for j in jobs]
        return {"xyz": np.concatenate([g[0] for g in got]), "samples": np.concatenate([g[1].reshape(-1) for g in got])}
    members, xyz, at = state["members"], state["xyz"], state["at"]
    if case["call"] == "batch":
        state["batch"].run(case["mcs"])
        for k, u in enumerate(members):
            u.get_coords(xyz[at[k]:at[k + 1]])
        return {"xyz": xyz}
    u = members[0]
    if case["call"] == "sample":
        obs = []
        for _ in range(case["samples"]):
            u.runSimulationOnGPU(case["mcs"])
            obs.append(u.observables_raw())
        return {"observables": obs, "xyz": u.get_coords(xyz)}
    u.runSimulationOnGPU(case["mcs"])
    return {"xyz": u.get_coords(xyz), "counters": list(u.stats().values())}


def work(case):
    """Bytes a pass cannot do without: every attempted move reads its monomer's lattice address, its
    bond code and the nine cells in front of it, every MCS; about one move in eight is made and
    writes address, code, two cells and its neighbours' codes; positions (12 B) and, where they
    are sampled, 13 B per monomer and sample come back once. No floating-point work."""
    systems = _systems(case)
    total = 0.0
    for k, s in enumerate(systems):
        bonds = float(s.nbr_count.mean())
        code = 4 if int(s.nbr_count.max()) <= 3 else 8
        mcs = _steps_of_job(case, k) if case["call"] == "serve" else case["mcs"] * max(case["samples"], 1)
        move = 4 + code + 9 / 8 + (4 + code + 2 / 8 + bonds * code) / 8
        looks = case["samples"] + (-(-mcs // case["every"]) if case["every"] else 0)
        total += s.n * (mcs * move + 12 + 13 * looks)
    return {"bytes": total, "flops": 0.0}


def exact(case, seed):
    """Every output is a whole number: passes compare bit for bit, no value in 64 bits applies."""
    return None
