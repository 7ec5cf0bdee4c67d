"""What the performance of this framework is measured on: the work of one MD step and of a rebuild, called through the
public entry points as a simulation calls them, over the sizes of the repository's configurations, tests and benchmark.

A case is one of these kinds:

  graph      radius graph over all atoms (edge list, shifts, degrees; optionally squared distances), every MD step of a
             single-GPU run
  owned      the graph a rank builds over [owned | ghost] positions for its own atoms, every MD step of a multi-GPU run
  rebuild    space-filling-curve partition plus the halo maps of one rank, at every repartition
  refresh    the distributed builder's refresh for one rank: degrees, degree-weighted partition, edges at cutoff + skin for
             its atoms, halo lists from these edges, edges filtered down to the cutoff
  kdtree     the other partitioner
  exchange   one message-passing layer: node embeddings to the ghosts, and the reverse sum of their gradients (two ranks
             driven from one process: all first halves, then all second halves)
  langevin   one integrator step (both halves) with the drift word

Edge lists, labels, halo lists and copied rows are compared value by value; the order of the edges is part of the result.
"""

import math

import torch

import dynamis_b200 as D
from dynamis_b200 import integrators
from dynamis_b200.partition import select_eq

FCC_A = 3.615        # lattice constants of the synthetic copper and silicon crystals
SI_A = 5.431
LIQUID_DENSITY = 0.1


def listed():
    return [
        # a small molecule box: launches and host time are all there is
        {"name": "graph_liquid_1k", "kind": "graph", "system": "liquid", "atoms": 1000, "radius": 5.0, "f64": False, "dist": False},
        # the CPU-runnable configuration: 20^3 cells of copper
        {"name": "graph_fcc_32k", "kind": "graph", "system": "fcc", "cells": 20, "radius": 6.0, "f64": False, "dist": False},
        # squared distances asked for as well (the writer that recomputes them), a medium size
        {"name": "graph_dist_131k", "kind": "graph", "system": "liquid", "atoms": 131_071, "radius": 5.0, "f64": False, "dist": True},
        # float64 positions in a triclinic cell
        {"name": "graph_si_f64_500k", "kind": "graph", "system": "si", "cells": 50, "radius": 6.0, "f64": True, "dist": False},
        # the benchmark's workload
        {"name": "graph_liquid_1m", "kind": "graph", "system": "liquid", "atoms": 1_000_000, "radius": 5.0, "f64": False, "dist": False},
        # the largest single-GPU system of the configurations' liquid
        {"name": "graph_liquid_4m", "kind": "graph", "system": "liquid", "atoms": 4_000_000, "radius": 5.0, "f64": False, "dist": False},
        # one rank's share of the 8-rank copper workload, 12 A halo, shifts in the model's sign and Cartesian
        {"name": "owned_fcc_1m_of_8m", "kind": "owned", "cells": 126, "ranks": 8, "radius": 6.0, "halo": 12.0},
        # repartition and halo rebuild of a million atoms on 8 ranks
        {"name": "rebuild_1m_w8", "kind": "rebuild", "atoms": 1_000_000, "ranks": 8, "radius": 5.0, "buffer": 1.0},
        # a rank's refresh with a skin, odd size
        {"name": "refresh_250k_w4", "kind": "refresh", "atoms": 250_007, "ranks": 4, "radius": 5.0, "buffer": 1.0},
        {"name": "kdtree_1m_w8", "kind": "kdtree", "atoms": 1_000_000, "ranks": 8},
        # 128-wide embeddings of half a million atoms per rank
        {"name": "exchange_f128_500k", "kind": "exchange", "rows": 500_000, "halo": 150_000, "width": 128},
        {"name": "langevin_1m", "kind": "langevin", "atoms": 1_000_000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["graph", "graph", "graph", "graph", "owned", "rebuild", "refresh", "kdtree", "exchange", "langevin"])
    if kind == "graph":
        system = rng.choice(["liquid", "liquid", "fcc", "si"])
        case = {"kind": kind, "system": system, "radius": rng.choice([4.5, 5.0, 5.5, 6.0]), "f64": rng.random() < 0.25,
                "dist": rng.random() < 0.2}
        if system == "liquid":
            case["atoms"] = _log(rng, 500, 1_500_000)
        else:
            case["cells"] = _log(rng, 6, 60 if system == "fcc" else 50)
        return case
    if kind == "owned":
        return {"kind": kind, "cells": _log(rng, 30, 105), "ranks": rng.choice([4, 8]), "radius": 6.0,
                "halo": rng.choice([6.5, 8.0, 12.0])}
    if kind == "rebuild":
        return {"kind": kind, "atoms": _log(rng, 20_000, 1_500_000), "ranks": rng.choice([2, 4, 5, 8]), "radius": 5.0, "buffer": rng.choice([0.5, 1.0])}
    if kind == "refresh":
        return {"kind": kind, "atoms": _log(rng, 20_000, 500_000), "ranks": rng.choice([2, 4, 8]), "radius": 5.0, "buffer": rng.choice([0.5, 1.0])}
    if kind == "kdtree":
        return {"kind": kind, "atoms": _log(rng, 20_000, 2_000_000), "ranks": rng.choice([2, 3, 4, 8, 13, 16])}
    if kind == "exchange":
        rows = _log(rng, 20_000, 600_000)
        return {"kind": kind, "rows": rows, "halo": int(rows * rng.uniform(0.1, 0.4)), "width": rng.choice([3, 16, 64, 65, 128, 256])}
    return {"kind": kind, "atoms": _log(rng, 1000, 4_000_000)}


# ---------------------------------------------------------------------------------------------- systems
_FCC = [[0.0, 0.0, 0.0], [0.5, 0.5, 0.0], [0.5, 0.0, 0.5], [0.0, 0.5, 0.5]]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _renumber(pos, gen, chunk):
    """The same atoms under other numbers: chunks of consecutive atoms in the order that the seed gives.  A system then has
    the same number of edges for every seed.  Chunks of one for a liquid, whose numbers say nothing about places; of 32 for
    a crystal, whose neighbouring numbers lie near one another."""
    n = pos.size(0)
    starts = torch.randperm(-(-n // chunk), generator=gen, device="cuda") * chunk
    order = (starts[:, None] + torch.arange(chunk, device="cuda")[None]).reshape(-1)
    return pos[order[order < n]].contiguous()


def _lattice(nx, ny, nz, basis):
    """Sites in units of the conventional cell, cell by cell."""
    dev = "cuda"
    grid = torch.meshgrid(torch.arange(nx, device=dev), torch.arange(ny, device=dev), torch.arange(nz, device=dev), indexing="ij")
    corner = torch.stack([g.reshape(-1) for g in grid], dim=1).to(torch.float64)
    return (corner[:, None, :] + torch.tensor(basis, dtype=torch.float64, device=dev)[None]).reshape(-1, 3)


def _liquid(atoms, gen, dtype):
    length = (atoms / LIQUID_DENSITY) ** (1.0 / 3.0)
    pos = torch.rand(atoms, 3, generator=_generator(1002), device="cuda", dtype=torch.float64) * length
    return _renumber(pos.to(dtype), gen, 1), torch.eye(3, dtype=torch.float64).mul(length).to(dtype)


def _jittered(sites, sigma, gen, dtype):
    sites += torch.randn(sites.shape, generator=_generator(1001), device="cuda", dtype=torch.float64) * sigma
    return _renumber(sites.to(dtype), gen, 32)


def _fcc(cells, gen, dtype):
    pos = _jittered(_lattice(cells, cells, cells, _FCC) * FCC_A, 0.1, gen, dtype)
    return pos, torch.eye(3, dtype=torch.float64).mul(cells * FCC_A).to(dtype)


def _si(cells, gen, dtype):
    """Sheared diamond-lattice silicon, half as high as wide."""
    n = [cells, cells, max(cells // 2, 3)]
    cell = torch.tensor([[n[0] * SI_A, 0.0, 0.0], [0.2 * n[0] * SI_A, n[1] * SI_A, 0.0], [0.1 * n[0] * SI_A, 0.0, n[2] * SI_A]],
                        dtype=torch.float64)
    frac = _lattice(n[0], n[1], n[2], _FCC + [[x + 0.25 for x in b] for b in _FCC]) / torch.tensor(n, dtype=torch.float64, device="cuda")
    return _jittered(frac @ cell.cuda(), 0.05, gen, dtype), cell.to(dtype)


def _system(case, gen):
    dtype = torch.float64 if case["f64"] else torch.float32
    if case["system"] == "liquid":
        return _liquid(case["atoms"], gen, dtype)
    return (_fcc if case["system"] == "fcc" else _si)(case["cells"], gen, dtype)


def _atoms(case):
    if "atoms" in case:
        return case["atoms"]
    if case.get("system") == "si":
        return 8 * case["cells"] ** 2 * max(case["cells"] // 2, 3)
    return 4 * case["cells"] ** 3


# ---------------------------------------------------------------------------------------------- prepare
def _prepare_owned(case, gen):
    pos, cell = _fcc(case["cells"], gen, torch.float32)
    own = torch.nonzero(D.sfc_partition_labels(pos, None, case["ranks"], 0) == 0).reshape(-1)
    length = float(cell[0, 0])
    lo, hi = pos[own].min(dim=0).values, pos[own].max(dim=0).values
    away = ((pos - (lo + hi) / 2 + length / 2) % length - length / 2).abs() - (hi - lo) / 2
    near = (away <= case["halo"]).all(dim=1)
    near[own] = False
    both = torch.cat([pos[own], pos[torch.nonzero(near).reshape(-1)]]).contiguous()
    return {"pos": both, "cell": cell, "pbc": torch.tensor([True] * 3), "local": own.numel()}


def _prepare_exchange(case, gen):
    rows, halo, width = case["rows"], case["halo"], case["width"]
    ranks, feats, grads = [], [], []
    for r in range(2):
        # an ascending list of distinct rows goes to the other rank
        send = torch.sort(torch.randperm(rows, generator=gen, device="cuda")[:halo]).values
        offsets = torch.tensor([0, halo if r == 1 else 0, halo])
        ex = D.FeatureExchanger()
        ranks.append((ex, ex.local_setup(offsets, send, offsets, rows, width, r, 2, torch.device("cuda", torch.cuda.current_device()))))
        feats.append(torch.randn(rows, width, generator=gen, device="cuda"))
        grads.append(torch.randn(rows + halo, width, generator=gen, device="cuda"))
    for ex, _ in ranks:
        ex.connect([meta for _, meta in ranks])
    return {"ranks": [ex for ex, _ in ranks], "feats": feats, "grads": grads}


def prepare(case, seed):
    gen, kind = _generator(seed), case["kind"]
    pbc = torch.tensor([True] * 3)
    if kind == "graph":
        pos, cell = _system(case, gen)
        state = {"pos": pos, "cell": cell, "pbc": pbc}
    elif kind == "owned":
        state = _prepare_owned(case, gen)
    elif kind in ("rebuild", "refresh"):
        pos, cell = _liquid(case["atoms"], gen, torch.float32)
        env, config, mol = D.DistEnvironment(), D.SimulationConfig(), D.MolecularInfo()
        env.global_rank, env.world_size = 1, case["ranks"]
        config.cutoff, config.ghost_cutoff_buffer, config.cell, config.pbc = case["radius"], case["buffer"], cell, pbc
        mol.num_atoms, mol.atom_positions = case["atoms"], pos
        mol.atom_vertex_numbers = torch.arange(case["atoms"], dtype=torch.int64, device="cuda")
        state = {"pos": pos, "cell": cell, "pbc": pbc, "env": env, "config": config, "mol": mol, "partitioner": D.SFCPartitioner()}
    elif kind == "kdtree":
        state = {"pos": _liquid(case["atoms"], gen, torch.float32)[0]}
    elif kind == "exchange":
        state = _prepare_exchange(case, gen)
    else:
        pos, _ = _liquid(case["atoms"], gen, torch.float32)
        vel, frc = (torch.randn(pos.shape, generator=gen, device="cuda") * s for s in (0.05, 1.0))
        state = {"pos": pos, "vel": vel, "frc": frc, "mass": torch.rand(case["atoms"], generator=gen, device="cuda") * 60.0 + 1.0,
                 "noise": [torch.randn(pos.shape, generator=gen, device="cuda") for _ in range(2)],
                 "watch": integrators.DriftWatch(pos, vel, 0.5), "step": integrators.Langevin(0.5, 0.01, 0.025)}
    state["case"] = dict(case)
    return state


# ---------------------------------------------------------------------------------------------- run
def _run_rebuild(s):
    info = s["partitioner"].partition(s["mol"], s["env"])
    s["partitioner"].build_halo_maps(info, s["mol"], s["env"], s["config"])
    return [info.partition_id, info.partition_indices, info.atom_counts, info.send_offsets, info.send_local_indices, info.recv_offsets,
            info.recv_ghost_indices, info.recv_atom_global, info.interior_mask, info.global_send_recv_matrix]


def _run_refresh(s):
    case, rank = s["case"], s["env"].global_rank
    pos, cell, pbc, ranks = s["pos"], s["cell"], s["pbc"], s["env"].world_size
    degrees = D.radius_graph_pbc_counts_ex(pos, cell, pbc, case["radius"])
    labels = D.sfc_partition_labels(pos, degrees, ranks, 0)
    mine = select_eq(labels, rank)
    outer, shifts, _, _ = D.radius_graph_pbc_ex(pos, cell, pbc, case["radius"] + case["buffer"], 0, False, mine)
    halo = D.extract_halo_info(outer, labels, mine, rank, ranks, case["atoms"])
    edges, edge_shifts = D.filter_edges_to_radius(outer, shifts, pos, cell, case["radius"])
    return [degrees, labels, mine, list(halo), edges, edge_shifts]


def _run_exchange(s):
    ranks = s["ranks"]
    begun = [ex.forward_begin(x) for ex, x in zip(ranks, s["feats"])]
    forward = [ex.forward_end(*b) for ex, b in zip(ranks, begun)]
    begun = [ex.backward_begin(g) for ex, g in zip(ranks, s["grads"])]
    backward = [ex.backward_end(*b) for ex, b in zip(ranks, begun)]
    return [forward, backward]


def _run_langevin(s):
    s["step"].halfstep1_(s["pos"], s["vel"], s["frc"], s["mass"], s["noise"][0], 0.5, drift=s["watch"])
    s["step"].halfstep2_(s["vel"], s["frc"], s["mass"], s["noise"][1], 0.5)
    return [s["pos"], s["vel"], s["watch"].flag]


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "graph":
        if case["dist"]:
            return D.radius_graph_pbc_with_dist(s["pos"], s["cell"], s["pbc"], case["radius"])
        return D.radius_graph_pbc_ex(s["pos"], s["cell"], s["pbc"], case["radius"], 0, False)
    if kind == "owned":
        return D.owned_graph(s["pos"], s["cell"], s["pbc"], case["radius"], s["local"])
    if kind == "kdtree":
        return D.kdtree_partition_labels(s["pos"], None, case["ranks"])
    return {"rebuild": _run_rebuild, "refresh": _run_refresh, "exchange": _run_exchange, "langevin": _run_langevin}[kind](s)


# ---------------------------------------------------------------------------------------------- work and tolerance
def _degree(density, radius):
    return density * 4.0 / 3.0 * math.pi * radius ** 3


def work(case):
    kind, flop = case["kind"], 8.0  # operations of one distance test
    if kind == "exchange":
        rows, halo, row = case["rows"], case["halo"], 4 * case["width"]
        # per rank: forward reads its rows and the send list, writes owned and ghost rows; the reverse reads the gradients, writes the sums
        return {"bytes": 2.0 * (row * (rows + rows + halo) + 8 * halo + row * (rows + halo + rows)), "flops": 2.0 * halo * case["width"]}
    n = float(_atoms(case))
    if kind == "graph":
        density = {"liquid": LIQUID_DENSITY, "fcc": 4.0 / FCC_A ** 3, "si": 8.0 / SI_A ** 3}[case["system"]]
        edges, real = n * _degree(density, case["radius"]), 8 if case["f64"] else 4
        return {"bytes": 3 * real * n + 4 * n + edges * (28 + (real if case["dist"] else 0)), "flops": flop * edges}
    if kind == "owned":
        own = n / case["ranks"]
        side, edges = (own * FCC_A ** 3 / 4.0) ** (1.0 / 3.0), own * _degree(4.0 / FCC_A ** 3, case["radius"])
        both = min(n, (side + 2 * case["halo"]) ** 3 * 4.0 / FCC_A ** 3)
        return {"bytes": 12 * both + 40 * edges, "flops": flop * edges}
    if kind in ("rebuild", "refresh"):
        outer, own = case["radius"] + case["buffer"], n / case["ranks"]
        side = (own / LIQUID_DENSITY) ** (1.0 / 3.0)
        halo = 2.0 * ((side + 2 * outer) ** 3 * LIQUID_DENSITY - own)
        if kind == "rebuild":
            return {"bytes": 12 * n + 8 * n + 8 * own + own + 8 * halo, "flops": flop * n * _degree(LIQUID_DENSITY, outer)}
        return {"bytes": 12 * n + 4 * n + 8 * n + 9 * own + 8 * halo + 28 * own * _degree(LIQUID_DENSITY, case["radius"]),
                "flops": flop * (n * _degree(LIQUID_DENSITY, case["radius"]) + own * _degree(LIQUID_DENSITY, outer))}
    if kind == "kdtree":
        return {"bytes": 12 * n + 8 * n, "flops": n * math.log2(case["ranks"])}
    # positions, forces, two noise arrays, mass, reference and previous velocities in; positions, velocities, previous velocities out
    return {"bytes": n * (12 * 7 + 4 + 12 * 3), "flops": 60.0 * n}


def tolerance(case):
    """Whole numbers, copied rows and unit shifts are exact.  Where sums or products are rounded the bounds are about four
    times the differences from the same path evaluated in 64 bits (squared distances: 1.3e-7 and at most 2.1e-6 in float32,
    9e-17 in float64; integrator: 6.5e-8 and 2.7e-7; reverse sums and Cartesian shifts: one rounding)."""
    if case["kind"] == "graph" and case["dist"]:
        return {"rel": 5e-16, "max": 2e-15} if case["f64"] else {"rel": 6e-7, "max": 1e-5}
    if case["kind"] == "langevin":
        return {"rel": 3e-7, "max": 2e-6}
    if case["kind"] in ("owned", "exchange"):
        return {"rel": 1e-7, "max": 5e-7}
    return "exact"
