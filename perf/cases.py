"""Performance cases: the work users of nabladyn_b200 have it do, through its public calls.

Each case is a dict of plain values; ``kind`` names the call:

* ``efv``: ``quantity.energy_force_virial`` of a Lennard-Jones model over a neighbor list;
* ``fit``: one Lennard-Jones training evaluation, ``training.predict`` and ``loss`` with the
  gradient in sigma and epsilon;
* ``list``: ``NeighborList.update`` of a frame that needs a rebuild, or ``allocate``;
* ``schnet``: ``quantity.energy_force_virial`` of a SchNet model;
* ``schnet_fit``: one SchNet training step, ``training.loss_and_gradient``;
* ``md``: ``md.nve`` / ``md.nvt`` of Lennard-Jones argon, a stretch of steps and the state;
* ``serve``: ``serving.ReplicaServer.serve`` of a batch of uneven replicas.

``listed`` gives the cases with names, ``draw`` one more of the same ranges, ``prepare`` a
case's inputs and what a program keeps between calls, ``run`` one call, ``work`` the bytes and
operations a call cannot do without, ``exact`` the float64 values written in plain torch.
"""

import dataclasses
import math

import numpy as np
import torch

from nabladyn_b200 import md, potential, quantity, serving, training
from nabladyn_b200.neighbors import NeighborList

DEVICE = "cuda"
CUTOFF, SKIN, JITTER = 1.0, 0.1, 0.02
ARGON_DENSITY, ARGON_MASS = 21.1, 39.948
TIMESTEP, TEMPERATURE, TIMESCALE = 0.004, 120.0, 0.1
BOLTZMANN = 0.00831446261815324
BEAD_CUTOFF, BEAD_DENSITY, BEAD_JITTER, FEATURES = 1.2, 10.0, 0.03, 64
# Lennard-Jones rows (0, 0), (0, 1), (1, 1), ... for up to three types.
SIGMA = {1: (0.34,), 2: (0.34, 0.32, 0.30), 3: (0.34, 0.32, 0.33, 0.30, 0.31, 0.32)}
EPSILON = {1: (0.996,), 2: (0.996, 0.8, 0.6), 3: (0.996, 0.8, 0.9, 0.6, 0.7, 0.8)}
CHANNELS = ("energy", "forces", "virial")
DTYPES = {"f32": torch.float32, "f64": torch.float64}


def listed():
    return [
        # A single small evaluation in float64: minimisers, checks and scripts call it one
        # frame at a time, so it is latency that counts.
        {"name": "efv_argon_512_f64", "kind": "efv", "atoms": 512, "types": 1, "dtype": "f64",
         "aspect": 1.0},
        # An ordinary mixture frame of an odd size.
        {"name": "efv_mixture_27k_f32", "kind": "efv", "atoms": 27431, "types": 2,
         "dtype": "f32", "aspect": 1.25},
        # The largest frame: the million-atom argon box.
        {"name": "efv_argon_1m_f32", "kind": "efv", "atoms": 1048576, "types": 1,
         "dtype": "f32", "aspect": 1.0},
        # One update of a Lennard-Jones fit: 64 frames of a two-type mixture.
        {"name": "fit_mixture_64x4096_f32", "kind": "fit", "frames": 64, "atoms": 4096,
         "types": 2, "dtype": "f32"},
        # A user's own loop over frames of the large box: every frame rebuilds the list.
        {"name": "list_update_1m_f32", "kind": "list", "call": "update", "atoms": 1048576,
         "dtype": "f32", "skin": 0.1, "aspect": 1.0},
        # A first list of a small odd system in float64, as every new frame set begins.
        {"name": "list_allocate_2k_f64", "kind": "list", "call": "allocate", "atoms": 2003,
         "dtype": "f64", "skin": 0.1, "aspect": 1.0},
        # The coarse-grained bead system, one evaluation.
        {"name": "schnet_efv_32k", "kind": "schnet", "atoms": 32768, "types": 1, "blocks": 3,
         "gaussians": 50},
        # A small odd bead system of two types.
        {"name": "schnet_efv_2k", "kind": "schnet", "atoms": 2111, "types": 2, "blocks": 3,
         "gaussians": 50},
        # A training step of the bead network over four frames.
        {"name": "schnet_fit_4x32k", "kind": "schnet_fit", "frames": 4, "atoms": 32768,
         "types": 1, "blocks": 3, "gaussians": 50},
        # The headline molecular dynamics: the million-atom box at constant energy.
        {"name": "md_nve_1m", "kind": "md", "ensemble": "nve", "atoms": 1048576, "steps": 20,
         "dtype": "f32"},
        # The small box at constant temperature, a stretch between samples.
        {"name": "md_nvt_512", "kind": "md", "ensemble": "nvt", "atoms": 512, "steps": 100,
         "dtype": "f32"},
        # Many uneven replicas in flight at once.
        {"name": "serve_512", "kind": "serve", "requests": 512, "steps": 100},
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("efv", "fit", "list", "schnet", "schnet_fit", "md", "serve"))
    if kind in ("efv", "list"):
        dtype = rng.choice(("f32", "f32", "f64"))
        case = {"kind": kind, "atoms": _log_uniform(rng, 400, 1048576 if dtype == "f32" else 400000),
                "dtype": dtype, "aspect": rng.choice((1.0, 1.1, 1.25))}
        if kind == "efv":
            return {**case, "types": rng.choice((1, 2, 3))}
        return {**case, "call": rng.choice(("update", "update", "allocate")),
                "skin": rng.choice((0.05, 0.1, 0.15))}
    if kind == "fit":
        dtype = rng.choice(("f32", "f32", "f64"))
        return {"kind": kind, "frames": _log_uniform(rng, 2, 64 if dtype == "f32" else 24),
                "atoms": _log_uniform(rng, 400, 4096), "types": rng.choice((1, 2, 3)),
                "dtype": dtype}
    if kind == "schnet":
        return {"kind": kind, "atoms": _log_uniform(rng, 343, 32768),
                "types": rng.choice((1, 2, 4)), "blocks": rng.choice((1, 2, 3)),
                "gaussians": rng.choice((20, 33, 50, 64))}
    if kind == "schnet_fit":
        return {"kind": kind, "frames": rng.choice((1, 2, 3, 4)),
                "atoms": _log_uniform(rng, 343, 32768), "types": rng.choice((1, 2, 4)),
                "blocks": rng.choice((1, 2, 3)), "gaussians": rng.choice((20, 33, 50, 64))}
    if kind == "md":
        dtype = rng.choice(("f32", "f32", "f64"))
        atoms = _log_uniform(rng, 400, 1000000 if dtype == "f32" else 100000)
        return {"kind": kind, "ensemble": rng.choice(("nve", "nvt")), "atoms": atoms,
                "steps": rng.randint(5, 20) if atoms > 50000 else rng.randint(20, 60),
                "dtype": dtype}
    return {"kind": kind, "requests": _log_uniform(rng, 16, 512), "steps": rng.randint(20, 100)}


# -- inputs ---------------------------------------------------------------------------------


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _lattice(atoms, density, aspect):
    """Lattice sites (float64) filling a box, and its lengths: face-centered cubic for 4 k^3
    atoms, else a simple-cubic grid of at least that many sites (the caller drops some)."""
    length = (atoms / density) ** (1.0 / 3.0)
    lengths = torch.tensor([length * aspect, length, length / aspect], dtype=torch.float64,
                           device=DEVICE)
    side = round((atoms / 4) ** (1.0 / 3.0))
    base = [[0.25, 0.25, 0.25]]
    if 4 * side**3 == atoms:
        base = [[0.25, 0.25, 0.25], [0.75, 0.75, 0.25], [0.75, 0.25, 0.75], [0.25, 0.75, 0.75]]
    else:
        side = math.ceil(round(atoms ** (1.0 / 3.0), 6))
        base = [[0.5, 0.5, 0.5]]
    axis = torch.arange(side, dtype=torch.float64, device=DEVICE)
    grid = torch.cartesian_prod(axis, axis, axis)
    base = torch.tensor(base, dtype=torch.float64, device=DEVICE)
    sites = (grid[:, None, :] + base).reshape(-1, 3) / side * lengths
    return sites, lengths


def _sites(atoms, density, aspect):
    """The lattice sites of ``atoms`` atoms (the same ones for every seed) and the box."""
    sites, lengths = _lattice(atoms, density, aspect)
    order = torch.randperm(sites.shape[0], generator=_generator(atoms), device=DEVICE)
    return sites[order[:atoms].sort()[0]], lengths


def _frames(count, atoms, density, jitter, dtype, generator, aspect=1.0):
    """``count`` jittered frames [count, N, 3] of one lattice and the cell [3]; atoms may lie a
    little outside the cell, as a user's may."""
    sites, lengths = _sites(atoms, density, aspect)
    noise = torch.randn((count, atoms, 3), dtype=torch.float64, generator=generator,
                        device=DEVICE)
    return (sites + jitter * noise).to(dtype), lengths.to(dtype)


def _lj_parameters(types, dtype):
    return (torch.tensor(SIGMA[types], dtype=dtype, device=DEVICE),
            torch.tensor(EPSILON[types], dtype=dtype, device=DEVICE))


def _types(atoms, types, generator):
    return torch.randint(types, (atoms,), generator=generator, device=DEVICE)


def _schnet_weights(types, blocks, gaussians, generator):
    """Float32 weights of a SchNet under its state-dict names."""
    def matrix(out, width):
        bound = math.sqrt(6.0 / (out + width))
        u = torch.rand((out, width), dtype=torch.float64, generator=generator, device=DEVICE)
        return ((2.0 * u - 1.0) * bound).float()

    def vector(width, scale=0.05):
        return (scale * torch.randn(width, dtype=torch.float64, generator=generator,
                                    device=DEVICE)).float()

    weights = {"embedding": vector((types, FEATURES), 1.0)}
    for b in range(blocks):
        name = f"blocks.{b}."
        weights[name + "atoms.weight"] = matrix(FEATURES, FEATURES)
        for layer, width in (("filter1", gaussians), ("filter2", FEATURES),
                             ("update1", FEATURES), ("update2", FEATURES)):
            weights[name + layer + ".weight"] = matrix(FEATURES, width)
            weights[name + layer + ".bias"] = vector(FEATURES)
    weights["readout1.weight"] = matrix(FEATURES // 2, FEATURES)
    weights["readout1.bias"] = vector(FEATURES // 2)
    weights["readout2.weight"] = matrix(1, FEATURES // 2)
    weights["readout2.bias"] = vector(1)
    return weights


def _inputs(case, seed):
    """A case's inputs from the seed alone (no call of the framework)."""
    kind, generator = case["kind"], _generator(seed)
    dtype = DTYPES[case.get("dtype", "f32")]
    if kind == "efv":
        types = _types(case["atoms"], case["types"], generator)
        x, cell = _frames(1, case["atoms"], ARGON_DENSITY, JITTER, dtype, generator,
                          case["aspect"])
        return {"types": types, "positions": x[0], "cell": cell}
    if kind == "list":
        x, cell = _frames(2, case["atoms"], ARGON_DENSITY, JITTER, dtype, generator,
                          case["aspect"])
        return {"frames": x, "cell": cell}
    if kind == "fit":
        types = _types(case["atoms"], case["types"], generator)
        x, cell = _frames(case["frames"], case["atoms"], ARGON_DENSITY, JITTER, dtype, generator)
        cells = cell.expand(case["frames"], 3).contiguous()
        # Labels of the exact parameters; the fit starts up to 10 % away.
        sigma, epsilon = _lj_parameters(case["types"], torch.float64)
        labels = [_lj_exact(x[f].double(), cell.double(), types, sigma, epsilon)
                  for f in range(case["frames"])]
        labels = {name: torch.stack([row[k] for row in labels]).to(dtype)
                  for k, name in enumerate(CHANNELS)}
        off = 0.9 + 0.2 * torch.rand(2, sigma.numel(), dtype=torch.float64, generator=generator,
                                     device=DEVICE)
        return {"types": types, "positions": x, "cells": cells, "labels": labels,
                "sigma": (sigma * off[0]).to(dtype), "epsilon": (epsilon * off[1]).to(dtype),
                "scales": _scales(labels)}
    if kind in ("schnet", "schnet_fit"):
        types = _types(case["atoms"], case["types"], generator)
        frames = case.get("frames", 1)
        x, cell = _frames(frames, case["atoms"], BEAD_DENSITY, BEAD_JITTER, torch.float32,
                          generator)
        weights = _schnet_weights(case["types"], case["blocks"], case["gaussians"], generator)
        got = {"types": types, "positions": x, "cell": cell, "weights": weights}
        if kind == "schnet_fit":
            # Labels from another network of the same size.
            teacher = _schnet_weights(case["types"], case["blocks"], case["gaussians"], generator)
            teacher = {name: w.double() for name, w in teacher.items()}
            rows = []
            for f in range(frames):
                values = _schnet_exact(x[f].double(), cell.double(), types, teacher,
                                       case["blocks"], case["gaussians"], False)
                rows.append([y.detach().float() for y in values])
            got["cells"] = cell.expand(frames, 3).contiguous()
            got["labels"] = {name: torch.stack([row[k] for row in rows])
                             for k, name in enumerate(CHANNELS)}
            got["scales"] = _scales(got["labels"])
        return got
    if kind == "md":
        x, cell = _frames(1, case["atoms"], ARGON_DENSITY, JITTER, dtype, generator)
        thermal = math.sqrt(BOLTZMANN * TEMPERATURE / ARGON_MASS)
        v = thermal * torch.randn((case["atoms"], 3), dtype=torch.float64, generator=generator,
                                  device=DEVICE)
        return {"positions": x[0], "cell": cell, "velocities": v.to(dtype),
                "masses": torch.full((case["atoms"],), ARGON_MASS, dtype=dtype, device=DEVICE)}
    raise ValueError(kind)


def _scales(labels):
    """The scales of a training loss: energy and virial by their spread over the frames, forces
    by their size."""
    found = {}
    for name, value in labels.items():
        value = value.double()
        rms = float(value.square().mean().sqrt())
        spread = rms
        if name != "forces":
            spread = float((value - value.mean(dim=0)).square().mean().sqrt())
        found[name] = spread or rms or 1.0
    return found


# -- the calls ------------------------------------------------------------------------------


def _lj_model(types, num_types, dtype, trainable=()):
    sigma, epsilon = _lj_parameters(num_types, dtype)
    return potential.lennard_jones(atom_types=types, sigma=sigma, epsilon=epsilon, cutoff=CUTOFF,
                                   trainable=trainable)


def _schnet_model(case, given, trainable):
    model = potential.schnet(atom_types=given["types"], num_types=case["types"],
                             cutoff=BEAD_CUTOFF, interactions=case["blocks"],
                             gaussians=case["gaussians"], trainable=trainable)
    model.load_state_dict(given["weights"])
    return model


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        # The sizes and settings of one request stream; the frames of this seed.
        rng = np.random.default_rng(seed)
        stream = serving.serving_requests(case["requests"], steps=case["steps"])
        requests = [dataclasses.replace(r, positions=r.positions + rng.normal(
            0.0, 0.01, r.positions.shape), velocities=rng.permutation(r.velocities))
            for r in stream]
        return {"kind": kind, "server": serving.ReplicaServer(), "requests": requests}
    given = _inputs(case, seed)
    state = {"kind": kind, "case": case, **given}
    if kind == "efv":
        model = _lj_model(given["types"], case["types"], given["positions"].dtype)
        pairs = NeighborList(CUTOFF, skin=SKIN)
        pairs.allocate(given["positions"], given["cell"])
        state.update(list=pairs, evaluate=quantity.energy_force_virial(model))
    elif kind == "list":
        state["turn"] = 0
        sites = _sites(case["atoms"], ARGON_DENSITY, case["aspect"])[0].to(given["cell"].dtype)
        pairs = NeighborList(CUTOFF, skin=case["skin"])
        if case["call"] == "update":
            # Sized on the lattice, with room for any of its frames.
            pairs = NeighborList(CUTOFF, skin=case["skin"], capacity_multiplier=1.4)
            pairs.allocate(sites, given["cell"])
            state["list"] = pairs
        else:
            # Each frame's pairs go into one index of a fixed width, as a data set keeps them.
            pairs.allocate(sites, given["cell"])
            columns = math.ceil(1.4 * pairs.pair_capacity)
            state["index"] = torch.zeros((2, columns), dtype=torch.int32, device=DEVICE)
    elif kind == "fit":
        state["model"] = _lj_model(given["types"], case["types"], given["positions"].dtype,
                                   ("sigma", "epsilon"))
        state["stack"] = training.pair_stack(given["positions"], given["cells"], CUTOFF)
    elif kind == "schnet":
        model = _schnet_model(case, given, False)
        pairs = NeighborList(BEAD_CUTOFF, skin=SKIN)
        pairs.allocate(given["positions"][0], given["cell"])
        state.update(list=pairs, evaluate=quantity.energy_force_virial(model))
    elif kind == "schnet_fit":
        model = _schnet_model(case, given, True)
        state.update(model=model,
                     parameters={k: v.detach().clone() for k, v in model.named_parameters()},
                     stack=training.pair_stack(given["positions"], given["cells"], BEAD_CUTOFF))
    elif kind == "md":
        types = torch.zeros(case["atoms"], dtype=torch.int64, device=DEVICE)
        model = _lj_model(types, 1, given["positions"].dtype)
        frame = (model, given["positions"], given["velocities"], given["masses"], given["cell"])
        if case["ensemble"] == "nve":
            state["simulation"] = md.nve(*frame, timestep=TIMESTEP, skin=SKIN)
        else:
            state["simulation"] = md.nvt(*frame, timestep=TIMESTEP, skin=SKIN,
                                         temperature=TEMPERATURE, thermostat_timescale=TIMESCALE)
    return state


def run(state):
    kind = state["kind"]
    if kind == "efv":
        energy, forces, virial = state["evaluate"](state["positions"], state["cell"],
                                                   state["list"].tensors())
        return {"energy": energy, "forces": forces, "virial": virial}
    if kind == "schnet":
        energy, forces, virial = state["evaluate"](state["positions"][0], state["cell"],
                                                   state["list"].tensors())
        return {"energy": energy, "forces": forces, "virial": virial}
    if kind == "list":
        case, frames = state["case"], state["frames"]
        state["turn"] ^= 1
        if case["call"] == "update":
            # The other frame: atoms moved by more than half the skin, so the list rebuilds.
            state["list"].update(frames[state["turn"]], state["cell"])
            return state["list"].tensors().index
        pairs = NeighborList(CUTOFF, skin=case["skin"])
        pairs.allocate(frames[state["turn"]], state["cell"])
        index = pairs.tensors().index
        state["index"][:, :index.shape[1]] = index
        return state["index"]
    if kind == "fit":
        parameters = {name: state[name].detach().clone().requires_grad_(True)
                      for name in ("sigma", "epsilon")}
        predicted = training.predict(state["model"], parameters, state["positions"],
                                     state["cells"], (state["stack"],), CHANNELS)
        weights = {name: 1.0 for name in CHANNELS}
        value, _ = training.loss(predicted, state["labels"], weights, state["scales"])
        value.backward()
        return {"loss": value.detach(), "sigma": parameters["sigma"].grad,
                "epsilon": parameters["epsilon"].grad,
                "predicted": {name: x.detach() for name, x in predicted.items()}}
    if kind == "schnet_fit":
        weights = {name: 1.0 for name in CHANNELS}
        value, gradient = training.loss_and_gradient(
            state["model"], state["parameters"], state["positions"], state["cells"],
            (state["stack"],), state["labels"], weights, state["scales"])
        return {"loss": value, "gradient": gradient}
    if kind == "md":
        simulation = state["simulation"]
        simulation.run(state["case"]["steps"])
        frame = simulation.state()
        # The unwrapped path, as a diffusion analysis takes it.
        path = frame.positions + frame.images.to(frame.positions.dtype) * frame.cell
        return {"path": path, "velocities": frame.velocities, "forces": frame.forces}
    results = sorted(state["server"].serve(state["requests"], realtime=False),
                     key=lambda r: r.name)
    cells = {r.name: r.cell for r in state["requests"]}
    return {
        "path": np.concatenate([r.positions + r.images * np.float32(cells[r.name])
                                for r in results]).astype(np.float32),
        "velocities": np.concatenate([r.velocities for r in results]),
        "energy": np.array([r.energy for r in results]),
        "steps": np.array([r.steps for r in results]),
    }


# -- what a call cannot do without ----------------------------------------------------------


def _half_pairs(atoms, density, radius):
    return 0.5 * atoms * density * 4.0 / 3.0 * math.pi * radius**3


def work(case):
    kind = case["kind"]
    real = 8 if case.get("dtype") == "f64" else 4
    if kind == "efv":
        n = case["atoms"]
        listed_pairs = _half_pairs(n, ARGON_DENSITY, CUTOFF + SKIN)
        return {"bytes": 6 * real * n + 8 * listed_pairs,
                "flops": 45 * _half_pairs(n, ARGON_DENSITY, CUTOFF)}
    if kind == "list":
        n = case["atoms"]
        # Positions in; every column of the index out, at least 1.25 times the pairs.
        listed_pairs = _half_pairs(n, ARGON_DENSITY, CUTOFF + case["skin"])
        return {"bytes": 3 * real * n + 8 * 1.25 * listed_pairs, "flops": 10 * listed_pairs}
    if kind == "fit":
        n, frames = case["atoms"], case["frames"]
        pairs = _half_pairs(n, ARGON_DENSITY, CUTOFF)
        # Positions and labels in, predicted forces out; the pairs read forward and backward.
        return {"bytes": frames * (9 * real * n + 16 * pairs), "flops": frames * 110 * pairs}
    if kind in ("schnet", "schnet_fit"):
        n, blocks = case["atoms"], case["blocks"]
        pairs = _half_pairs(n, BEAD_DENSITY, BEAD_CUTOFF)
        dense = FEATURES * FEATURES
        per_pair = 2 * (case["gaussians"] * FEATURES + dense)  # one filter network
        per_atom = 2 * 3 * dense
        listed_pairs = _half_pairs(n, BEAD_DENSITY, BEAD_CUTOFF + SKIN)
        if kind == "schnet":
            return {"bytes": 24 * n + 8 * listed_pairs,
                    "flops": blocks * 2 * (per_pair * pairs + per_atom * n)}
        frames = case["frames"]
        # E, F and W; then a tangent pass and a reverse pass of two streams with the filter
        # weights' gradients: the filter network 2 + 2 + 2 * 2 + 2 times over.
        return {"bytes": frames * (36 * n + 8 * pairs),
                "flops": frames * blocks * 10 * (per_pair * pairs + per_atom * n)}
    if kind == "md":
        n, steps = case["atoms"], case["steps"]
        # A step reads x and v and writes x, v and F; every pair is evaluated once.
        return {"bytes": steps * 15 * real * n,
                "flops": steps * 45 * _half_pairs(n, ARGON_DENSITY, CUTOFF)}
    mean = (16384 - 64) / math.log(16384 / 64)  # of the log-uniform sizes
    atom_steps = case["requests"] * case["steps"] * mean
    return {"bytes": 60 * atom_steps, "flops": 45 * _half_pairs(atom_steps, 20.0, CUTOFF)}


# -- float64 values in plain torch ----------------------------------------------------------


def _minimum_image(d, cell):
    return d - cell * torch.round(d / cell)


def _pairs64(x, cell, radius):
    """(i, j) of every pair closer than ``radius``, each once: all pairs of a small system, else
    the atoms of neighboring bins against each other."""
    n = x.shape[0]
    x = torch.remainder(x, cell)
    dims = [int(length // radius) for length in cell.tolist()]
    found = []
    if n <= 4500 or min(dims) < 3:
        for begin in range(0, n, 2048):
            rows = torch.arange(begin, min(n, begin + 2048), device=x.device)
            d = _minimum_image(x[rows][:, None, :] - x[None], cell)
            hit = (d.square().sum(-1) < radius * radius) & (
                rows[:, None] < torch.arange(n, device=x.device)[None])
            i, j = hit.nonzero(as_tuple=True)
            found.append(torch.stack([rows[i], j]))
        return torch.cat(found, dim=1)
    size = torch.tensor(dims, device=x.device)
    at = torch.minimum((x / cell * size).long(), size - 1)
    flat = (at[:, 0] * dims[1] + at[:, 1]) * dims[2] + at[:, 2]
    bins = math.prod(dims)
    counts = torch.bincount(flat, minlength=bins)
    order = flat.argsort()
    start = counts.cumsum(0) - counts
    most = int(counts.max())
    table = torch.full((bins, most), -1, dtype=torch.int64, device=x.device)
    table[flat[order], torch.arange(n, device=x.device) - start[flat[order]]] = order
    offsets = [(0, 0, 0)] + [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)
                             if (a, b, c) > (0, 0, 0)]
    chunk = max(1, 30_000_000 // (most * most))
    upper = torch.ones((most, most), dtype=torch.bool, device=x.device).triu(1)
    for offset in offsets:
        shift = torch.tensor(offset, device=x.device)
        for begin in range(0, bins, chunk):
            home = torch.arange(begin, min(bins, begin + chunk), device=x.device)
            place = torch.stack([home // (dims[1] * dims[2]), home // dims[2] % dims[1],
                                 home % dims[2]], dim=1)
            there = (place + shift) % size
            other = (there[:, 0] * dims[1] + there[:, 1]) * dims[2] + there[:, 2]
            a, b = table[home], table[other]
            d = _minimum_image(x[a][:, :, None, :] - x[b][:, None, :, :], cell)
            hit = (d.square().sum(-1) < radius * radius) & (a >= 0)[:, :, None] & (
                b >= 0)[:, None, :]
            if offset == (0, 0, 0):
                hit &= upper
            c, i, j = hit.nonzero(as_tuple=True)
            found.append(torch.stack([a[c, i], b[c, j]]))
    return torch.cat(found, dim=1)


def _lj_rows(types, i, j, sigma):
    count = {1: 1, 3: 2, 6: 3}[sigma.numel()]
    low, high = torch.minimum(types[i], types[j]), torch.maximum(types[i], types[j])
    return low * (2 * count - low - 1) // 2 + high


def _lj_terms(d, r2, sigma, epsilon):
    """(pair energies, f / r) of squared distances, sigma and epsilon per pair."""
    s2 = sigma * sigma
    p6 = (s2 / r2) ** 3
    c6 = (s2 / CUTOFF**2) ** 3
    return (4 * epsilon * (p6 * p6 - p6) - 4 * epsilon * (c6 * c6 - c6),
            24 * epsilon * (2 * p6 * p6 - p6) / r2)


def _lj_exact(x, cell, types, sigma, epsilon, pairs=None):
    """(E, F, W) of float64 positions, differentiable in sigma and epsilon."""
    pairs = _pairs64(x, cell, CUTOFF) if pairs is None else pairs
    energy, virial = 0.0, 0.0
    forces = torch.zeros_like(x)
    for begin in range(0, pairs.shape[1], 1 << 24):
        i, j = pairs[:, begin:begin + (1 << 24)]
        d = _minimum_image(x[i] - x[j], cell)
        r2 = d.square().sum(-1)
        near = r2 < CUTOFF**2
        i, j, d, r2 = i[near], j[near], d[near], r2[near]
        row = _lj_rows(types, i, j, sigma)
        u, f = _lj_terms(d, r2, sigma[row], epsilon[row])
        f = f[:, None] * d
        energy = energy + u.sum()
        virial = virial + f.T @ d
        forces = forces.index_add(0, i, f).index_add(0, j, -f)
    return energy, forces, virial


def _softplus(x):
    return torch.nn.functional.softplus(x, threshold=60.0) - math.log(2.0)


def _schnet_exact(x, cell, types, weights, blocks, gaussians, second_order):
    """(E, F, W) of a SchNet in float64; with ``second_order`` differentiable in the weights."""
    i, j = _pairs64(x, cell, BEAD_CUTOFF)
    d = _minimum_image(x[i] - x[j], cell)
    r = d.square().sum(-1).sqrt().requires_grad_(True)
    envelope = 0.5 * (torch.cos(r * (math.pi / BEAD_CUTOFF)) + 1.0)
    width = BEAD_CUTOFF / (gaussians - 1)
    centres = torch.arange(gaussians, dtype=torch.float64, device=x.device) * width
    basis = torch.exp(-0.5 * ((r[:, None] - centres) / width).square())
    h = weights["embedding"][types]
    for b in range(blocks):
        def dense(y, layer):
            y = y @ weights[f"blocks.{b}.{layer}.weight"].T
            return y + weights.get(f"blocks.{b}.{layer}.bias", 0.0)

        values = dense(h, "atoms")
        filters = dense(_softplus(dense(basis, "filter1")), "filter2") * envelope[:, None]
        message = torch.zeros_like(h).index_add(0, i, filters * values[j])
        message = message.index_add(0, j, filters * values[i])
        h = h + dense(_softplus(dense(message, "update1")), "update2")
    y = _softplus(h @ weights["readout1.weight"].T + weights["readout1.bias"])
    energy = (y @ weights["readout2.weight"].T + weights["readout2.bias"]).sum()
    slope, = torch.autograd.grad(energy, r, create_graph=second_order)
    pull = (slope / r.detach())[:, None] * d
    forces = torch.zeros_like(x).index_add(0, i, -pull).index_add(0, j, pull)
    return energy, forces, -(pull.T @ d)


def _loss_exact(predicted, labels, scales, frames):
    """One frame's share of the training loss."""
    return sum(((x - labels[name].double()) / scales[name]).square().mean()
               for name, x in zip(CHANNELS, predicted)) / frames


def _chain_half(kinetic, q, p, mass, degrees, thermal, dt):
    """Half a step of a Nose-Hoover chain of three; returns the velocities' factor."""
    def force(k, energy):
        return (2.0 * energy - degrees * thermal if k == 0
                else p[k - 1] ** 2 / mass[k - 1] - thermal)

    quarter = 0.25 * dt
    p[2] += quarter * force(2, kinetic)
    damp = [0.0, 0.0]
    for k in (1, 0):
        damp[k] = math.exp(-0.125 * dt * p[k + 1] / mass[k + 1])
        p[k] = damp[k] * (damp[k] * p[k] + quarter * force(k, kinetic))
    factor = math.exp(-0.5 * dt * p[0] / mass[0])
    kinetic *= factor * factor
    for k in range(3):
        q[k] += 0.5 * dt * p[k] / mass[k]
    for k in (0, 1):
        p[k] = damp[k] * (damp[k] * p[k] + quarter * force(k, kinetic))
    p[2] += quarter * force(2, kinetic)
    return factor


def _md_exact(case, given):
    x, v = given["positions"].double(), given["velocities"].double()
    cell, m = given["cell"].double(), ARGON_MASS
    n = x.shape[0]
    v = v - v.mean(dim=0)
    types = torch.zeros(n, dtype=torch.int64, device=x.device)
    sigma, epsilon = (p.double() for p in _lj_parameters(1, given["positions"].dtype))
    thermostat = case["ensemble"] == "nvt"
    thermal, degrees = BOLTZMANN * TEMPERATURE, 3 * n - 3
    mass = [degrees * thermal * TIMESCALE**2, thermal * TIMESCALE**2, thermal * TIMESCALE**2]
    q, p = [0.0] * 3, [0.0] * 3
    margin, reference, pairs = 0.2, None, None

    def forces():
        nonlocal reference, pairs
        if pairs is None or float((x - reference).square().sum(-1).max()) > (margin / 2) ** 2:
            reference, pairs = x, _pairs64(x, cell, CUTOFF + margin)
        return _lj_exact(x, cell, types, sigma, epsilon, pairs)[1]

    f = forces()
    for _ in range(case["steps"]):
        if thermostat:
            v = v * _chain_half(0.5 * m * float(v.square().sum()), q, p, mass, degrees, thermal,
                                TIMESTEP)
        v = v + 0.5 * TIMESTEP / m * f
        x = x + TIMESTEP * v
        f = forces()
        v = v + 0.5 * TIMESTEP / m * f
        if thermostat:
            v = v * _chain_half(0.5 * m * float(v.square().sum()), q, p, mass, degrees, thermal,
                                TIMESTEP)
    return {"path": x, "velocities": v, "forces": f}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("serve", "list"):
        return None  # minutes of dense float64 dynamics; whole numbers
    given = _inputs(case, seed)
    if kind == "efv":
        dtype = given["positions"].dtype
        sigma, epsilon = (p.double() for p in _lj_parameters(case["types"], dtype))
        return dict(zip(CHANNELS, _lj_exact(given["positions"].double(), given["cell"].double(),
                                            given["types"], sigma, epsilon)))
    if kind == "fit":
        sigma = given["sigma"].double().requires_grad_(True)
        epsilon = given["epsilon"].double().requires_grad_(True)
        total, rows = 0.0, []
        for f in range(case["frames"]):
            predicted = _lj_exact(given["positions"][f].double(), given["cells"][f].double(),
                                  given["types"], sigma, epsilon)
            labels = {name: given["labels"][name][f] for name in CHANNELS}
            value = _loss_exact(predicted, labels, given["scales"], case["frames"])
            value.backward()
            total += float(value.detach())
            rows.append([y.detach() for y in predicted])
        return {"loss": total, "sigma": sigma.grad, "epsilon": epsilon.grad,
                "predicted": {name: torch.stack([row[k] for row in rows])
                              for k, name in enumerate(CHANNELS)}}
    if kind in ("schnet", "schnet_fit"):
        weights = {name: w.double() for name, w in given["weights"].items()}
        cell = given["cell"].double()
        if kind == "schnet":
            got = _schnet_exact(given["positions"][0].double(), cell, given["types"], weights,
                                case["blocks"], case["gaussians"], False)
            return {name: y.detach() for name, y in zip(CHANNELS, got)}
        weights = {name: w.requires_grad_(True) for name, w in weights.items()}
        total = 0.0
        for f in range(case["frames"]):
            predicted = _schnet_exact(given["positions"][f].double(), cell, given["types"],
                                      weights, case["blocks"], case["gaussians"], True)
            labels = {name: given["labels"][name][f] for name in CHANNELS}
            value = _loss_exact(predicted, labels, given["scales"], case["frames"])
            value.backward()
            total += float(value.detach())
        return {"loss": total, "gradient": {name: w.grad for name, w in weights.items()}}
    return _md_exact(case, given)
