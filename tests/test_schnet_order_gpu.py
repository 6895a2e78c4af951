"""The SchNet kernels' FP32 sums keep their order: results bit for bit those of the kernels that
took a thread per pair.

Messages, their reverse and forces are sums over an atom's pairs, and their operands' rounding to
BF16 turns a last bit into a visible change, so the order of a sum is part of the result. It is
fixed within a warp's 32 rows (row by row along a run of one first atom, features in column order
in the sum over features); only the atomics that join the runs of several warps arrive in any
order. So the systems here are stars: every leaf is in one pair and a center's pairs lie in the
rows of at most two warps. Every feature sum then takes at most two atomics onto zero, 0 + a + b
in either order, and the outputs below have one value: no tolerance. Forces on the centers (an
atomic per pair) and the atom-wise weights' gradients (atomics over tiles) do not.

tests/golden/schnet_stars.npz holds the outputs of those kernels (the library as of commit
8935124), written by ``python tests/test_schnet_order_gpu.py FILE`` with it.
"""

import sys

import numpy as np
import pytest
import torch

from nabladyn_b200 import potential, quantity, training
from nabladyn_b200.neighbors import NeighborPairs
from oracle import schnet as oracle

pytestmark = pytest.mark.gpu

CUTOFF, CELL = 1.2, (7.0, 8.5, 6.25)
# pairs at least, leaves per center at most, blocks, Gaussians, types, loss channels
CASES = {
    "long": (700, 31, 3, 50, 2, ("energy", "virial")),
    "short": (300, 9, 2, 64, 1, ("energy", "virial")),
    "one_tile": (90, 31, 1, 20, 4, ("energy", "virial")),
    "dimers": (200, 1, 2, 33, 2, ("energy", "forces", "virial")),  # each force one atomic
}


def stars(rng, pairs, most):
    """Positions, the [2, C] index and which atoms are centers."""
    x, first, second = [], [], []
    while len(first) < pairs:
        center = len(x)
        x.append(rng.random_sample(3) * CELL)
        for _ in range(rng.randint(1, most + 1)):
            d = rng.standard_normal(3)
            first.append(center)
            second.append(len(x))
            x.append(x[center] + d * (rng.uniform(0.3, 1.15) / np.linalg.norm(d)))
    centers = np.zeros(len(x), dtype=bool)
    centers[first] = True
    return np.array(x), np.array([first, second], dtype=np.int32), centers


def evaluate(case, device):
    """The outputs that have one value, by name."""
    pairs, most, blocks, gaussians, types, channels = CASES[case]
    rng = np.random.RandomState(sorted(CASES).index(case))
    positions, index, centers = stars(rng, pairs, most)
    n = len(positions)
    model = potential.schnet(
        atom_types=torch.tensor(rng.randint(0, types, n), device=device), num_types=types,
        cutoff=CUTOFF, interactions=blocks, gaussians=gaussians, trainable=True)
    state = model.state_dict()
    for name, parameter in model.named_parameters():
        shape = tuple(parameter.shape)
        scale = 1.0 if name == "embedding" else (np.sqrt(2.0 / sum(shape)) if len(shape) == 2
                                                 else 0.05)
        state[name] = torch.tensor(scale * rng.standard_normal(shape), dtype=torch.float32)
    model.load_state_dict(state)
    x = torch.tensor(positions, dtype=torch.float32, device=device)
    cell = torch.tensor(CELL, dtype=torch.float32, device=device)
    columns = torch.tensor(index, device=device)
    e, f, w = quantity.energy_force_virial(model)(x, cell, NeighborPairs(columns, n, CUTOFF))
    leaves = torch.tensor(~centers, device=device)
    out = {"energy": e, "forces": f[leaves], "virial": w}
    labels = {"energy": rng.standard_normal(1), "forces": rng.standard_normal((1, n, 3)),
              "virial": rng.standard_normal((1, 3, 3))}
    ones = dict.fromkeys(channels, 1.0)
    out["loss"], gradient = training.loss_and_gradient(
        model, {k: v.detach().clone() for k, v in model.named_parameters()}, x[None], cell[None],
        (columns[None].contiguous(),),
        {k: torch.tensor(labels[k], dtype=torch.float32, device=device) for k in channels},
        ones, ones)
    out.update({k: v for k, v in gradient.items() if "filter" in k})
    return {k: v.detach().cpu().numpy() for k, v in out.items()}


@pytest.mark.parametrize("case", list(CASES))
def test_sums_keep_their_order(cuda, case):
    golden = np.load("tests/golden/schnet_stars.npz")
    for name, value in evaluate(case, cuda).items():
        np.testing.assert_array_equal(value, golden[f"{case}:{name}"], err_msg=name)


def test_energy_virial_and_loss_over_several_runs(cuda):
    """343 beads over all pairs, where every atomic order is open: each of eight runs within the
    bounds of the BF16 operands (those of the single-run tests: energy 3e-3 kJ/mol per atom,
    virial 1e-2, loss 1e-2 relative)."""
    golden = dict(np.load("tests/golden/schnet_343.npz"))
    fit = dict(np.load("tests/golden/schnet_fit_gradient.npz"))
    n = golden["positions"].shape[0]
    index = np.stack(np.triu_indices(n, 1)).astype(np.int32)
    model = potential.schnet(atom_types=torch.tensor(golden["atom_types"], device=cuda),
                             num_types=2, cutoff=CUTOFF, trainable=True)
    weights = {k: v.detach().double().cpu().numpy() for k, v in model.state_dict().items()}
    e64, _, w64 = oracle.energy_force_virial(golden["positions"], golden["cell"], *index,
                                             golden["atom_types"], weights, CUTOFF, 50, 3)
    columns = torch.tensor(index, device=cuda)
    x = torch.tensor(golden["positions"], dtype=torch.float32, device=cuda)
    cell = torch.tensor(golden["cell"], dtype=torch.float32, device=cuda)
    channels = ("energy", "forces", "virial")
    for _ in range(8):
        e, _, w = quantity.energy_force_virial(model)(x, cell, NeighborPairs(columns, n, CUTOFF))
        assert abs(float(e) - e64) <= 3e-3 * n
        assert np.linalg.norm(w.cpu().numpy() - w64) <= 1e-2 * np.linalg.norm(w64)
        loss, _ = training.loss_and_gradient(
            model, {k: v.detach().clone() for k, v in model.named_parameters()},
            torch.tensor(fit["positions"], dtype=torch.float32, device=cuda),
            torch.tensor(fit["cells"], dtype=torch.float32, device=cuda),
            (columns.expand(fit["positions"].shape[0], 2, -1).contiguous(),),
            {k: torch.tensor(fit[f"label:{k}"], dtype=torch.float32, device=cuda)
             for k in channels},
            dict.fromkeys(channels, 1.0), dict(zip(channels, fit["scales"].tolist())))
        assert float(loss) == pytest.approx(float(fit["loss"]), rel=1e-2)


if __name__ == "__main__":
    np.savez_compressed(sys.argv[1], **{f"{case}:{name}": value for case in CASES
                                        for name, value in evaluate(case, "cuda").items()})
