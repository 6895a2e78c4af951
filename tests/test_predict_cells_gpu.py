"""training.predict of Lennard-Jones with cells of another dtype than the positions (both are taken
in the wider one), and cells that do not belong to the frames (refused before any launch).

Tolerance: the same float64 arithmetic on the same values, 1e-12 of the scale (float64 atomics).
"""

import pytest
import torch

from nabladyn_b200 import lattice, potential, training

pytestmark = pytest.mark.gpu


@pytest.fixture
def frames(cuda):
    x, cell = lattice.fcc(4, 4 * 0.5745, 0.02, seed=3)
    x = torch.tensor(x, dtype=torch.float32, device=cuda)
    positions = torch.stack([x, x + 0.3])
    cells = torch.tensor(cell, dtype=torch.float64, device=cuda).expand(2, 3).contiguous()
    model = potential.lennard_jones(
        atom_types=torch.zeros(len(x), dtype=torch.int64, device=cuda),
        sigma=torch.tensor([0.34], dtype=torch.float64, device=cuda),
        epsilon=torch.tensor([0.996], dtype=torch.float64, device=cuda), cutoff=1.0,
        trainable=("sigma", "epsilon"))
    stack = training.pair_stack(positions.double(), cells, 1.0)
    return model, positions, cells, (stack,)


CHANNELS = ("energy", "forces", "virial")


@pytest.mark.parametrize("wide", ("cells", "positions"))
def test_mixed_types_take_the_wider(frames, wide):
    model, positions, cells, stacks = frames
    cells = cells.float().double()  # the same values in both types
    want = training.predict(model, {}, positions.double(), cells, stacks, CHANNELS)
    given = (positions, cells) if wide == "cells" else (positions.double(), cells.float())
    got = training.predict(model, {}, *given, stacks, CHANNELS)
    for name in CHANNELS:
        assert got[name].dtype == torch.float64
        torch.testing.assert_close(got[name], want[name], rtol=0.0,
                                   atol=1e-12 * float(want[name].detach().abs().max()))


def test_cells_of_other_frames_are_refused(frames):
    model, positions, cells, stacks = frames
    for bad in (cells[0], cells[:1], torch.cat([cells, cells]), cells.cpu(), cells[:, :2]):
        with pytest.raises(ValueError, match="cells must be"):
            training.predict(model, {}, positions.double(), bad, stacks, CHANNELS)
