"""A training loss of many blocks has the same bits each time (its block sums meet in the blocks'
order), as the means it stands for have."""

import pytest
import torch

from nabladyn_b200 import training

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frames, atoms", [(3, 1000), (16, 2111), (64, 4096)])
def test_loss_repeats(cuda, frames, atoms):
    generator = torch.Generator(cuda).manual_seed(frames)
    draw = lambda: {  # noqa: E731
        name: torch.randn(shape, generator=generator, dtype=torch.float64, device=cuda)
        for name, shape in (("energy", (frames,)), ("forces", (frames, atoms, 3)),
                            ("virial", (frames, 3, 3)))}
    predicted, labels = draw(), draw()
    ones = dict.fromkeys(predicted, 1.0)
    runs = []
    for _ in range(40):
        total, terms = training.loss(predicted, labels, ones, ones)
        runs.append(torch.stack([total, *terms.values()]))
    assert all(torch.equal(run, runs[0]) for run in runs)
