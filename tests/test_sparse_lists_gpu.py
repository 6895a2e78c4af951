"""Lists of gases, whose bins mostly hold no or few atoms: a warp per bin with atoms, several bins
per CTA, against the oracle (pair sets) and against the route of ordinary lists (the same columns
bit for bit; a list with room for more than twelve columns per atom takes it). Bins that do not fit
a warp's staging (128 candidates, 32 atoms, 512 pairs) lie among the empty ones in one case."""

import math

import numpy as np
import pytest
import torch

from nabladyn_b200 import space
from nabladyn_b200.neighbors import NeighborList
from oracle import neighbors as on

pytestmark = pytest.mark.gpu

RADIUS = 1.1


@pytest.mark.parametrize("dtype", (torch.float32, torch.float64))
@pytest.mark.parametrize("lengths, background, cluster", [
    ((12.0, 12.5, 13.0), 3000, 0),    # a bin per CTA
    ((60.0, 40.0, 41.0), 700, 0),     # 14 bins per CTA
    ((60.0, 40.0, 41.0), 9, 0),
    ((40.0, 40.0, 40.0), 30000, 600),  # a dense bin among sparse ones
    ((2.6, 100.0, 100.0), 2000, 0),   # minimum images
    ((90.0, 90.0, 90.0), 2500, 40),   # 32 bins per CTA
])
def test_gases_match_the_oracle_and_the_general_route(cuda, dtype, lengths, background, cluster):
    rng = np.random.default_rng(background + cluster)
    box = np.asarray(lengths)
    positions = rng.uniform(-0.2, 1.2, (background, 3)) * box
    n = background + cluster
    close = background // 3  # some pairs in any gas
    positions[:close] = positions[-close:] + rng.uniform(0.1, 0.5, (close, 3))
    positions = np.concatenate([positions, 0.4 * box + rng.uniform(0.0, 0.6, (cluster, 3))])
    x = torch.tensor(positions, dtype=dtype, device=cuda)
    cell = torch.tensor(box, dtype=dtype, device=cuda)

    def check(listed, frame, lattice):
        index, total = listed.tensors().index.cpu().numpy(), listed.num_pairs
        first, second, path = on.pairs(space.wrap(frame, lattice)[0].cpu().numpy(),
                                       lattice.cpu().numpy(), RADIUS)
        assert path == "grid" and total == len(first)
        np.testing.assert_array_equal(on.pair_set(index[0, :total], index[1, :total]),
                                      on.pair_set(first, second))
        columns = np.arange(total, index.shape[1])
        np.testing.assert_array_equal(index[:, total:], [columns % n] * 2)
        return index[:, :total]

    gas = NeighborList(RADIUS, skin=0.0, capacity_multiplier=1.5)
    gas.allocate(x, cell)
    assert gas.pair_capacity <= 12 * n
    roomy = NeighborList(RADIUS, skin=0.0, capacity_multiplier=math.ceil(13 * n / gas.num_pairs))
    roomy.allocate(x, cell)
    assert roomy.pair_capacity > 12 * n
    # The same frame, a moved one, and one of a smaller cell, which takes fewer bins than the list has.
    frames = ((x, cell), (x + 0.3, cell), ((0.93 * x).contiguous(), (0.93 * cell).contiguous()))
    for k, (frame, lattice) in enumerate(frames):
        if k:
            gas.update(frame, lattice)
            roomy.update(frame, lattice)
        np.testing.assert_array_equal(check(gas, frame, lattice), check(roomy, frame, lattice))
    assert gas._rebuild_count == 3
    held = gas._device_tensors()
    frame, lattice = frames[-1]
    assert torch.equal(held["reference_positions"], space.wrap(frame, lattice)[0])
    assert torch.equal(held["reference_cell"], lattice)
