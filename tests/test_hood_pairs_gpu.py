"""The grid path's pair build where a home bin does not fit its staging: more than 32 atoms per
bin, more than 512 candidates (several chunks), more than 3,072 pairs of 32 atoms, a short axis
(minimum images) with dense bins, atoms past every face. Pair sets, counts and order against the
oracle: sets bit for bit, each first atom's columns together and in ascending list order twice."""

import numpy as np
import pytest
import torch

from nabladyn_b200 import space
from nabladyn_b200.neighbors import NeighborList
from oracle import neighbors as on

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", (torch.float32, torch.float64))
@pytest.mark.parametrize("lengths, radius, background, cluster", [
    ((4.5, 4.5, 4.5), 1.1, 1300, 0),      # ordinary bins, 4 per axis
    ((4.5, 4.5, 4.5), 1.1, 3000, 0),      # 47 atoms per bin, some 600 candidates
    ((4.5, 4.5, 4.5), 1.1, 200, 1200),    # one bin of over a thousand atoms
    ((5.7, 2.6, 3.4), 1.1, 2200, 300),    # two bins on an axis, dense
    ((9.0, 4.6, 4.6), 0.5, 900, 5),       # many nearly empty bins
])
def test_dense_and_short_grids_match_the_oracle(cuda, dtype, lengths, radius, background,
                                                cluster):
    rng = np.random.default_rng(background + cluster)
    box = np.asarray(lengths)
    positions = rng.uniform(-0.2, 1.2, (background, 3)) * box
    dense = 0.05 * box + rng.uniform(0.0, 0.6, (cluster, 3))
    positions = np.concatenate([positions, dense])
    x = torch.tensor(positions, dtype=dtype, device=cuda)
    cell = torch.tensor(box, dtype=dtype, device=cuda)
    listed = NeighborList(radius, skin=0.0)
    listed.allocate(x, cell)
    index = listed.tensors().index.cpu().numpy()
    total = listed.num_pairs
    first, second, path = on.pairs(space.wrap(x, cell)[0].cpu().numpy(), cell.cpu().numpy(), radius)
    assert path == "grid" and total == len(first)
    np.testing.assert_array_equal(on.pair_set(index[0, :total], index[1, :total]),
                                  on.pair_set(first, second))
    runs = np.flatnonzero(np.diff(index[0, :total])) + 1
    starts = index[0, np.concatenate([[0], runs])]
    assert len(np.unique(starts)) == len(starts)  # each first atom's columns are together
    # An update that rebuilds (another frame, then this one again) gives the same columns.
    listed.update(x + 0.3, cell)
    listed.update(x, cell)
    assert listed._rebuild_count == 3
    np.testing.assert_array_equal(listed.tensors().index.cpu().numpy(), index)


def test_a_frame_of_non_finite_coordinates_is_refused(cuda):
    """Every coordinate NaN or infinite, so that all atoms would share a bin: refused, and the
    list stays usable for the next frame."""
    listed = NeighborList(1.0, skin=0.1)
    cell = torch.full((3,), 20.0, device=cuda)
    bad = torch.full((150000, 3), float("nan"), device=cuda)
    bad[::2] = float("inf")
    with pytest.raises(ValueError, match="positions must be finite"):
        listed.allocate(bad, cell)
    with pytest.raises(RuntimeError, match="allocate"):
        listed.tensors()
    one = 20.0 * torch.rand((1000, 3), device=cuda)
    one[77, 1] = -float("inf")
    with pytest.raises(ValueError, match="positions must be finite"):
        listed.allocate(one, cell)
    one[77, 1] = 3.0
    listed.allocate(one, cell)
    assert listed.num_pairs > 0


@pytest.mark.parametrize("dtype", (torch.float32, torch.float64))
def test_first_frame_starts_the_list(cuda, dtype):
    """Strided positions far outside the cell: the reference frame is the wrapped one, and an
    update with the same frame reuses its pairs."""
    generator = torch.Generator().manual_seed(5)
    wide = 60.0 * torch.randn((900, 3), generator=generator, dtype=torch.float64)
    x = torch.stack([wide, wide], dim=-1).to(dtype).to(cuda)[..., 0]
    cell = torch.tensor([9.0, 5.1, 4.7], dtype=dtype, device=cuda)
    listed = NeighborList(1.0, skin=0.1)
    listed.allocate(x, cell)
    held = listed._device_tensors()
    assert torch.equal(held["reference_positions"], space.wrap(x, cell)[0])
    assert torch.equal(held["reference_cell"], cell) and held["limits"].tolist() == [8, 4, 4]
    listed.update(x, cell)
    assert listed._rebuild_count == 1


@pytest.mark.parametrize("multiplier", (1.0, 1.3, 40.0))
@pytest.mark.parametrize("atoms", (1300, 40001))
def test_columns_past_the_total_are_self_pairs(cuda, atoms, multiplier):
    """The padding that some CTAs of the fill write: column k holds (k mod N, k mod N), after a
    tight, an ordinary and a roomy capacity (the largest takes more padding CTAs), and after an
    update that rebuilds."""
    rng = np.random.default_rng(atoms)
    side = (atoms / 14.0) ** (1 / 3)
    cell = torch.full((3,), side, device=cuda)
    x = torch.tensor(rng.uniform(0, side, (atoms, 3)), dtype=torch.float32, device=cuda)
    listed = NeighborList(1.0, skin=0.0, capacity_multiplier=multiplier)
    listed.allocate(x, cell)
    for _ in range(2):
        index = listed.tensors().index.cpu().numpy()
        columns = np.arange(listed.num_pairs, index.shape[1])
        np.testing.assert_array_equal(index[:, listed.num_pairs:], [columns % atoms] * 2)
        listed.update(x + 0.3, cell)
