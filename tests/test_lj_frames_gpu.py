"""nd_lj_frames, its parameter backward and nd_wrap against plain torch float64 on the same inputs, where the kernels can
go wrong: capacities around the 4 columns of a lane and the 128 of a warp (so the second row
starts at every offset from a 16-byte boundary), columns in any order, self-pairs and indices
outside the atoms between live ones, one to three frames and types, positions outside the cell.

Tolerances: a float64 sum of a few thousand terms of one magnitude keeps 1e-12 of its scale;
float32 pair terms carry a few roundings (6e-8 each) of quantities that cancel at most tenfold,
so 1e-5 of the scale.
"""

import math

import pytest
import torch

from nabladyn_b200 import space
from nabladyn_b200.potential._lennard_jones import evaluate_frames, pair_index
from nabladyn_b200.training._predict import _BatchLJ

pytestmark = pytest.mark.gpu

CUTOFF = 1.0


def system(frames, atoms, capacity, types, dtype, device, grouped):
    """Frames of atoms at least 0.3 nm apart on a jittered lattice, partly outside the cell, and
    random columns with padding and invalid ones among them."""
    generator = torch.Generator().manual_seed(1000 * atoms + capacity + types)
    side = math.ceil(atoms ** (1 / 3))
    axis = torch.arange(side, dtype=torch.float64)
    length = max(2.2, 0.36 * side)
    sites = torch.cartesian_prod(axis, axis, axis)[:atoms] * (length / side)
    x = sites + 0.01 * torch.rand((frames, atoms, 3), generator=generator, dtype=torch.float64)
    x += length * torch.randint(-2, 3, (frames, atoms, 1), generator=generator)
    cells = torch.full((frames, 3), length, dtype=torch.float64)
    index = torch.randint(0, atoms, (frames, 2, capacity), generator=generator)
    if grouped:
        index[:, 0] = index[:, 0].sort(dim=1)[0]
    bad = torch.rand((frames, capacity), generator=generator)
    index[:, 1] = torch.where(bad < 0.1, index[:, 0], index[:, 1])
    index[:, 0] = torch.where((bad >= 0.1) & (bad < 0.13), torch.tensor(atoms), index[:, 0])
    index[:, 1] = torch.where((bad >= 0.13) & (bad < 0.16), torch.tensor(-1), index[:, 1])
    kinds = torch.randint(0, types, (atoms,), generator=generator)
    rows = types * (types + 1) // 2
    sigma = 0.3 + 0.04 * torch.rand(rows, generator=generator, dtype=torch.float64)
    epsilon = 0.5 + 0.5 * torch.rand(rows, generator=generator, dtype=torch.float64)
    return (x.to(dtype).to(device), cells.to(dtype).to(device),
            index.to(torch.int32).to(device), kinds.to(device),
            sigma.to(dtype).to(device), epsilon.to(dtype).to(device))


def reference(x, cells, index, kinds, types, sigma, epsilon):
    """E, F, W of the frames by float64 torch operations."""
    x, cells, sigma, epsilon = (t.double() for t in (x, cells, sigma, epsilon))
    out = []
    for f in range(x.shape[0]):
        i, j = index[f].long()
        n = x.shape[1]
        keep = (i != j) & (i >= 0) & (i < n) & (j >= 0) & (j < n)
        i, j = i[keep], j[keep]
        d = x[f][i] - x[f][j]
        d = d - cells[f] * torch.round(d / cells[f])
        r2 = d.square().sum(-1)
        near = r2 < CUTOFF**2
        i, j, d, r2 = i[near], j[near], d[near], r2[near]
        row = pair_index(kinds[i], kinds[j], types)
        p6 = (sigma[row] ** 2 / r2) ** 3
        c6 = sigma[row] ** 6
        e = 4 * epsilon[row] * (p6 * p6 - p6 - c6 * c6 + c6)
        pull = (24 * epsilon[row] * (2 * p6 * p6 - p6) / r2)[:, None] * d
        forces = torch.zeros_like(x[f]).index_add(0, i, pull).index_add(0, j, -pull)
        out.append((e.sum(), forces, pull.T @ d))
    return [torch.stack(part) for part in zip(*out)]


@pytest.mark.parametrize("dtype", (torch.float32, torch.float64))
@pytest.mark.parametrize("frames, atoms, capacity, types, grouped", [
    (1, 2, 1, 1, True), (1, 7, 3, 1, True), (2, 9, 5, 2, False), (3, 40, 127, 1, True),
    (1, 40, 128, 3, True), (2, 65, 129, 2, True), (3, 130, 1023, 3, False),
    (1, 130, 1025, 1, True), (2, 500, 40002, 2, True), (1, 500, 200003, 3, True),
])
def test_frames_match_float64(cuda, dtype, frames, atoms, capacity, types, grouped):
    x, cells, index, kinds, sigma, epsilon = system(frames, atoms, capacity, types, dtype, cuda,
                                                    grouped)
    got = evaluate_frames(x, cells, index, kinds.to(torch.int32), types, sigma, epsilon, CUTOFF,
                          True)[:3]
    wrapped = space.wrapped_only(x, cells)
    again = evaluate_frames(wrapped, cells, index, kinds.to(torch.int32), types, sigma, epsilon,
                            CUTOFF, False)[:3]
    want = reference(wrapped, cells, index, kinds, types, sigma, epsilon)
    tolerance = 1e-12 if dtype == torch.float64 else 1e-5
    for values in (got, again):
        for value, exact in zip(values, want):
            assert value.dtype == dtype and value.shape == exact.shape
            scale = float(exact.abs().max()) + 1.0
            assert float((value.double() - exact).abs().max()) <= tolerance * scale


@pytest.mark.parametrize("dtype", (torch.float32, torch.float64))
@pytest.mark.parametrize("frames, atoms, capacity, types, grouped", [
    (1, 2, 1, 1, True), (2, 9, 5, 2, False), (3, 40, 255, 1, True), (2, 65, 257, 3, True),
    (1, 130, 70001, 8, False),
])
def test_parameter_gradients_match_float64(cuda, dtype, frames, atoms, capacity, types, grouped):
    """The backward of arbitrary adjoints of E, F and W, one to thirty-six parameter rows. The
    rows' sums are float64; the float32 inputs' geometry carries float32 roundings."""
    x, cells, index, kinds, sigma, epsilon = system(frames, atoms, capacity, types, dtype, cuda,
                                                    grouped)
    generator = torch.Generator().manual_seed(capacity)
    adjoints = [torch.randn(shape, generator=generator, dtype=torch.float64).to(dtype).to(cuda)
                for shape in ((frames,), (frames, atoms, 3), (frames, 3, 3))]
    parameters = [p.clone().requires_grad_(True) for p in (sigma, epsilon)]
    values = _BatchLJ.apply(*parameters, x, cells, index, kinds.to(torch.int32), types, CUTOFF)
    got = torch.autograd.grad(values, parameters, adjoints, retain_graph=True)
    again = torch.autograd.grad(values, parameters, adjoints)
    exact_parameters = [p.double().requires_grad_(True) for p in (sigma, epsilon)]
    exact = reference(space.wrapped_only(x, cells), cells, index, kinds, types,
                      *exact_parameters)
    want = torch.autograd.grad(exact, exact_parameters, [a.double() for a in adjoints])
    # A row's terms may cancel: the scale is their size, about that of the largest row.
    tolerance = 1e-11 if dtype == torch.float64 else 1e-4
    for value, second, exact_value in zip(got, again, want):
        assert value.dtype == dtype
        scale = float(exact_value.abs().max()) + 1.0
        assert float((value.double() - exact_value).abs().max()) <= tolerance * scale
        assert float((second.double() - exact_value).abs().max()) <= tolerance * scale


@pytest.mark.parametrize("dtype", (torch.float32, torch.float64))
def test_wrap_has_the_rounding_of_space_wrap(cuda, dtype):
    generator = torch.Generator().manual_seed(3)
    x = 40.0 * torch.randn((3, 1001, 3), generator=generator, dtype=torch.float64)
    cells = torch.tensor([[2.3, 3.1, 7.7], [36.77, 2.9, 5.5], [1e-3, 1e4, 11.0]])
    x, cells = x.to(dtype).to(cuda), cells.to(dtype).to(cuda)
    x[0, 0] = cells[0]
    x[0, 1] = -torch.finfo(dtype).tiny
    x[1, 0, 0] = float("nan")
    x[2, 5, 1] = float("inf")
    want = torch.stack([space.wrap(x[f], cells[f])[0] for f in range(3)])
    assert torch.equal(space.wrapped_only(x, cells).nan_to_num(-1.0), want.nan_to_num(-1.0))
    strided = torch.empty((1001, 6), dtype=dtype, device=cuda)[:, ::2]
    strided.copy_(x[1])
    assert torch.equal(space.wrapped_only(strided, cells[1]).nan_to_num(-1.0),
                       want[1].nan_to_num(-1.0))
