"""The float32 partial sums of E and W in nd_lj_frames. With every column the same pair (dimers of
one displacement), a sum of C columns differs from C times one column only by the sums'
roundings, which then all go one way.

A thread that adds m equal terms one after another is off by at most (m + 1) / 2 roundings of
2^-24; the bound is that of 2,048 threads an SM over the 148 SMs, each adding its columns one by
one, plus two for the outputs' own rounding.
"""

import pytest
import torch

from nabladyn_b200.potential._lennard_jones import evaluate_frames

pytestmark = pytest.mark.gpu

COLUMNS, DIMERS = 48_000_003, 4096


@pytest.mark.parametrize("displacement", [
    (0.21, 0.23, 0.22), (0.31, -0.17, 0.26), (-0.13, 0.41, 0.19), (0.27, 0.29, -0.33),
    (0.193, 0.237, 0.281), (0.347, 0.111, 0.203), (0.299, -0.251, 0.157), (0.171, 0.353, 0.117),
])
def test_sums_of_equal_terms(cuda, displacement):
    cell = torch.tensor([[64.0, 64.0, 64.0]], device=cuda)
    step = torch.tensor(displacement, device=cuda)
    x = torch.zeros((1, 2 * DIMERS, 3), device=cuda)  # at the origin, so the difference is exact
    x[0, 1::2] = step
    x = torch.where(x < 0, x + 64.0, x)
    one = torch.ones(1, device=cuda)
    first = (2 * (torch.arange(COLUMNS, device=cuda) % DIMERS)).to(torch.int32)
    index = torch.stack([first, first + 1])[None]
    kinds = torch.zeros(2 * DIMERS, dtype=torch.int32, device=cuda)

    def evaluate(columns):
        energy, _, virial, _ = evaluate_frames(x, cell, columns, kinds, 1, 0.34 * one, one, 1.0,
                                               False)
        return torch.cat([energy.double(), virial.double().reshape(-1)])

    total, term = evaluate(index), evaluate(index[..., :1].contiguous())
    added = COLUMNS / (148 * 2048)
    bound = ((added + 1) / 2 + 2) * 2.0**-24
    error = ((total - COLUMNS * term) / (COLUMNS * term)).abs()
    assert float(error.max()) <= bound, (error / bound).tolist()
