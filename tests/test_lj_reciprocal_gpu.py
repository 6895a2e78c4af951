"""The float32 pair arithmetic of nd_lj_frames takes 1 / r^2 as the rounded quotient.

A frame of one pair along x with sigma = 0.5, epsilon = 1 and cutoff 16 has
E = 4 (p^2 - p) + 2^-28, p = q^3, q = 0.25 / r^2: everything but 1 / r^2, q^2 and p is exact or
rounded once, so the bits of E follow from float32 operations on the host. 65,535 distances a
call, 16 calls: a million mantissas. Whether p^2 - p is fused is the compiler's choice, one for
all pairs.
"""

import numpy as np
import pytest
import torch

from nabladyn_b200.potential._lennard_jones import evaluate_frames

pytestmark = pytest.mark.gpu

FRAMES = 65535


def test_energy_bits_follow_from_the_rounded_quotient(cuda):
    rng = np.random.default_rng(11)
    fused = separate = True
    index = torch.tensor([[[0], [1]]], dtype=torch.int32, device=cuda).expand(FRAMES, 2, 1).contiguous()
    cells = torch.full((FRAMES, 3), 64.0, device=cuda)
    kinds = torch.zeros(2, dtype=torch.int32, device=cuda)
    for _ in range(16):
        r = rng.uniform(0.4, 0.7, FRAMES).astype(np.float32)
        x = torch.zeros((FRAMES, 2, 3), device=cuda)
        x[:, 1, 0] = torch.tensor(r, device=cuda)
        energy = evaluate_frames(x, cells, index, kinds, 1, torch.tensor([0.5], device=cuda),
                                 torch.ones(1, device=cuda), 16.0, False)[0].cpu().numpy()
        inverse = np.float32(1) / (r * r)
        q = np.float32(0.25) * inverse
        p = (q * q) * q
        wide = p.astype(np.float64)
        for name, t in (("fused", (wide * wide - wide).astype(np.float32)), ("separate", p * p - p)):
            bits = (4.0 * t.astype(np.float64) + 2.0**-28).astype(np.float32)
            same = np.array_equal(bits, energy)
            fused, separate = (fused and same, separate) if name == "fused" else (fused, separate and same)
    assert fused or separate
