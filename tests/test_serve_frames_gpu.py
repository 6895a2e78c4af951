"""Frames into and out of the replica server's pool: requests of zero steps come back as they
went in, at the sizes where a CTA's rows end unevenly, in one batch over both lanes.

Tolerances: the velocity of the center of mass is a float64 sum in another order than numpy's,
so a float32 velocity may round to its neighbor (one unit in the last place, 2^-23 relative of
the larger of the velocity and the center's); positions are wrapped in float32 (two roundings of
at most |x| 2^-24 each on the way in and one on the way out); the kinetic energy is a float64
sum of positive terms (N 2^-53 relative) over those velocities (2^-22)."""

import ctypes

import numpy as np
import pytest

from nabladyn_b200._native import Replica
from nabladyn_b200.serving import ReplicaRequest, ReplicaServer

pytestmark = pytest.mark.gpu

SIZES = (2, 31, 33, 511, 512, 513, 1025, 4099)


def request_of(atoms, dtype, seed):
    rng = np.random.default_rng(seed)
    side = max(3.0, (atoms / 20.0) ** (1 / 3))
    positions = rng.uniform(-side, 2 * side, (atoms, 3)).astype(dtype)
    return ReplicaRequest(positions=positions, velocities=rng.normal(0.5, 0.3, (atoms, 3)),
                          masses=rng.uniform(1.0, 50.0, atoms).astype(dtype),
                          cell=np.array([side, 1.25 * side, 1.5 * side]), temperature=120.0,
                          steps=0, name=atoms, epsilon=0.0)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_frames_come_back(cuda, dtype):
    requests = [request_of(atoms, dtype, atoms) for atoms in SIZES]
    server = ReplicaServer(device=cuda, budget_bytes=64 << 20, max_slots=16, large_atoms=600)
    results = {r.name: r for r in server.serve(requests, realtime=False)}
    table = server.table.view(server.max_slots, -1).cpu().numpy()
    records = {r.num_atoms: r for r in (Replica.from_buffer_copy(row.tobytes()) for row in table)}
    for request in requests:
        result = results[request.name]
        mass = np.asarray(request.masses, dtype=np.float64)
        velocity = request.velocities.astype(np.float64)
        center = (mass[:, None] * velocity).sum(axis=0) / mass.sum()
        expected = (velocity - center).astype(np.float32)
        bound = 2.0**-23 * np.maximum(np.abs(expected), np.abs(center))
        assert np.all(np.abs(result.velocities - expected) <= bound)
        cell = request.cell.astype(np.float32)
        assert np.all((result.positions >= 0) & (result.positions < cell))
        unwrapped = result.positions.astype(np.float64) + result.images * cell.astype(np.float64)
        assert np.all(np.abs(unwrapped - request.positions)
                      <= 4 * 2.0**-24 * (np.abs(request.positions) + cell))
        kinetic = 0.5 * (mass[:, None] * expected.astype(np.float64) ** 2).sum()
        assert records[request.name].thermostat[6] == pytest.approx(kinetic, rel=2.0**-21)
